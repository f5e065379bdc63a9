// Prints the batched walk's launch under a limit on blocks of 256 threads per SM:
// for every line "smem per_sm blocks descriptors" of the input the kernel's blocks
// per SM, threads per block and grid.  Host code only.
#include <cstdio>

#include "../ptwalker_gb300/csrc/batch_kernels.cuh"

int main()
{
    ptw_graph g;
    g.num_sms = 152;
    unsigned long long smem, nd;
    unsigned per_sm, blocks;
    while (std::scanf("%llu %u %u %llu", &smem, &per_sm, &blocks, &nd) == 4) {
        ptw::BatchLaunch l{};
        l.block = l.most = smem ? ptw::kBatchRowsBlock : 256;
        l.smem = smem;
        l.per_sm = (int)per_sm;
        ptw::limit_blocks(l, blocks);
        const unsigned grid = ptw::batch_grid(&g, l, nd);
        std::printf("%d %d %u\n", l.per_sm, l.block, grid);
    }
}
