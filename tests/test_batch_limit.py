"""ptw_batch_tune.blocks_per_sm on the CPU: the batched walk's launch has at most that
many times 256 threads per SM, whichever kernel runs."""
import os
import subprocess

import pytest

from ptwalker_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 152


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("bin") / "batch_limit")
    r = subprocess.run([_build._nvcc(), *_build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-o", exe,
                        os.path.join(HERE, "batch_limit.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(rows):
        r = subprocess.run([exe], input="".join("%d %d %d %d\n" % x for x in rows), capture_output=True, text=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]

    return run


def test_threads_per_sm(launches):
    rows = [(smem, per_sm, blocks, nd) for smem, fits in ((0, (1, 5, 8)), (20_000, (1, 2)))
            for per_sm in fits for blocks in (0, 1, 2, 3, 4, 5, 6, 7, 64) for nd in (1, 500, 10_000, 1_000_000)]
    got = launches(rows)
    assert len(got) == len(rows)
    for (smem, fit, blocks, nd), (per_sm, block, grid) in zip(rows, got):
        assert 1 <= per_sm <= fit and block % 32 == 0 and 32 <= block <= (768 if smem else 256)
        assert 1 <= grid <= SMS * per_sm
        most = (768 if smem else 256) * fit  # threads of an SM that the kernel allows
        if blocks:
            assert per_sm * block <= 256 * blocks
            most = min(most, 256 * blocks)
        if nd == 1_000_000:  # enough work: the limit is used, but for less than a warp per block
            assert per_sm * block > most - 32 * per_sm and grid == SMS * per_sm
