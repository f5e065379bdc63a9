// Path walks on the plain columns (DeepWalk in walk.cu, node2vec in
// node2vec.cu): helpers.
#pragma once

#include "ptw_internal.cuh"

namespace ptw {
namespace {

// A walker's path row, written from registers: four positions at a time with
// one 16-byte store where the row's addresses allow it (the row may start at
// any 4-byte address), single words at its ends.
struct PathOut {
    int32_t *row;
    uint32_t skew;  // position p is word (skew + p) % 4 of a 16-byte group
    int32_t b0, b1, b2, b3;

    __device__ __forceinline__ void start(int32_t *r)
    {
        row = r;
        skew = (uint32_t)(reinterpret_cast<uintptr_t>(r) >> 2) & 3;
        b0 = b1 = b2 = b3 = 0;
    }
    // Position p (called in order from 0).
    __device__ __forceinline__ void put(uint32_t p, int32_t x)
    {
        const uint32_t s = (skew + p) & 3;
        b0 = s == 0 ? x : b0;
        b1 = s == 1 ? x : b1;
        b2 = s == 2 ? x : b2;
        if (s == 3) {
            b3 = x;
            if (p >= 3) {
                *reinterpret_cast<int4 *>(row + p - 3) = make_int4(b0, b1, b2, b3);
            } else {
                row[p] = b3;
                if (p >= 1) row[p - 1] = b2;
                if (p >= 2) row[p - 2] = b1;
            }
        }
    }
    // The last position put was L - 1.
    __device__ __forceinline__ void finish(uint32_t L)
    {
        const uint32_t s = (skew + L - 1) & 3;
        if (s == 3) return;
        row[L - 1] = s == 0 ? b0 : s == 1 ? b1 : b2;
        if (s >= 1 && L >= 2) row[L - 2] = s == 1 ? b0 : b1;
        if (s == 2 && L >= 3) row[L - 3] = b0;
    }
};

}  // namespace
}  // namespace ptw
