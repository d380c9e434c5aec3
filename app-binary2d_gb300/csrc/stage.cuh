// stage.cuh — what the stage kernels share: periodic indexes and the failure key.
#pragma once

#include "physics.cuh"
#include "runtime.cuh"
#include "tma.cuh"

namespace b2d {

// A double-float value of the compensated FP32 state.
struct df32 { float hi, lo; };

__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// Failure key of a zone: the reference surfaces the error of the first
// block, in mesh.block_indexes() order, whose 3x3 neighbour join fails
// (scheme.rs:126, 161-165); within that block the first failing neighbour
// in neighbour order (mesh.rs:101-110), within that neighbour the first
// failing zone in row-major order (scheme.rs:190-197).  The smallest key
// over all failing zones of the earliest failing stage is that error:
//   stage:10 | run:8 | block:16 | neighbour order:4 | zone:24 | code:2
__device__ __forceinline__ unsigned long long error_key(int stage, int run, const RunDev& rd, int gi, int gj, int code)
{
    const int nb = rd.nb, bs = rd.bs;
    const int ni = gi / bs, nj = gj / bs;
    const unsigned long long zone = (unsigned long long)((gi % bs) * bs + (gj % bs));
    unsigned long long best = ~0ull;
    for (int di = -1; di <= 1; ++di)
        for (int dj = -1; dj <= 1; ++dj) {
            int bi = (ni - di + nb) % nb, bj = (nj - dj + nb) % nb;   // n = b + (di, dj)
            unsigned long long k = ((unsigned long long)stage << 54) | ((unsigned long long)run << 46) |
                                   ((unsigned long long)(bi * nb + bj) << 30) |
                                   ((unsigned long long)((di + 1) * 3 + (dj + 1)) << 26) | (zone << 2) |
                                   (unsigned long long)code;
            best = k < best ? k : best;
        }
    return best;
}

// Whether stage `stage` is to be left out: the advance was abandoned when it
// began, or an earlier stage of it failed.  A failure in this stage does not
// count, whoever found it: all of its zones are looked at, so that the smallest
// key does not depend on which CTAs run first.
__device__ __forceinline__ bool left_out(const Failure* failure, int stage)
{
    const volatile Failure* f = failure;
    const unsigned long long key = f->key, abandoned = f->abandoned;
    return abandoned || key < (unsigned long long)stage << 54;
}

}  // namespace b2d
