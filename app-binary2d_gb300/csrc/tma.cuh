// tma.cuh — shared-memory addresses for asynchronous copies, and the read-set check.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b2d {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Read-set check.  A build with B2D_POISON defined fills every stage kernel's
// dynamic shared memory with quiet NaN before the kernel uses it (each 32-bit
// word, so an FP64 slot reads as NaN too), and the FP32 kernel also sets the
// neighbours that its outermost lanes do not have to NaN.
// A slot that a zone's update reads without the kernel having written it, or
// a guard-column value that reaches a zone's update, then turns that zone NaN;
// a poisoned build that reproduces the normal build's states bit for bit shows
// that neither happens.  Without B2D_POISON this is empty.
__device__ __forceinline__ void poison_dynamic_smem(unsigned char* base)
{
#ifdef B2D_POISON
    uint32_t bytes;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(bytes));
    for (uint32_t i = 4 * threadIdx.x; i + 4 <= bytes; i += 4 * blockDim.x)
        *(uint32_t*)(base + i) = 0x7fc00000u;
    __syncthreads();
#else
    (void)base;
#endif
}

__device__ __forceinline__ float poison_or(float v)
{
#ifdef B2D_POISON
    (void)v;
    return __int_as_float(0x7fc00000);
#else
    return v;
#endif
}

}  // namespace b2d
