// Device functions that the SIRT kernels share (sirt.cu, sirt_slices.cu, sirt_small.cu).
#pragma once

#include "sirt_internal.cuh"

namespace synk {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ int stop_of(const SirtProblem &q, int s) {
    return *(volatile const int *)(q.stop_iter + s);
}
__device__ __forceinline__ double res2_of(const SirtProblem &q, int s, int it) {
    return *(volatile const double *)(q.res2 + (size_t)s * (q.iterations + 1) + it);
}

// BP (the update) of iteration it: the slice is below its count and neither
// stopped before nor converged at x_it.
__device__ __forceinline__ bool bp_needed(double tol2, const SirtProblem &q, int s, int it) {
    if (it >= q.iterations) return false;
    if (tol2 <= 0.0) return true;
    if (stop_of(q, s) < it) return false;
    return !(res2_of(q, s, it) <= tol2 * q.b2[s]);
}

// Number of listed corner-clipping rays of a problem.
__device__ __forceinline__ int graze_count(const SirtProblem &q) { return __ldg(q.goff + 4); }

// Backprojection terms of the listed rays that clip corner `corner` of slice
// s, summed by the calling warp (lanes over the list, combined in a fixed
// order); every lane returns the sum.
__device__ __forceinline__ float corner_terms_warp(const SirtProblem &q, int s, int corner) {
    const int lane = threadIdx.x & 31;
    const int n = __ldg(q.goff + corner + 1) - __ldg(q.goff + corner);
    const float *t = q.gcontrib + (size_t)s * 4 * q.graze_capc + (size_t)corner * q.graze_capc;
    float acc = 0.0f;
    for (int i = lane; i < n; i += 32) acc = __fadd_rn(acc, t[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    return acc;
}

}  // namespace synk
