// Cells of an array in the reference's layout (FP64, variable fastest: NV
// consecutive doubles per cell) through shared memory. A thread that reads its
// own cell's NV doubles makes NV warp loads of 32 addresses 8 NV bytes apart, each
// touching every cache line of the warp's cells; here a CTA's run of NT cells
// moves as NV * NT consecutive doubles, and a thread takes its cell from shared
// memory (NV odd: no bank conflict; NV = 4: two-way).
#pragma once
#include "vb_ns.h"
#include <cuda_runtime.h>

namespace VB_NS {

// cells [c0, c0 + n) of `a` (n <= NT) -> s; the caller synchronises
template <int NV, int NT> __device__ __forceinline__ void aos_in(const double* __restrict__ a, long long c0, int n, double* s) {
    const double* p = a + c0 * NV;
    if (n == NT) {
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k * NT + threadIdx.x] = p[k * NT + threadIdx.x];
    } else {
        for (int e = threadIdx.x; e < n * NV; e += NT) s[e] = p[e];
    }
}
// s -> cells [c0, c0 + n) of `a`
template <int NV, int NT> __device__ __forceinline__ void aos_out(double* __restrict__ a, long long c0, int n, const double* s) {
    double* p = a + c0 * NV;
    if (n == NT) {
#pragma unroll
        for (int k = 0; k < NV; ++k) p[k * NT + threadIdx.x] = s[k * NT + threadIdx.x];
    } else {
        for (int e = threadIdx.x; e < n * NV; e += NT) p[e] = s[e];
    }
}

}  // namespace VB_NS
