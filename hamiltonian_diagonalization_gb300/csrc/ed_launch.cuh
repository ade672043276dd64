// Kernel launches with the count kept, and what the solvers' steps share on
// the device: the products' clock and the start of a restart cycle.
#pragma once

#include "ed_internal.h"

namespace edgb {

template <class... P, class... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    kernel<<<grid, block, smem, st>>>(args...);
    count_launch();
    ED_CUDA(cudaGetLastError());
}

// The device clock in ns, for the products' share of a solve: the kernel
// before a product leaves the latest end of its blocks, the one after it its
// start.  (Event nodes around every product cost a captured cycle 12 us a
// step.)
__device__ __forceinline__ void stamp(unsigned long long* at)
{
    if (at && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        atomicMax(at, t);
    }
}

namespace {

// Start of a restart cycle: zero its coefficients and flags.
__global__ void __launch_bounds__(256) k_cycle_begin(double* __restrict__ coef, int64_t count, int* __restrict__ flags, int nflags,
                                                     unsigned long long* __restrict__ started)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) coef[i] = 0.0;
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < nflags; i += blockDim.x) flags[i] = 0;
    stamp(started);
}

// Time in ns between the stamps (started, ended) of steps [k, m).
inline double stamped_ns(const std::vector<unsigned long long>& t, int k, int m)
{
    double s = 0.0;
    for (int j = k; j < m; ++j)
        if (t[2 * j + 1] > t[2 * j]) s += (double)(t[2 * j + 1] - t[2 * j]);
    return s;
}

}  // namespace

}  // namespace edgb
