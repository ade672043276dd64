// Row-blocked fixed-point copy of a full-storage CRS (ed_spmv.cu).
//
// Eight consecutive rows are stored together in steps of four elements a row:
// lane l of a warp holds elements 4 j + (l & 3) of row l / 4 in step j, so a
// step's values and columns are each one aligned run of 32 entries, padded
// with zeros to the block's longest row (4.5 % more entries at N=11, 2S=30).
// A warp reading CRS rows directly starts each row's run at any offset, which
// costs the loads of 32 elements 7.6 L1 wavefronts where this layout takes 3,
// and k_spmv_fix is bound by those wavefronts; of the shapes of 32 elements,
// 8 x 4 also meets the fewest lines of x (10.9 on average at N=10, 2S=27;
// 4 x 8 12.1, 16 x 2 11.6, 1 x 32 23.3).
//
// Columns of 16 + 8 bits in two planes instead of 32 are slower in spite of
// the fewer bytes (730 against 679 us at N=11, 2S=30: one wavefront more).
#pragma once

#include "ed_fixed.cuh"

namespace edgb {
namespace {

constexpr int kBlkRows = 8, kBlkCols = 32 / kBlkRows;

__global__ void k_blk_steps(const int64_t* __restrict__ rowptr, int64_t n, int64_t blocks, int64_t* __restrict__ steps)
{
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < blocks; g += (int64_t)gridDim.x * blockDim.x) {
        int64_t longest = 0;
        for (int64_t r = g * kBlkRows; r < min(n, (g + 1) * kBlkRows); ++r) longest = max(longest, rowptr[r + 1] - rowptr[r]);
        steps[g] = (longest + kBlkCols - 1) / kBlkCols;
    }
}

// The sum over the lanes of one row.
__device__ __forceinline__ __int128 blk_row_sum(__int128 acc)
{
#pragma unroll
    for (int s = kBlkCols / 2; s > 0; s >>= 1) {
        const long long hi = (long long)(acc >> 64);
        const unsigned long long lo = (unsigned long long)acc;
        const long long ohi = __shfl_xor_sync(0xffffffffu, hi, s);
        const unsigned long long olo = __shfl_xor_sync(0xffffffffu, lo, s);
        acc += (__int128)(((unsigned __int128)(unsigned long long)ohi << 64) | olo);
    }
    return acc;
}

// Columns and values in the steps' order, fixed point at the exponent E.
__global__ void __launch_bounds__(256) k_blk_fill(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                                                  const double* __restrict__ val, int64_t n, int64_t blocks,
                                                  const int64_t* __restrict__ off, int E,
                                                  int32_t* __restrict__ ocol, int64_t* __restrict__ oval)
{
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < blocks; g += nw) {
        const int64_t r = g * kBlkRows + lane / kBlkCols;
        const int64_t s = r < n ? rowptr[r] : 0;
        const int len = r < n ? (int)(rowptr[r + 1] - s) : 0;
        const int64_t o = off[g];
        const int steps = (int)(off[g + 1] - o);
#pragma unroll 8
        for (int j = 0; j < steps; ++j) {
            const int k = j * kBlkCols + lane % kBlkCols;
            const int64_t at = (o + j) * 32 + lane;
            ocol[at] = k < len ? col[s + k] : 0;
            oval[at] = k < len ? fix_pair(val[s + k], E) : 0;
        }
    }
}

// y = A x, a warp a block of rows.  The columns of the next U steps are
// fetched with the current ones' values, so that an iteration waits for one
// memory access instead of two (112.0 -> 103.2 us at N=10, 2S=27 with the two
// conversion passes).  The stream of 12 bytes an entry bounds it: GB300,
// k_spmv_fix / this kernel: 0.07M rows (N=9, 2S=25) 39.0 / 33.9 us, 0.25M
// (N=10, 2S=27) 120.3 / 103.2, 0.61M (N=11, 2S=28) 304 / 264.5, 1.37M (N=11,
// 2S=30) 774 / 674 (6.5 TB/s).  U = 5 / 7 / 8: 104.5 / 109.9 / 107.8 at N=10;
// 3 CTAs per SM 110.9.
template <int U, int MINB>
__global__ void __launch_bounds__(256, MINB) k_spmv_blk(const int64_t* __restrict__ off, const int32_t* __restrict__ col,
                                                        const int2* __restrict__ aq, const int2* __restrict__ xq,
                                                        const int* __restrict__ xexp, int ea, double* __restrict__ y,
                                                        int64_t n, int64_t blocks)
{
    static_assert(U <= 8, "eight elements' products fit the int64 partial sums");
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int ex = __ldg(xexp);
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < blocks; g += nw) {
        const int64_t o = off[g];
        const int steps = (int)(off[g + 1] - o);
        const int2* ap = aq + o * 32 + lane;
        const int32_t* cp = col + o * 32 + lane;
        __int128 acc = 0;
        int c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = u < steps ? __ldcs(cp + u * 32) : 0;
        for (int j = 0; j < steps; j += U) {
            int2 a[U], x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                a[u] = j + u < steps ? __ldcs(ap + (j + u) * 32) : make_int2(0, 0);
                x[u] = __ldg(xq + c[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) c[u] = j + U + u < steps ? __ldcs(cp + (j + U + u) * 32) : 0;
            long long p2 = 0, p1 = 0, p0 = 0;
#pragma unroll
            for (int u = 0; u < U; ++u) fix_mac(a[u], x[u], p2, p1, p0);
            acc += fix_combine(p2, p1, p0);
        }
        acc = blk_row_sum(acc);
        const int64_t r = g * kBlkRows + lane / kBlkCols;
        if (lane % kBlkCols == 0 && r < n)
            y[r] = ex < 2047 ? round_i128(acc, ea + ex - 2160) : __longlong_as_double(0x7FF8000000000000ll);
    }
}

}  // namespace
}  // namespace edgb
