// Column sums of a row-major [rows, width] matrix, one block per 32 columns and row range, in a fixed order.
#pragma once

#include "cgnn_common.cuh"

namespace cgnn {

constexpr int COLSUM_WARPS = 8;
constexpr int COLSUM_UNROLL = 8;

// out[blockIdx.y, c] = sum of x[r, c] over the block's rows: a lane per column, warp w adds rows w, w + 8, ...
// with COLSUM_UNROLL loads in flight, and the warps' sums meet in shared memory in warp order.
template <typename T>
__global__ void __launch_bounds__(COLSUM_WARPS * 32) colsum_kernel(const T *x, int64_t rows, int64_t rows_per_block,
                                                                   int64_t width, T *out) {
    __shared__ T sums[COLSUM_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t c = (int64_t)blockIdx.x * 32 + lane;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_block;
    const int64_t r1 = min(rows, r0 + rows_per_block);
    T s = T(0);
    if (c < width) {
        const T *column = x + c;
        int64_t r = r0 + warp;
        for (; r + (COLSUM_UNROLL - 1) * COLSUM_WARPS < r1; r += COLSUM_UNROLL * COLSUM_WARPS) {
            T v[COLSUM_UNROLL];
#pragma unroll
            for (int u = 0; u < COLSUM_UNROLL; ++u) v[u] = column[(r + u * COLSUM_WARPS) * width];
#pragma unroll
            for (int u = 0; u < COLSUM_UNROLL; ++u) s += v[u];
        }
        for (; r < r1; r += COLSUM_WARPS) s += column[r * width];
    }
    sums[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && c < width) {
        s = sums[0][lane];
#pragma unroll
        for (int w = 1; w < COLSUM_WARPS; ++w) s += sums[w][lane];
        out[(int64_t)blockIdx.y * width + c] = s;
    }
}

}  // namespace cgnn
