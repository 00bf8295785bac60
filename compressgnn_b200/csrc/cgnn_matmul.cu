// out[M, N] = A^T B for tall row-major A [K, M] and B [K, N], fp32: the weight gradient of a Linear over the
// representatives (K of them, tens of thousands; M and N are layer widths).
//
// What bounds it is FP32 arithmetic and the shared-memory reads that feed it (2 K M N operations; A and B are read once or
// twice from cache) -- if enough blocks are at work: the output has a handful of tiles, so K is split over the
// whole GPU and the partial products are added in split order by a second kernel (deterministic, no atomics).  Both operands are
// contiguous along their output dimension, so a stage of MM_KC rows goes to shared memory as it lies
// (16-byte cp.async, or 4-byte ones for rows that are no whole vectors) and every lane's operand reads are
// 128-bit and free of bank conflicts.  A thread owns 8 x 8 outputs as pairs updated by fma.rn.f32x2 (each half the
// IEEE fma of the scalar form), which leaves issue slots for the operand loads.  128 x 256 over 64 k
// rows: 158 us in the library's kernel, 90 here (48 TFLOP/s; under ncu issue slots 55 % busy, DRAM 13 %, 11 warps to an
// SM); 64 x 128 over 2.7 k rows: 26, and 10 here.
#include <algorithm>

#include "cgnn_colsum.cuh"

namespace cgnn {
namespace {

constexpr int MM_THREADS = 128;
constexpr int MM_TM = 64, MM_TN = 128;  // output tile of a block
constexpr int MM_KC = 16;               // rows of A and B per stage
constexpr int MM_STAGES = 3;
constexpr int MM_WAVE = 148 * 4;        // blocks resident at once: registers and 36 KB of shared memory allow 4 per SM

__device__ __forceinline__ uint32_t mm_shared(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mm_copy16(uint32_t dst, const float *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mm_copy4(uint32_t dst, const float *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Rows [k0, k0 + MM_KC) of one operand, columns [c0, c0 + TILE), zero outside [0, k_end) x [0, width).
template <int TILE, bool VEC>
__device__ __forceinline__ void mm_load(float *stage, const float *x, int64_t k0, int64_t k_end, int c0, int width) {
    constexpr int W = VEC ? 4 : 1, PER_ROW = TILE / W;
#pragma unroll
    for (int i = threadIdx.x; i < MM_KC * PER_ROW; i += MM_THREADS) {
        const int k = i / PER_ROW, c = (i % PER_ROW) * W;
        const bool inside = k0 + k < k_end && c0 + c < width;
        const float *src = inside ? x + (k0 + k) * width + c0 + c : x;
        if constexpr (VEC) mm_copy16(mm_shared(stage + k * TILE + c), src, inside ? 16 : 0);
        else mm_copy4(mm_shared(stage + k * TILE + c), src, inside ? 4 : 0);
    }
}

template <bool VEC_A, bool VEC_B>
__global__ void __launch_bounds__(MM_THREADS, 4) matmul_tn_kernel(const float *a, const float *b, int64_t K, int M, int N,
                                                                  int64_t k_per_split, float *out) {
    __shared__ __align__(16) float as[MM_STAGES][MM_KC][MM_TM];
    __shared__ __align__(16) float bs[MM_STAGES][MM_KC][MM_TN];
    const int tiles_n = (N + MM_TN - 1) / MM_TN;
    const int m0 = (int)(blockIdx.x / tiles_n) * MM_TM, n0 = (int)(blockIdx.x % tiles_n) * MM_TN;
    const int64_t k_begin = (int64_t)blockIdx.y * k_per_split, k_end = min(K, k_begin + k_per_split);
    const int stages = k_end > k_begin ? (int)((k_end - k_begin + MM_KC - 1) / MM_KC) : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = (lane & 7) + 8 * (warp & 1);   // columns tx * 4 .. + 3 and 64 + tx * 4 .. + 3
    const int ty = (lane >> 3) + 4 * (warp >> 1); // rows    ty * 4 .. + 3 and 32 + ty * 4 .. + 3
    auto load = [&](int s) {
        if (s < stages) {
            const int64_t k0 = k_begin + (int64_t)s * MM_KC;
            mm_load<MM_TM, VEC_A>(&as[s % MM_STAGES][0][0], a, k0, k_end, m0, M);
            mm_load<MM_TN, VEC_B>(&bs[s % MM_STAGES][0][0], b, k0, k_end, n0, N);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < MM_STAGES - 1; ++s) load(s);
    for (int s = 0; s < stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(MM_STAGES - 2) : "memory");
        __syncthreads();  // stage s has landed for every thread, and stage s - 1 has been read by every thread
        load(s + MM_STAGES - 1);
        const int st = s % MM_STAGES;
#pragma unroll
        for (int k = 0; k < MM_KC; ++k) {
            const float4 a0 = *reinterpret_cast<const float4 *>(&as[st][k][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&as[st][k][32 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4 *>(&bs[st][k][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4 *>(&bs[st][k][64 + tx * 4]);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float2 bv[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                                  make_float2(b1.z, b1.w)};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(make_float2(av[i], av[i]), bv[j], acc[i][j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float *o = out + (int64_t)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + (i < 4 ? ty * 4 + i : 32 + ty * 4 + i - 4);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + (j < 2 ? tx * 4 + 2 * j : 64 + tx * 4 + 2 * (j - 2));
            if (n < N) o[(int64_t)m * N + n] = acc[i][j].x;
            if (n + 1 < N) o[(int64_t)m * N + n + 1] = acc[i][j].y;
        }
    }
}

int64_t matmul_tiles(int64_t M, int64_t N) { return ceil_div(M, MM_TM) * ceil_div(N, MM_TN); }

// One wave of blocks, but no split shorter than 4 stages.
int64_t matmul_splits(int64_t K, int64_t M, int64_t N) {
    return std::max<int64_t>(1, std::min<int64_t>(MM_WAVE / matmul_tiles(M, N), K / (4 * MM_KC)));
}

}  // namespace
}  // namespace cgnn

using namespace cgnn;

extern "C" {

size_t cgnn_matmul_tn_scratch_bytes(int64_t K, int64_t M, int64_t N) {
    if (K <= 0 || M <= 0 || N <= 0) return 0;
    const int64_t splits = matmul_splits(K, M, N);
    return splits == 1 ? 0 : (size_t)splits * (size_t)M * (size_t)N * sizeof(float);
}

int cgnn_matmul_tn(int64_t K, int64_t M, int64_t N, const float *a, const float *b, float *out, void *scratch,
                   size_t scratch_bytes, cgnn_stream_t stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    CGNN_REQUIRE(K >= 0 && M >= 0 && N >= 0 && M <= INT32_MAX / 2 && N <= INT32_MAX / 2, "matmul_tn: bad sizes");
    if (M == 0 || N == 0) return CGNN_OK;
    CGNN_REQUIRE(out != nullptr && (K == 0 || (a != nullptr && b != nullptr)), "matmul_tn: null pointer");
    if (K == 0) {
        CGNN_CUDA(cudaMemsetAsync(out, 0, (size_t)M * (size_t)N * sizeof(float), stream));
        return CGNN_OK;
    }
    const int64_t splits = matmul_splits(K, M, N);
    const int64_t per_split = ceil_div(ceil_div(K, splits), MM_KC) * MM_KC;
    CGNN_REQUIRE(splits == 1 || (scratch != nullptr && scratch_bytes >= cgnn_matmul_tn_scratch_bytes(K, M, N)),
                 "matmul_tn: scratch too small");
    CGNN_REQUIRE(matmul_tiles(M, N) < (1ll << 31), "matmul_tn: grid too large");
    float *product = splits == 1 ? out : static_cast<float *>(scratch);
    const dim3 grid((unsigned)matmul_tiles(M, N), (unsigned)splits);
    auto whole = [](const float *p, int64_t width) { return width % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool va = whole(a, M), vb = whole(b, N);
    if (va && vb) matmul_tn_kernel<true, true><<<grid, MM_THREADS, 0, stream>>>(a, b, K, (int)M, (int)N, per_split, product);
    else if (va) matmul_tn_kernel<true, false><<<grid, MM_THREADS, 0, stream>>>(a, b, K, (int)M, (int)N, per_split, product);
    else if (vb) matmul_tn_kernel<false, true><<<grid, MM_THREADS, 0, stream>>>(a, b, K, (int)M, (int)N, per_split, product);
    else matmul_tn_kernel<false, false><<<grid, MM_THREADS, 0, stream>>>(a, b, K, (int)M, (int)N, per_split, product);
    CGNN_LAUNCH_CHECK();
    if (splits > 1) {
        colsum_kernel<float><<<(unsigned)ceil_div(M * N, 32), COLSUM_WARPS * 32, 0, stream>>>(product, splits, splits, M * N,
                                                                                               out);
        CGNN_LAUNCH_CHECK();
    }
    return CGNN_OK;
}

}  // extern "C"
