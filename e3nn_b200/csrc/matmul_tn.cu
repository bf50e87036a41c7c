// out[m, n] = scale * sum_z x[z, m] g[z, n] in fp32: the weight gradient of a dense layer (many rows z, a narrow x).
//
// Bound by the FP32 pipe: 64 x 1472 entries over 429,000 rows are 81 GFLOP, 1.1 ms at 148 x 128 multiply-adds a clock, while
// the rows are 2.6 GB, 0.4 ms.  A block owns 64 x 256 entries, 8 x 16 a thread, which read 6 x 16 bytes of shared memory for 64
// packed multiply-adds (FFMA2: half the issue slots); rows arrive by cp.async four stages ahead.  The rows are split over
// whole waves, up to eight; a block sums 2,048 rows at a time in registers and adds the runs in its partial matrix, and a
// second kernel adds the partial matrices, all in a fixed order: the error stays below that of the library's fp32 product,
// which sums longer runs (429,000 rows: 8.1e-7 against 1.7e-6; 3.2 million: 8.9e-7 against 4.6e-6).
// Against that product, 64 x 1472: 5,000 rows 51 -> 35 us, 15,600 127 -> 71, 105,000 500 -> 404, 429,000 1690 -> 1582.  With
// 8 x 8 a thread 39, 76, 419 and 1609 us; FFMA in place of FFMA2 is 5 - 10 % slower than that.
#include "common.cuh"

#include <algorithm>

namespace e3b {
namespace {

constexpr int kTnM = 64, kTnRows = 16, kTnStages = 4, kTnThreads = 128;
constexpr int64_t kTnMostRows = 2048;     // rows summed in registers

template <int TN>
__host__ __device__ constexpr int tn_stage_floats() { return kTnRows * (kTnM + TN); }

template <int BYTES>
__device__ __forceinline__ void tn_copy(float* dst, const float* src, bool live) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(live ? 4 : 0) : "memory");
}

// TN: columns of a block, 128 or 256.  VEC: widths are multiples of 4 and both bases 16-byte aligned
template <int TN, bool VEC>
__device__ __forceinline__ void tn_fetch(float* sx, float* sg, const float* __restrict__ x, const float* __restrict__ g, int64_t z0,
                                         int64_t z_end, int m0, int n0, int M, int N) {
    constexpr int V = VEC ? 4 : 1, QX = kTnM / V, QG = TN / V;
#pragma unroll 4
    for (int i = threadIdx.x; i < kTnRows * QX; i += kTnThreads) {
        const int r = i / QX, c = (i % QX) * V;
        const bool live = z0 + r < z_end && m0 + c < M;
        tn_copy<4 * V>(sx + r * kTnM + c, live ? x + (z0 + r) * M + m0 + c : x, live);
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < kTnRows * QG; i += kTnThreads) {
        const int r = i / QG, c = (i % QG) * V;
        const bool live = z0 + r < z_end && n0 + c < N;
        tn_copy<4 * V>(sg + r * TN + c, live ? g + (z0 + r) * N + n0 + c : g, live);
    }
}

// RUNS: a block has more than kTnMostRows rows and adds one run of them after another in its entries of `out`.
template <int TN, bool VEC, bool RUNS>
__global__ void __launch_bounds__(kTnThreads, TN == 128 ? 3 : 2) matmul_tn_kernel(const float* __restrict__ x, const float* __restrict__ g, int64_t Z, int M,
                                                                  int N, int64_t rows_per_split, float scale, float* __restrict__ out) {
    extern __shared__ __align__(16) float smem[];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    constexpr int NP = TN / 32;             // pairs of columns a thread owns: 4 columns of every 64
    const int n0 = blockIdx.x * TN, m0 = blockIdx.y * kTnM;
    const int64_t z_begin = static_cast<int64_t>(blockIdx.z) * rows_per_split;
    const int64_t z_end = z_begin + rows_per_split < Z ? z_begin + rows_per_split : Z;
    const int64_t steps = (z_end - z_begin + kTnRows - 1) / kTnRows;
    float2 acc[8][NP];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < NP; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    auto fetch = [&](int64_t step) {
        float* s = smem + (step % kTnStages) * tn_stage_floats<TN>();
        if (step < steps) tn_fetch<TN, VEC>(s, s + kTnRows * kTnM, x, g, z_begin + step * kTnRows, z_end, m0, n0, M, N);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < kTnStages - 1; ++s) fetch(s);
    constexpr int64_t kRun = kTnMostRows / kTnRows;
    int64_t from = 0;
    do {
        const int64_t to = RUNS && from + kRun < steps ? from + kRun : steps;
        for (int64_t step = from; step < to; ++step) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kTnStages - 2) : "memory");
            __syncthreads();            // this stage has landed for everyone; the stage fetched next is free
            fetch(step + kTnStages - 1);
            const float* sx = smem + (step % kTnStages) * tn_stage_floats<TN>();
            const float* sg = sx + kTnRows * kTnM;
#pragma unroll
            for (int k = 0; k < kTnRows; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(sx + k * kTnM + ty * 4);
                const float4 a1 = *reinterpret_cast<const float4*>(sx + k * kTnM + 32 + ty * 4);
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                float2 b[NP];
#pragma unroll
                for (int j = 0; j < NP / 2; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(sg + k * TN + 64 * j + tx * 4);
                    b[2 * j] = make_float2(v.x, v.y);
                    b[2 * j + 1] = make_float2(v.z, v.w);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < NP; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i], a[i]), b[j], acc[i][j]);
            }
        }
        float* o = out + static_cast<int64_t>(blockIdx.z) * M * N;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + (i >> 2) * 32 + ty * 4 + (i & 3);
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                const int n = n0 + (j >> 1) * 64 + tx * 4 + (j & 1) * 2;
                float* p = o + static_cast<int64_t>(m) * N + n;
                const bool add = RUNS && from > 0;
                if (n < N) p[0] = add ? fmaf(scale, acc[i][j].x, p[0]) : scale * acc[i][j].x;
                if (n + 1 < N) p[1] = add ? fmaf(scale, acc[i][j].y, p[1]) : scale * acc[i][j].y;
                if (RUNS) acc[i][j] = make_float2(0.0f, 0.0f);
            }
        }
        if (RUNS) from = to;
    } while (RUNS && from < steps);
}

__global__ void __launch_bounds__(256) matmul_tn_sum_kernel(const float* __restrict__ partial, int splits, int64_t count, float scale,
                                                            float* __restrict__ out) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float v = 0.0f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) v += partial[s * count + i];
    out[i] = scale * v;
}

struct TnPlan { int64_t rows; int splits, tiles_m, tiles_n, tn; };

TnPlan tn_plan(int64_t Z, int M, int N) {
    TnPlan p;
    p.tiles_m = (M + kTnM - 1) / kTnM;
    // 256 columns a block (a third more multiply-adds per byte of shared memory) unless they leave
    // more than an eighth of the work to padding
    const int n128 = (N + 127) / 128, n256 = (N + 255) / 256;
    p.tn = 16 * n256 <= 9 * n128 ? 256 : 128;
    p.tiles_n = p.tn == 256 ? n256 : n128;
    const int64_t tiles = static_cast<int64_t>(p.tiles_m) * p.tiles_n, chunks = ceil_div(Z, 4 * kTnRows);
    int64_t wave = (p.tn == 256 ? 2 : 3) * kNumSMs / tiles;      // splits that fill the chip once
    wave = wave < 1 ? 1 : wave;
    const int64_t splits = std::min(chunks, wave * std::min<int64_t>(8, ceil_div(Z, wave * kTnMostRows)));   // (the partials stay small)
    p.rows = ceil_div(chunks, splits) * 4 * kTnRows;
    p.splits = static_cast<int>(ceil_div(Z, p.rows));
    return p;
}

}  // namespace
}  // namespace e3b

extern "C" int64_t e3b_matmul_tn_scratch_bytes(int64_t rows, int m, int n) {
    if (rows <= 0 || m <= 0 || n <= 0) return 0;
    const e3b::TnPlan p = e3b::tn_plan(rows, m, n);
    return p.splits > 1 ? static_cast<int64_t>(sizeof(float)) * p.splits * m * n : 0;
}

extern "C" int e3b_matmul_tn(const float* x, const float* g, int64_t rows, int m, int n, float scale, float* out, void* scratch,
                             int64_t scratch_bytes, void* stream) {
    using namespace e3b;
    if (rows < 0 || m < 0 || n < 0) return fail(E3B_ERR_ARG, "matmul_tn: negative size");
    if (m == 0 || n == 0) return E3B_OK;
    if (!out) return fail(E3B_ERR_ARG, "matmul_tn: null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t count = static_cast<int64_t>(m) * n;
    if (rows == 0) {
        E3B_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float) * count, s));
        return E3B_OK;
    }
    if (!x || !g) return fail(E3B_ERR_ARG, "matmul_tn: null pointer");
    const TnPlan p = tn_plan(rows, m, n);
    if (p.tiles_m > 65535) return fail(E3B_ERR_ARG, "matmul_tn: m too large");
    if (p.splits > 1 && (!scratch || scratch_bytes < e3b_matmul_tn_scratch_bytes(rows, m, n)))
        return fail(E3B_ERR_ARG, "matmul_tn: scratch too small");
    const bool vec = m % 4 == 0 && n % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(g)) & 15) == 0;
    const dim3 grid(p.tiles_n, p.tiles_m, p.splits);
    const int smem = kTnStages * static_cast<int>(sizeof(float)) * (p.tn == 256 ? tn_stage_floats<256>() : tn_stage_floats<128>());
    const bool runs = p.rows > kTnMostRows;
    auto kernel = p.tn == 256 ? (vec ? (runs ? matmul_tn_kernel<256, true, true> : matmul_tn_kernel<256, true, false>)
                                     : (runs ? matmul_tn_kernel<256, false, true> : matmul_tn_kernel<256, false, false>))
                              : (vec ? (runs ? matmul_tn_kernel<128, true, true> : matmul_tn_kernel<128, true, false>)
                                     : (runs ? matmul_tn_kernel<128, false, true> : matmul_tn_kernel<128, false, false>));
    E3B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    float* to = p.splits > 1 ? static_cast<float*>(scratch) : out;
    kernel<<<grid, kTnThreads, smem, s>>>(x, g, rows, m, n, p.rows, p.splits > 1 ? 1.0f : scale, to);
    if (p.splits > 1)
        matmul_tn_sum_kernel<<<static_cast<unsigned>(ceil_div(count, 256)), 256, 0, s>>>(to, p.splits, count, scale, out);
    return check_launch("matmul_tn");
}
