// Weight-shared contractions in fp32 on register tiles: 'uvw' products and the per-irrep Linear (forward and transposed),
// their weight gradient, and both operand gradients of a 'uvw' product.
//
// dense.cu describes the contraction; the kernels here read the second part of a dense plan (built by
// e3nn_b200/o3/_dense_plan.py, its word offset is the plan's last word), which lists whole paths instead of single
// contraction entries, so that a path's Clebsch-Gordan coupling is applied to 32 channels at a time:
//
//     T_p[z, k, i] = sum_j C_ijk x2[z, v, j]                (once per row and path)
//     A[z, k, u]   = sum_i T_p[z, k, i] x1[z, u, i]         (Linear: A = c x1, k = i)
//     out[z, w, k] = sum_{p, v, u} A[z, k, u] W_p[u, v, w]
//
// x1 and x2 are the call's operands, or exchanged (`swapped`: the operand with more channels goes first, see the builder).
//
// Second part: header of 14 words { n_groups, groups, n_chunks, chunks, n_paths, paths, n_in, in_groups, d1max, d3max,
// in_paths, covered, swapped, channels of all chunks } (word offsets into the plan), then
//   groups    x 6 : out_off, mul_out, dim3, first chunk, chunks, 0
//   chunks    x 6 : path, x1 offset of its first channel, channels (<= 32), x2 offset or -1, weight base, 1 = T changes
//   paths     x 16: d1, d2, d3, weight strides over u and w, ki segments, j segments, x1off, m1, x2off, m2, out_off, mo,
//                   weight base, stride over v, coefficient (Linear)
//   in_groups x 5 : x1off, m1, d1, first in_path, in_paths   (the paths that leave one input irrep)
//   segments      : word offsets s[0..n] of (index, coefficient) pairs: (j, C) per (k, i); (i * d3 + k, C) per j
#include "common.cuh"
#include "dense_plan.cuh"
#include "gate_act.cuh"

#include <utility>

namespace e3b {
namespace {

constexpr int kThreads = 128;
constexpr int kKC = 32;            // channels of a chunk
constexpr int kLda = kKC + 4;      // floats between the rows of a staged operand: 16-byte rows, 8 rows cover all banks
constexpr int kTM = 8, kTN = 4;    // accumulators of a thread: rows x output channels
constexpr int kMaxGroups = 32;

struct Part2 {
    const int32_t* plan;
    const int32_t* h;
    __host__ __device__ explicit Part2(const int32_t* p) : plan(p), h(p + p[p[6] - 1]) {}
    __host__ __device__ int n_groups() const { return h[0]; }
    __host__ __device__ const int32_t* group(int g) const { return plan + h[1] + 6 * g; }
    __host__ __device__ const int32_t* chunk(int c) const { return plan + h[3] + 6 * c; }
    __host__ __device__ const int32_t* path(int p) const { return plan + h[5] + 16 * p; }
    __host__ __device__ int n_in() const { return h[6]; }
    __host__ __device__ const int32_t* in_group(int g) const { return plan + h[7] + 5 * g; }
    __host__ __device__ int d1max() const { return h[8]; }
    __host__ __device__ int d3max() const { return h[9]; }
    __host__ __device__ int in_path(int n) const { return plan[h[10] + n]; }
    __host__ __device__ bool covers_x1() const { return h[11] != 0; }
    __host__ __device__ bool swapped() const { return h[12] != 0; }
    __host__ __device__ int d1row() const { return plan[swapped() ? 2 : 1]; }
    __host__ __device__ int d2row() const { return plan[swapped() ? 1 : 2]; }
    __host__ __device__ int n_chunks() const { return h[2]; }
    __host__ __device__ int channels() const { return h[13]; }      // of all chunks
};

// T[zl][k * d1 + i] of a tile of nz rows (row stride ldt).
__device__ __forceinline__ void stage_coupling(const int32_t* plan, const int32_t* path, const float* __restrict__ x2, int d2row,
                                               int x2off, int64_t z0, int nz, int64_t Z, float* sT, int ldt) {
    const int n = path[0] * path[2];
    const int32_t* seg = plan + path[5];
    for (int idx = threadIdx.x; idx < nz * n; idx += kThreads) {
        const int zl = idx / n, ki = idx - zl * n;
        float t = 0.0f;
        if (z0 + zl < Z) {
            const float* y = x2 + (z0 + zl) * d2row + x2off;
            for (int s = seg[ki]; s < seg[ki + 1]; s += 2) t = fmaf(__int_as_float(plan[s + 1]), y[plan[s]], t);
        }
        sT[zl * ldt + ki] = t;
    }
}

// A[(zl * d3 + k) * lda + u] of one chunk for the tile's nz rows; channels past `len` and rows past Z are zero.
// A warp takes the 32 channels of one row at a time (its loads are one contiguous stretch of the row).
template <int D1>
__device__ __forceinline__ void stage_rows_d(const float* __restrict__ x1, int d1row, int x1off, int len, int64_t z0, int nz, int64_t Z,
                                             int d3, bool coupled, float coef, const float* sT, int ldt, float* sA, int lda) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kAhead = D1 <= 3 ? 4 : 2;
    for (int zb = warp * kAhead; zb < nz; zb += (kThreads / 32) * kAhead) {
        float x[kAhead][D1];
#pragma unroll
        for (int r = 0; r < kAhead; ++r) {
            const bool live = zb + r < nz && z0 + zb + r < Z && lane < len;
            const float* p = x1 + (z0 + zb + r) * d1row + x1off + lane * D1;
#pragma unroll
            for (int i = 0; i < D1; ++i) x[r][i] = live ? __ldg(p + i) : 0.0f;
        }
#pragma unroll
        for (int r = 0; r < kAhead; ++r) {
            const int zl = zb + r;
            if (zl >= nz) break;
            float* a = sA + static_cast<size_t>(zl) * d3 * lda + lane;
            if (!coupled) {
#pragma unroll
                for (int i = 0; i < D1; ++i) a[i * lda] = coef * x[r][i];
            } else {
                const float* t = sT + zl * ldt;
                for (int k = 0; k < d3; ++k) {
                    float v = 0.0f;
#pragma unroll
                    for (int i = 0; i < D1; ++i) v = fmaf(t[k * D1 + i], x[r][i], v);
                    a[k * lda] = v;
                }
            }
        }
    }
}

__device__ void stage_rows_any(const float* __restrict__ x1, int d1row, int x1off, int d1, int len, int64_t z0, int nz, int64_t Z, int d3,
                               bool coupled, float coef, const float* sT, int ldt, float* sA, int lda) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int zl = warp; zl < nz; zl += kThreads / 32) {
        const bool live = z0 + zl < Z && lane < len;
        const float* p = x1 + (z0 + zl) * d1row + x1off + lane * d1;
        for (int k = 0; k < d3; ++k) {
            float v = 0.0f;
            if (live) {
                if (!coupled) v = coef * p[k];
                else for (int i = 0; i < d1; ++i) v = fmaf(sT[zl * ldt + k * d1 + i], p[i], v);
            }
            sA[(zl * d3 + k) * lda + lane] = v;
        }
    }
}

__device__ __forceinline__ void stage_rows(int d1, const float* __restrict__ x1, int d1row, int x1off, int len, int64_t z0, int nz,
                                           int64_t Z, int d3, bool coupled, float coef, const float* sT, int ldt, float* sA, int lda) {
    switch (d1) {
        case 1: stage_rows_d<1>(x1, d1row, x1off, len, z0, nz, Z, d3, coupled, coef, sT, ldt, sA, lda); break;
        case 3: stage_rows_d<3>(x1, d1row, x1off, len, z0, nz, Z, d3, coupled, coef, sT, ldt, sA, lda); break;
        case 5: stage_rows_d<5>(x1, d1row, x1off, len, z0, nz, Z, d3, coupled, coef, sT, ldt, sA, lda); break;
        case 7: stage_rows_d<7>(x1, d1row, x1off, len, z0, nz, Z, d3, coupled, coef, sT, ldt, sA, lda); break;
        default: stage_rows_any(x1, d1row, x1off, d1, len, z0, nz, Z, d3, coupled, coef, sT, ldt, sA, lda);
    }
}

// W[kk][n] of a chunk: kKC x BN, zero outside len x cols.
template <int BN>
__device__ __forceinline__ void stage_weights(const float* __restrict__ W, int su, int sw, int len, int cols, float* sW) {
    constexpr int ld = BN + 4;
    for (int idx = threadIdx.x; idx < kKC * BN; idx += kThreads) {
        // consecutive threads along the direction that is contiguous in memory
        const int kk = sw == 1 ? idx / BN : idx % kKC, n = sw == 1 ? idx % BN : idx / kKC;
        sW[kk * ld + n] = (kk < len && n < cols) ? __ldg(W + static_cast<int64_t>(kk) * su + static_cast<int64_t>(n) * sw) : 0.0f;
    }
}

// ---------------------------------------------------------------------------------------------- forward, any irrep
struct FwdLaunch {
    int n;                               // groups of this launch
    int first_block[kMaxGroups + 1];
    int16_t group[kMaxGroups];
    int16_t bn[kMaxGroups];              // columns of a tile: 16, 32, 64 or 128
};

__host__ __device__ inline int tile_rows(int bn) { return kTM * kTN * kThreads / bn; }

// One tile: rows (z, k) of tile_rows(BN) / d3 consecutive z, BN output channels, the whole contraction.
template <int BN>
__device__ __forceinline__ void fwd_tile(const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                         const float* __restrict__ W, float* __restrict__ out, int64_t Z, int tile, int accumulate,
                                         float* smem) {
    constexpr int CX = BN / kTN, LX = CX < 8 ? CX : 8, LY = 32 / LX, WC = CX / LX, RY = kThreads / CX, BM = RY * kTM;
    constexpr int ldw = BN + 4;
    const int out_off = g[0], mo = g[1], d3 = g[2], d1row = P.d1row(), d2row = P.d2row(), dout = P.plan[3];
    const int col_blocks = (mo + BN - 1) / BN, tz = BM / d3;
    const int64_t z0 = static_cast<int64_t>(tile / col_blocks) * tz;
    const int c0 = (tile % col_blocks) * BN, cols = min(BN, mo - c0);
    float* sA = smem;
    float* sW = smem + BM * kLda;
    float* sT = sW + kKC * ldw;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % WC) * LX + lane % LX, ty = (warp / WC) * LY + lane / LX;

    float acc[kTM][kTN];
#pragma unroll
    for (int i = 0; i < kTM; ++i)
#pragma unroll
        for (int j = 0; j < kTN; ++j) acc[i][j] = 0.0f;
    // the rows of the tile past nz * d3 are read (and never stored): they must not hold non-finite leftovers
    for (int idx = tid; idx < (BM - tz * d3) * kLda; idx += kThreads) sA[tz * d3 * kLda + idx] = 0.0f;

    // sums of up to 32 entries, over several chunks where the paths have fewer channels, in accumulators of their own: the
    // rounding error grows with sqrt(32) + sqrt(K / 32)
    float part[kTM][kTN];
#pragma unroll
    for (int i = 0; i < kTM; ++i)
#pragma unroll
        for (int j = 0; j < kTN; ++j) part[i][j] = 0.0f;
    int held = 0;
    for (int c = 0; c < g[4]; ++c) {
        const int32_t* ch = P.chunk(g[3] + c);
        const int32_t* path = P.path(ch[0]);
        const int len = ch[2], d1 = path[0], ldt = (d1 * d3) | 1;
        const bool coupled = ch[3] >= 0;
        __syncthreads();
        if (coupled && ch[5]) {
            stage_coupling(P.plan, path, x2, d2row, ch[3], z0, tz, Z, sT, ldt);
            __syncthreads();
        }
        stage_weights<BN>(W + ch[4] + static_cast<int64_t>(c0) * path[4], path[3], path[4], len, cols, sW);
        stage_rows(d1, x1, d1row, ch[1], len, z0, tz, Z, d3, coupled, __int_as_float(path[15]), sT, ldt, sA, kLda);
        __syncthreads();
        const int kend = (len + 3) & ~3;
#pragma unroll 1
        for (int kk = 0; kk < kend; kk += 4) {
            float4 w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const float4*>(sW + (kk + q) * ldw + tx * kTN);
#pragma unroll
            for (int i = 0; i < kTM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(sA + (ty + RY * i) * kLda + kk);
                const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    part[i][0] = fmaf(av[q], w[q].x, part[i][0]);
                    part[i][1] = fmaf(av[q], w[q].y, part[i][1]);
                    part[i][2] = fmaf(av[q], w[q].z, part[i][2]);
                    part[i][3] = fmaf(av[q], w[q].w, part[i][3]);
                }
            }
        }
        held += len;
        if (c + 1 < g[4] && held + P.chunk(g[3] + c + 1)[2] <= kKC) continue;
        held = 0;
#pragma unroll
        for (int i = 0; i < kTM; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) { acc[i][j] += part[i][j]; part[i][j] = 0.0f; }
    }
    __syncthreads();
    // the tile in output order, then contiguous row segments
    float* sO = smem;
    const int seg = cols * d3;
#pragma unroll
    for (int i = 0; i < kTM; ++i) {
        const int r = ty + RY * i, zl = r / d3, k = r - zl * d3;
        if (zl >= tz) continue;
#pragma unroll
        for (int j = 0; j < kTN; ++j) {
            const int n = tx * kTN + j;
            if (n < cols) sO[zl * seg + n * d3 + k] = acc[i][j];
        }
    }
    __syncthreads();
    for (int zl = warp; zl < tz; zl += kThreads / 32) {
        if (z0 + zl >= Z) break;
        float* o = out + (z0 + zl) * dout + out_off + c0 * d3;
        for (int e = lane; e < seg; e += 32) o[e] = accumulate ? o[e] + sO[zl * seg + e] : sO[zl * seg + e];
    }
}

__global__ void __launch_bounds__(kThreads) dense_tile_fwd_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                  const float* __restrict__ x2, const float* __restrict__ W,
                                                                  float* __restrict__ out, int64_t Z, int accumulate, FwdLaunch L) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* g = P.group(L.group[s]);
    const int tile = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (L.bn[s]) {
        case 16: fwd_tile<16>(P, g, x1, x2, W, out, Z, tile, accumulate, smem); break;
        case 32: fwd_tile<32>(P, g, x1, x2, W, out, Z, tile, accumulate, smem); break;
        case 64: fwd_tile<64>(P, g, x1, x2, W, out, Z, tile, accumulate, smem); break;
        default: fwd_tile<128>(P, g, x1, x2, W, out, Z, tile, accumulate, smem); break;
    }
}

// Columns of a tile: the narrowest that holds the group's channels in one pass, so that the coupled operand is built once;
// at most 64 where one row's components would not fit the rows of a wider tile (l = 16 and up).
constexpr int kMostDim = 64;
inline int columns_for(int mo, int d3) { return mo <= 16 ? 16 : mo <= 32 ? 32 : (mo <= 64 || d3 > tile_rows(128)) ? 64 : 128; }

// ---------------------------------------------------------------------------------------------- weight gradient, any irrep
// grad_W_p[u, v, w] += sum_{z, k} A[z, k, u] grad_out[z, w, k]: a block owns the K entries of up to 128 / 64 / 32 channels
// (whole chunks) x 32 / 64 / 128 output channels in registers and walks every splits-th tile of 64 (z, k) rows.
constexpr int kBwRows = 64;

struct BwdWLaunch {
    int n;
    int first_block[kMaxGroups + 1];
    int splits[kMaxGroups];
    int16_t group[kMaxGroups];
    int16_t bw[kMaxGroups];              // output channels of a block: 32, 64 or 128
};

template <int BW>
__device__ __forceinline__ void bwd_w_block(const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                            const float* __restrict__ gout, float* __restrict__ grad_w, int64_t Z, int block, int splits,
                                            float* smem) {
    constexpr int KB = 4096 / BW, NCH = KB / kKC, lda = KB + 4, ldg = BW + 4;
    constexpr int CX = BW / kTN, LX = 8, LY = 4, WC = CX / LX;
    const int out_off = g[0], mo = g[1], d3 = g[2], d1row = P.d1row(), d2row = P.d2row(), dout = P.plan[3];
    const int kblocks = (g[4] + NCH - 1) / NCH, wblocks = (mo + BW - 1) / BW, tz = kBwRows / d3, rows = tz * d3;
    const int split = block / (kblocks * wblocks), rest = block % (kblocks * wblocks);
    const int ch0 = (rest / wblocks) * NCH, nch = min(NCH, g[4] - ch0);
    const int w0 = (rest % wblocks) * BW, cols = min(BW, mo - w0);
    float* sA = smem;
    float* sG = smem + kBwRows * lda;
    float* sT = sG + kBwRows * ldg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % WC) * LX + (lane & 7), ty = (warp / WC) * LY + (lane >> 3);

    float acc[kTM][kTN];
#pragma unroll
    for (int i = 0; i < kTM; ++i)
#pragma unroll
        for (int j = 0; j < kTN; ++j) acc[i][j] = 0.0f;

    const int64_t tiles = (Z + tz - 1) / tz;
    for (int64_t tile = split; tile < tiles; tile += splits) {
        const int64_t z0 = tile * tz;
        __syncthreads();
        for (int c = 0; c < nch; ++c) {
            const int32_t* ch = P.chunk(g[3] + ch0 + c);
            const int32_t* path = P.path(ch[0]);
            const int d1 = path[0], ldt = (d1 * d3) | 1;
            const bool coupled = ch[3] >= 0;
            if (coupled && (ch[5] || c == 0)) {
                __syncthreads();      // the previous chunk's readers of sT
                stage_coupling(P.plan, path, x2, d2row, ch[3], z0, tz, Z, sT, ldt);
                __syncthreads();
            }
            stage_rows(d1, x1, d1row, ch[1], ch[2], z0, tz, Z, d3, coupled, __int_as_float(path[15]), sT, ldt, sA + c * kKC, lda);
        }
        // cotangent columns: [(z, k)][w]
        for (int zl = warp; zl < tz; zl += kThreads / 32) {
            const float* gr = gout + (z0 + zl) * dout + out_off + w0 * d3;
            const bool live = z0 + zl < Z;
            for (int e = lane; e < BW * d3; e += 32) {
                const int w = e / d3, k = e - w * d3;
                sG[(zl * d3 + k) * ldg + w] = (live && w < cols) ? __ldg(gr + e) : 0.0f;
            }
        }
        __syncthreads();
        float part[kTM][kTN];
#pragma unroll
        for (int i = 0; i < kTM; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) part[i][j] = 0.0f;
        if (ty * kTM < nch * kKC) {
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
                const float4 a0 = *reinterpret_cast<const float4*>(sA + r * lda + ty * kTM);
                const float4 a1 = *reinterpret_cast<const float4*>(sA + r * lda + ty * kTM + 4);
                const float4 b = *reinterpret_cast<const float4*>(sG + r * ldg + tx * kTN);
                const float av[kTM] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                const float bv[kTN] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < kTM; ++i)
#pragma unroll
                    for (int j = 0; j < kTN; ++j) part[i][j] = fmaf(av[i], bv[j], part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < kTM; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) acc[i][j] += part[i][j];
    }
#pragma unroll
    for (int i = 0; i < kTM; ++i) {
        const int kk = ty * kTM + i, c = kk / kKC, u = kk - c * kKC;
        if (c >= nch) continue;
        const int32_t* ch = P.chunk(g[3] + ch0 + c);
        if (u >= ch[2]) continue;
        const int32_t* path = P.path(ch[0]);
        float* p = grad_w + ch[4] + static_cast<int64_t>(u) * path[3] + static_cast<int64_t>(w0 + tx * kTN) * path[4];
#pragma unroll
        for (int j = 0; j < kTN; ++j)
            if (tx * kTN + j < cols) atomicAdd(p + static_cast<int64_t>(j) * path[4], acc[i][j]);
    }
}

__global__ void __launch_bounds__(kThreads, 4) dense_tile_bwd_w_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                    const float* __restrict__ x2, const float* __restrict__ gout,
                                                                    float* __restrict__ grad_w, int64_t Z, BwdWLaunch L) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* g = P.group(L.group[s]);
    const int block = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (L.bw[s]) {
        case 32: bwd_w_block<32>(P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
        case 64: bwd_w_block<64>(P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
        default: bwd_w_block<128>(P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
    }
}

// ---------------------------------------------------------------------------------------------- irreps of l <= 3
// For output irreps of dimension D3 <= 7 (compile time) operands stay in row order, [z][channel * D + component], the
// order they have in memory: a thread owns whole rows z, so 4 channels of one row are D3 aligned 16-byte reads, the
// sum over components needs no transposed copy, rows arrive by cp.async while the chunk before is multiplied, and
// results leave as 16-byte stores.  (The form above, used for l > 3, transposes every chunk into (z, k) rows with
// loads that wait for memory one after another: 1.86 ms for the weight gradient of a 6336 -> 1024 Linear on 16,384
// rows, 13 GFLOP.)
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool live) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// dst[z * ld + e] <- src[z * row + e], e < n (zero for n <= e < width and for z >= nz_live), z < BZ; width, ld % 4 == 0.
template <int BZ>
__device__ __forceinline__ void fetch_rows(float* dst, int ld, const float* __restrict__ src, int row, int n, int width, int nz_live) {
    if ((row & 3) == 0 && (n & 3) == 0 && aligned16(src)) {
        const int q = width >> 2;
        for (int idx = threadIdx.x; idx < BZ * q; idx += kThreads) {
            const int z = idx / q, e = (idx - z * q) * 4;
            const bool live = z < nz_live && e < n;
            cp_async16(dst + z * ld + e, live ? src + static_cast<int64_t>(z) * row + e : src, live);
        }
    } else {
        for (int idx = threadIdx.x; idx < BZ * width; idx += kThreads) {
            const int z = idx / width, e = idx - z * width;
            const bool live = z < nz_live && e < n;
            cp_async4(dst + z * ld + e, live ? src + static_cast<int64_t>(z) * row + e : src, live);
        }
    }
}

// dst[kk * ld + n] <- W[kk * su + n * sw], kk < 32, n < BN, zero outside len x cols.
template <int BN>
__device__ __forceinline__ void fetch_weights(float* dst, int ld, const float* __restrict__ W, int su, int sw, int len, int cols) {
    if (sw == 1 && (su & 3) == 0 && (cols & 3) == 0 && aligned16(W)) {
        for (int idx = threadIdx.x; idx < kKC * BN / 4; idx += kThreads) {
            const int kk = idx / (BN / 4), n = (idx % (BN / 4)) * 4;
            const bool live = kk < len && n < cols;
            cp_async16(dst + kk * ld + n, live ? W + static_cast<int64_t>(kk) * su + n : W, live);
        }
    } else {
        for (int idx = threadIdx.x; idx < kKC * BN; idx += kThreads) {
            const int kk = sw == 1 ? idx / BN : idx % kKC, n = sw == 1 ? idx % BN : idx / kKC;
            const bool live = kk < len && n < cols;
            cp_async4(dst + kk * ld + n, live ? W + static_cast<int64_t>(kk) * su + static_cast<int64_t>(n) * sw : W, live);
        }
    }
}

// T[z][k * d1 + i] of BZ rows from the second operand's rows in shared memory.
template <int BZ>
__device__ __forceinline__ void couple_rows(const int32_t* plan, const int32_t* path, const float* sY, int ldy, int x2off, float* sT, int ldt) {
    const int n = path[0] * path[2];
    const int32_t* seg = plan + path[5];
    for (int idx = threadIdx.x; idx < BZ * n; idx += kThreads) {
        const int z = idx / n, ki = idx - z * n;
        const float* y = sY + z * ldy + x2off;
        float t = 0.0f;
        for (int s = seg[ki]; s < seg[ki + 1]; s += 2) t = fmaf(__int_as_float(plan[s + 1]), y[plan[s]], t);
        sT[z * ldt + ki] = t;
    }
}

// A[z][u * D3 + k] = sum_i T[z][k * D1 + i] X[z][u * D1 + i], u < 32.
template <int D3, int D1, int BZ>
__device__ __forceinline__ void build_rows_d(const float* sX, int ldx, const float* sT, int ldt, float* sA, int lda) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int z = warp; z < BZ; z += kThreads / 32) {
        float x[D1];
#pragma unroll
        for (int i = 0; i < D1; ++i) x[i] = sX[z * ldx + lane * D1 + i];
        const float* t = sT + z * ldt;
#pragma unroll
        for (int k = 0; k < D3; ++k) {
            float v = 0.0f;
#pragma unroll
            for (int i = 0; i < D1; ++i) v = fmaf(t[k * D1 + i], x[i], v);
            sA[z * lda + lane * D3 + k] = v;
        }
    }
}

template <int D3, int BZ>
__device__ __forceinline__ void build_rows(int d1, const float* sX, int ldx, const float* sT, int ldt, float* sA, int lda) {
    switch (d1) {
        case 1: build_rows_d<D3, 1, BZ>(sX, ldx, sT, ldt, sA, lda); break;
        case 3: build_rows_d<D3, 3, BZ>(sX, ldx, sT, ldt, sA, lda); break;
        case 5: build_rows_d<D3, 5, BZ>(sX, ldx, sT, ldt, sA, lda); break;
        default: build_rows_d<D3, 7, BZ>(sX, ldx, sT, ldt, sA, lda); break;
    }
}

// Rows of a forward tile.  TX threads share a row (8 channels each); a thread owns rows_per_thread rows.
template <int D3, int TX, bool COUPLED>
__host__ __device__ constexpr int rows_per_thread() {
    // uncoupled: up to 56 accumulators; coupled: at most 32 rows a block, so that the chunk of the first operand and the
    // coupled chunk (32 x 7 floats a row each) leave room for several blocks on an SM
    return COUPLED ? (D3 == 1 ? TX / 4 : D3 == 3 ? (TX >= 8 ? 2 : 1) : 1) : (D3 == 1 ? 4 : D3 == 3 ? 2 : 1);
}

__host__ __device__ constexpr int pad_row(int floats) { return floats + 4; }      // rows 4 banks apart

template <int D3, int TX, bool COUPLED>
constexpr int fwd_rows() { return kThreads / TX * rows_per_thread<D3, TX, COUPLED>(); }

// Shared floats of a forward tile: two row buffers, two weight buffers, coupling, second operand.
template <int D3, int TX, bool COUPLED>
inline size_t fwd_floats(int d1max, int d2row) {
    constexpr int BZ = fwd_rows<D3, TX, COUPLED>();
    const size_t w = 2 * kKC * (8 * TX + 4);
    if (!COUPLED) return w + 2 * static_cast<size_t>(BZ) * pad_row(32 * D3);
    return w + static_cast<size_t>(BZ) * (pad_row(32 * d1max) + pad_row(32 * D3) + (d1max * D3 | 1) + (d2row | 1));
}

// NARROW: some chunk has fewer than 32 channels.
template <int D3, int TX, bool COUPLED, bool GATE, bool NARROW>
__device__ __forceinline__ void fwd_rows_tile(const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                              const float* __restrict__ W, float* __restrict__ out, int64_t Z, int tile, int accumulate,
                                              const DenseGateEpilogue& ep, float* smem) {
    constexpr int ZPT = rows_per_thread<D3, TX, COUPLED>(), TZ = kThreads / TX, BZ = TZ * ZPT, BN = 8 * TX, ldw = BN + 4;
    const int out_off = g[0], mo = g[1], nch = g[4], d1row = P.d1row(), d2row = P.d2row(), dout = P.plan[3];
    const int col_blocks = (mo + BN - 1) / BN;
    const int64_t z0 = static_cast<int64_t>(tile / col_blocks) * BZ;
    const int live = static_cast<int>(min(static_cast<int64_t>(BZ), Z - z0));
    const int c0 = (tile % col_blocks) * BN, cols = min(BN, mo - c0);
    const int ldx = pad_row(32 * (COUPLED ? P.d1max() : D3)), ldy = d2row | 1;
    constexpr int lda = pad_row(32 * D3);
    float* sW = smem;                                        // [2][32][ldw]
    float* sX = smem + 2 * kKC * ldw;                        // coupled: one chunk of x1; uncoupled: [2] chunks
    float* sA = sX + BZ * ldx;                               // coupled operand
    float* sT = sA + BZ * lda;
    float* sY = sT + (COUPLED ? BZ * (P.d1max() * D3 | 1) : 0);
    const int tid = threadIdx.x, tx = tid % TX, tz = tid / TX;

    auto fetch = [&](int c) {
        const int32_t* ch = P.chunk(g[3] + c);
        const int32_t* path = P.path(ch[0]);
        const int d1 = COUPLED ? path[0] : D3;
        fetch_rows<BZ>(sX + (COUPLED ? 0 : (c & 1) * BZ * ldx), ldx, x1 + z0 * d1row + ch[1], d1row, ch[2] * d1, 32 * d1, live);
        fetch_weights<BN>(sW + (c & 1) * kKC * ldw, ldw, W + ch[4] + static_cast<int64_t>(c0) * path[4], path[3], path[4], ch[2], cols);
        cp_async_commit();
    };

    float acc[ZPT][D3][8];
#pragma unroll
    for (int p = 0; p < ZPT; ++p)
#pragma unroll
        for (int k = 0; k < D3; ++k)
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[p][k][n] = 0.0f;

    // sums of up to 32 entries, over several chunks where the paths have fewer channels, in accumulators of their own: the
    // rounding error grows with sqrt(32) + sqrt(K / 32)
    float part[ZPT][D3][8];
#pragma unroll
    for (int p = 0; p < ZPT; ++p)
#pragma unroll
        for (int k = 0; k < D3; ++k)
#pragma unroll
            for (int n = 0; n < 8; ++n) part[p][k][n] = 0.0f;
    int held = 0;

    if (COUPLED)
        for (int idx = tid; idx < BZ * d2row; idx += kThreads) {
            const int z = idx / d2row, e = idx - z * d2row;
            cp_async4(sY + z * ldy + e, z < live ? x2 + (z0 + z) * d2row + e : x2, z < live);
        }
    fetch(0);
    for (int c = 0; c < nch; ++c) {
        const int32_t* ch = P.chunk(g[3] + c);
        const int32_t* path = P.path(ch[0]);
        const float* A = sX + (c & 1) * BZ * ldx;
        float coef = 1.0f;
        if (COUPLED) {
            const int d1 = path[0], ldt = (d1 * D3) | 1;
            cp_async_wait<0>();
            __syncthreads();          // this chunk is there; everyone is done with the previous coupled operand
            if (ch[5]) {
                couple_rows<BZ>(P.plan, path, sY, ldy, ch[3], sT, ldt);
                __syncthreads();
            }
            build_rows<D3, BZ>(d1, sX, ldx, sT, ldt, sA, lda);
            __syncthreads();
            if (c + 1 < nch) fetch(c + 1);
            A = sA;
        } else {
            coef = __int_as_float(path[15]);
            if (c + 1 < nch) { fetch(c + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
            __syncthreads();
        }
        const float* w = sW + (c & 1) * kKC * ldw;
        const int uend = (ch[2] + 3) & ~3;
#pragma unroll 1
        for (int u = 0; u < uend; u += 4) {
            float wv[4][8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 lo = *reinterpret_cast<const float4*>(w + (u + q) * ldw + tx * 4);
                const float4 hi = *reinterpret_cast<const float4*>(w + (u + q) * ldw + BN / 2 + tx * 4);
                wv[q][0] = lo.x; wv[q][1] = lo.y; wv[q][2] = lo.z; wv[q][3] = lo.w;
                wv[q][4] = hi.x; wv[q][5] = hi.y; wv[q][6] = hi.z; wv[q][7] = hi.w;
            }
#pragma unroll
            for (int p = 0; p < ZPT; ++p) {
                float a[4 * D3];
#pragma unroll
                for (int e = 0; e < D3; ++e) {
                    const float4 t = *reinterpret_cast<const float4*>(A + (tz + TZ * p) * (COUPLED ? lda : ldx) + u * D3 + 4 * e);
                    a[4 * e] = t.x; a[4 * e + 1] = t.y; a[4 * e + 2] = t.z; a[4 * e + 3] = t.w;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int k = 0; k < D3; ++k)
#pragma unroll
                        for (int n = 0; n < 8; ++n) part[p][k][n] = fmaf(a[q * D3 + k], wv[q][n], part[p][k][n]);
            }
        }
        held += ch[2];
        bool keep = NARROW && c + 1 < nch && held + P.chunk(g[3] + c + 1)[2] <= kKC;
        if (!COUPLED && keep) keep = P.path(P.chunk(g[3] + c + 1)[0])[15] == path[15];      // one coefficient
        if (!keep) {
            held = 0;
#pragma unroll
            for (int p = 0; p < ZPT; ++p)
#pragma unroll
                for (int k = 0; k < D3; ++k)
#pragma unroll
                    for (int n = 0; n < 8; ++n) { acc[p][k][n] = fmaf(coef, part[p][k][n], acc[p][k][n]); part[p][k][n] = 0.0f; }
        }
        if (!COUPLED) __syncthreads();          // the buffers are fetched into again
    }
    const bool vec = (dout & 3) == 0 && (cols & 3) == 0 && aligned16(out + out_off + c0 * D3) && !accumulate;
#pragma unroll
    for (int p = 0; p < ZPT; ++p) {
        const int z = tz + TZ * p;
        if (z >= live) continue;
        float* o = out + (z0 + z) * dout + out_off + c0 * D3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n0 = h * (BN / 2) + tx * 4;
            if (n0 >= cols) continue;
            if (GATE) {
                // one table entry per channel (its components are consecutive columns and share the gate)
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    if (n0 + n >= cols) continue;
                    const int col = out_off + (c0 + n0 + n) * D3;
                    const int4 e = __ldg(reinterpret_cast<const int4*>(ep.tbl) + col);      // kind, destination, activation, gate slot
                    if (e.x == 1) {
                        const float gate = ep.gates[(z0 + z) * ep.n_slots + e.w];
#pragma unroll
                        for (int k = 0; k < D3; ++k) ep.final_out[(z0 + z) * ep.dout_final + e.y + k] = acc[p][k][4 * h + n] * gate;
                    } else if (e.x == 0 || e.x == 2) {
                        const float v = ep.cst[col] * gate_act(e.z, acc[p][0][4 * h + n]);
                        if (e.x == 0) ep.final_out[(z0 + z) * ep.dout_final + e.y] = v;
                        else ep.gates[(z0 + z) * ep.n_slots + e.w] = v;
                    }
                }
            } else if (vec) {
#pragma unroll
                for (int e = 0; e < D3; ++e) {
                    // element 4 e + r of the 4 channels' run is channel (4 e + r) / D3, component (4 e + r) % D3
                    float4 t;
                    t.x = acc[p][(4 * e) % D3][4 * h + (4 * e) / D3];
                    t.y = acc[p][(4 * e + 1) % D3][4 * h + (4 * e + 1) / D3];
                    t.z = acc[p][(4 * e + 2) % D3][4 * h + (4 * e + 2) / D3];
                    t.w = acc[p][(4 * e + 3) % D3][4 * h + (4 * e + 3) / D3];
                    *reinterpret_cast<float4*>(o + n0 * D3 + 4 * e) = t;
                }
            } else {
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    if (n0 + n >= cols) continue;
#pragma unroll
                    for (int k = 0; k < D3; ++k) {
                        float* q = o + (n0 + n) * D3 + k;
                        *q = accumulate ? *q + acc[p][k][4 * h + n] : acc[p][k][4 * h + n];
                    }
                }
            }
        }
    }
}

struct FwdShape { int rows; size_t floats; };

template <int D3, bool COUPLED>
inline FwdShape fwd_shape_tx(int tx, int d1max, int d2row) {
    if (tx == 4) return {fwd_rows<D3, 4, COUPLED>(), fwd_floats<D3, 4, COUPLED>(d1max, d2row)};
    if (tx == 8) return {fwd_rows<D3, 8, COUPLED>(), fwd_floats<D3, 8, COUPLED>(d1max, d2row)};
    return {fwd_rows<D3, 16, COUPLED>(), fwd_floats<D3, 16, COUPLED>(d1max, d2row)};
}

template <bool COUPLED>
inline FwdShape fwd_shape(int d3, int tx, int d1max, int d2row) {
    switch (d3) {
        case 1: return fwd_shape_tx<1, COUPLED>(tx, d1max, d2row);
        case 3: return fwd_shape_tx<3, COUPLED>(tx, d1max, d2row);
        case 5: return fwd_shape_tx<5, COUPLED>(tx, d1max, d2row);
        default: return fwd_shape_tx<7, COUPLED>(tx, d1max, d2row);
    }
}

template <int D3, bool COUPLED, bool GATE, bool NARROW>
__device__ __forceinline__ void fwd_rows_tx(int tx, const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                            const float* __restrict__ W, float* __restrict__ out, int64_t Z, int tile, int accumulate,
                                            const DenseGateEpilogue& ep, float* smem) {
    if (tx == 4) fwd_rows_tile<D3, 4, COUPLED, GATE, NARROW>(P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem);
    else if (tx == 8) fwd_rows_tile<D3, 8, COUPLED, GATE, NARROW>(P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem);
    else fwd_rows_tile<D3, 16, COUPLED, GATE, NARROW>(P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem);
}

struct RowsLaunch {
    int n;                               // groups of this launch
    int first_block[kMaxGroups + 1];
    int splits[kMaxGroups];              // (weight gradient)
    int16_t group[kMaxGroups];
    int16_t shape[kMaxGroups];           // forward: threads a row; weight gradient: output channels of a block
};

template <bool COUPLED, bool GATE, bool NARROW>
__global__ void __launch_bounds__(kThreads, 3) dense_rows_fwd_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                     const float* __restrict__ x2, const float* __restrict__ W,
                                                                     float* __restrict__ out, int64_t Z, int accumulate, RowsLaunch L,
                                                                     DenseGateEpilogue ep) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* g = P.group(L.group[s]);
    const int tile = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (g[2]) {
        case 1: fwd_rows_tx<1, COUPLED, GATE, NARROW>(L.shape[s], P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem); break;
        case 3: fwd_rows_tx<3, COUPLED, GATE, NARROW>(L.shape[s], P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem); break;
        case 5: fwd_rows_tx<5, COUPLED, GATE, NARROW>(L.shape[s], P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem); break;
        default: fwd_rows_tx<7, COUPLED, GATE, NARROW>(L.shape[s], P, g, x1, x2, W, out, Z, tile, accumulate, ep, smem); break;
    }
}

// ---- weight gradient: 4096 = KB x BW entries of one group in registers (8 x 4 a thread), rows streamed
template <int D3, bool COUPLED>
__host__ __device__ constexpr int wgrad_rows() { return COUPLED ? 8 : D3 == 1 ? 32 : D3 == 3 ? 16 : 8; }

template <int D3, int BW, bool COUPLED>
inline size_t wgrad_floats(int d1max, int d2row) {
    constexpr int KB = 4096 / BW, BZ = wgrad_rows<D3, COUPLED>(), NCH = KB / kKC;
    const size_t gbuf = 2 * static_cast<size_t>(BZ) * pad_row(BW * D3);
    if (!COUPLED) return gbuf + 2 * static_cast<size_t>(BZ) * pad_row(KB * D3);
    return gbuf + static_cast<size_t>(BZ) * (pad_row(KB * d1max) + pad_row(KB * D3) + NCH * (d1max * D3 | 1) + 2 * (d2row | 1));
}

template <int D3, int BW, bool COUPLED>
__device__ __forceinline__ void wgrad_block(const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                            const float* __restrict__ gout, float* __restrict__ grad_w, int64_t Z, int block, int splits,
                                            float* smem) {
    constexpr int KB = 4096 / BW, NCH = KB / kKC, BZ = wgrad_rows<D3, COUPLED>(), ldg = pad_row(BW * D3), lda = pad_row(KB * D3);
    constexpr int CX = BW / kTN, WC = CX / 8;
    const int out_off = g[0], mo = g[1], d1row = P.d1row(), d2row = P.d2row(), dout = P.plan[3];
    const int kblocks = (g[4] + NCH - 1) / NCH, wblocks = (mo + BW - 1) / BW;
    const int split = block / (kblocks * wblocks), rest = block % (kblocks * wblocks);
    const int ch0 = (rest / wblocks) * NCH, nch = min(NCH, g[4] - ch0);
    const int w0 = (rest % wblocks) * BW, cols = min(BW, mo - w0);
    const int d1max = P.d1max(), ldx = COUPLED ? pad_row(KB * d1max) : lda, ldy = d2row | 1, ldt = COUPLED ? (d1max * D3 | 1) : 0;
    float* sG = smem;                                   // [2][BZ][ldg]
    float* sX = smem + 2 * BZ * ldg;                    // uncoupled: [2][BZ][lda]; coupled: one set of x1 chunks
    float* sA = sX + BZ * ldx;
    float* sT = sA + BZ * lda;                          // [NCH][BZ][ldt]
    float* sY = sT + NCH * BZ * ldt;                    // [2][BZ][ldy]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % WC) * 8 + (lane & 7), ty = (warp / WC) * 4 + (lane >> 3);

    auto fetch = [&](int64_t tile, int buf) {
        const int64_t z0 = tile * BZ;
        const int live = static_cast<int>(min(static_cast<int64_t>(BZ), Z - z0));
        int col = 0;
        for (int c = 0; c < nch; ++c) {
            const int32_t* ch = P.chunk(g[3] + ch0 + c);
            const int d1 = COUPLED ? P.path(ch[0])[0] : D3;
            fetch_rows<BZ>(sX + (COUPLED ? 0 : buf * BZ * lda) + col, ldx, x1 + z0 * d1row + ch[1], d1row, ch[2] * d1, 32 * d1, live);
            col += 32 * d1;
        }
        fetch_rows<BZ>(sG + buf * BZ * ldg, ldg, gout + z0 * dout + out_off + w0 * D3, dout, cols * D3, BW * D3, live);
        if (COUPLED)
            for (int idx = tid; idx < BZ * d2row; idx += kThreads) {
                const int z = idx / d2row, e = idx - z * d2row;
                cp_async4(sY + (buf * BZ + z) * ldy + e, z < live ? x2 + (z0 + z) * d2row + e : x2, z < live);
            }
        cp_async_commit();
    };

    float acc[kTM][kTN];
#pragma unroll
    for (int i = 0; i < kTM; ++i)
#pragma unroll
        for (int j = 0; j < kTN; ++j) acc[i][j] = 0.0f;

    const int64_t tiles = (Z + BZ - 1) / BZ;
    int buf = 0;
    if (split < tiles) fetch(split, 0);
    for (int64_t tile = split; tile < tiles; tile += splits, buf ^= 1) {
        const bool more = tile + splits < tiles;
        const float* A = sX + buf * BZ * lda;
        if (COUPLED) {
            cp_async_wait<0>();
            __syncthreads();
            for (int c = 0; c < nch; ++c) {
                const int32_t* ch = P.chunk(g[3] + ch0 + c);
                if (ch[5] || c == 0) {
                    const int32_t* path = P.path(ch[0]);
                    couple_rows<BZ>(P.plan, path, sY + buf * BZ * ldy, ldy, ch[3], sT + c * BZ * ldt, (path[0] * D3) | 1);
                }
            }
            __syncthreads();
            int col = 0, tc = 0;
            for (int c = 0; c < nch; ++c) {
                const int32_t* ch = P.chunk(g[3] + ch0 + c);
                const int d1 = P.path(ch[0])[0];
                if (ch[5] || c == 0) tc = c;
                build_rows<D3, BZ>(d1, sX + col, ldx, sT + tc * BZ * ldt, (d1 * D3) | 1, sA + c * kKC * D3, lda);
                col += 32 * d1;
            }
            __syncthreads();
            if (more) fetch(tile + splits, buf ^ 1);
            A = sA;
        } else {
            if (more) { fetch(tile + splits, buf ^ 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
            __syncthreads();
        }
        const float* G = sG + buf * BZ * ldg;
        if (ty * kTM < nch * kKC) {
            float part[kTM][kTN];
#pragma unroll
            for (int i = 0; i < kTM; ++i)
#pragma unroll
                for (int j = 0; j < kTN; ++j) part[i][j] = 0.0f;
#pragma unroll 1
            for (int z = 0; z < BZ; ++z) {
                float b[kTN * D3];
#pragma unroll
                for (int e = 0; e < D3; ++e) {
                    const float4 t = *reinterpret_cast<const float4*>(G + z * ldg + tx * kTN * D3 + 4 * e);
                    b[4 * e] = t.x; b[4 * e + 1] = t.y; b[4 * e + 2] = t.z; b[4 * e + 3] = t.w;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float a[4 * D3];
#pragma unroll
                    for (int e = 0; e < D3; ++e) {
                        const float4 t = *reinterpret_cast<const float4*>(A + z * lda + (ty * kTM + 4 * h) * D3 + 4 * e);
                        a[4 * e] = t.x; a[4 * e + 1] = t.y; a[4 * e + 2] = t.z; a[4 * e + 3] = t.w;
                    }
#pragma unroll
                    for (int k = 0; k < D3; ++k)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < kTN; ++j) part[4 * h + i][j] = fmaf(a[i * D3 + k], b[j * D3 + k], part[4 * h + i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < kTM; ++i)
#pragma unroll
                for (int j = 0; j < kTN; ++j) acc[i][j] += part[i][j];
        }
        if (!COUPLED) __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kTM; ++i) {
        const int kk = ty * kTM + i, c = kk / kKC, u = kk - c * kKC;
        if (c >= nch) continue;
        const int32_t* ch = P.chunk(g[3] + ch0 + c);
        if (u >= ch[2]) continue;
        const int32_t* path = P.path(ch[0]);
        const float coef = COUPLED ? 1.0f : __int_as_float(path[15]);
        const int sw = path[4], n0 = tx * kTN;
        float* p = grad_w + ch[4] + static_cast<int64_t>(u) * path[3] + static_cast<int64_t>(w0 + n0) * sw;
        if (sw == 1 && n0 + kTN <= cols && aligned16(p)) {
            atomicAdd(reinterpret_cast<float4*>(p), make_float4(coef * acc[i][0], coef * acc[i][1], coef * acc[i][2], coef * acc[i][3]));
        } else {
#pragma unroll
            for (int j = 0; j < kTN; ++j)
                if (n0 + j < cols) atomicAdd(p + static_cast<int64_t>(j) * sw, coef * acc[i][j]);
        }
    }
}

template <int D3, bool COUPLED>
inline size_t wgrad_floats_bw(int bw, int d1max, int d2row) {
    return bw == 32 ? wgrad_floats<D3, 32, COUPLED>(d1max, d2row) : bw == 64 ? wgrad_floats<D3, 64, COUPLED>(d1max, d2row)
                                                                             : wgrad_floats<D3, 128, COUPLED>(d1max, d2row);
}

template <bool COUPLED>
inline FwdShape wgrad_shape(int d3, int bw, int d1max, int d2row) {
    switch (d3) {
        case 1: return {wgrad_rows<1, COUPLED>(), wgrad_floats_bw<1, COUPLED>(bw, d1max, d2row)};
        case 3: return {wgrad_rows<3, COUPLED>(), wgrad_floats_bw<3, COUPLED>(bw, d1max, d2row)};
        case 5: return {wgrad_rows<5, COUPLED>(), wgrad_floats_bw<5, COUPLED>(bw, d1max, d2row)};
        default: return {wgrad_rows<7, COUPLED>(), wgrad_floats_bw<7, COUPLED>(bw, d1max, d2row)};
    }
}

template <int D3, bool COUPLED>
__device__ __forceinline__ void wgrad_bw(int bw, const Part2& P, const int32_t* g, const float* __restrict__ x1, const float* __restrict__ x2,
                                         const float* __restrict__ gout, float* __restrict__ grad_w, int64_t Z, int block, int splits,
                                         float* smem) {
    if (bw == 32) wgrad_block<D3, 32, COUPLED>(P, g, x1, x2, gout, grad_w, Z, block, splits, smem);
    else if (bw == 64) wgrad_block<D3, 64, COUPLED>(P, g, x1, x2, gout, grad_w, Z, block, splits, smem);
    else wgrad_block<D3, 128, COUPLED>(P, g, x1, x2, gout, grad_w, Z, block, splits, smem);
}

template <bool COUPLED>
__global__ void __launch_bounds__(kThreads, 4) dense_rows_wgrad_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                       const float* __restrict__ x2, const float* __restrict__ gout,
                                                                       float* __restrict__ grad_w, int64_t Z, RowsLaunch L) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* g = P.group(L.group[s]);
    const int block = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (g[2]) {
        case 1: wgrad_bw<1, COUPLED>(L.shape[s], P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
        case 3: wgrad_bw<3, COUPLED>(L.shape[s], P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
        case 5: wgrad_bw<5, COUPLED>(L.shape[s], P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
        default: wgrad_bw<7, COUPLED>(L.shape[s], P, g, x1, x2, gout, grad_w, Z, block, L.splits[s], smem); break;
    }
}

// ---------------------------------------------------------------------------------------------- operand gradients
// Both operand gradients of a 'uvw' product come from one intermediate per path:
//     Q[z, u, k]       = sum_w W_p[u, v, w] g[z, w, k]
//     grad_x1[z, u, i] += sum_k T_p[z, k, i] Q[z, u, k]
//     M[z, i, k]       = sum_u x1[z, u, i] Q[z, u, k],   grad_x2[z, v, j] += sum_{i, k} C_ijk M[z, i, k]
// A block owns one input irrep's 32 channels for 32 rows; a thread owns one row and 8 channels for every k and i, so
// the sums over k stay in its registers, and the sums over u cross 4 lanes.  Its share of grad_x2 goes to a partial of its
// own; a second kernel adds the partials in a fixed order (10,000 rows, three partials of nine columns: 2 us more than float
// atomics, whose sum varies from call to call).
constexpr int kBxZ = 32, kBxU = 8;
constexpr int kBxRun = 32;         // additions to an entry of grad_x1 in a register before it is put away (one run of 300: 1.5
                                   // to 2.5 times the error against 64 bits)

struct BwdXLaunch {
    int n;
    int first_block[kMaxGroups + 1];
    int first_part[kMaxGroups];          // of all blocks of 32 channels of the first operand, the group's first
    int16_t group[kMaxGroups];
};

struct BwdXShared {
    float *g, *w, *t, *m, *g2;      // g: [2] cotangent chunks, w: [2] weight chunks [channel of w][channel of u]
    int ldt, ldm, ld2, g_floats;    // g_floats: one cotangent buffer
};

// The walk over (path, second-operand channel, chunk of 32 output channels); the next step is fetched while one is used.
struct BwdXStep {
    int n, v, c0;
    const int32_t* path;
};

__device__ __forceinline__ bool bwd_x_next(const Part2& P, const int32_t* in, BwdXStep& s) {
    s.c0 += kKC;
    if (s.c0 < s.path[12]) return true;
    s.c0 = 0;
    if (++s.v < s.path[10]) return true;
    s.v = 0;
    if (++s.n >= in[4]) return false;
    s.path = P.path(P.in_path(in[3] + s.n));
    return true;
}

__device__ __forceinline__ void bwd_x_fetch(const Part2& P, const BwdXStep& s, const float* __restrict__ W, const float* __restrict__ gout,
                                            int64_t z0, int live, int u0, int nu, const BwdXShared& S, int buf) {
    const int d3 = s.path[2], su = s.path[3], sw = s.path[4], len = min(kKC, s.path[12] - s.c0), dout = P.plan[3];
    fetch_rows<kBxZ>(S.g + buf * S.g_floats, pad_row(32 * d3), gout + z0 * dout + s.path[11] + s.c0 * d3, dout, len * d3, 32 * d3, live);
    const float* w = W + s.path[13] + static_cast<int64_t>(u0) * su + static_cast<int64_t>(s.v) * s.path[14] + static_cast<int64_t>(s.c0) * sw;
    float* dst = S.w + buf * kKC * kLda;
    for (int idx = threadIdx.x; idx < kKC * 32; idx += kThreads) {
        const int ww = idx & 31, u = idx >> 5;
        const bool ok = ww < len && u < nu;
        cp_async4(dst + ww * kLda + u, ok ? w + static_cast<int64_t>(u) * su + static_cast<int64_t>(ww) * sw : W, ok);
    }
    cp_async_commit();
}

// One step: the chunk's share of Q and, at once, what it adds to both gradients (both are linear in Q, and a chunk's sum
// of 32 terms is then the only long chain of additions).
template <int D1, int D3, bool NEED1, bool NEED2>
__device__ __forceinline__ void bwd_x_step(const Part2& P, const BwdXStep& s, const float* __restrict__ xrow, bool xvec, int nu,
                                           const BwdXShared& S, int buf, float (&gx)[D1][kBxU]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 3, ty = warp * 8 + (lane >> 2);
    constexpr int ldg = pad_row(32 * D3), ldt = (D1 * D3) | 1;
    const float* G = S.g + buf * S.g_floats + ty * ldg;
    const float* w = S.w + buf * kKC * kLda + tx * kBxU;
    float q[D3][kBxU];
#pragma unroll
    for (int k = 0; k < D3; ++k)
#pragma unroll
        for (int u = 0; u < kBxU; ++u) q[k][u] = 0.0f;
    const int end = (min(kKC, s.path[12] - s.c0) + 3) & ~3;
#pragma unroll 1
    for (int c = 0; c < end; c += 4) {
        float a[4 * D3];
#pragma unroll
        for (int e = 0; e < D3; ++e) {
            const float4 t = *reinterpret_cast<const float4*>(G + c * D3 + 4 * e);
            a[4 * e] = t.x; a[4 * e + 1] = t.y; a[4 * e + 2] = t.z; a[4 * e + 3] = t.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 lo = *reinterpret_cast<const float4*>(w + (c + r) * kLda);
            const float4 hi = *reinterpret_cast<const float4*>(w + (c + r) * kLda + 4);
            const float wv[kBxU] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int k = 0; k < D3; ++k)
#pragma unroll
                for (int u = 0; u < kBxU; ++u) q[k][u] = fmaf(a[r * D3 + k], wv[u], q[k][u]);
        }
    }
    if (NEED1) {
#pragma unroll
        for (int k = 0; k < D3; ++k)
#pragma unroll
            for (int i = 0; i < D1; ++i) {
                const float t = S.t[ty * ldt + k * D1 + i];
#pragma unroll
                for (int u = 0; u < kBxU; ++u) gx[i][u] = fmaf(t, q[k][u], gx[i][u]);
            }
    }
    if (NEED2) {
        float m[D1 * D3];
#pragma unroll
        for (int e = 0; e < D1 * D3; ++e) m[e] = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float x[4 * D1];      // 4 channels of the row (cached: every path reads them again)
#pragma unroll
            for (int e = 0; e < D1; ++e) {
                const int at = (tx * kBxU + 4 * h) * D1 + 4 * e;
                if (xvec) {
                    const float4 t = at < nu * D1 ? __ldg(reinterpret_cast<const float4*>(xrow + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    x[4 * e] = t.x; x[4 * e + 1] = t.y; x[4 * e + 2] = t.z; x[4 * e + 3] = t.w;
                } else {
#pragma unroll
                    for (int r = 0; r < 4; ++r) x[4 * e + r] = at + r < nu * D1 ? __ldg(xrow + at + r) : 0.0f;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < D1; ++i)
#pragma unroll
                    for (int k = 0; k < D3; ++k) m[i * D3 + k] = fmaf(x[u * D1 + i], q[k][4 * h + u], m[i * D3 + k]);
        }
#pragma unroll
        for (int e = 0; e < D1 * D3; ++e) {
            m[e] += __shfl_xor_sync(0xffffffffu, m[e], 1);
            m[e] += __shfl_xor_sync(0xffffffffu, m[e], 2);
            if (tx == (e & 3)) S.m[ty * S.ldm + e] = m[e];
        }
        __syncwarp();
        // the 8 rows of a warp are its own: no barrier
        const int d2 = s.path[1], x2off = s.path[9] + s.v * d2;
        const int32_t* seg = P.plan + s.path[6];
        for (int t = lane; t < 8 * d2; t += 32) {
            const int zl = warp * 8 + t / d2, j = t % d2;
            float r = 0.0f;
            for (int e = seg[j]; e < seg[j + 1]; e += 2) r = fmaf(__int_as_float(P.plan[e + 1]), S.m[zl * S.ldm + P.plan[e]], r);
            S.g2[zl * S.ld2 + x2off + j] += r;
        }
        __syncwarp();
    }
}

// RUNS: some block of the first operand takes more than kBxRun additions (put away in between).
template <int D1, bool NEED1, bool NEED2, bool RUNS>
__device__ __forceinline__ void bwd_x_block(const Part2& P, const int32_t* in, const float* __restrict__ x1, const float* __restrict__ x2,
                                            const float* __restrict__ W, const float* __restrict__ gout, float* __restrict__ g1,
                                            float* __restrict__ g2, float* __restrict__ partial, int64_t Z, int block, int first_part,
                                            const BwdXShared& S) {
    const int x1off = in[0], m1 = in[1], ublocks = (m1 + 31) / 32;
    const int64_t z0 = static_cast<int64_t>(block / ublocks) * kBxZ;
    const int u0 = (block % ublocks) * 32, nu = min(32, m1 - u0);
    const int d1row = P.d1row(), d2row = P.d2row();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 3, ty = warp * 8 + (lane >> 2);
    float gx[D1][kBxU];
#pragma unroll
    for (int i = 0; i < D1; ++i)
#pragma unroll
        for (int u = 0; u < kBxU; ++u) gx[i][u] = 0.0f;
    const int live = static_cast<int>(min(static_cast<int64_t>(kBxZ), Z - z0));
    if (NEED2)
        for (int idx = lane; idx < 8 * S.ld2; idx += 32) S.g2[warp * 8 * S.ld2 + idx] = 0.0f;
    const float* xrow = x1 + (z0 + min(ty, live - 1)) * d1row + x1off + u0 * D1;
    const bool xvec = (d1row & 3) == 0 && (nu & 3) == 0 && aligned16(x1 + x1off);

    BwdXStep step{0, 0, 0, P.path(P.in_path(in[3]))};
    bwd_x_fetch(P, step, W, gout, z0, live, u0, nu, S, 0);
    // wide second operands: the sums so far are put away in grad_x1 now and then, so that the runs of additions stay short
    int run = 0;
    bool away = false;
    float* orow = RUNS ? g1 + (z0 + min(ty, live - 1)) * d1row + x1off + u0 * D1 : nullptr;
    for (int buf = 0;; buf ^= 1) {
        BwdXStep next = step;
        const bool more = bwd_x_next(P, in, next);
        if (more) bwd_x_fetch(P, next, W, gout, z0, live, u0, nu, S, buf ^ 1);
        if (NEED1 && step.c0 == 0)
            stage_coupling(P.plan, step.path, x2, d2row, step.path[9] + step.v * step.path[1], z0, kBxZ, Z, S.t, (D1 * step.path[2]) | 1);
        if (more) cp_async_wait<1>(); else cp_async_wait<0>();
        __syncthreads();
        switch (step.path[2]) {
            case 1: bwd_x_step<D1, 1, NEED1, NEED2>(P, step, xrow, xvec, nu, S, buf, gx); break;
            case 3: bwd_x_step<D1, 3, NEED1, NEED2>(P, step, xrow, xvec, nu, S, buf, gx); break;
            case 5: bwd_x_step<D1, 5, NEED1, NEED2>(P, step, xrow, xvec, nu, S, buf, gx); break;
            default: bwd_x_step<D1, 7, NEED1, NEED2>(P, step, xrow, xvec, nu, S, buf, gx); break;
        }
        __syncthreads();      // the buffers and the coupling are written again
        if (!more) break;
        if (RUNS && (run += step.path[2]) >= kBxRun) {
#pragma unroll
            for (int u = 0; u < kBxU; ++u)
#pragma unroll
                for (int i = 0; i < D1; ++i) {
                    float* o = orow + (tx * kBxU + u) * D1 + i;
                    if (ty < live && tx * kBxU + u < nu) *o = away ? *o + gx[i][u] : gx[i][u];
                    gx[i][u] = 0.0f;
                }
            run = 0;
            away = true;
        }
        step = next;
    }
    if (NEED1) {
        // [row][u * D1 + i] over the cotangent buffers, then contiguous row segments
        constexpr int ld = 32 * D1 + 1;
#pragma unroll
        for (int i = 0; i < D1; ++i)
#pragma unroll
            for (int u = 0; u < kBxU; ++u) S.g[ty * ld + (tx * kBxU + u) * D1 + i] = gx[i][u];
        __syncwarp();
        for (int r = 0; r < 8; ++r) {
            const int zl = warp * 8 + r;
            if (z0 + zl >= Z) break;
            float* o = g1 + (z0 + zl) * d1row + x1off + u0 * D1;
            for (int e = lane; e < nu * D1; e += 32) o[e] = RUNS && away ? o[e] + S.g[zl * ld + e] : S.g[zl * ld + e];
        }
    }
    if (NEED2) {
        __syncwarp();
        for (int r = 0; r < 8; ++r) {
            const int zl = warp * 8 + r;
            if (z0 + zl >= Z) break;
            float* o = (partial ? partial + (first_part + block % ublocks) * Z * d2row : g2) + (z0 + zl) * d2row;
            for (int e = lane; e < d2row; e += 32) {
                if (partial) o[e] = S.g2[zl * S.ld2 + e];
                else atomicAdd(o + e, S.g2[zl * S.ld2 + e]);
            }
        }
    }
}

template <bool NEED1, bool NEED2, bool RUNS>
__global__ void __launch_bounds__(kThreads, 3) dense_tile_bwd_x_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                       const float* __restrict__ x2, const float* __restrict__ W,
                                                                       const float* __restrict__ gout, float* __restrict__ g1,
                                                                       float* __restrict__ g2, float* __restrict__ partial, int64_t Z,
                                                                       int g_floats, BwdXLaunch L) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    BwdXShared S;
    S.ldt = (P.d1max() * P.d3max()) | 1;
    S.ldm = S.ldt;
    S.ld2 = P.d2row() | 1;
    S.g_floats = g_floats;
    S.g = smem;
    S.w = S.g + 2 * g_floats;
    S.t = S.w + 2 * kKC * kLda;
    S.m = S.t + kBxZ * S.ldt;
    S.g2 = S.m + (NEED2 ? kBxZ * S.ldm : 0);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* in = P.in_group(L.group[s]);
    const int block = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (in[2]) {
        case 1: bwd_x_block<1, NEED1, NEED2, RUNS>(P, in, x1, x2, W, gout, g1, g2, partial, Z, block, L.first_part[s], S); break;
        case 3: bwd_x_block<3, NEED1, NEED2, RUNS>(P, in, x1, x2, W, gout, g1, g2, partial, Z, block, L.first_part[s], S); break;
        case 5: bwd_x_block<5, NEED1, NEED2, RUNS>(P, in, x1, x2, W, gout, g1, g2, partial, Z, block, L.first_part[s], S); break;
        default: bwd_x_block<7, NEED1, NEED2, RUNS>(P, in, x1, x2, W, gout, g1, g2, partial, Z, block, L.first_part[s], S); break;
    }
}

// out[i] = sum of partial[0..parts)[i], i < count.
__global__ void __launch_bounds__(256) dense_bwd_x_sum_kernel(const float* __restrict__ partial, int parts, int64_t count, float* __restrict__ out) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float v = 0.0f;
#pragma unroll 4
    for (int p = 0; p < parts; ++p) v += partial[p * count + i];
    out[i] = v;
}

constexpr int kMaxShared = 227 * 1024;

// Blocks of 32 channels of the first operand, each with a partial of grad_x2.
inline int bwd_x_parts(const Part2& P) {
    int parts = 0;
    for (int g = 0; g < P.n_in(); ++g) parts += (P.in_group(g)[1] + 31) / 32;
    return parts;
}

// Rows whose partials are held at a time: at most 128 MB of them, at least 16 row tiles.
inline int64_t bwd_x_slab(const Part2& P, int parts, int64_t rows) {
    const int64_t fit = (int64_t{128} << 20) / (static_cast<int64_t>(sizeof(float)) * parts * std::max(P.d2row(), 1)) / kBxZ * kBxZ;
    return std::min<int64_t>(rows, std::max<int64_t>(fit, 16 * kBxZ));
}

// Floats of one cotangent buffer of dense_tile_bwd_x_kernel; the two together later hold the grad_x1 tile.
inline int bwd_x_g_floats(int d1max, int d3max) {
    return std::max(kBxZ * pad_row(32 * d3max), ((kBxZ * (32 * d1max + 1) + 1) / 2 + 3) & ~3);
}

inline size_t bwd_x_shared(const Part2& P, bool need2) {
    const int ldt = (P.d1max() * P.d3max()) | 1;
    size_t f = 2 * static_cast<size_t>(bwd_x_g_floats(P.d1max(), P.d3max())) + 2 * kKC * kLda + kBxZ * ldt;
    if (need2) f += static_cast<size_t>(kBxZ) * (ldt + (P.d2row() | 1));
    return f * sizeof(float);
}

// Under eight channels a chunk the table-driven kernel (dense.cu), whose contraction index runs over all pairs of channels, is
// the faster one: 10,000 rows of 4 x 4 -> 64 channels, l <= 2, 169 against 187 us, 100,000 rows of 1 x 1 -> 1, 294 against 504;
// with eight (30,000 rows of 8 x 8 -> 64) 1,313 against 1,051.
// A Linear goes there when an output has many such chunks, each with its copies and a barrier: 30,000 rows of 300 x 1 channel
// 648 -> 255 us; a few (4x0e+4x1o) are 17 us on the tiles against 79.
constexpr int64_t kFewChannels = 8;
constexpr int kFewChannelsChunks = 24;

bool too_many_blocks(int64_t blocks) { return blocks > 2147483647LL; }

}  // namespace

// Whether every group of the plan suits the row kernels: l <= 3 on both sides of every path.
static bool rows_plan(const Part2& P) {
    if (P.d1max() > 7 || P.d3max() > 7) return false;
    for (int g = 0; g < P.n_groups(); ++g)
        if (P.group(g)[2] > 7) return false;
    return true;
}

// Whether the tile of every group that has work fits a block's shared memory.
template <typename ShapeOf>
static bool all_groups_fit(const Part2& P, const ShapeOf& shape_of) {
    for (int n = 0; n < P.n_groups(); ++n) {
        const int32_t* g = P.group(n);
        if (g[1] != 0 && g[4] != 0 && shape_of(g).floats * sizeof(float) > static_cast<size_t>(kMaxShared)) return false;
    }
    return true;
}

// A plan couples a second operand in all of its paths (a product) or in none (a Linear).
static bool coupled_plan(const Part2& P) { return P.h[2] > 0 && P.chunk(0)[3] >= 0; }

// Launches go out up to kMaxGroups groups at a time.  *done = false: nothing was launched, because a group needs more shared
// memory than a block can have (a very wide second operand).
// pass: 0 every group, 1 the groups of scalars, 2 the others.  Scalar groups with Gate go out one launch each, in plan order: a
// gated scalar then finds the gates of an earlier irrep written (blocks of one grid have no order among them).
template <bool COUPLED, bool GATE>
static int launch_rows_fwd(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                           float* out, int64_t Z, int accumulate, const DenseGateEpilogue& ep, int pass, cudaStream_t s, bool* done) {
    const Part2 P(plan_host);
    const int most = GATE && pass == 1 ? 1 : kMaxGroups;
    const bool narrow = P.channels() < kKC * P.n_chunks();
    // the narrowest tile that holds the group's channels in one pass, so that the coupled operand is built once
    auto threads_a_row = [](const int32_t* g) { return g[1] <= 32 ? 4 : g[1] <= 64 ? 8 : 16; };
    auto shape_of = [&](const int32_t* g) { return fwd_shape<COUPLED>(g[2], threads_a_row(g), P.d1max(), P.d2row()); };
    *done = all_groups_fit(P, shape_of);
    if (!*done) return E3B_OK;
    int g0 = 0;
    while (g0 < P.n_groups()) {
        RowsLaunch L;
        L.n = 0;
        int64_t blocks = 0;
        size_t floats = 0;
        for (; g0 < P.n_groups() && L.n < most; ++g0) {
            const int32_t* g = P.group(g0);
            if (g[1] == 0 || g[4] == 0 || (pass == 1 && g[2] != 1) || (pass == 2 && g[2] == 1)) continue;
            const int tx = threads_a_row(g);
            const FwdShape shape = shape_of(g);
            L.first_block[L.n] = static_cast<int>(blocks);
            L.group[L.n] = static_cast<int16_t>(g0);
            L.shape[L.n] = static_cast<int16_t>(tx);
            blocks += ceil_div(Z, shape.rows) * ceil_div(g[1], 8 * tx);
            if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_fwd: too many rows");
            floats = std::max(floats, shape.floats);
            ++L.n;
        }
        if (L.n == 0) continue;
        L.first_block[L.n] = static_cast<int>(blocks);
        const size_t bytes = floats * sizeof(float);
        auto kernel = narrow ? dense_rows_fwd_kernel<COUPLED, GATE, true> : dense_rows_fwd_kernel<COUPLED, GATE, GATE>;
        E3B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, weight, out, Z, accumulate, L, ep);
        if (int rc = check_launch("e3b_dense_fwd")) return rc;
    }
    return E3B_OK;
}

// As launch_rows_fwd, for the weight gradient.
template <bool COUPLED>
static int launch_rows_wgrad(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* gout,
                             float* grad_w, int64_t Z, cudaStream_t s, bool* done) {
    const Part2 P(plan_host);
    auto channels_of = [](const int32_t* g) { return g[1] <= 32 ? 32 : g[1] <= 64 ? 64 : 128; };
    auto shape_of = [&](const int32_t* g) { return wgrad_shape<COUPLED>(g[2], channels_of(g), P.d1max(), P.d2row()); };
    *done = all_groups_fit(P, shape_of);
    if (!*done) return E3B_OK;
    int g0 = 0;
    while (g0 < P.n_groups()) {
        RowsLaunch L;
        L.n = 0;
        int64_t blocks = 0, work[kMaxGroups], total_work = 0, tiles[kMaxGroups], parts[kMaxGroups];
        size_t floats = 0;
        for (; g0 < P.n_groups() && L.n < kMaxGroups; ++g0) {
            const int32_t* g = P.group(g0);
            if (g[1] == 0 || g[4] == 0) continue;
            const int bw = channels_of(g);
            const FwdShape shape = shape_of(g);
            L.group[L.n] = static_cast<int16_t>(g0);
            L.shape[L.n] = static_cast<int16_t>(bw);
            parts[L.n] = ceil_div(g[4], 4096 / bw / kKC) * ceil_div(g[1], bw);
            tiles[L.n] = ceil_div(Z, shape.rows);
            work[L.n] = parts[L.n] * tiles[L.n] * shape.rows * g[2];
            total_work += work[L.n];
            floats = std::max(floats, shape.floats);
            ++L.n;
        }
        if (L.n == 0) continue;
        const size_t bytes = floats * sizeof(float);
        // one wave of resident blocks over all groups, in proportion to their rows x components
        const int64_t resident = kNumSMs * std::max<int64_t>(1, std::min<int64_t>(4, kMaxShared / static_cast<int64_t>(bytes + 1024)));
        for (int n = 0; n < L.n; ++n) {
            const int64_t share = resident * work[n] / total_work;
            L.splits[n] = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(tiles[n], share / parts[n])));
            L.first_block[n] = static_cast<int>(blocks);
            blocks += parts[n] * L.splits[n];
        }
        L.first_block[L.n] = static_cast<int>(blocks);
        if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_bwd_w: too many blocks");
        auto kernel = dense_rows_wgrad_kernel<COUPLED>;
        E3B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, gout, grad_w, Z, L);
        if (int rc = check_launch("e3b_dense_bwd_w")) return rc;
    }
    return E3B_OK;
}

int launch_dense_rows_gate(const int32_t* plan_host, const int32_t* plan_dev, const float* x, const float* weight,
                           const DenseGateEpilogue& ep, int64_t Z, cudaStream_t s, bool* done) {
    const Part2 P(plan_host);
    *done = false;
    if (!rows_plan(P) || coupled_plan(P)) return E3B_OK;
    // scalars and gates first: the gated irreps read the activated gates of the same rows
    if (int rc = launch_rows_fwd<false, true>(plan_host, plan_dev, x, nullptr, weight, nullptr, Z, 0, ep, 1, s, done)) return rc;
    if (!*done) return E3B_OK;
    return launch_rows_fwd<false, true>(plan_host, plan_dev, x, nullptr, weight, nullptr, Z, 0, ep, 2, s, done);
}

bool few_channels(const int32_t* plan_host) {
    const Part2 P(plan_host);
    if (P.channels() >= kFewChannels * P.n_chunks()) return false;
    if (coupled_plan(P)) return true;
    if (plan_host[4] != P.n_groups()) return false;      // a transposed Linear whose first part adds up groups
    int most = 0;
    for (int g = 0; g < P.n_groups(); ++g) most = std::max(most, P.group(g)[4]);
    return most > kFewChannelsChunks;
}

// The table-driven kernel contracts 64 pairs of channels and up to 128 output channels a block, however they come about; the
// register tiles take a chunk of 32 channels for every channel of the second operand, half as fast beyond 64 output channels.
// Both sides in microseconds a row as measured (l <= 2), and what the table takes to start: 30,000 rows of 4 x 4 -> 4 channels 422
// (table) and 1,789 us, 8 x 8 -> 64 1,613 / 3,729, 16 x 16 -> 16 5,780 / 7,723, but 16 x 3 -> 16 1,260 / 1,083, 32 x 8 -> 32 5,947 /
// 3,627 and 32 x 1 -> 32 816 / 270; 2,000 rows: 4 x 4 -> 4 95 / 129, 16 x 16 -> 16 433 / 526, 2 x 2 -> 2 85 / 64.
bool pairs_bwd_w(const int32_t* plan_host, int64_t num_rows) {
    const Part2 P(plan_host);
    if (!coupled_plan(P)) return false;
    const int32_t* first = plan_host + plan_host[7];
    double chunks = 0.0, blocks = 0.0;
    for (int n = 0; n < P.n_groups(); ++n) {
        const int mo = P.group(n)[1], wide = (mo + 127) / 128;
        if (first[6 * n + 2] > kBwRows) return false;
        chunks += P.group(n)[4] * wide * (mo > 64 ? 1.5 : 1.0);
        blocks += (first[6 * n + 3] + 63) / 64 * wide;
    }
    chunks /= std::max(P.n_groups(), 1);
    blocks /= std::max(P.n_groups(), 1);
    return static_cast<double>(num_rows) * ((chunks > 12.0 ? 0.0036 : 0.0028) * chunks - 0.0124 * blocks) > 45.0;
}

int launch_dense_tile_fwd(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                          float* out, int64_t Z, int accumulate, cudaStream_t s) {
    const Part2 P(plan_host);
    if (P.swapped()) std::swap(x1, x2);
    if (rows_plan(P)) {
        bool done = false;
        const DenseGateEpilogue none{nullptr, nullptr, nullptr, nullptr, 0, 0};
        const int rc = coupled_plan(P)
                           ? launch_rows_fwd<true, false>(plan_host, plan_dev, x1, x2, weight, out, Z, accumulate, none, 0, s, &done)
                           : launch_rows_fwd<false, false>(plan_host, plan_dev, x1, x2, weight, out, Z, accumulate, none, 0, s, &done);
        if (rc != E3B_OK || done) return rc;
    }
    int g0 = 0;
    while (g0 < P.n_groups()) {
        FwdLaunch L;
        L.n = 0;
        int64_t blocks = 0;
        size_t floats = 0;
        for (; g0 < P.n_groups() && L.n < kMaxGroups; ++g0) {
            const int32_t* g = P.group(g0);
            if (g[1] == 0 || g[4] == 0) continue;
            const int bn = columns_for(g[1], g[2]), bm = tile_rows(bn);
            if (g[2] > kMostDim) return fail(E3B_ERR_UNSUPPORTED, "dense_fwd: irrep dimension %d too large", g[2]);
            L.first_block[L.n] = static_cast<int>(blocks);
            L.group[L.n] = static_cast<int16_t>(g0);
            L.bn[L.n] = static_cast<int16_t>(bn);
            blocks += ceil_div(Z, bm / g[2]) * ceil_div(g[1], bn);
            if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_fwd: too many rows");
            const int tz = bm / g[2];
            floats = std::max(floats, static_cast<size_t>(bm * kLda + kKC * (bn + 4)) + static_cast<size_t>(tz) * (P.d1max() * g[2] | 1));
            ++L.n;
        }
        if (L.n == 0) continue;
        L.first_block[L.n] = static_cast<int>(blocks);
        const int bytes = static_cast<int>(floats * sizeof(float));
        if (bytes > kMaxShared) return fail(E3B_ERR_UNSUPPORTED, "dense_fwd: irrep dimensions too large");
        E3B_CUDA_TRY(cudaFuncSetAttribute(dense_tile_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        dense_tile_fwd_kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, weight, out, Z, accumulate, L);
        if (int rc = check_launch("e3b_dense_fwd")) return rc;
    }
    return E3B_OK;
}

int launch_dense_tile_bwd_w(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* gout,
                            float* grad_w, int64_t Z, cudaStream_t s) {
    const Part2 P(plan_host);
    if (P.swapped()) std::swap(x1, x2);
    if (rows_plan(P)) {
        bool done = false;
        const int rc = coupled_plan(P) ? launch_rows_wgrad<true>(plan_host, plan_dev, x1, x2, gout, grad_w, Z, s, &done)
                                       : launch_rows_wgrad<false>(plan_host, plan_dev, x1, x2, gout, grad_w, Z, s, &done);
        if (rc != E3B_OK || done) return rc;
    }
    int g0 = 0;
    while (g0 < P.n_groups()) {
        BwdWLaunch L;
        L.n = 0;
        int64_t blocks = 0, work[kMaxGroups], total_work = 0;
        size_t floats = 0;
        int parts[kMaxGroups];
        int64_t tiles[kMaxGroups];
        for (; g0 < P.n_groups() && L.n < kMaxGroups; ++g0) {
            const int32_t* g = P.group(g0);
            if (g[1] == 0 || g[4] == 0) continue;
            if (g[2] > kBwRows) return fail(E3B_ERR_UNSUPPORTED, "dense_bwd_w: irrep dimension %d too large", g[2]);
            const int bw = g[1] <= 32 ? 32 : g[1] <= 64 ? 64 : 128, nch = 4096 / bw / kKC, tz = kBwRows / g[2];
            L.group[L.n] = static_cast<int16_t>(g0);
            L.bw[L.n] = static_cast<int16_t>(bw);
            parts[L.n] = static_cast<int>(ceil_div(g[4], nch) * ceil_div(g[1], bw));
            tiles[L.n] = ceil_div(Z, tz);
            work[L.n] = parts[L.n] * tiles[L.n];
            total_work += work[L.n];
            floats = std::max(floats, static_cast<size_t>(kBwRows) * (4096 / bw + 4 + bw + 4) + static_cast<size_t>(tz) * (P.d1max() * g[2] | 1));
            ++L.n;
        }
        if (L.n == 0) continue;
        // four blocks per SM over all groups, split in proportion to their tiles
        for (int n = 0; n < L.n; ++n) {
            const int64_t share = (static_cast<int64_t>(kNumSMs) * 4 * work[n] + total_work - 1) / total_work;
            L.splits[n] = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(tiles[n], (share + parts[n] - 1) / parts[n])));
            L.first_block[n] = static_cast<int>(blocks);
            blocks += static_cast<int64_t>(parts[n]) * L.splits[n];
        }
        L.first_block[L.n] = static_cast<int>(blocks);
        if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_bwd_w: too many blocks");
        const int bytes = static_cast<int>(floats * sizeof(float));
        if (bytes > kMaxShared) return fail(E3B_ERR_UNSUPPORTED, "dense_bwd_w: irrep dimensions too large");
        E3B_CUDA_TRY(cudaFuncSetAttribute(dense_tile_bwd_w_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        dense_tile_bwd_w_kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, gout, grad_w, Z, L);
        if (int rc = check_launch("e3b_dense_bwd_w")) return rc;
    }
    return E3B_OK;
}

template <bool NEED1, bool NEED2>
static int launch_bwd_x(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                        const float* gout, float* g1, float* g2, float* partial, int64_t Z, cudaStream_t s) {
    const Part2 P(plan_host);
    const size_t bytes = bwd_x_shared(P, NEED2);
    bool runs = false;
    for (int n = 0; n < P.n_in(); ++n) {
        const int32_t* in = P.in_group(n);
        int64_t adds = 0;
        for (int q = 0; q < in[4]; ++q) {
            const int32_t* path = P.path(P.in_path(in[3] + q));
            adds += static_cast<int64_t>(path[10]) * ((path[12] + kKC - 1) / kKC) * path[2];
        }
        runs = runs || adds > kBxRun;
    }
    int g0 = 0, part = 0;
    while (g0 < P.n_in()) {
        BwdXLaunch L;
        L.n = 0;
        int64_t blocks = 0;
        for (; g0 < P.n_in() && L.n < kMaxGroups; ++g0) {
            const int32_t* in = P.in_group(g0);
            L.first_block[L.n] = static_cast<int>(blocks);
            L.first_part[L.n] = part;
            L.group[L.n] = static_cast<int16_t>(g0);
            part += (in[1] + 31) / 32;
            blocks += ceil_div(Z, kBxZ) * ceil_div(in[1], 32);
            if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_bwd_x: too many rows");
            ++L.n;
        }
        L.first_block[L.n] = static_cast<int>(blocks);
        auto kernel = runs ? dense_tile_bwd_x_kernel<NEED1, NEED2, NEED1> : dense_tile_bwd_x_kernel<NEED1, NEED2, false>;
        E3B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, weight, gout, g1, g2, partial, Z,
                                                                      bwd_x_g_floats(P.d1max(), P.d3max()), L);
        if (int rc = check_launch("e3b_dense_bwd_x")) return rc;
    }
    return E3B_OK;
}

}  // namespace e3b

extern "C" int e3b_dense_bwd_x_supported(const int32_t* plan_host) {
    using namespace e3b;
    if (!whole_plan(plan_host)) return 0;
    const Part2 P(plan_host);
    return P.n_in() > 0 && P.d1max() <= 7 && P.d3max() <= 7 && bwd_x_shared(P, true) <= static_cast<size_t>(kMaxShared);
}

namespace e3b {
// Operands in the plan's order.  partial: nullptr (grad_x2 by atomics) or bwd_x_parts() x rows x d2 floats (grad_x2 itself when there is one part).
static int bwd_x_rows(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight, const float* gout,
                      float* g1, float* g2, float* partial, int64_t Z, cudaStream_t s) {
    if (g1 && g2) return launch_bwd_x<true, true>(plan_host, plan_dev, x1, x2, weight, gout, g1, g2, partial, Z, s);
    if (g1) return launch_bwd_x<true, false>(plan_host, plan_dev, x1, x2, weight, gout, g1, g2, partial, Z, s);
    return launch_bwd_x<false, true>(plan_host, plan_dev, x1, x2, weight, gout, g1, g2, partial, Z, s);
}

static int bwd_x(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight, const float* gout,
                 float* g1, float* g2, int64_t Z, bool ordered, void* scratch, int64_t scratch_bytes, void* stream) {
    if (!whole_plan(plan_host)) return fail(E3B_ERR_ARG, "dense_bwd_x: bad plan (one without its second part has to be built again)");
    if (Z < 0) return fail(E3B_ERR_ARG, "dense_bwd_x: negative row count");
    if (Z == 0 || (!g1 && !g2)) return E3B_OK;
    if (!plan_dev || !x1 || !x2 || !weight || !gout) return fail(E3B_ERR_ARG, "dense_bwd_x: null pointer");
    if (!e3b_dense_bwd_x_supported(plan_host)) return fail(E3B_ERR_UNSUPPORTED, "dense_bwd_x: irreps above l = 3 or too wide");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Part2 P(plan_host);
    if (P.swapped()) {
        std::swap(x1, x2);
        std::swap(g1, g2);
    }
    const int64_t d1 = P.d1row(), d2 = P.d2row(), dout = plan_host[3];
    const int parts = bwd_x_parts(P);
    if (g1 && !P.covers_x1()) E3B_CUDA_TRY(cudaMemsetAsync(g1, 0, sizeof(float) * Z * d1, s));
    if (!g2 || parts == 1) return bwd_x_rows(plan_host, plan_dev, x1, x2, weight, gout, g1, g2, g2, Z, s);
    if (!ordered) {
        E3B_CUDA_TRY(cudaMemsetAsync(g2, 0, sizeof(float) * Z * d2, s));
        return bwd_x_rows(plan_host, plan_dev, x1, x2, weight, gout, g1, g2, nullptr, Z, s);
    }
    const int64_t slab = bwd_x_slab(P, parts, Z);
    if (!scratch || scratch_bytes < static_cast<int64_t>(sizeof(float)) * parts * slab * d2) return fail(E3B_ERR_ARG, "dense_bwd_x: scratch too small");
    float* partial = static_cast<float*>(scratch);
    for (int64_t z = 0; z < Z; z += slab) {
        const int64_t n = std::min(slab, Z - z), count = n * d2;
        if (int rc = bwd_x_rows(plan_host, plan_dev, x1 + z * d1, x2 + z * d2, weight, gout + z * dout, g1 ? g1 + z * d1 : nullptr, g2 + z * d2,
                                partial, n, s))
            return rc;
        dense_bwd_x_sum_kernel<<<static_cast<unsigned>(ceil_div(count, 256)), 256, 0, s>>>(partial, parts, count, g2 + z * d2);
        if (int rc = check_launch("e3b_dense_bwd_x")) return rc;
    }
    return E3B_OK;
}
}  // namespace e3b

extern "C" int64_t e3b_dense_bwd_x_scratch_bytes(const int32_t* plan_host, int64_t num_rows) {
    using namespace e3b;
    if (!e3b_dense_bwd_x_supported(plan_host) || num_rows <= 0) return 0;
    const Part2 P(plan_host);
    const int parts = bwd_x_parts(P);
    return parts == 1 ? 0 : static_cast<int64_t>(sizeof(float)) * parts * bwd_x_slab(P, parts, num_rows) * P.d2row();
}

extern "C" int e3b_dense_bwd_x(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                               const float* grad_out, float* grad_x1, float* grad_x2, int64_t num_rows, void* stream) {
    return e3b::bwd_x(plan_host, plan_dev, x1, x2, weight, grad_out, grad_x1, grad_x2, num_rows, false, nullptr, 0, stream);
}

extern "C" int e3b_dense_bwd_x_ordered(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                                       const float* grad_out, float* grad_x1, float* grad_x2, int64_t num_rows, void* scratch,
                                       int64_t scratch_bytes, void* stream) {
    return e3b::bwd_x(plan_host, plan_dev, x1, x2, weight, grad_out, grad_x1, grad_x2, num_rows, true, scratch, scratch_bytes, stream);
}
