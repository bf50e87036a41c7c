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
// Second part: header of 12 words { n_groups, groups, n_chunks, chunks, n_paths, paths, n_in, in_groups, d1max, d3max,
// in_paths, covered } (word offsets into the plan), then
//   groups    x 6 : out_off, mul_out, dim3, first chunk, chunks, 0
//   chunks    x 6 : path, x1 offset of its first channel, channels (<= 32), x2 offset or -1, weight base, 1 = T changes
//   paths     x 16: d1, d2, d3, weight strides over u and w, ki segments, j segments, x1off, m1, x2off, m2, out_off, mo,
//                   weight base, stride over v, coefficient (Linear)
//   in_groups x 5 : x1off, m1, d1, first in_path, in_paths   (the paths that leave one input irrep)
//   segments      : word offsets s[0..n] of (index, coefficient) pairs: (j, C) per (k, i); (i * d3 + k, C) per j
#include "common.cuh"
#include "dense_plan.cuh"

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

// ---------------------------------------------------------------------------------------------- forward
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
    const int out_off = g[0], mo = g[1], d3 = g[2], d1row = P.plan[1], d2row = P.plan[2], dout = P.plan[3];
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
        // the chunk's sum in accumulators of its own: the rounding error grows with sqrt(32) + sqrt(K / 32)
        float part[kTM][kTN];
#pragma unroll
        for (int i = 0; i < kTM; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) part[i][j] = 0.0f;
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
#pragma unroll
        for (int i = 0; i < kTM; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) acc[i][j] += part[i][j];
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

// Columns of a tile: the narrowest that holds the group's channels in one pass, so that the coupled operand is built once.
inline int columns_for(int mo) { return mo <= 16 ? 16 : mo <= 32 ? 32 : mo <= 64 ? 64 : 128; }

// ---------------------------------------------------------------------------------------------- weight gradient
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
    const int out_off = g[0], mo = g[1], d3 = g[2], d1row = P.plan[1], d2row = P.plan[2], dout = P.plan[3];
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

// ---------------------------------------------------------------------------------------------- operand gradients
// Both operand gradients of a 'uvw' product come from one intermediate per path:
//     Q[z, u, k]       = sum_w W_p[u, v, w] g[z, w, k]
//     grad_x1[z, u, i] += sum_k T_p[z, k, i] Q[z, u, k]
//     M[z, i, k]       = sum_u x1[z, u, i] Q[z, u, k],   grad_x2[z, v, j] += sum_{i, k} C_ijk M[z, i, k]
// A block owns one input irrep's 32 channels for 32 rows; a thread owns one row and 8 channels for every k and i, so
// the sums over k stay in its registers, and the sums over u cross 4 lanes.
constexpr int kBxZ = 32, kBxU = 8;

struct BwdXLaunch {
    int n;
    int first_block[kMaxGroups + 1];
    int16_t group[kMaxGroups];
};

struct BwdXShared {
    float *a, *w, *x, *t, *m, *g2;
    int ldx, ldt, ldm, ld2;
};

template <int D1, int D3, bool NEED1, bool NEED2>
__device__ __forceinline__ void bwd_x_path(const Part2& P, const int32_t* path, const float* __restrict__ x2, const float* __restrict__ W,
                                           const float* __restrict__ gout, int64_t z0, int64_t Z, int u0, int nu, const BwdXShared& S,
                                           float (&gx)[D1][kBxU]) {
    const int su = path[3], sw = path[4], x2off = path[9], m2 = path[10], out_off = path[11], mo = path[12], wbase = path[13], sv = path[14];
    const int d2 = path[1], d2row = P.plan[2], dout = P.plan[3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 3, ty = warp * 8 + (lane >> 2);
    const int ldt = (D1 * D3) | 1;
    for (int v = 0; v < m2; ++v) {
        float q[D3][kBxU];
#pragma unroll
        for (int k = 0; k < D3; ++k)
#pragma unroll
            for (int u = 0; u < kBxU; ++u) q[k][u] = 0.0f;
        for (int c0 = 0; c0 < mo; c0 += kKC) {
            const int len = min(kKC, mo - c0);
            __syncthreads();
            if (NEED1 && c0 == 0) stage_coupling(P.plan, path, x2, d2row, x2off + v * d2, z0, kBxZ, Z, S.t, ldt);
            // W[w][u]
            for (int idx = tid; idx < kKC * 32; idx += kThreads) {
                const int ww = idx & 31, u = idx >> 5;
                S.w[ww * kLda + u] = (ww < len && u < nu) ? __ldg(W + wbase + static_cast<int64_t>(u0 + u) * su + static_cast<int64_t>(v) * sv
                                                                  + static_cast<int64_t>(c0 + ww) * sw) : 0.0f;
            }
            if (v == 0 || mo > kKC) stage_rows_d<D3>(gout, dout, out_off + c0 * D3, len, z0, kBxZ, Z, D3, false, 1.0f, nullptr, 0, S.a, kLda);
            __syncthreads();
            float part[D3][kBxU];
#pragma unroll
            for (int k = 0; k < D3; ++k)
#pragma unroll
                for (int u = 0; u < kBxU; ++u) part[k][u] = 0.0f;
            const int kend = (len + 3) & ~3;
#pragma unroll 1
            for (int kk = 0; kk < kend; kk += 4) {
                float w[4][kBxU];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float4 lo = *reinterpret_cast<const float4*>(S.w + (kk + s) * kLda + tx * kBxU);
                    const float4 hi = *reinterpret_cast<const float4*>(S.w + (kk + s) * kLda + tx * kBxU + 4);
                    w[s][0] = lo.x; w[s][1] = lo.y; w[s][2] = lo.z; w[s][3] = lo.w;
                    w[s][4] = hi.x; w[s][5] = hi.y; w[s][6] = hi.z; w[s][7] = hi.w;
                }
#pragma unroll
                for (int k = 0; k < D3; ++k) {
                    const float4 a = *reinterpret_cast<const float4*>(S.a + (ty * D3 + k) * kLda + kk);
                    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int s = 0; s < 4; ++s)
#pragma unroll
                        for (int u = 0; u < kBxU; ++u) part[k][u] = fmaf(av[s], w[s][u], part[k][u]);
                }
            }
#pragma unroll
            for (int k = 0; k < D3; ++k)
#pragma unroll
                for (int u = 0; u < kBxU; ++u) q[k][u] += part[k][u];
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
#pragma unroll
            for (int i = 0; i < D1; ++i) {
                float m[D3];
#pragma unroll
                for (int k = 0; k < D3; ++k) m[k] = 0.0f;
#pragma unroll
                for (int u = 0; u < kBxU; ++u) {
                    const float x = S.x[ty * S.ldx + (tx * kBxU + u) * D1 + i];
#pragma unroll
                    for (int k = 0; k < D3; ++k) m[k] = fmaf(x, q[k][u], m[k]);
                }
#pragma unroll
                for (int k = 0; k < D3; ++k) {
                    m[k] += __shfl_xor_sync(0xffffffffu, m[k], 1);
                    m[k] += __shfl_xor_sync(0xffffffffu, m[k], 2);
                    if (tx == 0) S.m[ty * S.ldm + i * D3 + k] = m[k];
                }
            }
            __syncwarp();
            // the 8 rows of a warp are its own: no barrier
            const int32_t* seg = P.plan + path[6];
            for (int t = lane; t < 8 * d2; t += 32) {
                const int zl = warp * 8 + t / d2, j = t % d2;
                float s = 0.0f;
                for (int e = seg[j]; e < seg[j + 1]; e += 2) s = fmaf(__int_as_float(P.plan[e + 1]), S.m[zl * S.ldm + P.plan[e]], s);
                S.g2[zl * S.ld2 + x2off + v * d2 + j] += s;
            }
            __syncwarp();
        }
    }
}

template <int D1, bool NEED1, bool NEED2>
__device__ __forceinline__ void bwd_x_block(const Part2& P, const int32_t* in, const float* __restrict__ x1, const float* __restrict__ x2,
                                            const float* __restrict__ W, const float* __restrict__ gout, float* __restrict__ g1,
                                            float* __restrict__ g2, int64_t Z, int block, const BwdXShared& S) {
    const int x1off = in[0], m1 = in[1], ublocks = (m1 + 31) / 32;
    const int64_t z0 = static_cast<int64_t>(block / ublocks) * kBxZ;
    const int u0 = (block % ublocks) * 32, nu = min(32, m1 - u0);
    const int d1row = P.plan[1], d2row = P.plan[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 3, ty = warp * 8 + (lane >> 2);
    float gx[D1][kBxU];
#pragma unroll
    for (int i = 0; i < D1; ++i)
#pragma unroll
        for (int u = 0; u < kBxU; ++u) gx[i][u] = 0.0f;
    if (NEED2) {
        for (int zl = warp; zl < kBxZ; zl += kThreads / 32) {
            const float* p = x1 + (z0 + zl) * d1row + x1off + u0 * D1;
            for (int e = lane; e < 32 * D1; e += 32) S.x[zl * S.ldx + e] = (z0 + zl < Z && e < nu * D1) ? __ldg(p + e) : 0.0f;
            for (int e = lane; e < d2row; e += 32) S.g2[zl * S.ld2 + e] = 0.0f;
        }
    }
    for (int n = 0; n < in[4]; ++n) {
        const int32_t* path = P.path(P.in_path(in[3] + n));
        switch (path[2]) {
            case 1: bwd_x_path<D1, 1, NEED1, NEED2>(P, path, x2, W, gout, z0, Z, u0, nu, S, gx); break;
            case 3: bwd_x_path<D1, 3, NEED1, NEED2>(P, path, x2, W, gout, z0, Z, u0, nu, S, gx); break;
            case 5: bwd_x_path<D1, 5, NEED1, NEED2>(P, path, x2, W, gout, z0, Z, u0, nu, S, gx); break;
            default: bwd_x_path<D1, 7, NEED1, NEED2>(P, path, x2, W, gout, z0, Z, u0, nu, S, gx); break;
        }
    }
    if (NEED1) {
        __syncthreads();
        // [row][u * D1 + i] over the staged cotangent, then contiguous row segments
        constexpr int ld = 32 * D1 + 1;
#pragma unroll
        for (int i = 0; i < D1; ++i)
#pragma unroll
            for (int u = 0; u < kBxU; ++u) S.a[ty * ld + (tx * kBxU + u) * D1 + i] = gx[i][u];
        __syncwarp();
        for (int r = 0; r < 8; ++r) {
            const int zl = warp * 8 + r;
            if (z0 + zl >= Z) break;
            float* o = g1 + (z0 + zl) * d1row + x1off + u0 * D1;
            for (int e = lane; e < nu * D1; e += 32) o[e] = S.a[zl * ld + e];
        }
    }
    if (NEED2) {
        __syncwarp();
        for (int r = 0; r < 8; ++r) {
            const int zl = warp * 8 + r;
            if (z0 + zl >= Z) break;
            for (int e = lane; e < d2row; e += 32) atomicAdd(g2 + (z0 + zl) * d2row + e, S.g2[zl * S.ld2 + e]);
        }
    }
}

template <bool NEED1, bool NEED2>
__global__ void __launch_bounds__(kThreads, 2) dense_tile_bwd_x_kernel(const int32_t* __restrict__ plan, const float* __restrict__ x1,
                                                                       const float* __restrict__ x2, const float* __restrict__ W,
                                                                       const float* __restrict__ gout, float* __restrict__ g1,
                                                                       float* __restrict__ g2, int64_t Z, int a_floats, BwdXLaunch L) {
    extern __shared__ __align__(16) float smem[];
    const Part2 P(plan);
    BwdXShared S;
    S.ldx = 32 * P.d1max() + 1;
    S.ldt = (P.d1max() * P.d3max()) | 1;
    S.ldm = S.ldt;
    S.ld2 = plan[2] | 1;
    S.a = smem;
    S.w = S.a + a_floats;
    S.t = S.w + kKC * kLda;
    S.x = S.t + kBxZ * S.ldt;
    S.m = S.x + (NEED2 ? kBxZ * S.ldx : 0);
    S.g2 = S.m + (NEED2 ? kBxZ * S.ldm : 0);
    int s = 0;
    while (s + 1 < L.n && static_cast<int>(blockIdx.x) >= L.first_block[s + 1]) ++s;
    const int32_t* in = P.in_group(L.group[s]);
    const int block = static_cast<int>(blockIdx.x) - L.first_block[s];
    switch (in[2]) {
        case 1: bwd_x_block<1, NEED1, NEED2>(P, in, x1, x2, W, gout, g1, g2, Z, block, S); break;
        case 3: bwd_x_block<3, NEED1, NEED2>(P, in, x1, x2, W, gout, g1, g2, Z, block, S); break;
        case 5: bwd_x_block<5, NEED1, NEED2>(P, in, x1, x2, W, gout, g1, g2, Z, block, S); break;
        default: bwd_x_block<7, NEED1, NEED2>(P, in, x1, x2, W, gout, g1, g2, Z, block, S); break;
    }
}

constexpr int kMaxShared = 227 * 1024;

// Floats of the operand buffer of dense_tile_bwd_x_kernel: the staged cotangent, later the grad_x1 tile.
inline int bwd_x_a_floats(int d1max, int d3max) { return std::max(kBxZ * d3max * kLda, (kBxZ * (32 * d1max + 1) + 3) & ~3); }

inline size_t bwd_x_shared(const int32_t* plan, int d1max, int d3max, bool need2) {
    const int ldt = (d1max * d3max) | 1;
    size_t f = bwd_x_a_floats(d1max, d3max) + kKC * kLda + kBxZ * ldt;
    if (need2) f += static_cast<size_t>(kBxZ) * (32 * d1max + 1) + kBxZ * ldt + kBxZ * (plan[2] | 1);
    return f * sizeof(float);
}

bool too_many_blocks(int64_t blocks) { return blocks > 2147483647LL; }

}  // namespace

int launch_dense_tile_fwd(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                          float* out, int64_t Z, int accumulate, cudaStream_t s) {
    const Part2 P(plan_host);
    int g0 = 0;
    while (g0 < P.n_groups()) {
        FwdLaunch L;
        L.n = 0;
        int64_t blocks = 0;
        size_t floats = 0;
        for (; g0 < P.n_groups() && L.n < kMaxGroups; ++g0) {
            const int32_t* g = P.group(g0);
            if (g[1] == 0 || g[4] == 0) continue;
            const int bn = columns_for(g[1]), bm = tile_rows(bn);
            if (g[2] > bm) return fail(E3B_ERR_UNSUPPORTED, "dense_fwd: irrep dimension %d too large", g[2]);
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
                        const float* gout, float* g1, float* g2, int64_t Z, cudaStream_t s) {
    const Part2 P(plan_host);
    const size_t bytes = bwd_x_shared(plan_host, P.d1max(), P.d3max(), NEED2);
    int g0 = 0;
    while (g0 < P.n_in()) {
        BwdXLaunch L;
        L.n = 0;
        int64_t blocks = 0;
        for (; g0 < P.n_in() && L.n < kMaxGroups; ++g0) {
            const int32_t* in = P.in_group(g0);
            L.first_block[L.n] = static_cast<int>(blocks);
            L.group[L.n] = static_cast<int16_t>(g0);
            blocks += ceil_div(Z, kBxZ) * ceil_div(in[1], 32);
            if (too_many_blocks(blocks)) return fail(E3B_ERR_ARG, "dense_bwd_x: too many rows");
            ++L.n;
        }
        L.first_block[L.n] = static_cast<int>(blocks);
        auto kernel = dense_tile_bwd_x_kernel<NEED1, NEED2>;
        E3B_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
        kernel<<<static_cast<unsigned>(blocks), kThreads, bytes, s>>>(plan_dev, x1, x2, weight, gout, g1, g2, Z,
                                                                      bwd_x_a_floats(P.d1max(), P.d3max()), L);
        if (int rc = check_launch("e3b_dense_bwd_x")) return rc;
    }
    return E3B_OK;
}

}  // namespace e3b

extern "C" int e3b_dense_bwd_x_supported(const int32_t* plan_host) {
    using namespace e3b;
    if (!plan_host || plan_host[0] != kDenseMagic) return 0;
    const Part2 P(plan_host);
    return P.n_in() > 0 && P.d1max() <= 7 && P.d3max() <= 7 && bwd_x_shared(plan_host, P.d1max(), P.d3max(), true) <= static_cast<size_t>(kMaxShared);
}

extern "C" int e3b_dense_bwd_x(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                               const float* grad_out, float* grad_x1, float* grad_x2, int64_t num_rows, void* stream) {
    using namespace e3b;
    if (!plan_host || plan_host[0] != kDenseMagic) return fail(E3B_ERR_ARG, "dense_bwd_x: bad plan");
    if (num_rows < 0) return fail(E3B_ERR_ARG, "dense_bwd_x: negative row count");
    if (num_rows == 0 || (!grad_x1 && !grad_x2)) return E3B_OK;
    if (!plan_dev || !x1 || !x2 || !weight || !grad_out) return fail(E3B_ERR_ARG, "dense_bwd_x: null pointer");
    if (!e3b_dense_bwd_x_supported(plan_host)) return fail(E3B_ERR_UNSUPPORTED, "dense_bwd_x: irreps above l = 3 or too wide");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Part2 P(plan_host);
    if (grad_x1 && !P.covers_x1()) E3B_CUDA_TRY(cudaMemsetAsync(grad_x1, 0, sizeof(float) * num_rows * plan_host[1], s));
    if (grad_x2) E3B_CUDA_TRY(cudaMemsetAsync(grad_x2, 0, sizeof(float) * num_rows * plan_host[2], s));
    if (grad_x1 && grad_x2) return launch_bwd_x<true, true>(plan_host, plan_dev, x1, x2, weight, grad_out, grad_x1, grad_x2, num_rows, s);
    if (grad_x1) return launch_bwd_x<true, false>(plan_host, plan_dev, x1, x2, weight, grad_out, grad_x1, grad_x2, num_rows, s);
    return launch_bwd_x<false, true>(plan_host, plan_dev, x1, x2, weight, grad_out, grad_x1, grad_x2, num_rows, s);
}
