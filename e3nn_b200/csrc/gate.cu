// Gate non-linearity on rows of irreps features: the step after the Linear in every model
// (e3nn/nn/_gate.py:35-144 with e3nn/nn/_activation.py:9-111 and the 'uuu' product of
// e3nn/o3/_tensor_product/_sub.py ElementwiseTensorProduct, which for a scalar second operand is a plain
// per-channel multiplication):
//
//   out = [ c_i * phi_i(scalars_i) ]  (+)  [ gated_j * c_j * phi_j(gates_j) ]
//
// The reference runs an Extract (three narrow + cat), two Activations (narrow + cat per block) and a
// generated tensor product; here one elementwise kernel per direction reads a row once and writes it once.
// The irreps bookkeeping lives on the host: per OUTPUT column {input column, gate column or -1,
// activation code, constant}, per INPUT column {kind, first output column, count, partner column}.
#include "common.cuh"
#include "gate_act.cuh"

namespace e3b {
namespace {

// A thread owns one column (its table entry stays in registers) and walks the rows: consecutive threads touch
// consecutive addresses, no per-element index arithmetic beyond one multiply-add per row.
// out_tbl[j] = {input column, gate column or -1, activation code}, out_cst[j] = constant
__global__ void __launch_bounds__(256) gate_fwd_kernel(const float* __restrict__ x, const int32_t* __restrict__ out_tbl,
                                                       const float* __restrict__ out_cst, float* __restrict__ out, int64_t rows,
                                                       int din, int dout) {
    const int j = blockIdx.y * blockDim.x + threadIdx.x;
    if (j >= dout) return;
    const int src = out_tbl[3 * j], gate = out_tbl[3 * j + 1], act = out_tbl[3 * j + 2];
    const float cst = out_cst[j];
    // four rows per trip: their loads are independent and in flight together
    for (int64_t z0 = static_cast<int64_t>(blockIdx.x) * 4; z0 < rows; z0 += static_cast<int64_t>(gridDim.x) * 4) {
        float v[4], gv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t z = z0 + r < rows ? z0 + r : rows - 1;
            v[r] = x[z * din + src];
            gv[r] = gate < 0 ? 0.0f : x[z * din + gate];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (z0 + r < rows) out[(z0 + r) * dout + j] = gate < 0 ? cst * gate_act(act, v[r]) : v[r] * (cst * gate_act(act, gv[r]));
    }
}

// One thread per CHANNEL (a scalar, or the 2l+1 components of a gated channel): the gate's activation, the only
// transcendental work of the row, is evaluated once per channel instead of once per column, forward and backward.
// ch_tbl[q] = {first input column, count (1 or 2l+1), gate column or -1, activation code, first output column},
// ch_cst[q] = constant.  Lanes are consecutive channels, i.e. adjacent runs of 2l+1 floats: full lines are used.
// Bound by HBM; the components of two rows are loaded before the first is used (COUNT is a compile-time 1, 3, 5 or 7;
// 0: any count, one component after the other).
// 20,011 rows of 256x0e+64x1o+64x2e+64x3o: 43 -> 34 us forward, gradient 96 (a thread per column) -> 53 us.
struct GateChannel {
    int src, cnt, gate, act, dst;
    float cst;
};

template <int COUNT>
__device__ __forceinline__ void gate_fwd_rows(const GateChannel& c, const float* __restrict__ x, float* __restrict__ out, int64_t rows,
                                              int din, int dout) {
    constexpr int N = COUNT > 0 ? COUNT : 1;
    for (int64_t z0 = static_cast<int64_t>(blockIdx.x) * 2; z0 < rows; z0 += static_cast<int64_t>(gridDim.x) * 2) {
        float v[2][N], gv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float* xr = x + (z0 + r < rows ? z0 + r : rows - 1) * din;
            gv[r] = c.gate < 0 ? 0.0f : xr[c.gate];
            if (COUNT > 0) {
#pragma unroll
                for (int m = 0; m < N; ++m) v[r][m] = xr[c.src + m];
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (z0 + r >= rows) break;
            const float* xr = x + (z0 + r) * din + c.src;
            float* orow = out + (z0 + r) * dout + c.dst;
            if (c.gate < 0) {
                orow[0] = c.cst * gate_act(c.act, COUNT > 0 ? v[r][0] : xr[0]);
                continue;
            }
            const float f = c.cst * gate_act(c.act, gv[r]);
            if (COUNT > 0) {
#pragma unroll
                for (int m = 0; m < N; ++m) orow[m] = v[r][m] * f;
            } else {
                for (int m = 0; m < c.cnt; ++m) orow[m] = xr[m] * f;
            }
        }
    }
}

template <int COUNT>
__device__ __forceinline__ void gate_bwd_rows(const GateChannel& c, const float* __restrict__ x, const float* __restrict__ gout,
                                              float* __restrict__ gin, int64_t rows, int din, int dout) {
    constexpr int N = COUNT > 0 ? COUNT : 1;
    for (int64_t z0 = static_cast<int64_t>(blockIdx.x) * 2; z0 < rows; z0 += static_cast<int64_t>(gridDim.x) * 2) {
        float v[2][N], g[2][N], gv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t z = z0 + r < rows ? z0 + r : rows - 1;
            gv[r] = c.gate < 0 ? 0.0f : x[z * din + c.gate];
            if (COUNT > 0) {
#pragma unroll
                for (int m = 0; m < N; ++m) { v[r][m] = x[z * din + c.src + m]; g[r][m] = gout[z * dout + c.dst + m]; }
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (z0 + r >= rows) break;
            const float* xr = x + (z0 + r) * din + c.src;
            const float* gr = gout + (z0 + r) * dout + c.dst;
            float* ir = gin + (z0 + r) * din;
            if (c.gate < 0) {
                ir[c.src] = (COUNT > 0 ? g[r][0] : gr[0]) * c.cst * gate_act_grad(c.act, COUNT > 0 ? v[r][0] : xr[0]);
                continue;
            }
            const float f = c.cst * gate_act(c.act, gv[r]);
            float acc = 0.0f;
            if (COUNT > 0) {
#pragma unroll
                for (int m = 0; m < N; ++m) { ir[c.src + m] = g[r][m] * f; acc = fmaf(g[r][m], v[r][m], acc); }
            } else {
                for (int m = 0; m < c.cnt; ++m) { ir[c.src + m] = gr[m] * f; acc = fmaf(gr[m], xr[m], acc); }
            }
            ir[c.gate] = acc * c.cst * gate_act_grad(c.act, gv[r]);
        }
    }
}

__device__ __forceinline__ GateChannel gate_channel(const int32_t* __restrict__ ch_tbl, const float* __restrict__ ch_cst, int q) {
    return {ch_tbl[5 * q], ch_tbl[5 * q + 1], ch_tbl[5 * q + 2], ch_tbl[5 * q + 3], ch_tbl[5 * q + 4], ch_cst[q]};
}

__global__ void __launch_bounds__(256) gate_fwd_channel_kernel(const float* __restrict__ x, const int32_t* __restrict__ ch_tbl,
                                                               const float* __restrict__ ch_cst, float* __restrict__ out,
                                                               int64_t rows, int din, int dout, int nch) {
    const int q = blockIdx.y * blockDim.x + threadIdx.x;
    if (q >= nch) return;
    const GateChannel c = gate_channel(ch_tbl, ch_cst, q);
    switch (c.cnt) {
        case 1: gate_fwd_rows<1>(c, x, out, rows, din, dout); break;
        case 3: gate_fwd_rows<3>(c, x, out, rows, din, dout); break;
        case 5: gate_fwd_rows<5>(c, x, out, rows, din, dout); break;
        case 7: gate_fwd_rows<7>(c, x, out, rows, din, dout); break;
        default: gate_fwd_rows<0>(c, x, out, rows, din, dout); break;
    }
}

// Every input column belongs to exactly one channel (its components or its gate).
__global__ void __launch_bounds__(256) gate_bwd_channel_kernel(const float* __restrict__ x, const float* __restrict__ gout,
                                                               const int32_t* __restrict__ ch_tbl, const float* __restrict__ ch_cst,
                                                               float* __restrict__ gin, int64_t rows, int din, int dout, int nch) {
    const int q = blockIdx.y * blockDim.x + threadIdx.x;
    if (q >= nch) return;
    const GateChannel c = gate_channel(ch_tbl, ch_cst, q);
    switch (c.cnt) {
        case 1: gate_bwd_rows<1>(c, x, gout, gin, rows, din, dout); break;
        case 3: gate_bwd_rows<3>(c, x, gout, gin, rows, din, dout); break;
        case 5: gate_bwd_rows<5>(c, x, gout, gin, rows, din, dout); break;
        case 7: gate_bwd_rows<7>(c, x, gout, gin, rows, din, dout); break;
        default: gate_bwd_rows<0>(c, x, gout, gin, rows, din, dout); break;
    }
}

// in_tbl[c] = {kind, first output column, count, partner, activation code}, in_cst[c] = constant:
// kind 0 = scalar, 1 = gated component (partner = its gate's input column, activation of that gate),
// 2 = gate (count = 2l+1 components of its channel, partner = input column of the first component),
// 3 = column no output depends on
__global__ void __launch_bounds__(256) gate_bwd_kernel(const float* __restrict__ x, const float* __restrict__ gout,
                                                       const int32_t* __restrict__ in_tbl, const float* __restrict__ in_cst,
                                                       float* __restrict__ gin, int64_t rows, int din, int dout) {
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= din) return;
    const int kind = in_tbl[5 * c], o0 = in_tbl[5 * c + 1], cnt = in_tbl[5 * c + 2], partner = in_tbl[5 * c + 3],
              act = in_tbl[5 * c + 4];
    const float cst = in_cst[c];
    for (int64_t z = blockIdx.x; z < rows; z += gridDim.x) {
        const float* xr = x + z * din;
        const float* gr = gout + z * dout;
        float g = 0.0f;
        if (kind == 0) {
            g = gr[o0] * cst * gate_act_grad(act, xr[c]);
        } else if (kind == 1) {
            g = gr[o0] * (cst * gate_act(act, xr[partner]));
        } else if (kind == 2) {
            float acc = 0.0f;
            for (int m = 0; m < cnt; ++m) acc = fmaf(gr[o0 + m], xr[partner + m], acc);
            g = acc * cst * gate_act_grad(act, xr[c]);
        }
        gin[z * din + c] = g;
    }
}

// grid: y covers the columns in blocks of 256, x walks the rows with enough blocks to fill the machine
dim3 gate_grid(int64_t rows, int cols) {
    const int ny = (cols + 255) / 256;
    int64_t nx = (static_cast<int64_t>(kNumSMs) * 16 + ny - 1) / ny;
    if (nx > rows) nx = rows;
    if (nx < 1) nx = 1;
    return dim3(static_cast<unsigned>(nx), static_cast<unsigned>(ny));
}

}  // namespace
}  // namespace e3b

extern "C" int e3b_gate_fwd(const float* x, const int32_t* out_table, const float* out_const, float* out, int64_t rows,
                            int din, int dout, void* stream) {
    using namespace e3b;
    if (rows < 0 || din < 0 || dout < 0) return fail(E3B_ERR_ARG, "gate_fwd: negative size");
    if (rows == 0 || dout == 0) return E3B_OK;
    if (!x || !out_table || !out_const || !out) return fail(E3B_ERR_ARG, "gate_fwd: null pointer");
    gate_fwd_kernel<<<gate_grid(rows, dout), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, out_table, out_const, out, rows, din, dout);
    return check_launch("gate_fwd");
}

extern "C" int e3b_gate_fwd_channels(const float* x, const int32_t* channel_table, const float* channel_const, float* out,
                                     int64_t rows, int din, int dout, int num_channels, void* stream) {
    using namespace e3b;
    if (rows < 0 || din < 0 || dout < 0 || num_channels < 0) return fail(E3B_ERR_ARG, "gate_fwd_channels: negative size");
    if (rows == 0 || num_channels == 0) return E3B_OK;
    if (!x || !channel_table || !channel_const || !out) return fail(E3B_ERR_ARG, "gate_fwd_channels: null pointer");
    gate_fwd_channel_kernel<<<gate_grid(rows, num_channels), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        x, channel_table, channel_const, out, rows, din, dout, num_channels);
    return check_launch("gate_fwd_channels");
}

extern "C" int e3b_gate_bwd(const float* x, const float* grad_out, const int32_t* in_table, const float* in_const,
                            float* grad_x, int64_t rows, int din, int dout, void* stream) {
    using namespace e3b;
    if (rows < 0 || din < 0 || dout < 0) return fail(E3B_ERR_ARG, "gate_bwd: negative size");
    if (rows == 0 || din == 0) return E3B_OK;
    if (!x || !grad_out || !in_table || !in_const || !grad_x) return fail(E3B_ERR_ARG, "gate_bwd: null pointer");
    gate_bwd_kernel<<<gate_grid(rows, din), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, grad_out, in_table, in_const, grad_x, rows, din, dout);
    return check_launch("gate_bwd");
}

extern "C" int e3b_gate_bwd_channels(const float* x, const float* grad_out, const int32_t* channel_table, const float* channel_const,
                                     float* grad_x, int64_t rows, int din, int dout, int num_channels, void* stream) {
    using namespace e3b;
    if (rows < 0 || din < 0 || dout < 0 || num_channels < 0) return fail(E3B_ERR_ARG, "gate_bwd_channels: negative size");
    if (rows == 0 || num_channels == 0) return E3B_OK;
    if (!x || !grad_out || !channel_table || !channel_const || !grad_x) return fail(E3B_ERR_ARG, "gate_bwd_channels: null pointer");
    gate_bwd_channel_kernel<<<gate_grid(rows, num_channels), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        x, grad_out, channel_table, channel_const, grad_x, rows, din, dout, num_channels);
    return check_launch("gate_bwd_channels");
}
