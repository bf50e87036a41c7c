// What dense.cu and dense_tile.cu share: the plan's magic word, the Gate epilogue and the register-tile launches.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

namespace e3b {

constexpr int kDenseMagic = 0x65336251;          // a plan with both parts
constexpr int kDenseMagicFirst = 0x65336250;     // the first part alone, as plans were before there was a second

inline bool whole_plan(const int32_t* plan) { return plan && plan[0] == kDenseMagic; }
inline bool any_plan(const int32_t* plan) { return plan && (plan[0] == kDenseMagic || plan[0] == kDenseMagicFirst); }

// Gate applied where the contraction's result is still in registers (Linear followed by Gate).  Column c of the
// contraction's output row is described by tbl[4 c ..] = {kind, destination column, activation, gate slot} and
// cst[c]: kind 0 = scalar: final[z, dst] = cst * act(v); kind 2 = gate: gates[z, slot] = cst * act(v);
// kind 1 = gated component: final[z, dst] = v * gates[z, slot] (its gate's launch ran before); kind 3 = unused.
struct DenseGateEpilogue {
    const int32_t* tbl;
    const float* cst;
    float* gates;       // [rows, n_slots] activated gates
    float* final_out;   // [rows, dout_final]
    int n_slots, dout_final;
};

// The Linear of a plan with Gate as its epilogue on the row kernels; *done = false: the plan has irreps of l > 3.
int launch_dense_rows_gate(const int32_t* plan_host, const int32_t* plan_dev, const float* x, const float* weight,
                           const DenseGateEpilogue& ep, int64_t num_rows, cudaStream_t s, bool* done);
// Whether the table-driven kernels of dense.cu are faster than the register tiles: forward, and for the weight gradient.
bool few_channels(const int32_t* plan_host);
bool pairs_bwd_w(const int32_t* plan_host, int64_t num_rows);
int launch_dense_tile_fwd(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                          float* out, int64_t num_rows, int accumulate, cudaStream_t s);
int launch_dense_tile_bwd_w(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* grad_out,
                            float* grad_weight, int64_t num_rows, cudaStream_t s);

}  // namespace e3b
