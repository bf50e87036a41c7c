// What dense.cu and dense_tile.cu share: the plan's magic word and the register-tile launches.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

namespace e3b {

constexpr int kDenseMagic = 0x65336250;

int launch_dense_tile_fwd(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* weight,
                          float* out, int64_t num_rows, int accumulate, cudaStream_t s);
int launch_dense_tile_bwd_w(const int32_t* plan_host, const int32_t* plan_dev, const float* x1, const float* x2, const float* grad_out,
                            float* grad_weight, int64_t num_rows, cudaStream_t s);

}  // namespace e3b
