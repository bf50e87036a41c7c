// Exclusive scan of int32 counts into int64 offsets, used by the neighbour-list builder.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace e3b {

// One block of 1024 threads covers kScanChunk counts.  Two launches (block sums, then every block adds up the sums
// before it and scans its own chunk) replace a single block that walked the whole array 1024 counts at a time with
// four barriers per step: 197 us for 262,144 counts, 6 us as two launches; up to one chunk the second launch alone.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanChunk = kScanThreads * kScanItems;

static inline int64_t scan_blocks(int64_t n) { return n > 0 ? (n + kScanChunk - 1) / kScanChunk : 1; }

// Sum over the block (all threads receive it); `buf` has 33 entries and may be reused after the call.
static __device__ __forceinline__ int64_t block_sum(int64_t v, int64_t* buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) buf[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int64_t w = lane < static_cast<int>(blockDim.x >> 5) ? buf[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (lane == 0) buf[32] = w;
    }
    __syncthreads();
    const int64_t r = buf[32];
    __syncthreads();
    return r;
}

static __global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int32_t* __restrict__ counts, int64_t n,
                                                                        int64_t* __restrict__ sums) {
    __shared__ int64_t buf[33];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanChunk;
    int64_t v = 0;
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        const int64_t i = base + r * kScanThreads + threadIdx.x;
        if (i < n) v += counts[i];
    }
    v = block_sum(v, buf);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

// offsets[n + 1]; `sums` as written by scan_sums_kernel (not read when there is one block).
static __global__ void __launch_bounds__(kScanThreads) scan_offsets_kernel(const int32_t* __restrict__ counts, int64_t n,
                                                                           const int64_t* __restrict__ sums,
                                                                           int64_t* __restrict__ offsets) {
    __shared__ int64_t buf[33];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int64_t before = 0;
    for (int64_t b = t; b < static_cast<int64_t>(blockIdx.x); b += kScanThreads) before += sums[b];
    if (blockIdx.x > 0) before = block_sum(before, buf);
    // a thread owns kScanItems consecutive counts
    const int64_t first = static_cast<int64_t>(blockIdx.x) * kScanChunk + static_cast<int64_t>(t) * kScanItems;
    int32_t v[kScanItems];
    int64_t mine = 0;
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        v[r] = first + r < n ? counts[first + r] : 0;
        mine += v[r];
    }
    int64_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) buf[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int64_t w = buf[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t up = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += up;
        }
        buf[lane] = w;
    }
    __syncthreads();
    int64_t at = before + (warp > 0 ? buf[warp - 1] : 0) + (incl - mine);
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        if (first + r < n) offsets[first + r] = at;
        at += v[r];
        if (first + r == n - 1) offsets[n] = at;
    }
}

// offsets[0..n] <- exclusive scan of counts[0..n); n > 0; `sums`: scan_blocks(n) words of scratch.
static inline void launch_exclusive_scan(const int32_t* counts, int64_t n, int64_t* sums, int64_t* offsets, cudaStream_t s) {
    const unsigned blocks = static_cast<unsigned>(scan_blocks(n));
    if (blocks > 1) scan_sums_kernel<<<blocks, kScanThreads, 0, s>>>(counts, n, sums);
    scan_offsets_kernel<<<blocks, kScanThreads, 0, s>>>(counts, n, sums, offsets);
}

}  // namespace e3b
