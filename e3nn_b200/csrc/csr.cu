// Destination-sorted CSR of an edge list: stable LSD radix sort of (dst, edge id) + row pointers.
//
// Integer, HBM-bound work.  Keys are the destination ids (range-checked, < 2^31), values the
// edge ids; 8-bit digits, ceil(bits(num_nodes-1)/8) passes.  A pass is three launches:
//   1. per-block digit histogram                     -> hist[digit][block]   (pass 0: while converting the input)
//   2. exclusive scan of every digit's row of hist, one block per digit, and the digit totals
//   3. stable scatter: a warp ranks its own contiguous part of the block's keys against per-warp digit counters
//      (equal digits by ballots, input order kept), the block's keys are put in digit order in shared memory and leave in
//      runs of consecutive addresses.
// Row pointers are a lower bound search of every node id in the sorted keys.
// 2,097,152 edges into 65,536 nodes: 484 us of kernels before this form (a single block scanned the histogram,
// 170 us per pass, and the row counts, 51 us; the scatter took 28 us per pass with four barriers per 256 keys).
// The result is bit-identical to argsort(dst, stable=True) / cumsum(bincount(dst)).
#include "common.cuh"

#include <mutex>

namespace e3b {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                          // keys per thread per block
constexpr int kSortChunk = kSortThreads * kSortItems;  // 2048 keys per block
constexpr int kRadix = 256;

struct CsrScratch {
    uint32_t* keys[2];
    uint32_t* vals[2];
    uint32_t* hist;    // [kRadix * nblocks]
    uint32_t* totals;  // [kRadix]
    int64_t nblocks;
};

__host__ inline int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

__host__ int64_t csr_layout(int64_t E, int64_t N, char* base, CsrScratch* out) {
    (void)N;
    const int64_t nblocks = ceil_div(E > 0 ? E : 1, kSortChunk);
    int64_t off = 0;
    auto take = [&](int64_t bytes) {
        char* p = base ? base + off : nullptr;
        off += align256(bytes);
        return p;
    };
    char* k0 = take(E * 4); char* k1 = take(E * 4);
    char* v0 = take(E * 4); char* v1 = take(E * 4);
    char* h = take(kRadix * nblocks * 4);
    char* t = take(kRadix * 4);
    if (out) {
        out->keys[0] = reinterpret_cast<uint32_t*>(k0); out->keys[1] = reinterpret_cast<uint32_t*>(k1);
        out->vals[0] = reinterpret_cast<uint32_t*>(v0); out->vals[1] = reinterpret_cast<uint32_t*>(v1);
        out->hist = reinterpret_cast<uint32_t*>(h);
        out->totals = reinterpret_cast<uint32_t*>(t);
        out->nblocks = nblocks;
    }
    return off;
}

// Digit histogram of one block's keys.  FIRST: the keys are made here, from the int64 destinations (out of range ->
// status and key 0).
template <bool FIRST>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const int64_t* __restrict__ dst, int64_t N, int32_t* status,
                                                                  uint32_t* __restrict__ keys, int64_t E, int shift,
                                                                  uint32_t* __restrict__ hist, int64_t nblocks) {
    __shared__ uint32_t h[kRadix];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kSortChunk;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int64_t i = base + r * kSortThreads + threadIdx.x;
        if (i >= E) break;
        uint32_t key;
        if (FIRST) {
            const int64_t d = dst[i];
            const bool ok = d >= 0 && d < N;
            if (!ok) atomicExch(status, 1);
            key = ok ? static_cast<uint32_t>(d) : 0u;
            keys[i] = key;
        } else {
            key = keys[i];
        }
        atomicAdd(&h[(key >> shift) & 0xffu], 1u);
    }
    __syncthreads();
    hist[static_cast<int64_t>(threadIdx.x) * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan over one warp's lanes and the block's warps; *total receives the block's sum.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        before += w < warp ? warp_sums[w] : 0u;
        sum += warp_sums[w];
    }
    __syncthreads();
    *total = sum;
    return before + incl - v;
}

// Block d: exclusive scan of hist[d][0..nblocks) in place, totals[d] = its sum.
__global__ void __launch_bounds__(kSortThreads) radix_scan_kernel(uint32_t* __restrict__ hist, int64_t nblocks,
                                                                  uint32_t* __restrict__ totals) {
    __shared__ uint32_t warp_sums[kSortWarps];
    uint32_t* row = hist + static_cast<int64_t>(blockIdx.x) * nblocks;
    uint32_t carry = 0;
    constexpr int kPer = 4;
    for (int64_t base = 0; base < nblocks; base += kSortThreads * kPer) {
        const int64_t i = base + static_cast<int64_t>(threadIdx.x) * kPer;
        uint32_t v[kPer], mine = 0;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            v[r] = i + r < nblocks ? row[i + r] : 0u;
            mine += v[r];
        }
        uint32_t sum;
        uint32_t at = carry + block_exclusive_scan(mine, warp_sums, &sum);
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            if (i + r < nblocks) row[i + r] = at;
            at += v[r];
        }
        carry += sum;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Stable scatter of one 8-bit digit.  FIRST: the values are the positions themselves.  LAST: the values also go to
// perm as int64 (the sorted keys are kept for the row pointers, the 32-bit values are not).
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kSortThreads) radix_scatter_kernel(const uint32_t* __restrict__ keys_in,
                                                                     const uint32_t* __restrict__ vals_in, int64_t E,
                                                                     int shift, const uint32_t* __restrict__ hist,
                                                                     const uint32_t* __restrict__ totals, int64_t nblocks,
                                                                     uint32_t* __restrict__ keys_out,
                                                                     uint32_t* __restrict__ vals_out,
                                                                     int64_t* __restrict__ perm) {
    __shared__ uint32_t cnt[kSortWarps][kRadix];    // digit counts of every warp, then the local slot of its first key
    __shared__ uint32_t out_base[kRadix];           // global slot of local slot 0 of a digit's run
    __shared__ uint32_t warp_sums[kSortWarps];
    __shared__ uint32_t skey[kSortChunk], sval[kSortChunk];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) cnt[w][t] = 0;
    const int64_t chunk0 = static_cast<int64_t>(blockIdx.x) * kSortChunk;
    const int have = static_cast<int>(E - chunk0 < kSortChunk ? E - chunk0 : kSortChunk);
    uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int q = warp * (32 * kSortItems) + r * 32 + lane;
        key[r] = q < have ? keys_in[chunk0 + q] : 0u;
        val[r] = FIRST ? static_cast<uint32_t>(chunk0 + q) : (q < have ? vals_in[chunk0 + q] : 0u);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const bool live = warp * (32 * kSortItems) + r * 32 + lane < have;
        const uint32_t digit = (key[r] >> shift) & 0xffu;
        // lanes of this warp holding the same digit, bit by bit (__match_any_sync in its place: 26 us a pass over 2,097,152
        // keys, now 16)
        uint32_t same = __ballot_sync(0xffffffffu, live);
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            const bool set = (digit >> bit) & 1u;
            const uint32_t votes = __ballot_sync(0xffffffffu, set);
            same &= set ? votes : ~votes;
        }
        const uint32_t before = live ? cnt[warp][digit] : 0u;
        rank[r] = before + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (live && (same >> lane) == 1u) cnt[warp][digit] = before + __popc(same);   // the highest lane of the set
        __syncwarp();
    }
    __syncthreads();
    // thread t owns digit t: its run's place in the block and in the output
    uint32_t mine = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) mine += cnt[w][t];
    uint32_t unused;
    uint32_t at = block_exclusive_scan(mine, warp_sums, &unused);
    const uint32_t digit_base = block_exclusive_scan(totals[t], warp_sums, &unused);
    out_base[t] = digit_base + hist[static_cast<int64_t>(t) * nblocks + blockIdx.x] - at;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = cnt[w][t];
        cnt[w][t] = at;
        at += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        if (warp * (32 * kSortItems) + r * 32 + lane < have) {
            const uint32_t slot = cnt[warp][(key[r] >> shift) & 0xffu] + rank[r];
            skey[slot] = key[r];
            sval[slot] = val[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int q = r * kSortThreads + t;
        if (q < have) {
            const uint32_t k = skey[q];
            const uint32_t pos = out_base[(k >> shift) & 0xffu] + static_cast<uint32_t>(q);
            keys_out[pos] = k;
            if (LAST) perm[pos] = static_cast<int64_t>(sval[q]);
            else vals_out[pos] = sval[q];
        }
    }
}

// rowptr[n] = number of sorted keys below n, n = 0..N.
__global__ void csr_rowptr_kernel(const uint32_t* __restrict__ keys, int64_t E, int64_t N, int64_t* __restrict__ rowptr) {
    const int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (n > N) return;
    int64_t lo = 0, hi = n == 0 ? 0 : E;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (static_cast<int64_t>(keys[mid]) < n) lo = mid + 1;
        else hi = mid;
    }
    rowptr[n] = lo;
}

// A single node: every edge already in place.
__global__ void csr_one_node_kernel(const int64_t* __restrict__ dst, int64_t E, int64_t* __restrict__ perm,
                                    int64_t* __restrict__ rowptr, int32_t* status) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (int64_t e = first; e < E; e += stride) {
        if (dst[e] != 0) atomicExch(status, 1);
        perm[e] = e;
    }
    if (first == 0) { rowptr[0] = 0; rowptr[1] = E; }
}

}  // namespace e3b

extern "C" int64_t e3b_csr_scratch_bytes(int64_t num_edges, int64_t num_nodes) {
    if (num_edges < 0 || num_nodes < 0) return 0;
    return e3b::csr_layout(num_edges, num_nodes, nullptr, nullptr);
}

extern "C" int e3b_csr_from_dst(const int64_t* dst, int64_t num_edges, int64_t num_nodes, int64_t* perm,
                                int64_t* rowptr, void* scratch, int64_t scratch_bytes, int32_t* status, void* stream) {
    using namespace e3b;
    const int64_t E = num_edges, N = num_nodes;
    if (E < 0 || N < 0) return fail(E3B_ERR_ARG, "csr: negative size");
    if (E >= (1LL << 31) || N >= (1LL << 31)) return fail(E3B_ERR_ARG, "csr: sizes must be below 2^31");
    if (!rowptr || !status || (E > 0 && (!dst || !perm))) return fail(E3B_ERR_ARG, "csr: null pointer");
    if (E > 0 && N == 0) return fail(E3B_ERR_ARG, "csr: edges but no nodes");
    const int64_t need = csr_layout(E, N, nullptr, nullptr);
    if (!scratch || scratch_bytes < need) return fail(E3B_ERR_ARG, "csr: scratch of %lld bytes needed, %lld given", (long long)need, (long long)scratch_bytes);
    if (reinterpret_cast<uintptr_t>(scratch) % 256 != 0) return fail(E3B_ERR_ARG, "csr: scratch must be 256-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CsrScratch sc;
    csr_layout(E, N, static_cast<char*>(scratch), &sc);

    E3B_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
    if (E == 0) {
        E3B_CUDA_TRY(cudaMemsetAsync(rowptr, 0, static_cast<size_t>(N + 1) * sizeof(int64_t), s));
        return E3B_OK;
    }
    int bits = 0;
    while (bits < 31 && ((N - 1) >> bits) != 0) ++bits;
    const int passes = (bits + 7) / 8;
    if (passes == 0) {
        csr_one_node_kernel<<<static_cast<int>(std::min<int64_t>(ceil_div(E, 256), kNumSMs * 8)), 256, 0, s>>>(dst, E, perm, rowptr, status);
        return check_launch("e3b_csr_from_dst");
    }
    const unsigned nb = static_cast<unsigned>(sc.nblocks);
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        const bool first = p == 0, last = p == passes - 1;
        if (first) radix_hist_kernel<true><<<nb, kSortThreads, 0, s>>>(dst, N, status, sc.keys[cur], E, shift, sc.hist, sc.nblocks);
        else radix_hist_kernel<false><<<nb, kSortThreads, 0, s>>>(nullptr, N, nullptr, sc.keys[cur], E, shift, sc.hist, sc.nblocks);
        radix_scan_kernel<<<kRadix, kSortThreads, 0, s>>>(sc.hist, sc.nblocks, sc.totals);
        auto scatter = first ? (last ? radix_scatter_kernel<true, true> : radix_scatter_kernel<true, false>)
                             : (last ? radix_scatter_kernel<false, true> : radix_scatter_kernel<false, false>);
        scatter<<<nb, kSortThreads, 0, s>>>(sc.keys[cur], sc.vals[cur], E, shift, sc.hist, sc.totals, sc.nblocks,
                                            sc.keys[cur ^ 1], sc.vals[cur ^ 1], perm);
        cur ^= 1;
    }
    csr_rowptr_kernel<<<static_cast<unsigned>(ceil_div(N + 1, 256)), 256, 0, s>>>(sc.keys[cur], E, N, rowptr);
    return check_launch("e3b_csr_from_dst");
}

// ------------------------------------------------------------------------------------------------
// Allocation-free variant: the scratch lives in this library's own device image.
//
// Some callers cannot hand over scratch memory because they cannot allocate any: code that
// runs inside a memory pool it does not own (an inference server's pre-sized arena), a plug-in
// invoked from a real-time loop where cudaMalloc's implicit device synchronisation is not
// acceptable, or a host language binding that has no device allocator of its own.  For them the
// work area is a fixed array in global memory that every GPU loading this library carries
// until the process exits (about 4.1 MiB).  The price is a hard size limit and a shared buffer.
namespace e3b {

constexpr int64_t kStaticCsrMaxEdges = 1 << 18;   // 262,144
constexpr int64_t kStaticCsrMaxNodes = 1 << 16;   // 65,536
// = csr_layout(kStaticCsrMaxEdges, kStaticCsrMaxNodes): 4 key/value buffers, digit histograms, digit totals
constexpr int64_t kStaticCsrBytes = 4 * (kStaticCsrMaxEdges * 4) + kRadix * (kStaticCsrMaxEdges / kSortChunk) * 4
                                    + kRadix * 4;

static __device__ __align__(256) unsigned char g_csr_static_scratch[kStaticCsrBytes];

constexpr int kMaxDevices = 64;
static void* g_csr_static_ptr[kMaxDevices] = {nullptr};
static std::mutex g_csr_static_mutex;

// Device address of the array on the current device.  In host code the array's name is only a
// handle for the runtime, never a device pointer: the address has to be asked for, once per
// device, while that device is current.
static int csr_static_address(void** out) {
    int dev = -1;
    E3B_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(E3B_ERR_UNSUPPORTED, "csr_static: device index %d not supported", dev);
    std::lock_guard<std::mutex> lock(g_csr_static_mutex);
    if (g_csr_static_ptr[dev] == nullptr) {
        void* p = nullptr;
        E3B_CUDA_TRY(cudaGetSymbolAddress(&p, g_csr_static_scratch));
        if (p == nullptr) return fail(E3B_ERR_CUDA, "csr_static: null symbol address");
        g_csr_static_ptr[dev] = p;
    }
    *out = g_csr_static_ptr[dev];
    return E3B_OK;
}

}  // namespace e3b

extern "C" int64_t e3b_csr_static_max_edges(void) { return e3b::kStaticCsrMaxEdges; }
extern "C" int64_t e3b_csr_static_max_nodes(void) { return e3b::kStaticCsrMaxNodes; }

extern "C" int e3b_csr_from_dst_static(const int64_t* dst, int64_t num_edges, int64_t num_nodes, int64_t* perm,
                                       int64_t* rowptr, int32_t* status, void* stream) {
    using namespace e3b;
    if (num_edges < 0 || num_nodes < 0) return fail(E3B_ERR_ARG, "csr_static: negative size");
    if (num_edges > kStaticCsrMaxEdges || num_nodes > kStaticCsrMaxNodes)
        return fail(E3B_ERR_ARG,
                    "csr_static: %lld edges / %lld nodes exceed the built-in work area (at most %lld edges and %lld nodes); "
                    "use e3b_csr_from_dst with caller-provided scratch",
                    (long long)num_edges, (long long)num_nodes, (long long)kStaticCsrMaxEdges, (long long)kStaticCsrMaxNodes);
    void* scratch = nullptr;
    const int rc = csr_static_address(&scratch);
    if (rc != E3B_OK) return rc;
    // The status word, which must start from zero, is cleared by the call below on
    // the caller's stream; the rest of the work area is fully overwritten before it is read.
    return e3b_csr_from_dst(dst, num_edges, num_nodes, perm, rowptr, scratch, kStaticCsrBytes, status, stream);
}
