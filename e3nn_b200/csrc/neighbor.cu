// Neighbour list of a periodic cubic box by a cell list, on the device.
//
// e3nn itself only ships an O(N^2) radius_graph (e3nn/nn/models/gate_points_2101.py:27-32) and states the
// periodic convention edge_vec = pos[src] - pos[dst] + shift
// (docs/guide/periodic_boundary_conditions.rst:134-136, gate_points_2101.py:328).  This builder produces,
// for every ordered pair with |pos[src] - pos[dst] + shift| <= cutoff (nearest image, src != dst), one
// edge; edges are sorted by destination, then by source, which is also the CSR order the fused
// convolution consumes (rowptr is an output).
//
// Integer work, HBM / latency bound, two passes because the edge count is not known in advance:
//   count: wrap positions into the box (fp64), bin atoms into cells of side box / floor(box / cutoff)
//          >= cutoff, exclusive scan of the cell counts, scatter the atoms (index and wrapped position) into cell
//          order, then one warp per atom counts its neighbours in the 27 surrounding cells -> rowptr (scan);
//   fill:  the same walk collects a row in shared memory, ranks its entries by source and writes (src, dst, shift)
//          at rowptr[dst] + rank, which removes the scatter's dependence on atomics order: the result is
//          bit-identical from run to run.
// A warp per atom: the 27 cells hold about 27 x 0.05 x 125 = 170 candidates of which 26 are neighbours, so the lanes
// test 32 candidates at a time from the cell-ordered copy of the positions (contiguous within a cell).  With one
// thread per atom, which walked the candidates one by one and sorted its row by insertion in global memory, the
// fill pass took 304 us for 256 atoms, 384 us for 4,001 and 2.07 ms for 262,144.
// Distances are evaluated in fp64 as (p_j - p_i) + image, the same value with the opposite sign from
// either end of a pair, so the list is symmetric by construction.
#include "common.cuh"
#include "scan.cuh"

namespace e3b {
namespace {

struct NeighborScratch {
    double* p;            // [N,3] wrapped positions
    double* p_cell;       // [N,3] the same in cell order
    int32_t* cell_of;     // [N]
    int32_t* cell_atoms;  // [N]
    int32_t* deg;         // [N]
    int32_t* cell_count;  // [C], then cell_fill [C] (one memset)
    int32_t* cell_fill;
    int64_t* cell_start;  // [C+1]
    int64_t* sums;        // block sums of the scans over C cells and N rows
};

__host__ __device__ inline size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

size_t carve(void* scratch, int64_t n, int64_t c, NeighborScratch* out) {
    unsigned char* b = static_cast<unsigned char*>(scratch);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = b ? b + off : nullptr;
        off += align256(bytes);
        return p;
    };
    NeighborScratch s;
    s.p = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    s.p_cell = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    s.cell_of = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n));
    s.cell_atoms = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n));
    s.deg = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * n));
    s.cell_count = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 2 * c));
    s.cell_fill = s.cell_count + c;
    s.cell_start = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * (c + 1)));
    s.sums = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * static_cast<size_t>(scan_blocks(c > n ? c : n))));
    if (out) *out = s;
    return off;
}

__global__ void wrap_bin_kernel(const float* __restrict__ pos, int64_t n, double box, int nc, double* __restrict__ p,
                                int32_t* __restrict__ cell_of, int32_t* __restrict__ cell_count) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double x = static_cast<double>(pos[i * 3 + a]);
        double w = x - floor(x / box) * box;
        if (w >= box) w -= box;
        if (w < 0.0) w = 0.0;
        p[i * 3 + a] = w;
        int q = static_cast<int>(w / box * nc);
        c[a] = q < 0 ? 0 : (q >= nc ? nc - 1 : q);
    }
    const int cell = (c[0] * nc + c[1]) * nc + c[2];
    cell_of[i] = cell;
    atomicAdd(cell_count + cell, 1);
}

__global__ void cell_scatter_kernel(const int32_t* __restrict__ cell_of, const double* __restrict__ p, int64_t n,
                                    const int64_t* __restrict__ cell_start, int32_t* __restrict__ cell_fill,
                                    int32_t* __restrict__ cell_atoms, double* __restrict__ p_cell) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int cell = cell_of[i];
    const int64_t slot = cell_start[cell] + atomicAdd(cell_fill + cell, 1);
    cell_atoms[slot] = static_cast<int32_t>(i);
    p_cell[slot * 3] = p[i * 3];
    p_cell[slot * 3 + 1] = p[i * 3 + 1];
    p_cell[slot * 3 + 2] = p[i * 3 + 2];
}

constexpr int kWalkWarps = 4;
constexpr int kRowCap = 256;   // row entries ranked in shared memory; longer rows are ranked by walking again

// The candidates of one atom: lane c < 27 holds cell c of the 3 x 3 x 3 block around it.
struct Candidates {
    int first;       // candidates in the cells before this lane's
    int64_t start;   // slot of this lane's cell
    int total;       // of all 27 cells
};

__device__ __forceinline__ Candidates candidates_of(int cell, int nc, const int64_t* __restrict__ cell_start, int lane) {
    const int cz = cell % nc, cy = (cell / nc) % nc, cx = cell / (nc * nc);
    int nx = cx + lane / 9 - 1, ny = cy + (lane / 3) % 3 - 1, nz = cz + lane % 3 - 1;
    nx += nx < 0 ? nc : 0; nx -= nx >= nc ? nc : 0;
    ny += ny < 0 ? nc : 0; ny -= ny >= nc ? nc : 0;
    nz += nz < 0 ? nc : 0; nz -= nz >= nc ? nc : 0;
    Candidates r{0, 0, 0};
    int count = 0;
    if (lane < 27) {
        const int64_t c = (static_cast<int64_t>(nx) * nc + ny) * nc + nz;
        r.start = cell_start[c];
        count = static_cast<int>(cell_start[c + 1] - r.start);
    }
    int incl = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    r.first = incl - count;
    r.total = __shfl_sync(0xffffffffu, incl, 31);
    return r;
}

// Candidate t (any t, all lanes call): the slot it sits in and its cell 0..26.  The last cell whose first
// candidate is <= t holds it (empty cells share `first` with the next one, the last of them wins).
__device__ __forceinline__ int64_t candidate_slot(const Candidates& c, int t, int* which) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const int mid = lo + step;
        const int f = __shfl_sync(0xffffffffu, c.first, mid < 27 ? mid : 26);
        if (mid < 27 && f <= t) lo = mid;
    }
    *which = lo;
    return __shfl_sync(0xffffffffu, c.start, lo) + (t - __shfl_sync(0xffffffffu, c.first, lo));
}

struct Image { double x, y, z; };

__device__ __forceinline__ Image image_of(int cell, int which, int nc, double box) {
    const int cz = cell % nc, cy = (cell / nc) % nc, cx = cell / (nc * nc);
    const int nx = cx + which / 9 - 1, ny = cy + (which / 3) % 3 - 1, nz = cz + which % 3 - 1;
    return {nx < 0 ? -box : (nx >= nc ? box : 0.0), ny < 0 ? -box : (ny >= nc ? box : 0.0), nz < 0 ? -box : (nz >= nc ? box : 0.0)};
}

// One warp per destination atom i of the rows [row0, row0 + nrows).  FILL == false: deg[i - row0] = number of
// neighbours.  FILL == true: writes the row's edges at rowptr[i - row0], sorted by source.
template <bool FILL>
__global__ void __launch_bounds__(32 * kWalkWarps) neighbor_walk_kernel(
        const float* __restrict__ pos, const double* __restrict__ p, const double* __restrict__ p_cell,
        const int32_t* __restrict__ cell_of, const int64_t* __restrict__ cell_start, const int32_t* __restrict__ cell_atoms,
        int64_t row0, int64_t nrows, double box, double cutoff2, int nc, int32_t* __restrict__ deg,
        const int64_t* __restrict__ rowptr, int64_t* __restrict__ edge_src, int64_t* __restrict__ edge_dst,
        float* __restrict__ shift) {
    __shared__ int32_t row_src[FILL ? kWalkWarps : 1][FILL ? kRowCap : 1];
    __shared__ uint8_t row_cell[FILL ? kWalkWarps : 1][FILL ? kRowCap : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t local = static_cast<int64_t>(blockIdx.x) * kWalkWarps + warp;
    if (local >= nrows) return;
    const int64_t i = row0 + local;
    const double pix = p[i * 3], piy = p[i * 3 + 1], piz = p[i * 3 + 2];
    const int cell = cell_of[i];
    const Candidates cand = candidates_of(cell, nc, cell_start, lane);

    // whether candidate t is a neighbour; all lanes call, lanes past the end get false
    auto test = [&](int t, int* j, int* which) {
        const int64_t slot = candidate_slot(cand, t < cand.total ? t : 0, which);
        if (t >= cand.total) return false;
        *j = cell_atoms[slot];
        const Image im = image_of(cell, *which, nc, box);
        const double dx = (p_cell[slot * 3] - pix) + im.x, dy = (p_cell[slot * 3 + 1] - piy) + im.y,
                     dz = (p_cell[slot * 3 + 2] - piz) + im.z;
        return *j != i && dx * dx + dy * dy + dz * dz <= cutoff2;
    };

    if (!FILL) {
        int count = 0;
        for (int t = lane; t - lane < cand.total; t += 32) {
            int j, which;
            count += test(t, &j, &which) ? 1 : 0;
        }
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0) deg[local] = count;
        return;
    }

    const int64_t base = rowptr[local];
    const int n = static_cast<int>(rowptr[local + 1] - base);
    // offset between the caller's coordinates and the wrapped ones (0 for atoms inside the box)
    const double oix = pix - static_cast<double>(pos[i * 3]), oiy = piy - static_cast<double>(pos[i * 3 + 1]),
                 oiz = piz - static_cast<double>(pos[i * 3 + 2]);
    auto store = [&](int64_t e, int j, int which) {
        const Image im = image_of(cell, which, nc, box);
        edge_src[e] = j;
        edge_dst[e] = i;
        // edge_vec = pos[src] - pos[dst] + shift must equal (p_j - p_i) + image
        shift[e * 3] = static_cast<float>((p[j * 3ll] - static_cast<double>(pos[j * 3ll])) - oix + im.x);
        shift[e * 3 + 1] = static_cast<float>((p[j * 3ll + 1] - static_cast<double>(pos[j * 3ll + 1])) - oiy + im.y);
        shift[e * 3 + 2] = static_cast<float>((p[j * 3ll + 2] - static_cast<double>(pos[j * 3ll + 2])) - oiz + im.z);
    };
    if (n <= kRowCap) {
        int have = 0;
        for (int t = lane; t - lane < cand.total; t += 32) {
            int j = 0, which = 0;
            const bool ok = test(t, &j, &which);
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            const int at = have + __popc(m & ((1u << lane) - 1u));
            if (ok && at < n) { row_src[warp][at] = j; row_cell[warp][at] = static_cast<uint8_t>(which); }
            have += __popc(m);
        }
        __syncwarp();
        for (int a = lane; a < n; a += 32) {
            const int j = row_src[warp][a];
            int rank = 0;
            for (int b = 0; b < n; ++b) rank += row_src[warp][b] < j ? 1 : 0;
            store(base + rank, j, row_cell[warp][a]);
        }
        return;
    }
    // a row too long for shared memory: every neighbour's rank is counted by one more walk over the candidates
    for (int t0 = 0; t0 < cand.total; t0 += 32) {
        int j = 0, which = 0;
        const bool ok = test(t0 + lane, &j, &which);
        unsigned m = __ballot_sync(0xffffffffu, ok);
        while (m != 0) {
            const int from = __ffs(m) - 1;
            m &= m - 1;
            const int key = __shfl_sync(0xffffffffu, j, from);
            int below = 0;
            for (int t = lane; t - lane < cand.total; t += 32) {
                int j2 = 0, w2 = 0;
                below += (test(t, &j2, &w2) && j2 < key) ? 1 : 0;
            }
            below = __reduce_add_sync(0xffffffffu, below);
            if (lane == from) store(base + below, j, which);
        }
    }
}

int cells_per_side(double box, double cutoff) {
    const double q = floor(box / cutoff);
    return q > 1024.0 ? 1024 : static_cast<int>(q);   // more cells than that only lengthens the scan
}

int check_rows(int64_t n, int64_t row0, int64_t row1) {
    if (row0 < 0 || row1 < row0 || row1 > n) return fail(E3B_ERR_ARG, "neighbor list: rows [%lld, %lld) outside [0, %lld)",
                                                          static_cast<long long>(row0), static_cast<long long>(row1), static_cast<long long>(n));
    return E3B_OK;
}

int check_neighbor_args(int64_t n, double box, double cutoff) {
    if (n < 0) return fail(E3B_ERR_ARG, "neighbor list: negative atom count");
    if (n > 2147483647LL) return fail(E3B_ERR_ARG, "neighbor list: more than 2^31 - 1 atoms");
    if (!(cutoff > 0.0) || !(box > 0.0)) return fail(E3B_ERR_ARG, "neighbor list: box and cutoff must be positive");
    if (box < 3.0 * cutoff)
        return fail(E3B_ERR_UNSUPPORTED, "neighbor list: the cell list needs box >= 3 x cutoff (box %g, cutoff %g)", box, cutoff);
    return E3B_OK;
}

}  // namespace
}  // namespace e3b

extern "C" int64_t e3b_neighbor_scratch_bytes(int64_t num_atoms, double box, double cutoff) {
    using namespace e3b;
    if (num_atoms < 0 || !(cutoff > 0.0) || box < 3.0 * cutoff) return -1;
    const int64_t nc = cells_per_side(box, cutoff);
    return static_cast<int64_t>(carve(nullptr, num_atoms, nc * nc * nc, nullptr));
}

extern "C" int e3b_neighbor_count(const float* pos, int64_t num_atoms, double box, double cutoff, void* scratch,
                                  int64_t scratch_bytes, int64_t* rowptr, void* stream) {
    return e3b_neighbor_count_rows(pos, num_atoms, box, cutoff, scratch, scratch_bytes, 0, num_atoms, rowptr, stream);
}

extern "C" int e3b_neighbor_count_rows(const float* pos, int64_t num_atoms, double box, double cutoff, void* scratch,
                                       int64_t scratch_bytes, int64_t row0, int64_t row1, int64_t* rowptr, void* stream) {
    using namespace e3b;
    if (int rc = check_neighbor_args(num_atoms, box, cutoff)) return rc;
    if (int rc = check_rows(num_atoms, row0, row1)) return rc;
    if (!rowptr) return fail(E3B_ERR_ARG, "neighbor_count: null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t nrows = row1 - row0;
    if (num_atoms == 0 || nrows == 0) {
        E3B_CUDA_TRY(cudaMemsetAsync(rowptr, 0, sizeof(int64_t), s));
        return E3B_OK;
    }
    const int nc = cells_per_side(box, cutoff);
    const int64_t cells = static_cast<int64_t>(nc) * nc * nc;
    if (!pos || !scratch) return fail(E3B_ERR_ARG, "neighbor_count: null pointer");
    if (scratch_bytes < static_cast<int64_t>(carve(nullptr, num_atoms, cells, nullptr)) || reinterpret_cast<uintptr_t>(scratch) % 256 != 0)
        return fail(E3B_ERR_ARG, "neighbor_count: scratch too small or not 256-byte aligned");
    NeighborScratch sc;
    carve(scratch, num_atoms, cells, &sc);
    E3B_CUDA_TRY(cudaMemsetAsync(sc.cell_count, 0, sizeof(int32_t) * 2 * cells, s));
    const int threads = 256;
    const unsigned grid = static_cast<unsigned>(ceil_div(num_atoms, threads));
    wrap_bin_kernel<<<grid, threads, 0, s>>>(pos, num_atoms, box, nc, sc.p, sc.cell_of, sc.cell_count);
    launch_exclusive_scan(sc.cell_count, cells, sc.sums, sc.cell_start, s);
    cell_scatter_kernel<<<grid, threads, 0, s>>>(sc.cell_of, sc.p, num_atoms, sc.cell_start, sc.cell_fill, sc.cell_atoms, sc.p_cell);
    neighbor_walk_kernel<false><<<static_cast<unsigned>(ceil_div(nrows, kWalkWarps)), 32 * kWalkWarps, 0, s>>>(
        pos, sc.p, sc.p_cell, sc.cell_of, sc.cell_start, sc.cell_atoms, row0, nrows, box, cutoff * cutoff, nc, sc.deg, nullptr,
        nullptr, nullptr, nullptr);
    launch_exclusive_scan(sc.deg, nrows, sc.sums, rowptr, s);
    return check_launch("neighbor_count");
}

extern "C" int e3b_neighbor_fill(const float* pos, int64_t num_atoms, double box, double cutoff, void* scratch,
                                 int64_t scratch_bytes, const int64_t* rowptr, int64_t* edge_src, int64_t* edge_dst,
                                 float* shift, void* stream) {
    return e3b_neighbor_fill_rows(pos, num_atoms, box, cutoff, scratch, scratch_bytes, 0, num_atoms, rowptr, edge_src, edge_dst,
                                  shift, stream);
}

extern "C" int e3b_neighbor_fill_rows(const float* pos, int64_t num_atoms, double box, double cutoff, void* scratch,
                                      int64_t scratch_bytes, int64_t row0, int64_t row1, const int64_t* rowptr, int64_t* edge_src,
                                      int64_t* edge_dst, float* shift, void* stream) {
    using namespace e3b;
    if (int rc = check_neighbor_args(num_atoms, box, cutoff)) return rc;
    if (int rc = check_rows(num_atoms, row0, row1)) return rc;
    const int64_t nrows = row1 - row0;
    if (num_atoms == 0 || nrows == 0) return E3B_OK;
    const int nc = cells_per_side(box, cutoff);
    const int64_t cells = static_cast<int64_t>(nc) * nc * nc;
    if (!pos || !scratch || !rowptr || !edge_src || !edge_dst || !shift) return fail(E3B_ERR_ARG, "neighbor_fill: null pointer");
    if (scratch_bytes < static_cast<int64_t>(carve(nullptr, num_atoms, cells, nullptr)) || reinterpret_cast<uintptr_t>(scratch) % 256 != 0)
        return fail(E3B_ERR_ARG, "neighbor_fill: scratch too small or not 256-byte aligned");
    NeighborScratch sc;
    carve(scratch, num_atoms, cells, &sc);
    neighbor_walk_kernel<true><<<static_cast<unsigned>(ceil_div(nrows, kWalkWarps)), 32 * kWalkWarps, 0, static_cast<cudaStream_t>(stream)>>>(
        pos, sc.p, sc.p_cell, sc.cell_of, sc.cell_start, sc.cell_atoms, row0, nrows, box, cutoff * cutoff, nc, sc.deg, rowptr,
        edge_src, edge_dst, shift);
    return check_launch("neighbor_fill");
}
