// neighbors.cu — cell keys, fluid reorder, cell-start table, neighbour lists and boundary psi.
//
// Reference: cuda_neighborsSearch (DFSPH_core_cuda.cu:2651-3024) with
// DFSPH_computeGridIdx_kernel (:1833-1848), DFSPH_CountingSortIds_kernel (:1851-1857),
// cuda_sortData (:2057-2120) and DFSPH_neighborsSearch_kernel<true> (:2219-2517), which iterates
// ITER_NEIGHBORS_FROM_STRUCTURE_LINEAR_ADVANCED (DFSPH_macro_cuda.h:136-155): every particle of the
// 27 cells around the particle's cell is tested with squaredNorm < H^2, self excluded for the fluid.
//
// Differences by design: 30-bit Morton keys sorted by a stable in-house radix sort (sort.cu)
// instead of a dense 256^3 histogram; a cell table sized to the scene's grid, cleared per step;
// neighbour lists with a checked capacity (the reference writes past MAX_NEIGHBOURS = 90 unchecked).
#include <algorithm>

#include "dfsph_state.cuh"
#include "sort.cuh"

namespace dfsph {

namespace {

template <class Real>
__device__ __forceinline__ bool particle_cell(Real x, Real y, Real z, const StepParams<Real>& p, int& cx, int& cy,
                                              int& cz) {
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) return false;
    cx = cell_coord(x, p.kern.H, p.off_x);
    cy = cell_coord(y, p.kern.H, p.off_y);
    cz = cell_coord(z, p.kern.H, p.off_z);
    return cx >= 0 && cy >= 0 && cz >= 0 && cx < p.dim_x && cy < p.dim_y && cz < p.dim_z;
}

__device__ __forceinline__ uint32_t cell_linear(int cx, int cy, int cz, int dim_x, int dim_y) {
    return (uint32_t)cx + (uint32_t)dim_x * ((uint32_t)cy + (uint32_t)dim_y * (uint32_t)cz);
}

// Cell keys and, for the sort that follows, the histograms of their 8-bit digits (hist: 256 words per
// pass, zero before the launch), counted in shared memory first. Launches bound the binning of a small
// set and memory that of a large one. Counting here, scanning in the sort's passes and the fused reorder
// below took it from nine launches to five with three digits: 38 -> 24 us at 27 k particles, 61 -> 44 us at
// 250 k, 95 -> 83 us at 1 M (as timed alone); the step 705 -> 691 us at 250 k, unchanged at 1 k. One, two
// and four keys per thread differ by less than the runs do from 27 k to 1 M; two halves the words that
// blocks add to the global histograms.
// The pass clears two buffers of the binning on the way (16-byte aligned). Few particles in a large domain
// have a table far larger than their keys: blocks are added until a thread clears no more than kClearPerThread
// words, up to kClearBlocks blocks (the resident ones). 1000 particles, a grid by the keys alone -> this one:
// binning with 200^3 cells 792 -> 34 us, with 400^3 5690 -> 118 us, with 20^3 unchanged. Where there are 512
// keys or more to 4096 words the two grids are the same.
constexpr uint32_t kKeysPerThread = 2;
constexpr size_t kClearPerThread = 16;
constexpr size_t kClearBlocks = 148 * 8;
__device__ __forceinline__ void clear_words(uint32_t* __restrict__ z, size_t words, size_t t, size_t stride) {
    uint4* __restrict__ v = reinterpret_cast<uint4*>(z);
    for (size_t k = t; k < words / 4; k += stride) v[k] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t k = (words & ~(size_t)3) + t; k < words; k += stride) z[k] = 0u;
}
template <class Real>
__global__ void __launch_bounds__(kBlock) cell_keys_kernel(const Vec4<Real>* __restrict__ pos, uint32_t n,
                                                           StepParams<Real> p, uint32_t* __restrict__ keys,
                                                           uint32_t* __restrict__ status, uint32_t* __restrict__ hist,
                                                           int passes, uint32_t* __restrict__ z0, size_t w0,
                                                           uint32_t* __restrict__ z1, size_t w1) {
    __shared__ uint32_t counted[kSortHistWords];
    DFSPH_PDL_ENTER;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    clear_words(z0, w0, t, stride);
    clear_words(z1, w1, t, stride);
    for (uint32_t k = threadIdx.x; k < kSortHistWords; k += kBlock) counted[k] = 0u;
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kKeysPerThread; ++u) {
        const uint32_t i = (blockIdx.x * kKeysPerThread + u) * kBlock + threadIdx.x;
        if (i >= n) break;
        const Vec4<Real> x = pos[i];
        int cx, cy, cz;
        uint32_t key;
        if (particle_cell(x.x, x.y, x.z, p, cx, cy, cz)) {
            key = morton3((uint32_t)cx, (uint32_t)cy, (uint32_t)cz);
        } else {
            key = kEscapedKey;
            const bool finite = isfinite(x.x) && isfinite(x.y) && isfinite(x.z);
            atomicOr(status, finite ? DFSPH_ST_ESCAPED : (DFSPH_ST_NONFINITE | DFSPH_ST_ESCAPED));
        }
        keys[i] = key;
        for (int d = 0; d < passes; ++d) atomicAdd(&counted[d * kSortDigits + ((key >> (8 * d)) & 255u)], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < (uint32_t)passes * kSortDigits; k += kBlock)
        if (counted[k]) atomicAdd(hist + k, counted[k]);
}

// Cell start/end from run boundaries of the sorted keys (replaces the dense histogram scan).
__device__ __forceinline__ void mark_cell_bounds(const uint32_t* __restrict__ keys, uint32_t n, uint32_t i, int dim_x,
                                                 int dim_y, int dim_z, uint2* __restrict__ table) {
    const uint32_t k = keys[i];
    if (k == kEscapedKey) return;
    const uint32_t cx = compact_bits10(k), cy = compact_bits10(k >> 1), cz = compact_bits10(k >> 2);
    if (cx >= (uint32_t)dim_x || cy >= (uint32_t)dim_y || cz >= (uint32_t)dim_z) return;
    const uint32_t lin = cell_linear((int)cx, (int)cy, (int)cz, dim_x, dim_y);
    if (i == 0 || keys[i - 1] != k) table[lin].x = i;
    if (i == n - 1 || keys[i + 1] != k) table[lin].y = i + 1;
}

// The end of a fluid binning in one launch: the reorder of the particles, the cell table, the state block
// with the reordered arrays' pointers, and the sort's histograms cleared for the next key pass.
template <class Real> struct FluidArrays {
    Vec4<Real>*pos, *vel;
    Real *kappa, *kappaV;
    uint32_t* id;
};
template <class Real>
__global__ void __launch_bounds__(kBlock) reorder_fluid_kernel(
    const uint32_t* __restrict__ perm, const uint32_t* __restrict__ sorted_keys, uint32_t n, const FluidArrays<Real> in,
    const FluidArrays<Real> out, uint2* __restrict__ table, uint32_t* __restrict__ hist, DevState<Real>* __restrict__ ds,
    const DevState<Real> state) {
    DFSPH_PDL_ENTER;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) publish_state(ds, state);
    if (blockIdx.x == gridDim.x - 1)
        for (uint32_t k = threadIdx.x; k < kSortHistWords; k += kBlock) hist[k] = 0u;
    if (i >= n) return;
    mark_cell_bounds(sorted_keys, n, i, state.p.dim_x, state.p.dim_y, state.p.dim_z, table);
    uint32_t j = perm[i];
    if (j >= n) j = i;  // only after a failed sort (flagged in the status word); stay in range
    out.pos[i] = in.pos[j];
    out.vel[i] = in.vel[j];
    out.kappa[i] = in.kappa[j];
    out.kappaV[i] = in.kappaV[j];
    out.id[i] = in.id[j];
}

template <class Real>
__global__ void __launch_bounds__(kBlock) reorder_pair_kernel(const uint32_t* __restrict__ perm, uint32_t n,
                                                              const Real* __restrict__ a_in,
                                                              const Real* __restrict__ b_in, Real* __restrict__ a_out,
                                                              Real* __restrict__ b_out) {
    DFSPH_PDL_ENTER;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t j = perm[i];
    if (j >= n) j = i;
    a_out[i] = a_in[j];
    b_out[i] = b_in[j];
}

// A cell-table run [r.x, r.y) of a set of `limit` particles. Checked builds verify it and raise
// DFSPH_ST_INDEX instead of scanning a run out of range; the unchecked build trusts the table.
__device__ __forceinline__ bool run_in_range(uint2 r, uint32_t limit, uint32_t* status) {
#ifdef DFSPH_CHECKED
    if (r.x > r.y || r.y > limit) {
        atomicOr(status, DFSPH_ST_INDEX);
        return false;
    }
#else
    (void)r;
    (void)limit;
    (void)status;
#endif
    return true;
}

#ifdef DFSPH_CHECKED
// Test hook of the checked build: replaces particle 0's first list entry by `value` (an index past the
// fluid count, inside the allocation), which the validation below must report.
__global__ void corrupt_first_neighbor_kernel(uint4* __restrict__ nbr, const uint32_t* __restrict__ counts,
                                              uint32_t value) {
    if (threadIdx.x == 0 && (counts[0] & 0xFFFFu) > 0) nbr[0].x = value;
}

// Validation of the lists before any pass gathers through them (checked build): a count past the
// table's capacity, a fluid entry >= n or a boundary entry >= n_boundary raises DFSPH_ST_INDEX and
// empties that particle's list, so no pass reads out of range. The passes themselves are the
// unchecked build's code, so a clean run gives the same bits.
__global__ void __launch_bounds__(kBlock) validate_neighbors_kernel(uint32_t* __restrict__ counts,
                                                                    const uint4* __restrict__ nbr, uint32_t n,
                                                                    uint32_t n_boundary, uint32_t stride, uint32_t cap,
                                                                    uint32_t* __restrict__ status) {
    DFSPH_PDL_ENTER;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = counts[i], nf = c & 0xFFFFu, nb = c >> 16;
    bool bad = nf + nb > cap;
    const uint32_t* __restrict__ words = reinterpret_cast<const uint32_t*>(nbr);
    const uint32_t b0 = 4u * slot_groups(nf), end = b0 + 4u * slot_groups(nb);  // fill-up slots are gathered too
    for (uint32_t k = 0; k < end && !bad; ++k) bad = words[slot_word(k, stride, i)] >= (k < b0 ? n : n_boundary);
    if (bad) {
        atomicOr(status, DFSPH_ST_INDEX);
        counts[i] = 0u;
    }
}
#endif

// Neighbour build: one thread per fluid particle; fluid neighbours (self excluded), then boundary
// neighbours, cells in a fixed order (z, y, x from -1 to +1), particles of a cell in sorted order.
//
// The pass is bound by instruction issue (about 216 candidate tests per particle for ~30 accepted), so
// a test is kept to the load, the predicate and a predicated append without a branch. Appends go to a
// column of shared memory (ListStage) and from there to the list a whole group (four slots, 16 bytes)
// at a time. The column holds 40 entries, more than most lists, and when a lane has to flush all lanes of
// the warp that scan with it do: with 24 entries and each lane for itself the flushes were a quarter of
// the pass's instructions. Measured at 1 M particles, static / moving walls: 336 / 348 us -> 304 / 319 us
// (386 us with a branch per accepted candidate and no column); 250 k 106 -> 97 us, 1 k 33 -> 29 us. Five
// or six blocks per SM instead of four, two, five or eight candidates per batch instead of four, and two
// particles of a cell per thread were slower or, for large scenes, at most 5 % faster.
constexpr uint32_t kStageSlots = 40;
constexpr uint32_t kScanBatch = 4;
constexpr int kBuildMinBlocks = 4;
static_assert(kScanBatch - 1 <= kScanPad, "a batch reads past the end of the last run");

// One part (fluid or boundary) of a thread's list while it is built.
struct ListStage {
    uint32_t* column;  // shared memory: entry k waits at column[k * kBlock]
    uint32_t top;      // kBlock times the entries waiting
    uint32_t written;  // entries flushed (a multiple of four)
    uint32_t cap;      // entries the list can take
    uint4* group;      // where the next group goes
    uint32_t stride;

    __device__ __forceinline__ void append(uint32_t j) {
        column[top] = j;
        top += kBlock;
    }
    __device__ __forceinline__ void store_group(uint32_t k) {  // k: kBlock times the first entry
        if (written < cap)
            *group = make_uint4(column[k], column[k + kBlock], column[k + 2 * kBlock], column[k + 3 * kBlock]);
        group += stride;
        written += 4;
    }
    // Writes the whole groups; fewer than four entries stay.
    __device__ __forceinline__ void flush() {
        uint32_t k = 0;
        for (; k + 4 * kBlock <= top; k += 4 * kBlock) store_group(k);
        for (uint32_t u = 0; k + u < top; u += kBlock) column[u] = column[k + u];
        top -= k;
    }
    // Ends the part: fills its last group up with `fill`, or with its last entry, and returns the number
    // of entries kept; the list continues at `group`.
    __device__ __forceinline__ uint32_t finish(bool last, uint32_t fill, bool& overflow) {
        flush();
        const uint32_t total = written + top / kBlock;
        if (top) {
            const uint32_t v = last ? column[top - kBlock] : fill;
            for (uint32_t k = top; k < 4 * kBlock; k += kBlock) column[k] = v;
            store_group(0);
        }
        overflow = overflow || total > cap;
        return min(total, cap);
    }
};

// Appends the candidates [j0, j1) of one cell that lie within H of particle i, in index order (the
// fluid skips i itself). The positions are loaded kScanBatch at a time so that several loads are in
// flight per thread (src has kScanPad elements to spare after its last).
template <class Real, bool kFluid>
__device__ __forceinline__ void scan_cell(const Vec4<Real>* __restrict__ src, uint32_t j0, uint32_t j1, uint32_t i,
                                          const Vec4<Real>& xi, Real H2, ListStage& st) {
    for (uint32_t jb = j0; jb < j1; jb += kScanBatch) {
        // (a hint: which lanes scan together does not change what any of them writes)
        if (__any_sync(__activemask(), st.top > (kStageSlots - kScanBatch) * kBlock)) st.flush();
        Vec4<Real> xj[kScanBatch];
#pragma unroll
        for (uint32_t u = 0; u < kScanBatch; ++u) xj[u] = ld4<Real>(src + jb + u);
#pragma unroll
        for (uint32_t u = 0; u < kScanBatch; ++u) {
            const uint32_t j = jb + u;
            if (pair_within(xi.x, xi.y, xi.z, xj[u].x, xj[u].y, xj[u].z, H2) & (j < j1) & (!kFluid | (j != i)))
                st.append(j);
        }
    }
}

// The 27 cells around (cx, cy, cz) of one cell table, a row of three at a time.
template <class Real, bool kFluid>
__device__ __forceinline__ void scan_cells(const Vec4<Real>* __restrict__ src, const uint2* __restrict__ tab, int cx,
                                           int cy, int cz, const StepParams<Real>& p, uint32_t limit, uint32_t* status,
                                           uint32_t i, const Vec4<Real>& xi, ListStage& st) {
    const Real H2 = p.H2;
#pragma unroll 1
    for (int k = 0; k < 9; ++k) {
        const int z = cz - 1 + k / 3, y = cy - 1 + k % 3;
        if ((uint32_t)z >= (uint32_t)p.dim_z || (uint32_t)y >= (uint32_t)p.dim_y) continue;
        const uint2* __restrict__ row = tab + cell_linear(0, y, z, p.dim_x, p.dim_y);
        uint2 r[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int x = cx - 1 + u;
            r[u] = (uint32_t)x < (uint32_t)p.dim_x ? row[x] : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (run_in_range(r[u], limit, status)) scan_cell<Real, kFluid>(src, r[u].x, r[u].y, i, xi, H2, st);
    }
}

template <class Real, bool kShift>
__global__ void __launch_bounds__(kBlock, kBuildMinBlocks) build_neighbors_kernel(const DevState<Real>* __restrict__ ds, uint32_t n,
                                                                 const uint2* __restrict__ ftab,
                                                                 const uint2* __restrict__ btab,
                                                                 const uint8_t* __restrict__ bnear) {
    __shared__ uint32_t stage[kStageSlots * kBlock];
    DFSPH_PDL_ENTER;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const StepParams<Real>& p = ds->p;
    const Vec4<Real>* __restrict__ bpos = ds->bpos;
    const Vec4<Real> xi = ds->pos[i];
    int cx, cy, cz;
    uint32_t nf = 0, nb = 0;
    bool overflow = false;
    if (particle_cell(xi.x, xi.y, xi.z, p, cx, cy, cz)) {
        ListStage st;
        st.column = stage + threadIdx.x;
        st.top = st.written = 0;
        st.cap = p.nbr_cap;
        st.group = ds->nbr + i;
        st.stride = p.nbr_stride;
        scan_cells<Real, true>(ds->pos, ftab, cx, cy, cz, p, n, ds->status, i, xi, st);
        nf = st.finish(false, i, overflow);
        st.group = ds->nbr + (size_t)slot_groups(nf) * p.nbr_stride + i;
        st.top = st.written = 0;
        st.cap = p.nbr_cap - nf;
        if (p.n_boundary > 0 && !kShift) {
            if (bnear[cell_linear(cx, cy, cz, p.dim_x, p.dim_y)])
                scan_cells<Real, false>(bpos, btab, cx, cy, cz, p, p.n_boundary, ds->status, i, xi, st);
        }
        if (p.n_boundary > 0 && kShift) {
            // The whole boundary has only translated by s since it was binned: the cells around the
            // binned cell of x_i - s, with one more layer on a side where x_i - s lies within 1e-3 of a
            // cell face (the binned and the current positions differ from s by rounding; the pair test
            // uses the current positions).
            int lo[3], hi[3], mid[3];
            bool query = true;
            const float q[3] = {__fsub_rn((float)xi.x, (float)p.bsx), __fsub_rn((float)xi.y, (float)p.bsy),
                                __fsub_rn((float)xi.z, (float)p.bsz)};
            const int off[3] = {p.off_x, p.off_y, p.off_z};
            const int dim[3] = {p.dim_x, p.dim_y, p.dim_z};
            const float Hf = (float)p.kern.H;
            bool inside = true;
            for (int a = 0; a < 3 && query; ++a) {
                const float t = __fadd_rn(__fdiv_rn(q[a], Hf), (float)off[a]);
                if (!(fabsf(t) < 1.0e8f)) {  // also NaN: no boundary neighbours, as off the grid
                    query = false;
                    break;
                }
                const float c = floorf(t), frac = t - c;
                mid[a] = (int)c;
                inside = inside && mid[a] >= 0 && mid[a] < dim[a];
                lo[a] = (int)c - 1 - (frac < 1e-3f ? 1 : 0);
                hi[a] = (int)c + 1 + (frac > 1.0f - 1e-3f ? 1 : 0);
            }
            // no boundary cell within two cells of the binned cell: nothing to look up
            if (query && inside && !bnear[cell_linear(mid[0], mid[1], mid[2], p.dim_x, p.dim_y)]) query = false;
            for (int z = query ? lo[2] : 1; query && z <= hi[2]; ++z) {
                if (z < 0 || z >= p.dim_z) continue;
                for (int y = lo[1]; y <= hi[1]; ++y) {
                    if (y < 0 || y >= p.dim_y) continue;
                    for (int x = lo[0]; x <= hi[0]; ++x) {
                        if (x < 0 || x >= p.dim_x) continue;
                        const uint2 r = btab[cell_linear(x, y, z, p.dim_x, p.dim_y)];
                        if (!run_in_range(r, p.n_boundary, ds->status)) continue;
                        scan_cell<Real, false>(bpos, r.x, r.y, i, xi, p.H2, st);
                    }
                }
            }
        }
        nb = st.finish(true, 0u, overflow);
    }
    if (overflow) atomicOr(ds->status, DFSPH_ST_NEIGHBOR_OVERFLOW);
    ds->counts[i] = nf | (nb << 16);
}

// The end of a boundary binning in one launch: the cell table, the marks of the cells within two cells
// (along each axis) of a cell that holds boundary particles, and the sort's histograms cleared for the next key
// pass. Fluid in an unmarked cell has no boundary neighbours, and the neighbour build skips their cell table.
// One thread per boundary particle; the first of each cell's run marks. Two launches and two memsets -> one
// launch: moving a part of the boundary 59 -> 46 us at 500 samples, 62 -> 53 us at 23 k, 74 -> 65 us at 56 k.
__global__ void __launch_bounds__(kBlock) boundary_cells_kernel(const uint32_t* __restrict__ keys, uint32_t nb,
                                                                int dim_x, int dim_y, int dim_z,
                                                                uint2* __restrict__ table,
                                                                uint8_t* __restrict__ bnear,
                                                                uint32_t* __restrict__ hist) {
    DFSPH_PDL_ENTER;
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == gridDim.x - 1)
        for (uint32_t k = threadIdx.x; k < kSortHistWords; k += kBlock) hist[k] = 0u;
    if (b >= nb) return;
    mark_cell_bounds(keys, nb, b, dim_x, dim_y, dim_z, table);
    const uint32_t k = keys[b];
    if (k == kEscapedKey || (b > 0 && keys[b - 1] == k)) return;
    const int cx = (int)compact_bits10(k), cy = (int)compact_bits10(k >> 1), cz = (int)compact_bits10(k >> 2);
    for (int z = max(cz - 2, 0); z <= min(cz + 2, dim_z - 1); ++z)
        for (int y = max(cy - 2, 0); y <= min(cy + 2, dim_y - 1); ++y)
            for (int x = max(cx - 2, 0); x <= min(cx + 2, dim_x - 1); ++x)
                bnear[cell_linear(x, y, z, dim_x, dim_y)] = 1;
}

// Akinci boundary psi (FluidModel::computeBoundaryPsi, FluidModel.cpp:233-258):
// psi_b = rho0 / (W0 + sum_{b' != b, |x_b - x_b'| < H} W(x_b - x_b')), accumulated in FP64.
template <class Real>
__global__ void __launch_bounds__(kBlock) boundary_psi_kernel(const Vec4<Real>* __restrict__ bpos_in,
                                                              Vec4<Real>* __restrict__ bpos_out, uint32_t nb,
                                                              StepParams<Real> p, const uint2* __restrict__ btab,
                                                              uint32_t* __restrict__ status) {
    DFSPH_PDL_ENTER;
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const Vec4<Real> xb = bpos_in[b];
    int cx, cy, cz;
    const double H = (double)p.kern.H;
    const double k = 8.0 / (3.14159265358979323846 * H * H * H);
    double delta = k;  // W(0)
    if (particle_cell(xb.x, xb.y, xb.z, p, cx, cy, cz)) {
        for (int dz = -1; dz <= 1; ++dz) {
            const int z = cz + dz;
            if (z < 0 || z >= p.dim_z) continue;
            for (int dy = -1; dy <= 1; ++dy) {
                const int y = cy + dy;
                if (y < 0 || y >= p.dim_y) continue;
                for (int dx = -1; dx <= 1; ++dx) {
                    const int x = cx + dx;
                    if (x < 0 || x >= p.dim_x) continue;
                    const uint2 r = btab[cell_linear(x, y, z, p.dim_x, p.dim_y)];
                    if (!run_in_range(r, nb, status)) continue;
                    for (uint32_t j = r.x; j < r.y; ++j) {
                        if (j == b) continue;
                        const Vec4<Real> xj = bpos_in[j];
                        if (pair_within(xb.x, xb.y, xb.z, xj.x, xj.y, xj.z, p.H2)) {
                            const double rx = (double)xb.x - (double)xj.x;
                            const double ry = (double)xb.y - (double)xj.y;
                            const double rz = (double)xb.z - (double)xj.z;
                            const double q = sqrt(rx * rx + ry * ry + rz * rz) / H;
                            double w = 0.0;
                            if (q <= 1.0) {
                                if (q <= 0.5) {
                                    w = k * (6.0 * q * q * q - 6.0 * q * q + 1.0);
                                } else {
                                    const double f = 1.0 - q;
                                    w = k * (2.0 * f * f * f);
                                }
                            }
                            delta += w;
                        }
                    }
                }
            }
        }
    } else {
        atomicOr(status, DFSPH_ST_BOUNDARY_OVERFLOW);
    }
    Vec4<Real> out = xb;
    out.w = (Real)((double)p.density0 / delta);
    bpos_out[b] = out;
}

template <class Real>
__global__ void __launch_bounds__(kBlock) scatter_by_id_kernel(const uint32_t* __restrict__ id, uint32_t n,
                                                               const Real* __restrict__ src, int comps,
                                                               int src_stride, Real* __restrict__ dst) {
    DFSPH_PDL_ENTER;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t t = id[i];
    for (int c = 0; c < comps; ++c) dst[(size_t)t * comps + c] = src[(size_t)i * src_stride + c];
}

}  // namespace

template <class Real>
void launch_cell_keys(const Vec4<Real>* pos, uint32_t n, const StepParams<Real>& p, uint32_t* keys, uint32_t* status,
                      uint32_t* hist, int passes, cudaStream_t s, uint32_t* clear0, size_t words0, uint32_t* clear1,
                      size_t words1) {
    constexpr uint32_t per_block = kBlock * kKeysPerThread;
    if (!n) return;
    const size_t clearing = std::min((words0 + words1) / (kBlock * kClearPerThread), kClearBlocks);
    const uint32_t blocks = std::max((n + per_block - 1) / per_block, (uint32_t)clearing);
    launch_pdl(cell_keys_kernel<Real>, blocks, kBlock, 0, s, pos, n, p, keys, status, hist, passes, clear0, words0, clear1,
               words1);
}
template <class Real>
void launch_reorder_fluid(const uint32_t* perm, const uint32_t* sorted_keys, uint32_t n, const Vec4<Real>* pos_in,
                          const Vec4<Real>* vel_in, const Real* kappa_in, const Real* kappaV_in, const uint32_t* id_in,
                          uint2* table, uint32_t* hist, DevState<Real>* d, const DevState<Real>& state, cudaStream_t s) {
    if (!n) return;
    const FluidArrays<Real> in{const_cast<Vec4<Real>*>(pos_in), const_cast<Vec4<Real>*>(vel_in), const_cast<Real*>(kappa_in),
                               const_cast<Real*>(kappaV_in), const_cast<uint32_t*>(id_in)};
    const FluidArrays<Real> out{state.pos, state.vel, state.kappa, state.kappaV, state.id};
    launch_pdl(reorder_fluid_kernel<Real>, grid_for(n), kBlock, 0, s, perm, sorted_keys, n, in, out, table, hist, d, state);
}
template <class Real>
void launch_reorder_pair(const uint32_t* perm, uint32_t n, const Real* a_in, const Real* b_in, Real* a_out,
                         Real* b_out, cudaStream_t s) {
    if (n) launch_pdl(reorder_pair_kernel<Real>, grid_for(n), kBlock, 0, s, perm, n, a_in, b_in, a_out, b_out);
}
void launch_boundary_cells(const uint32_t* sorted_keys, uint32_t nb, int dim_x, int dim_y, int dim_z, uint2* table,
                           uint8_t* near_boundary, uint32_t* hist, cudaStream_t s) {
    if (nb)
        launch_pdl(boundary_cells_kernel, grid_for(nb), kBlock, 0, s, sorted_keys, nb, dim_x, dim_y, dim_z, table,
                   near_boundary, hist);
}
template <class Real>
void launch_build_neighbors(const DevState<Real>* d, uint32_t n, const uint2* fluid_table, const uint2* boundary_table,
                            const uint8_t* near_boundary, cudaStream_t s, bool boundary_shifted) {
    if (!n) return;
    launch_pdl(boundary_shifted ? build_neighbors_kernel<Real, true> : build_neighbors_kernel<Real, false>, grid_for(n),
               kBlock, 0, s, d, n, fluid_table, boundary_table, near_boundary);
}
void launch_validate_neighbors(uint32_t* counts, const uint4* nbr, uint32_t n, uint32_t n_boundary, uint32_t stride,
                               uint32_t cap, uint32_t* status, cudaStream_t s) {
#ifdef DFSPH_CHECKED
    if (n) launch_pdl(validate_neighbors_kernel, grid_for(n), kBlock, 0, s, counts, nbr, n, n_boundary, stride, cap, status);
#else
    (void)counts;
    (void)nbr;
    (void)n;
    (void)n_boundary;
    (void)stride;
    (void)cap;
    (void)status;
    (void)s;
#endif
}
void launch_corrupt_first_neighbor(uint4* nbr, const uint32_t* counts, uint32_t value, cudaStream_t s) {
#ifdef DFSPH_CHECKED
    corrupt_first_neighbor_kernel<<<1, 32, 0, s>>>(nbr, counts, value);
#else
    (void)nbr;
    (void)counts;
    (void)value;
    (void)s;
#endif
}
template <class Real>
void launch_boundary_psi(const Vec4<Real>* bpos_in, Vec4<Real>* bpos_out, uint32_t nb, const StepParams<Real>& p,
                         const uint2* boundary_table, uint32_t* status, cudaStream_t s) {
    if (nb) launch_pdl(boundary_psi_kernel<Real>, grid_for(nb), kBlock, 0, s, bpos_in, bpos_out, nb, p, boundary_table, status);
}
template <class Real>
void launch_scatter_by_id(const uint32_t* id, uint32_t n, const Real* src, int comps, int src_stride, Real* dst,
                          cudaStream_t s) {
    if (n) launch_pdl(scatter_by_id_kernel<Real>, grid_for(n), kBlock, 0, s, id, n, src, comps, src_stride, dst);
}

#define DFSPH_INSTANTIATE_NEIGHBORS(R)                                                                               \
    template void launch_cell_keys<R>(const Vec4<R>*, uint32_t, const StepParams<R>&, uint32_t*, uint32_t*,          \
                                      uint32_t*, int, cudaStream_t, uint32_t*, size_t, uint32_t*, size_t);           \
    template void launch_reorder_fluid<R>(const uint32_t*, const uint32_t*, uint32_t, const Vec4<R>*, const Vec4<R>*, \
                                          const R*, const R*, const uint32_t*, uint2*, uint32_t*, DevState<R>*,      \
                                          const DevState<R>&, cudaStream_t);                                         \
    template void launch_build_neighbors<R>(const DevState<R>*, uint32_t, const uint2*, const uint2*, const uint8_t*, \
                                            cudaStream_t, bool);                                                     \
    template void launch_reorder_pair<R>(const uint32_t*, uint32_t, const R*, const R*, R*, R*, cudaStream_t);       \
    template void launch_boundary_psi<R>(const Vec4<R>*, Vec4<R>*, uint32_t, const StepParams<R>&, const uint2*,     \
                                         uint32_t*, cudaStream_t);                                                   \
    template void launch_scatter_by_id<R>(const uint32_t*, uint32_t, const R*, int, int, R*, cudaStream_t);

DFSPH_INSTANTIATE_NEIGHBORS(float)
DFSPH_INSTANTIATE_NEIGHBORS(double)

}  // namespace dfsph
