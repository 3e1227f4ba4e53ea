// Linked-cell full neighbour list build and layout kernels.
//
// Restates what the reference's Neighbor constructor obtains from
// Cabana::VerletList<FullNeighborTag, VerletLayout2D>
// (CabanaPD_Neighbor.hpp:44-66, 107-132): every particle is a candidate
// neighbour, rows exist for particles [begin, n), and j is a neighbour of i
// when |pos_j - pos_i|^2 <= cutoff^2. Compiled with --fmad=false so the
// squared distance rounds as a scalar evaluation does; the neighbour SET is
// therefore identical to the CPU oracle's.
//
// Steps: bounding box -> cell size (>= cutoff) -> cell index per particle ->
// counting sort into cells -> per-row count over the surrounding cells, with
// the longest row and the total -> per-row fill (in one pass with the count
// where an earlier build left a list to fill), rows sorted by ascending caller index (the
// order the oracle sums in) -> intact-bond bits.
#include <cub/cub.cuh>

#include <algorithm>
#include <climits>
#include <cstring>
#include <cmath>
#include <string>
#include <vector>

#include "cpd_internal.cuh"

namespace cpd {
namespace {

constexpr int kBlock = 256;
constexpr int kLocalRow = 256;  // rows up to this length are sorted in registers/local memory

inline int blocks_for(int64_t rows) { return (int)((rows + kBlock - 1) / kBlock); }

struct Grid {
    double lo[3];
    double cell;
    int32_t nc[3];
    int32_t R;  // visit radius in cells: every pair within the cutoff is at most R cells apart
};

// Bounding box of the positions x (+ disp, which are then written to y): a
// bounded grid (bbox_blocks) strides over the particles, so that few partials
// go to the host.
__global__ void __launch_bounds__(kBlock)
    k_bbox(const double* x, const double* disp, double* y, int64_t n, int64_t npad,
           double* partial)
{
    __shared__ double s[6][kBlock];
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        for (int d = 0; d < 3; d++) {
            double v = x[d * npad + i];
            if (disp) {
                v = v + disp[d * npad + i];
                y[d * npad + i] = v;
            }
            lo[d] = fmin(lo[d], v);
            hi[d] = fmax(hi[d], v);
        }
    for (int d = 0; d < 3; d++) {
        s[d][threadIdx.x] = lo[d];
        s[3 + d][threadIdx.x] = hi[d];
    }
    __syncthreads();
    for (int w = kBlock / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int d = 0; d < 3; d++) {
                s[d][threadIdx.x] = fmin(s[d][threadIdx.x], s[d][threadIdx.x + w]);
                s[3 + d][threadIdx.x] = fmax(s[3 + d][threadIdx.x], s[3 + d][threadIdx.x + w]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 6; c++) partial[6 * blockIdx.x + c] = s[c][0];
}

__device__ __forceinline__ void cell_coords(const Grid& g, double px, double py, double pz,
                                            int32_t c[3])
{
    const double p[3] = {px, py, pz};
    for (int d = 0; d < 3; d++) {
        double k = floor((p[d] - g.lo[d]) / g.cell);
        int32_t kk = (int32_t)fmax(0.0, fmin(k, (double)(g.nc[d] - 1)));
        c[d] = kk;
    }
}

__global__ void k_cell_index(const double* pos, int64_t n, int64_t npad, Grid g,
                             int32_t* cell, int32_t* cell_count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t c[3];
    cell_coords(g, pos[i], pos[npad + i], pos[2 * npad + i], c);
    const int32_t id = c[0] + g.nc[0] * (c[1] + g.nc[1] * c[2]);
    cell[i] = id;
    atomicAdd(cell_count + id, 1);
}

// The particles in cell order: their indices and, for the one-pass fill, their
// positions (one plane per component, so that the lanes of a warp, on
// neighbouring runs, read neighbouring values).
struct CellOrder {
    const double* pos;  // [3][n], or null
    const int32_t* index;
    int64_t n;
};
__global__ void __launch_bounds__(kBlock)
    k_cell_fill(const double* __restrict__ pos, int64_t npad, const int32_t* cell, int64_t n,
                const int32_t* cell_start, int32_t* cursor, double* sorted, int32_t* index)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t c = cell[i];
    const int32_t slot = cell_start[c] + atomicAdd(cursor + c, 1);
    if (sorted)
        for (int d = 0; d < 3; d++) sorted[d * n + slot] = pos[d * npad + i];
    index[slot] = (int32_t)i;
}

// Calls emit(j, dx, dy, dz) for every j != i within the cutoff: walks the
// (2R + 1)^2 lines of cells around particle i in increasing (z, y); the cells
// of one line are consecutive cell ids, so their particles are one contiguous
// run of the cell-sorted order. With cells about cutoff / 3 wide, a lattice
// holds about one particle per cell and an x-fastest lattice row is emitted
// in nearly ascending index order (the row sort then moves little).
// SORTED: candidates from the cell-sorted positions (co.pos), the index read of
// those within the cutoff only; otherwise through their index.
template <bool SORTED, typename Emit>
__device__ __forceinline__ void visit_neighbors(const double* __restrict__ pos, int64_t npad,
                                                const Grid& g, const int32_t* __restrict__ cell_start,
                                                const CellOrder& co, int64_t i,
                                                double rsqr, Emit&& emit)
{
    const double px = pos[i], py = pos[npad + i], pz = pos[2 * npad + i];
    int32_t c[3];
    cell_coords(g, px, py, pz, c);
    const int32_t cx0 = max(c[0] - g.R, 0), cx1 = min(c[0] + g.R, g.nc[0] - 1);
    for (int dz = -g.R; dz <= g.R; dz++) {
        const int32_t cz = c[2] + dz;
        if (cz < 0 || cz >= g.nc[2]) continue;
        for (int dy = -g.R; dy <= g.R; dy++) {
            const int32_t cy = c[1] + dy;
            if (cy < 0 || cy >= g.nc[1]) continue;
            const int64_t line = (int64_t)g.nc[0] * (cy + (int64_t)g.nc[1] * cz);
            const int32_t q1 = __ldg(cell_start + line + cx1 + 1);
            for (int32_t q = __ldg(cell_start + line + cx0); q < q1; q++) {
                int64_t j = i;
                if (!SORTED) {
                    j = __ldg(co.index + q);
                    if (j == i) continue;
                }
                const double ddx = (SORTED ? __ldg(co.pos + q) : pos[j]) - px;
                const double ddy = (SORTED ? __ldg(co.pos + co.n + q) : pos[npad + j]) - py;
                const double ddz =
                    (SORTED ? __ldg(co.pos + 2 * co.n + q) : pos[2 * npad + j]) - pz;
                const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
                if (!(d2 <= rsqr)) continue;
                if (SORTED) {
                    j = __ldg(co.index + q);
                    if (j == i) continue;
                }
                emit(j, ddx, ddy, ddz);
            }
        }
    }
}

// The longest of the calling block's rows and their sum into stats (one
// atomic each per warp with any row).
__device__ __forceinline__ void row_stats(int32_t cnt, unsigned long long* stats)
{
    const unsigned mx = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    const unsigned sum = __reduce_add_sync(0xffffffffu, (unsigned)cnt);
    if ((threadIdx.x & 31) == 0 && sum > 0) {
        atomicMax(stats, (unsigned long long)mx);
        atomicAdd(stats + 1, (unsigned long long)sum);
    }
}

// min_out (optional, 3 slots): per axis the smallest nonzero |x_j - x_i|
// over the accepted pairs (the bit patterns of non-negative doubles order
// like the values), the lattice spacing the mixed path's stencil needs.
// stats: [0] the longest row, [1] the sum of the row lengths.
template <bool SORTED>
__global__ void __launch_bounds__(kBlock)
    k_count(const double* pos, int64_t n, int64_t npad, int64_t begin, Grid g,
            const int32_t* cell_start, CellOrder co, double rsqr, int32_t* count,
            unsigned long long* min_out, unsigned long long* stats)
{
    __shared__ unsigned long long s_min[3][kBlock];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double m[3] = {INFINITY, INFINITY, INFINITY};
    int32_t cnt = 0;
    if (i < npad) {
        if (i >= begin && i < n)
            visit_neighbors<SORTED>(pos, npad, g, cell_start, co, i, rsqr,
                            [&](int64_t, double dx, double dy, double dz) {
                                cnt++;
                                if (min_out) {
                                    const double a0 = fabs(dx), a1 = fabs(dy), a2 = fabs(dz);
                                    if (a0 > 0.0) m[0] = fmin(m[0], a0);
                                    if (a1 > 0.0) m[1] = fmin(m[1], a1);
                                    if (a2 > 0.0) m[2] = fmin(m[2], a2);
                                }
                            });
        count[i] = cnt;
    }
    row_stats(cnt, stats);
    if (!min_out) return;  // uniform across the grid
    for (int d = 0; d < 3; ++d) s_min[d][threadIdx.x] = __double_as_longlong(m[d]);
    __syncthreads();
    for (int w = kBlock / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int d = 0; d < 3; ++d)
                s_min[d][threadIdx.x] = min(s_min[d][threadIdx.x], s_min[d][threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) atomicMin(min_out + d, s_min[d][0]);
}

// Count and fill in one pass into a list of `cap` columns that an earlier
// build left: rows of up to cap neighbours are complete and sorted by the
// neighbours' caller index (user_id, or the index itself); when the longest
// row (stats[0]) is longer, the caller takes k_fill on a longer list instead.
// Rows are sorted in place, so the list has at most kRefillRow columns. One
// walk over the cells instead of two: 0.47 ms for 4.0 M spheres with six
// contacts each, 0.78 + 0.72 ms by count and fill. Longer rows are k_fill's,
// which sorts them in local memory: per step with a rebuild, 100 thousand
// random points with rows of up to 23, 30, 46 and 78: 0.27, 0.36, 0.74 and 2.10
// ms in one pass, 0.26, 0.32, 0.52 and 1.02 by count and fill, in cells of the
// cutoff; 1.0 M points with rows of up to 24, 32 and 46: 1.25, 1.83 and 4.21
// against 1.56, 2.14 and 3.97.
constexpr int32_t kRefillRow = 32;
__global__ void __launch_bounds__(kBlock)
    k_refill(const double* pos, int64_t n, int64_t npad, int64_t begin, Grid g,
             const int32_t* cell_start, CellOrder co, double rsqr, int32_t* count,
             const int32_t* __restrict__ user_id, int32_t cap, int32_t* idx,
             unsigned long long* stats)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t cnt = 0;
    if (i < npad) {
        if (i >= begin && i < n) {
            visit_neighbors<true>(pos, npad, g, cell_start, co, i, rsqr,
                            [&](int64_t j, double, double, double) {
                                if (cnt < cap) {
                                    // Insert by key from the end of the row.
                                    const int32_t kv = user_id ? user_id[j] : (int32_t)j;
                                    int32_t b = cnt - 1;
                                    while (b >= 0) {
                                        const int32_t v = idx[(int64_t)b * npad + i];
                                        if ((user_id ? user_id[v] : v) <= kv) break;
                                        idx[(int64_t)(b + 1) * npad + i] = v;
                                        b--;
                                    }
                                    idx[(int64_t)(b + 1) * npad + i] = (int32_t)j;
                                }
                                cnt++;
                            });
            for (int32_t a = cnt; a < cap; a++) idx[(int64_t)a * npad + i] = (int32_t)i;
        }
        count[i] = cnt;
    }
    row_stats(cnt, stats);
}

// Fill row i and sort it by the caller index of the neighbour. Rows that fit
// kLocalRow are sorted in a thread-local array; longer rows are sorted in
// place in the column-major list.
template <bool SORTED>
__global__ void __launch_bounds__(kBlock)
    k_fill(const double* pos, int64_t n, int64_t npad, int64_t begin, Grid g,
           const int32_t* cell_start, CellOrder co, double rsqr,
           const int32_t* count, const int32_t* user_id, int32_t max_n, int32_t* idx)
{
    const int64_t i = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t cnt = count[i];
    auto key = [&](int32_t j) -> int32_t { return user_id ? user_id[j] : j; };
    if (cnt <= kLocalRow) {
        int32_t row[kLocalRow];
        int32_t k = 0;
        visit_neighbors<SORTED>(pos, npad, g, cell_start, co, i, rsqr,
                        [&](int64_t j, double, double, double) {
                            if (k < kLocalRow) row[k] = (int32_t)j;
                            k++;
                        });
        for (int32_t a = 1; a < cnt; a++) {
            const int32_t v = row[a];
            const int32_t kv = key(v);
            int32_t b = a - 1;
            while (b >= 0 && key(row[b]) > kv) {
                row[b + 1] = row[b];
                b--;
            }
            row[b + 1] = v;
        }
        for (int32_t a = 0; a < cnt; a++) idx[(int64_t)a * npad + i] = row[a];
    } else {
        int32_t k = 0;
        visit_neighbors<SORTED>(pos, npad, g, cell_start, co, i, rsqr,
                        [&](int64_t j, double, double, double) {
                            if (k < max_n) idx[(int64_t)k * npad + i] = (int32_t)j;
                            k++;
                        });
        for (int32_t a = 1; a < cnt; a++) {
            const int32_t v = idx[(int64_t)a * npad + i];
            const int32_t kv = key(v);
            int32_t b = a - 1;
            while (b >= 0 && key(idx[(int64_t)b * npad + i]) > kv) {
                idx[(int64_t)(b + 1) * npad + i] = idx[(int64_t)b * npad + i];
                b--;
            }
            idx[(int64_t)(b + 1) * npad + i] = v;
        }
    }
    for (int32_t a = cnt; a < max_n; a++) idx[(int64_t)a * npad + i] = (int32_t)i;
}

__global__ void k_init_mu(const int32_t* count, int64_t npad, int32_t nwords, uint32_t* mu)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npad) return;
    const int32_t cnt = count[i];
    for (int32_t w = 0; w < nwords; w++) {
        const int32_t left = cnt - 32 * w;
        uint32_t word = left >= 32 ? 0xffffffffu : (left <= 0 ? 0u : ((1u << left) - 1u));
        mu[(int64_t)w * npad + i] = word;
    }
}

__global__ void k_aos_to_soa(const double* aos, double* soa, int64_t n, int64_t npad,
                             int comps, const int32_t* perm)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t src = perm ? perm[k] : k;
    for (int d = 0; d < comps; d++) soa[d * npad + k] = aos[src * comps + d];
}

__global__ void k_fill_value(double* a, int64_t n, double v)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) a[k] = v;
}

// Caller-order int32 no-fail flags -> internal-order bytes.
__global__ void k_nofail_to_u8(const int32_t* src, uint8_t* dst, int64_t n, const int32_t* perm)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    dst[k] = src[perm ? perm[k] : k] != 0;
}

__global__ void k_soa_to_aos(const double* soa, double* aos, int64_t n, int64_t npad,
                             int comps, const int32_t* perm)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t dst = perm ? perm[k] : k;
    for (int d = 0; d < comps; d++) aos[dst * comps + d] = soa[d * npad + k];
}

// Row k of the internal list -> caller row perm[k], neighbour indices
// translated to caller indices (already in ascending caller order).
__global__ void k_ell_to_rows(const int32_t* count, const int32_t* idx, const uint32_t* mu,
                              int64_t n, int64_t npad, int32_t max_n, const int32_t* perm,
                              const int32_t* user_id, int32_t* out_counts, int32_t* out_idx,
                              int32_t* out_mu)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t row = perm ? perm[k] : k;
    const int32_t cnt = count[k];
    if (out_counts) out_counts[row] = cnt;
    for (int32_t a = 0; a < max_n; a++) {
        const bool valid = a < cnt;
        if (out_idx) {
            int32_t j = idx[(int64_t)a * npad + k];
            out_idx[row * max_n + a] = valid ? (user_id ? user_id[j] : j) : -1;
        }
        if (out_mu) {
            int32_t bit = 0;
            if (valid && mu) bit = (mu[(int64_t)(a >> 5) * npad + k] >> (a & 31)) & 1u;
            out_mu[row * max_n + a] = bit;
        }
    }
}

#define CPD_TRY(call)                                                           \
    do {                                                                        \
        cudaError_t e_ = (call);                                                \
        if (e_ != cudaSuccess) {                                                \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);           \
            return -1;                                                          \
        }                                                                       \
    } while (0)

}  // namespace

void free_neighbor_list(NeighborList& nl, cudaStream_t st)
{
    if (nl.count) dev_free(nl.count, st);
    if (nl.idx) dev_free(nl.idx, st);
    if (nl.mu) dev_free(nl.mu, st);
    nl = NeighborList{};
}

// Index delta from a row to its nearest neighbour straight along +y (same x
// and z within tol): the line pitch of an x-fastest lattice, used only to
// group bond-kernel warps (tile_view).
__global__ void k_row_pitch(const double* __restrict__ pos, int64_t npad, int64_t row,
                            const int32_t* __restrict__ count, const int32_t* __restrict__ idx,
                            double tol, long long* out)
{
    // One warp; ties go to the earliest neighbour of the row.
    const int lane = threadIdx.x;
    const int cnt = count[row];
    double best = INFINITY;
    long long d = 0;
    int at = INT_MAX;
    for (int k = lane; k < cnt; k += 32) {
        const int64_t j = idx[(int64_t)k * npad + row];
        const double dx = pos[j] - pos[row];
        const double dy = pos[npad + j] - pos[npad + row];
        const double dz = pos[2 * npad + j] - pos[2 * npad + row];
        if (fabs(dx) <= tol && fabs(dz) <= tol && dy > tol && dy < best) {
            best = dy;
            d = (long long)(j - row);
            at = k;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const long long od = __shfl_xor_sync(0xffffffffu, d, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (ob < best || (ob == best && oa < at)) {
            best = ob;
            d = od;
            at = oa;
        }
    }
    if (lane == 0) *out = d < 0 ? -d : d;
}

int build_neighbor_list(const double* x, const double* disp, int64_t n, int64_t npad,
                        int64_t begin, double cutoff, const int32_t* user_id,
                        bool with_mu, NeighborList& out, cudaStream_t st,
                        std::string& err, double* min_spacing)
{
    int launches = 0;
    PhaseTrace tr("list");
    const double* pos = x;
    double* y = nullptr;
    if (disp) {
        CPD_TRY(dev_alloc(&y, sizeof(double) * 3 * npad, st));
        pos = y;
    }
    // Bounding box (and the displaced positions).
    const int nb = std::min(blocks_for(n), 148 * 4);
    double* d_part = nullptr;
    CPD_TRY(dev_alloc(&d_part, sizeof(double) * 6 * nb, st));
    k_bbox<<<nb, kBlock, 0, st>>>(x, disp, y, n, npad, d_part);
    launches++;
    std::vector<double> part(6 * (size_t)nb);
    CPD_TRY(cudaMemcpyAsync(part.data(), d_part, sizeof(double) * 6 * nb,
                            cudaMemcpyDeviceToHost, st));
    CPD_TRY(cudaStreamSynchronize(st));
    CPD_TRY(dev_free(d_part, st));
    double lo[3], hi[3];
    for (int d = 0; d < 3; d++) {
        lo[d] = part[d];
        hi[d] = part[3 + d];
    }
    for (int b = 1; b < nb; b++)
        for (int d = 0; d < 3; d++) {
            lo[d] = std::min(lo[d], part[6 * b + d]);
            hi[d] = std::max(hi[d], part[6 * b + 3 + d]);
        }
    // A list of short rows that an earlier build left is filled as it is
    // counted.
    const bool refill = out.idx && out.cap > 0 && out.cap <= kRefillRow && !with_mu && !min_spacing;
    // Cells a little over a third of the cutoff wide (visit radius 3: 49 lines
    // of cells and 13 cutoffs cubed of candidates a row) where the grid then
    // holds few more cells than particles; else cells of the cutoff (9 lines,
    // 27 cutoffs cubed), or of 4/3, 8/3, ... of it. The 1e-9 margin keeps cutoff
    // / cell below the radius, so pairs within the cutoff are at most R cells
    // apart. (Cells of two thirds, which a grid too fine by up to eight times
    // would allow, mean 25 lines and 37 cutoffs cubed: 1.0 M random points with
    // mean rows of 24, count and fill, 5.0 ms against 4.0.)
    // The one-pass fill takes cells of the cutoff first: its walk is short of
    // loads in flight, and 9 lines are fewer dependent chains (1.0 M lattice
    // points, rows of 32: 2.23 vs 2.62 ms per step with a rebuild). Where even
    // those are too fine, either the rows are nearly empty (1.0 M points, mean
    // rows of 1: 0.51 ms in cells of 4/3, 0.82 of 2) or the box is: then most
    // lines of cells are looked up for nothing, and cells of 2 are faster (a
    // shell of 0.5 M points, mean rows of 1.7, 3.4 and 6.8: 1.18, 0.75 and 1.27
    // ms, 1.86, 1.09 and 1.94 in cells of 4/3). The earlier list's mean row
    // tells them apart.
    Grid g;
    auto fits = [&](double cell) {
        for (int d = 0; d < 3; d++) {
            double span = (hi[d] - lo[d]) / cell;
            g.nc[d] = (int32_t)std::max<int64_t>(1, std::min<int64_t>((int64_t)span + 1, 1 << 20));
        }
        return (double)g.nc[0] * g.nc[1] * g.nc[2] <= 4.0 * (double)n + 4096.0;
    };
    double cell = cutoff / 3.0 * (1.0 + 1e-9);
    bool whole = false;  // cells of the cutoff
    if (refill || !fits(cell)) {
        cell = cutoff * (1.0 + 1e-9);
        whole = fits(cell);
        if (!whole) {
            const bool hollow = refill && 2 * out.total >= 3 * (n - begin);
            for (cell *= hollow ? 2.0 : 4.0 / 3.0; !fits(cell);) cell *= 2.0;
        }
    }
    // The cell-sorted positions serve the one-pass fill and cells of the cutoff.
    // Elsewhere the walk is bound by how its lanes' candidates lie in memory, and
    // a lattice whose order is not x fastest has them side by side in its own
    // order and apart in the cells' (1.0 M points z fastest, rows of 32, cells of
    // a third: 2.6 ms per step with a rebuild, 3.6 with sorted positions).
    const bool by_cell = refill || whole;
    for (int d = 0; d < 3; d++) g.lo[d] = lo[d];
    g.cell = cell;
    g.R = std::max(1, (int32_t)std::ceil(cutoff / cell - 1e-9));
    const int64_t ncell = (int64_t)g.nc[0] * g.nc[1] * g.nc[2];

    int32_t *cellid = nullptr, *cell_count = nullptr, *cell_start = nullptr;
    int32_t* index = nullptr;
    double* sorted = nullptr;
    CPD_TRY(dev_alloc(&cellid, sizeof(int32_t) * n, st));
    CPD_TRY(dev_alloc(&cell_count, sizeof(int32_t) * (ncell + 1), st));
    CPD_TRY(dev_alloc(&cell_start, sizeof(int32_t) * (ncell + 1), st));
    CPD_TRY(dev_alloc(&index, sizeof(int32_t) * n, st));
    if (by_cell) CPD_TRY(dev_alloc(&sorted, sizeof(double) * 3 * n, st));
    CPD_TRY(cudaMemsetAsync(cell_count, 0, sizeof(int32_t) * (ncell + 1), st));
    k_cell_index<<<blocks_for(n), kBlock, 0, st>>>(pos, n, npad, g, cellid, cell_count);
    launches++;
    size_t tmp_bytes = 0;
    CPD_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cell_count, cell_start,
                                          (int)(ncell + 1), st));
    void* tmp = nullptr;
    CPD_TRY(dev_alloc(&tmp, tmp_bytes, st));
    CPD_TRY(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, cell_count, cell_start,
                                          (int)(ncell + 1), st));
    launches++;
    CPD_TRY(cudaMemsetAsync(cell_count, 0, sizeof(int32_t) * (ncell + 1), st));
    k_cell_fill<<<blocks_for(n), kBlock, 0, st>>>(pos, npad, cellid, n, cell_start, cell_count,
                                                  sorted, index);
    launches++;

    tr.mark("cells", st);
    // Row counts.
    if (!out.count) CPD_TRY(dev_alloc(&out.count, sizeof(int32_t) * npad, st));
    const double rsqr = cutoff * cutoff;
    const CellOrder co{sorted, index, n};
    // stats: the longest row and the rows' sum; then the smallest spacings.
    unsigned long long* d_stats = nullptr;
    CPD_TRY(dev_alloc(&d_stats, 5 * sizeof(unsigned long long), st));
    CPD_TRY(cudaMemsetAsync(d_stats, 0, 2 * sizeof(unsigned long long), st));
    CPD_TRY(cudaMemsetAsync(d_stats + 2, 0x7f, 3 * sizeof(unsigned long long), st));
    if (refill)
        k_refill<<<blocks_for(npad), kBlock, 0, st>>>(pos, n, npad, begin, g, cell_start, co,
                                                      rsqr, out.count, user_id, out.cap, out.idx,
                                                      d_stats);
    else
        (by_cell ? k_count<true> : k_count<false>)<<<blocks_for(npad), kBlock, 0, st>>>(
            pos, n, npad, begin, g, cell_start, co, rsqr, out.count,
            min_spacing ? d_stats + 2 : nullptr, d_stats);
    launches++;
    unsigned long long hstats[5];
    CPD_TRY(cudaMemcpyAsync(hstats, d_stats, sizeof(hstats), cudaMemcpyDeviceToHost, st));
    CPD_TRY(cudaStreamSynchronize(st));
    CPD_TRY(dev_free(d_stats, st));
    if (min_spacing)
        for (int d = 0; d < 3; ++d) std::memcpy(&min_spacing[d], &hstats[2 + d], sizeof(double));
    const int32_t max_n = (int32_t)hstats[0];
    const long long total = (long long)hstats[1];
    const bool filled = refill && max_n <= out.cap;
    tr.mark("count", st);
    // (Re)allocate the padded list when it grows.
    const int32_t cap = std::max(max_n, 1);
    if (!out.idx || cap > out.cap) {
        if (out.idx) CPD_TRY(dev_free(out.idx, st));
        out.idx = nullptr;
        CPD_TRY(dev_alloc(&out.idx, sizeof(int32_t) * (size_t)cap * npad, st));
        out.cap = cap;
        out.bytes = sizeof(int32_t) * (size_t)npad * (1 + (size_t)cap);
        if (with_mu) {
            if (out.mu) CPD_TRY(dev_free(out.mu, st));
            out.mu = nullptr;
            const int32_t nw = (cap + 31) / 32;
            CPD_TRY(dev_alloc(&out.mu, sizeof(uint32_t) * (size_t)nw * npad, st));
            out.bytes += sizeof(uint32_t) * (size_t)nw * npad;
        }
    }
    out.max_n = max_n;
    out.total = total;
    out.nwords = (max_n + 31) / 32;
    tr.mark("alloc", st);
    if (n > begin && !filled) {
        (by_cell ? k_fill<true> : k_fill<false>)<<<blocks_for(n - begin), kBlock, 0, st>>>(
            pos, n, npad, begin, g, cell_start, co, rsqr, out.count, user_id, max_n, out.idx);
        launches++;
    }
    if (with_mu && out.nwords > 0) {
        k_init_mu<<<blocks_for(npad), kBlock, 0, st>>>(out.count, npad, out.nwords, out.mu);
        launches++;
    }
    tr.mark("fill", st);
    // Lists on reference positions (PD bonds): the lattice line pitch at a
    // middle row.
    out.pitch = 0;
    if (!disp && n > begin && max_n > 0) {
        long long* d_pitch = nullptr;
        CPD_TRY(dev_alloc(&d_pitch, sizeof(long long), st));
        k_row_pitch<<<1, 32, 0, st>>>(pos, npad, begin + (n - begin) / 2, out.count, out.idx,
                                      1e-6 * cutoff, d_pitch);
        launches++;
        long long pitch = 0;
        CPD_TRY(cudaMemcpyAsync(&pitch, d_pitch, sizeof(pitch), cudaMemcpyDeviceToHost, st));
        CPD_TRY(cudaStreamSynchronize(st));
        CPD_TRY(dev_free(d_pitch, st));
        out.pitch = pitch;
    }
    CPD_TRY(cudaGetLastError());
    CPD_TRY(dev_free(tmp, st));
    CPD_TRY(dev_free(cellid, st));
    CPD_TRY(dev_free(cell_count, st));
    CPD_TRY(dev_free(cell_start, st));
    CPD_TRY(dev_free(index, st));
    if (sorted) CPD_TRY(dev_free(sorted, st));
    if (y) CPD_TRY(dev_free(y, st));
    return launches;
}

int launch_aos_to_soa(const double* aos, double* soa, int64_t n, int64_t npad, int comps,
                      const int32_t* perm, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_aos_to_soa<<<blocks_for(n), kBlock, 0, st>>>(aos, soa, n, npad, comps, perm);
    return 1;
}

int launch_fill_value(double* a, int64_t n, double v, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_fill_value<<<blocks_for(n), kBlock, 0, st>>>(a, n, v);
    return 1;
}

int launch_nofail_to_u8(const int32_t* src, uint8_t* dst, int64_t n, const int32_t* perm,
                        cudaStream_t st)
{
    if (n <= 0) return 0;
    k_nofail_to_u8<<<blocks_for(n), kBlock, 0, st>>>(src, dst, n, perm);
    return 1;
}

int launch_soa_to_aos(const double* soa, double* aos, int64_t n, int64_t npad, int comps,
                      const int32_t* perm, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_soa_to_aos<<<blocks_for(n), kBlock, 0, st>>>(soa, aos, n, npad, comps, perm);
    return 1;
}

int launch_ell_to_rows(const NeighborList& nl, int64_t n, int64_t npad, const int32_t* perm,
                       const int32_t* user_id, int32_t* counts, int32_t* indices,
                       int32_t* mu, cudaStream_t st)
{
    if (n <= 0) return 0;
    k_ell_to_rows<<<blocks_for(n), kBlock, 0, st>>>(nl.count, nl.idx, nl.mu, n, npad,
                                                     nl.max_n, perm, user_id, counts,
                                                     indices, mu);
    return 1;
}

}  // namespace cpd
