// Periodic cell-list neighbor graph on the device: receiver-major CSR whose per-receiver edge order
// is bin-stencil order (z outermost, x innermost), atoms of a bin in ascending index.  That is the
// order and the accepted edge set of the reference's builder
// (libsymmetrix/source/neighbor_graph_kokkos.cpp:39-405); the work split is different:
//   * atoms are put in bin order by one stable radix sort of (bin, atom) pairs, so bins need no
//     per-bin sort and the candidates of x-adjacent bins are contiguous in memory;
//   * one to eight warps own a receiver; for each (z, y) row of its share of the stencil a warp walks maximal runs of
//     x-adjacent bins that share a periodic image, 32 candidates at a time, and compacts the accepted
//     ones in order with a ballot and a prefix population count.
// The distance test is evaluated in double with round-to-nearest adds and multiplies that are never
// contracted into FMAs, in the operand order of the reference's expression, so that a pair at the
// cutoff is accepted or rejected exactly as an IEEE evaluation of that expression would.
#pragma once

#include "common.cuh"

namespace sxb {

struct CellGrid {
    int bins[3];
    int reach[3];
    int num_bins;
    double range[3];         // the cutoff in units of bins, a little more (see finish_cell_grid)
    double cutoff_squared;
};

// What a search starts from, in one launch instead of three fills and two copies: the cell pair in its place, empty bins, a clear
// status word.  For small graphs the launches and copies around the search cost more than the search: with this and the
// report below a list of 120 atoms takes 118 instead of 143 us, of 2,160 atoms 152 instead of 184.
struct CellPair {
    double cell[9], inverse[9];
};
__global__ void begin_search_kernel(CellPair pair, double* __restrict__ cell, double* __restrict__ inv_cell, int num_bins,
                                    int* __restrict__ bin_sizes, int items, long long* __restrict__ counts, int* __restrict__ status)
{
    const long k = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < 9) {
        cell[k] = pair.cell[k];
        inv_cell[k] = pair.inverse[k];
    }
    if (k <= num_bins) bin_sizes[k] = 0;
    if (k == 0) {
        counts[items] = 0;
        *status = 0;
    }
}

// The number of edges and the status word, written to the host through its mapping.
__global__ void report_search_kernel(const long long* __restrict__ total, const int* __restrict__ status, long long* __restrict__ host)
{
    host[0] = *total;
    host[1] = *status;
}

// Fractional coordinates wrapped into [0, 1), the wrap count per axis, the wrapped Cartesian position
// and the atom's bin; a non-finite coordinate raises bit 2 of the status word, one more than 2^31 - 1 cells
// away bit 5.
__global__ void wrap_and_bin_kernel(int n, CellGrid grid, const double* __restrict__ positions,
                                    const double* __restrict__ inv_cell, const double* __restrict__ cell,
                                    double* __restrict__ wrapped_pos, int* __restrict__ wrap_count,
                                    int* __restrict__ atom_bin, int* __restrict__ atom_index, int* __restrict__ bin_sizes,
                                    int* __restrict__ status)
{
    const int atom = blockIdx.x * blockDim.x + threadIdx.x;
    if (atom >= n) return;
    atom_index[atom] = atom;
    const double p[3] = {positions[3 * atom], positions[3 * atom + 1], positions[3 * atom + 2]};
    if (!isfinite(p[0]) || !isfinite(p[1]) || !isfinite(p[2])) {
        atomicOr(status, 4);
        atom_bin[atom] = 0;
        atomicAdd(bin_sizes, 1);
        for (int c = 0; c < 3; ++c) {
            wrapped_pos[3 * atom + c] = 0.0;
            wrap_count[3 * atom + c] = 0;
        }
        return;
    }
    double f[3];
    int b[3];
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        double s = __dmul_rn(p[0], inv_cell[axis]);
        s = __dadd_rn(s, __dmul_rn(p[1], inv_cell[3 + axis]));
        s = __dadd_rn(s, __dmul_rn(p[2], inv_cell[6 + axis]));
        if (!(fabs(s) < 2147483647.0)) {   // the count of cells does not fit an int (nor, below, a bin that is made from it)
            atomicOr(status, 32);
            s = 0.0;
        }
        const int w = static_cast<int>(floor(s));
        f[axis] = __dadd_rn(s, -static_cast<double>(w));
        wrap_count[3 * atom + axis] = w;
        b[axis] = min(grid.bins[axis] - 1, static_cast<int>(__dmul_rn(f[axis], static_cast<double>(grid.bins[axis]))));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double s = __dmul_rn(f[0], cell[c]);
        s = __dadd_rn(s, __dmul_rn(f[1], cell[3 + c]));
        s = __dadd_rn(s, __dmul_rn(f[2], cell[6 + c]));
        wrapped_pos[3 * atom + c] = s;
    }
    const int bin = (b[2] * grid.bins[1] + b[1]) * grid.bins[0] + b[0];
    atom_bin[atom] = bin;
    atomicAdd(bin_sizes + bin, 1);
}

// Wrapped positions gathered into bin order, so that a warp reads its candidates coalesced.
__global__ void gather_sorted_positions_kernel(int n, const int* __restrict__ sorted_atoms, const double* __restrict__ wrapped_pos,
                                               double* __restrict__ sorted_pos)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int atom = sorted_atoms[k];
    sorted_pos[3 * k] = wrapped_pos[3 * atom];
    sorted_pos[3 * k + 1] = wrapped_pos[3 * atom + 1];
    sorted_pos[3 * k + 2] = wrapped_pos[3 * atom + 2];
}

// Bin coordinate `raw` of an unbounded bin lattice folded into [0, extent): returns the folded
// coordinate and stores how many periods were removed (the periodic image of that bin).
__device__ __forceinline__ int fold_bin(int raw, int extent, int& image)
{
    image = raw >= 0 ? raw / extent : -((extent - 1 - raw) / extent);
    return raw - image * extent;
}

// First and last bin offset along an axis that can hold a neighbor: a bin whose gap to the receiver, in units of bins, is beyond
// `range` has none.  `inside` is where the receiver stands in its own bin, 0 to 1.
__device__ __forceinline__ void stencil_extent(double inside, double range, int reach, int& low, int& high)
{
    high = static_cast<int>(fmin(static_cast<double>(reach), floor(range + inside)));
    low = -static_cast<int>(fmin(static_cast<double>(reach), floor(range + 1.0 - inside)));
}

// kFill = false: counts[receiver * parts + part] = number of accepted candidates.
// kFill = true:  writes sources / shifts from offsets[receiver * parts + part] on, in candidate order.
// Both passes are serial chains of FP64 tests and ballots, 32 candidates a turn, so they are bound by the number of turns of a
// warp.  The reference's stencil reaches one bin further than a neighbor can stand; the bins out of the receiver's range are
// passed over (their candidates would all be rejected), and with few receivers the (z, y) rows are dealt to several warps.
// From host positions to a ready graph, whole stencil by one warp, then as it is: 120 atoms 253 -> 143 us, 2,160: 270 -> 184,
// 5,000: 373 -> 244, 20,480: 959 -> 485, 135,000: 4.55 -> 2.06 ms, with the copies around it as they were (6.5 A lists of about 99 neighbors; nodes sorted by a count).
template <bool kFill>
__global__ void __launch_bounds__(256)
receiver_edges_kernel(int num_receivers, int parts, CellGrid grid, const int* __restrict__ atom_bin, const int* __restrict__ bin_begin,
                      const int* __restrict__ sorted_atoms, const double* __restrict__ sorted_pos,
                      const double* __restrict__ wrapped_pos, const int* __restrict__ wrap_count,
                      const double* __restrict__ cell, const double* __restrict__ inv_cell, long long* __restrict__ counts,
                      const long long* __restrict__ offsets, int* __restrict__ sources, int* __restrict__ shifts)
{
    const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31u;
    const int receiver = item / parts, part = item - receiver * parts;
    if (receiver >= num_receivers) return;
    const int nx = grid.bins[0], ny = grid.bins[1], nz = grid.bins[2];
    const int home = atom_bin[receiver];
    const int hx = home % nx, hy = (home / nx) % ny, hz = home / (nx * ny);
    const double rx = wrapped_pos[3 * receiver], ry = wrapped_pos[3 * receiver + 1], rz = wrapped_pos[3 * receiver + 2];
    const int wrx = wrap_count[3 * receiver], wry = wrap_count[3 * receiver + 1], wrz = wrap_count[3 * receiver + 2];
    long long written = kFill ? offsets[item] : 0;

    int low[3], high[3];
    const int own[3] = {hx, hy, hz};
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        const double f = rx * inv_cell[axis] + ry * inv_cell[3 + axis] + rz * inv_cell[6 + axis];
        const double inside = fmin(1.0, fmax(0.0, f * grid.bins[axis] - own[axis]));
        stencil_extent(inside, grid.range[axis], grid.reach[axis], low[axis], high[axis]);
    }
    const int rows_y = high[1] - low[1] + 1;
    const long rows = static_cast<long>(rows_y) * (high[2] - low[2] + 1);
    const long row_begin = rows * part / parts, row_end = rows * (part + 1) / parts;
    for (long t = row_begin; t < row_end; ++t) {
        const int dz = low[2] + static_cast<int>(t / rows_y), dy = low[1] + static_cast<int>(t % rows_y);
        int iz, iy;
        const int bz = fold_bin(hz + dz, nz, iz), by = fold_bin(hy + dy, ny, iy);
        // image translation, one product per (axis, component); the sums below add them one at a time
        const double zx = __dmul_rn(static_cast<double>(iz), cell[6]), zy = __dmul_rn(static_cast<double>(iz), cell[7]),
                     zz = __dmul_rn(static_cast<double>(iz), cell[8]);
        const double yx = __dmul_rn(static_cast<double>(iy), cell[3]), yy = __dmul_rn(static_cast<double>(iy), cell[4]),
                     yz = __dmul_rn(static_cast<double>(iy), cell[5]);
        const int row = (bz * ny + by) * nx;
        int dx = low[0];
        while (dx <= high[0]) {
            int ix;
            const int bx = fold_bin(hx + dx, nx, ix);
            // bins bx .. bx+run-1 of this row share the image ix and are contiguous in bin order
            const int run = min(high[0] - dx + 1, nx - bx);
            const double xx = __dmul_rn(static_cast<double>(ix), cell[0]), xy = __dmul_rn(static_cast<double>(ix), cell[1]),
                         xz = __dmul_rn(static_cast<double>(ix), cell[2]);
            const bool home_image = ix == 0 && iy == 0 && iz == 0;
            const int first = bin_begin[row + bx], last = bin_begin[row + bx + run];
            for (int k0 = first; k0 < last; k0 += 32) {
                const int k = k0 + static_cast<int>(lane);
                bool accept = false;
                int source = -1;
                if (k < last) {
                    source = sorted_atoms[k];
                    double d = __dadd_rn(sorted_pos[3 * k], -rx);
                    d = __dadd_rn(__dadd_rn(__dadd_rn(d, xx), yx), zx);
                    double d2 = __dmul_rn(d, d);
                    d = __dadd_rn(sorted_pos[3 * k + 1], -ry);
                    d = __dadd_rn(__dadd_rn(__dadd_rn(d, xy), yy), zy);
                    d2 = __dadd_rn(d2, __dmul_rn(d, d));
                    d = __dadd_rn(sorted_pos[3 * k + 2], -rz);
                    d = __dadd_rn(__dadd_rn(__dadd_rn(d, xz), yz), zz);
                    d2 = __dadd_rn(d2, __dmul_rn(d, d));
                    accept = !(d2 > grid.cutoff_squared) && !(home_image && source == receiver);
                }
                const unsigned taken = __ballot_sync(0xffffffffu, accept);
                if constexpr (kFill) {
                    if (accept) {
                        const long long edge = written + __popc(taken & ((1u << lane) - 1u));
                        sources[edge] = source;
                        shifts[3 * edge] = ix - wrap_count[3 * source] + wrx;
                        shifts[3 * edge + 1] = iy - wrap_count[3 * source + 1] + wry;
                        shifts[3 * edge + 2] = iz - wrap_count[3 * source + 2] + wrz;
                    }
                }
                written += __popc(taken);
            }
            dx += run;
        }
    }
    if constexpr (!kFill) {
        if (lane == 0) counts[item] = written;
    }
}

// Re-expresses a CSR graph given in caller node order in the internal order (nodes grouped by
// element): receiver ``new`` is caller node ``original[new]``; its edge list keeps its order and
// its sources are renumbered.  ``edge_map[new_edge]`` = caller edge index.  With types > 1 the edges of a receiver are
// stably grouped by the active type of their source.
__global__ void permute_graph_kernel(int n, int types, const unsigned char* __restrict__ atype, const int* __restrict__ original,
                                     const int* __restrict__ internal_of,
                                     const int* __restrict__ old_first, const int* __restrict__ old_sources,
                                     const int* __restrict__ old_shifts, const int* __restrict__ new_first,
                                     int* __restrict__ new_sources, int* __restrict__ new_shifts, int* __restrict__ edge_map)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= n) return;
    const int old_node = original[warp];
    const int ob = old_first[old_node], count = old_first[old_node + 1] - ob;
    const int nb = new_first[warp];
    int written = 0;
    for (int a = 0; a < types; ++a)
        for (int t0 = 0; t0 < count; t0 += 32) {
            const int t = t0 + lane, source = t < count ? internal_of[old_sources[ob + t]] : -1;
            const bool take = source >= 0 && (types == 1 || atype[source] == a);
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int e = nb + written + __popc(mask & ((1u << lane) - 1u));
                new_sources[e] = source;
                edge_map[e] = ob + t;
                if (old_shifts != nullptr) {
                    const size_t to = 3 * static_cast<size_t>(e), from = 3 * static_cast<size_t>(ob + t);
                    new_shifts[to] = old_shifts[from];
                    new_shifts[to + 1] = old_shifts[from + 1];
                    new_shifts[to + 2] = old_shifts[from + 2];
                }
            }
            written += __popc(mask);
        }
}

__global__ void gather_counts_kernel(int n, const int* __restrict__ original, const int* __restrict__ old_first,
                                     int* __restrict__ new_counts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int o = original[i];
    new_counts[i] = old_first[o + 1] - old_first[o];
}

}  // namespace sxb
