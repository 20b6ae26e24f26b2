// Fixed-order accumulation for the reproducible mode.
//
// By default the gradient kernels add the source adjoint H1_adj_j and the force on the source atom with
// atomics, whose order varies from run to run (results agree to rounding only).  The reference instead
// walks a source-sorted schedule (source_offsets / source_edges, libsymmetrix/source/
// mace_kokkos_factorized_lifecycle.cpp:2133-2195) so that every sum has one order.  In the reproducible
// mode the gradient kernels leave one record per edge (source adjoint, directed force) and the kernels
// below sum the records over that same schedule: edges of a source in ascending edge index.  Two
// evaluations of the same input then give identical bits.
#pragma once

#include "common.cuh"

namespace sxb {

// H1_adj[node] = sum over the edges whose source is `node`, in schedule order, of the edge's record.
// One block per node, one thread per four floats of the row.  The block first compacts the node's schedule to the edges that
// left a record (those inside the cutoff), kScheduleChunk at a time, so that the sums read their records without a chain of
// three dependent loads in front of each: 64 -> 47 us at 1,080 atoms and 128 x 4 floats a row.
constexpr int kScheduleChunk = 128;
__global__ void __launch_bounds__(kScheduleChunk)
reduce_source_adjoint_kernel(int row_floats, const int* __restrict__ source_offsets, const int* __restrict__ source_edges,
                             const EdgeGeom* __restrict__ geom, float r_cut, const float* __restrict__ records,
                             float* __restrict__ H1_adj)
{
    __shared__ int edges[kScheduleChunk];
    __shared__ int warp_counts[kScheduleChunk / 32];
    const int node = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int end = source_offsets[node + 1];
    for (int q0 = 0; q0 < (row_floats >> 2); q0 += kScheduleChunk) {
        const int q = q0 + threadIdx.x;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = source_offsets[node]; k0 < end; k0 += kScheduleChunk) {
            const int e = k0 + static_cast<int>(threadIdx.x) < end ? source_edges[k0 + threadIdx.x] : -1;
            const bool active = e >= 0 && geom[e].r < r_cut;        // list-skin edges leave no record
            const unsigned mask = __ballot_sync(0xffffffffu, active);
            if (lane == 0) warp_counts[warp] = __popc(mask);
            __syncthreads();
            int slot = __popc(mask & ((1u << lane) - 1u)), count = 0;
#pragma unroll
            for (int w = 0; w < kScheduleChunk / 32; ++w) {
                if (w < warp) slot += warp_counts[w];
                count += warp_counts[w];
            }
            if (active) edges[slot] = e;
            __syncthreads();
            if (q < (row_floats >> 2)) {
#pragma unroll 8
                for (int k = 0; k < count; ++k) {
                    const float4 v = reinterpret_cast<const float4*>(records + static_cast<size_t>(edges[k]) * row_floats)[q];
                    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                }
            }
            __syncthreads();
        }
        if (q < (row_floats >> 2)) reinterpret_cast<float4*>(H1_adj + static_cast<size_t>(node) * row_floats)[q] = acc;
    }
}

// Sum over the warp by a fixed tree, the same on every run and in every lane.
__device__ __forceinline__ double warp_total(double v)
{
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) v += __shfl_xor_sync(0xffffffffu, v, offset);
    return v;
}

// Adds the lanes' force vectors to the warp's running sums: the n-th vector that is not zero goes to lane n % 32, whatever
// number of zero vectors (edges in the list's skin) lies between them.  `rank` counts them; `slots` is the warp's exchange area.
__device__ __forceinline__ void add_by_rank(const double (&f)[3], double (*__restrict__ slots)[3], int lane, int& rank, double (&sum)[3])
{
    const bool given = f[0] != 0.0 || f[1] != 0.0 || f[2] != 0.0;
    const unsigned mask = __ballot_sync(0xffffffffu, given);
    if (given)
#pragma unroll
        for (int q = 0; q < 3; ++q) slots[(rank + __popc(mask & ((1u << lane) - 1u))) & 31][q] = f[q];
    __syncwarp();
    if (((lane - rank) & 31) < __popc(mask))
#pragma unroll
        for (int q = 0; q < 3; ++q) sum[q] += slots[lane][q];
    __syncwarp();
    rank += __popc(mask);
}

// forces[node] = - sum over the node's own edges (it is their receiver) + sum over the edges it is the source of.  One warp
// per node: the edges of either list that carry a force are dealt to the lanes in ascending order, the lanes meet in a fixed
// tree.  (One thread per node left 1,080 atoms on nine blocks; this and the last stage below: 105 -> 33 us.)
constexpr int kNodeForceWarps = 4;
__global__ void __launch_bounds__(32 * kNodeForceWarps)
reduce_node_forces_kernel(int num_nodes, int num_receivers, const int* __restrict__ first, const int* __restrict__ source_offsets,
                          const int* __restrict__ source_edges, const double* __restrict__ edge_forces, double* __restrict__ forces)
{
    __shared__ double slots[kNodeForceWarps][32][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, node = blockIdx.x * kNodeForceWarps + warp;
    if (node >= num_nodes) return;
    double own[3] = {0.0, 0.0, 0.0}, f[3];
    int rank = 0;
    const int own_end = node < num_receivers ? first[node + 1] : 0;
    for (int e0 = node < num_receivers ? first[node] : 0; e0 < own_end; e0 += 32) {
#pragma unroll
        for (int q = 0; q < 3; ++q) f[q] = e0 + lane < own_end ? -edge_forces[3 * static_cast<size_t>(e0 + lane) + q] : 0.0;
        add_by_rank(f, slots[warp], lane, rank, own);
    }
    rank = 0;
    const int end = source_offsets[node + 1];
    for (int k0 = source_offsets[node]; k0 < end; k0 += 32) {
        const size_t e = k0 + lane < end ? source_edges[k0 + lane] : 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) f[q] = k0 + lane < end ? edge_forces[3 * e + q] : 0.0;
        add_by_rank(f, slots[warp], lane, rank, own);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double total = warp_total(own[q]);
        if (lane == 0) forces[3 * static_cast<size_t>(node) + q] = total;
    }
}

constexpr int kTotalsThreads = 256;

// Stage 1: block b sums f (x) xyz over its 256 edges and the node energies of its 256 receivers into
// partials[b][10] = [energy, virial 9]; the tree inside a block is the same on every run.
__global__ void __launch_bounds__(kTotalsThreads)
partial_totals_kernel(long num_edges, int num_receivers, const EdgeGeom* __restrict__ geom, const double* __restrict__ edge_forces,
                      const double* __restrict__ node_energies, double* __restrict__ partials)
{
    __shared__ double warp_sums[kTotalsThreads / 32][10];
    const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (idx < num_receivers) v[0] = node_energies[idx];
    if (idx < num_edges) {
        const EdgeGeom g = geom[idx];
        const double len = g.r;
        const double rx = len * g.ux, ry = len * g.uy, rz = len * g.uz;
        const double ex = edge_forces[3 * idx], ey = edge_forces[3 * idx + 1], ez = edge_forces[3 * idx + 2];
        v[1] = ex * rx; v[2] = ex * ry; v[3] = ex * rz;
        v[4] = ey * rx; v[5] = ey * ry; v[6] = ey * rz;
        v[7] = ez * rx; v[8] = ez * ry; v[9] = ez * rz;
    }
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1)
#pragma unroll
        for (int q = 0; q < 10; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], offset);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 10; ++q) warp_sums[warp][q] = v[q];
    __syncthreads();
    if (threadIdx.x < 10) {
        double s = 0.0;
        for (int w = 0; w < kTotalsThreads / 32; ++w) s += warp_sums[w][threadIdx.x];
        partials[static_cast<long>(blockIdx.x) * 10 + threadIdx.x] = s;
    }
}

// Stage 2: one warp per quantity adds the block partials, every lane each 32nd block in order, the lanes by a fixed tree; the
// result goes to slot 0 of the energy / virial slots (the other slots stay zero in this mode), which the closing kernel sums.
__global__ void __launch_bounds__(320) final_totals_kernel(int num_blocks, const double* __restrict__ partials,
                                                           double* __restrict__ energy_slots, double* __restrict__ virial_slots)
{
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
    for (int b = lane; b < num_blocks; b += 32) s += partials[static_cast<long>(b) * 10 + q];
    s = warp_total(s);
    if (lane != 0) return;
    if (q == 0) energy_slots[0] = s;
    else virial_slots[q - 1] = s;
}

__global__ void count_sources_kernel(long num_edges, const int* __restrict__ sources, int* __restrict__ counts)
{
    const long e = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e < num_edges) atomicAdd(counts + sources[e], 1);
}

__global__ void iota_kernel(long n, int* __restrict__ out)
{
    const long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[i] = static_cast<int>(i);
}

}  // namespace sxb
