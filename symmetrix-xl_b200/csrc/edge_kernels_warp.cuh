// Layer-0 edge kernels, warp-per-receiver form: one warp owns one receiver and every lane owns
// kVec consecutive channels (C = 32*kVec), so the channel-independent edge state read from shared
// memory, the gradient contraction and the 3-value force reduction are paid once per kVec channels,
// spline coefficients arrive as 128-bit loads, and a receiver needs no block-wide barrier at all.
// These kernels are bound by the load/store pipe (ncu: l1tex data-pipe wavefronts ~86 % of peak for
// the one-channel-per-thread form), which is what this layout relieves.
// Math and reference citations: see edge_kernels.cuh (layer 0 forward/reverse,
// libsymmetrix/source/mace.cpp:1356-1403 and 1486-1559).
#pragma once

#include <type_traits>

#include "edge_kernels_pairs.cuh"

namespace sxb {

constexpr int kWarpChunk = 32;        // edges staged per pass: one per lane
constexpr int kWarpsPerBlock = 4;

template <bool kGradient>
struct alignas(16) WarpChunk {
    float4 y[kWarpChunk][4];
    float4 gx[kGradient ? kWarpChunk : 1][4];
    float4 gy[kGradient ? kWarpChunk : 1][4];
    float4 gz[kGradient ? kWarpChunk : 1][4];
    float4 misc[kWarpChunk];      // x = spline offset, yzw = unit direction
    int2 index[kWarpChunk];       // x = coefficient base or -1, y = source
    float len[kGradient ? kWarpChunk : 1];
    float dens[kGradient ? kWarpChunk : 1];   // d/dr of the density spline (0 without density scaling)
    float force[kGradient ? kWarpChunk : 1][3];
};

template <bool kGradient>
__device__ __forceinline__ void fill_warp_chunk(WarpChunk<kGradient>& s, int lane, int begin, int count,
                                                const int* __restrict__ sources, const EdgeGeom* __restrict__ geom,
                                                const unsigned char* __restrict__ atype, int type_i, int num_active,
                                                const SplineGrid& grid, int functions,
                                                const float* __restrict__ density_table = nullptr, int density_types = 1)
{
    if (lane < count) {
        const int e = begin + lane;
        const EdgeGeom g = geom[e];
        const int j = sources[e];
        if (!(g.r < grid.r_cut)) {
            s.index[lane] = make_int2(-1, j);
        } else {
            int interval;
            float x;
            spline_point(grid, g.r, interval, x);
            const int pair = type_i * num_active + atype[j];
            s.index[lane] = make_int2((pair * grid.intervals + interval) * 4 * functions, j);
            s.misc[lane] = make_float4(x, g.ux, g.uy, g.uz);
            const float inv_r = 1.0f / g.r;
            if constexpr (kGradient) {
                harmonics16<true>(g.ux, g.uy, g.uz, inv_r, reinterpret_cast<float*>(s.y[lane]), reinterpret_cast<float*>(s.gx[lane]),
                                  reinterpret_cast<float*>(s.gy[lane]), reinterpret_cast<float*>(s.gz[lane]));
                s.len[lane] = g.r;
                s.dens[lane] = density_table != nullptr
                                   ? scalar_spline_derivative(density_table, (type_i * density_types + (density_types > 1 ? atype[j] : 0)) * grid.intervals + interval, x)
                                   : 0.0f;
            } else {
                harmonics16<false>(g.ux, g.uy, g.uz, inv_r, reinterpret_cast<float*>(s.y[lane]), nullptr, nullptr, nullptr);
            }
        }
    }
}

template <int kVec>
struct VecLoad;
template <>
struct VecLoad<1> {
    static __device__ __forceinline__ void load(const float* p, float* out) { out[0] = *p; }
    static __device__ __forceinline__ void store(float* p, const float* in) { *p = in[0]; }
};
template <>
struct VecLoad<2> {
    static __device__ __forceinline__ void load(const float* p, float* out)
    {
        const float2 v = *reinterpret_cast<const float2*>(p);
        out[0] = v.x; out[1] = v.y;
    }
    static __device__ __forceinline__ void store(float* p, const float* in) { *reinterpret_cast<float2*>(p) = make_float2(in[0], in[1]); }
};
template <>
struct VecLoad<4> {
    static __device__ __forceinline__ void load(const float* p, float* out)
    {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    }
    static __device__ __forceinline__ void store(float* p, const float* in)
    {
        *reinterpret_cast<float4*>(p) = make_float4(in[0], in[1], in[2], in[3]);
    }
};

// The same as channel pairs.
template <int kPairs>
struct PairLoad;
template <>
struct PairLoad<1> {
    static __device__ __forceinline__ void load(const float* p, f2* out) { out[0] = *reinterpret_cast<const f2*>(p); }
};
template <>
struct PairLoad<2> {
    static __device__ __forceinline__ void load(const float* p, f2* out)
    {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
        out[0] = v.x; out[1] = v.y;
    }
};

// ---------------------------------------------------------------------------------------------
template <int kVec>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
l0_forward_warp_kernel(int num_nodes, int node0, int parts, bool parts_by_active, const int* __restrict__ first,
                       const int* __restrict__ sources, const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype,
                       int num_active, SplineGrid grid, const float* __restrict__ table, float* __restrict__ A0,
                       const float* __restrict__ inv_scale)
{
    constexpr int C = 32 * kVec, F = 4 * C;
    __shared__ WarpChunk<false> chunks[kWarpsPerBlock];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // parts = 1: a warp per receiver; parts = kWarpsPerBlock: the block's warps share one receiver
    const int slot = blockIdx.x * kWarpsPerBlock + warp;
    const int local = slot / parts, part = slot % parts;    // receiver inside the tile
    if (local >= num_nodes) return;                         // whole blocks when parts > 1
    const int i = node0 + local;                            // graph-wide receiver index
    WarpChunk<false>& s = chunks[warp];
    const int k = lane * kVec;
    const int type_i = atype[i];
    const int2 range = parts_by_active && parts > 1 ? active_edge_part(first, geom, grid.r_cut, i, part, parts)
                                                    : edge_part(first, i, part, parts);
    const int begin = range.x, end = range.y;
    float acc[16][kVec];
#pragma unroll
    for (int lm = 0; lm < 16; ++lm)
#pragma unroll
        for (int v = 0; v < kVec; ++v) acc[lm][v] = 0.0f;
    for (int chunk = begin; chunk < end; chunk += kWarpChunk) {
        const int count = min(kWarpChunk, end - chunk);
        __syncwarp();
        fill_warp_chunk<false>(s, lane, chunk, count, sources, geom, atype, type_i, num_active, grid, F);
        __syncwarp();
        for (int t = 0; t < count; ++t) {
            const int base = s.index[t].x;
            if (base < 0) continue;
            const float x = s.misc[t].x, xx = x * x, xxx = xx * x;
            const float* c = table + base + k;
            float y[16];
            load16(s.y[t], y);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                float c0[kVec], c1[kVec], c2[kVec], c3[kVec];
                VecLoad<kVec>::load(c + l * C, c0);
                VecLoad<kVec>::load(c + F + l * C, c1);
                VecLoad<kVec>::load(c + 2 * F + l * C, c2);
                VecLoad<kVec>::load(c + 3 * F + l * C, c3);
#pragma unroll
                for (int v = 0; v < kVec; ++v) {
                    const float R = cubic(c0[v], c1[v], c2[v], c3[v], x, xx, xxx);
#pragma unroll
                    for (int lm = l * l; lm < (l + 1) * (l + 1); ++lm) acc[lm][v] = fmaf(R, y[lm], acc[lm][v]);
                }
            }
        }
    }
    if (parts > 1) {
        // every warp leaves its sums in shared memory; the warps of the receiver then add up a share of the rows each, in
        // part order
        extern __shared__ float part_rows[];                // [kWarpsPerBlock][16][C]
#pragma unroll
        for (int lm = 0; lm < 16; ++lm) VecLoad<kVec>::store(part_rows + (warp * 16 + lm) * C + k, acc[lm]);
        __syncthreads();
        const float scale = inv_scale != nullptr ? inv_scale[i] : 1.0f;
        const float* rows = part_rows + (warp - part) * 16 * C + k;
        for (int lm = part; lm < 16; lm += parts) {
            float sum[kVec], v[kVec];
            VecLoad<kVec>::load(rows + lm * C, sum);
            for (int r = 1; r < parts; ++r) {
                VecLoad<kVec>::load(rows + (r * 16 + lm) * C, v);
#pragma unroll
                for (int q = 0; q < kVec; ++q) sum[q] += v[q];
            }
#pragma unroll
            for (int q = 0; q < kVec; ++q) sum[q] *= scale;
            VecLoad<kVec>::store(A0 + (static_cast<size_t>(local) * 16 + lm) * C + k, sum);
        }
        return;
    }
    if (inv_scale != nullptr) {   // density scaling, mace.cpp:1562-1584
        const float scale = inv_scale[i];
#pragma unroll
        for (int lm = 0; lm < 16; ++lm)
#pragma unroll
            for (int v = 0; v < kVec; ++v) acc[lm][v] *= scale;
    }
    float* out = A0 + static_cast<size_t>(local) * 16 * C + k;
#pragma unroll
    for (int lm = 0; lm < 16; ++lm) VecLoad<kVec>::store(out + lm * C, acc[lm]);
}

// lane t finishes edge t of a chunk: directed force dE/d(xyz_ij) = -(sum), scatter and virial
template <typename Chunk>
__device__ __forceinline__ void finish_warp_chunk(const Chunk& s, int lane, int chunk, int count, float density_coef, const ForceOutputs& out,
                                                  double& rfx, double& rfy, double& rfz, double* vir)
{
    if (lane < count && s.index[lane].x >= 0) {
        const float4 u = s.misc[lane];
        const float dens = density_coef * s.dens[lane];   // dE/d(xyz) += (A_adj . A) / (1 + rho) * s'(r) * rhat
        const double ex = -static_cast<double>(s.force[lane][0] - dens * u.y);
        const double ey = -static_cast<double>(s.force[lane][1] - dens * u.z);
        const double ez = -static_cast<double>(s.force[lane][2] - dens * u.w);
        const int j = s.index[lane].y;
        if (out.atom_forces != nullptr) {
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(j), ex);
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(j) + 1, ey);
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(j) + 2, ez);
        }
        rfx -= ex; rfy -= ey; rfz -= ez;
        const double len = s.len[lane];
        const float4 m = s.misc[lane];
        const double rx = len * m.y, ry = len * m.z, rz = len * m.w;
        vir[0] += ex * rx; vir[1] += ex * ry; vir[2] += ex * rz;
        vir[3] += ey * rx; vir[4] += ey * ry; vir[5] += ey * rz;
        vir[6] += ez * rx; vir[7] += ez * ry; vir[8] += ez * rz;
        if (out.edge_forces != nullptr) {
            double* ef = out.edge_forces + 3 * static_cast<size_t>(chunk + lane);
            if (out.accumulate_edge) { ef[0] += ex; ef[1] += ey; ef[2] += ez; }
            else { ef[0] = ex; ef[1] = ey; ef[2] = ez; }
        }
    } else if (lane < count && out.edge_forces != nullptr && !out.accumulate_edge) {
        double* ef = out.edge_forces + 3 * static_cast<size_t>(chunk + lane);
        ef[0] = ef[1] = ef[2] = 0.0;
    }
}

// receiver total and virial: one reduction per receiver and part
__device__ __forceinline__ void finish_warp_receiver(int lane, int i, const ForceOutputs& out, double rfx, double rfy, double rfz, double* vir)
{
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        rfx += __shfl_xor_sync(0xffffffffu, rfx, offset);
        rfy += __shfl_xor_sync(0xffffffffu, rfy, offset);
        rfz += __shfl_xor_sync(0xffffffffu, rfz, offset);
#pragma unroll
        for (int q = 0; q < 9; ++q) vir[q] += __shfl_xor_sync(0xffffffffu, vir[q], offset);
    }
    if (lane == 0 && out.atom_forces != nullptr) {
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(i), rfx);
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(i) + 1, rfy);
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(i) + 2, rfz);
        const int slot = i % kVirialSlots;
#pragma unroll
        for (int q = 0; q < 9; ++q) atomicAdd(out.virial_slots + slot * 9 + q, vir[q]);
    }
}

// ---------------------------------------------------------------------------------------------
// Edge state of the gradient: harmonics as pairs (Y, Y) and gradients per component, the layout of edge_kernels_pairs.cuh.
struct alignas(16) WarpPairChunk {
    float2 y[kWarpChunk][kPairSlots];
    float g[kWarpChunk][kGradSlots];
    float4 misc[kWarpChunk];      // x = spline offset, yzw = unit direction
    int2 index[kWarpChunk];       // x = coefficient base or -1, y = source
    float len[kWarpChunk];
    float dens[kWarpChunk];       // d/dr of the density spline (0 without density scaling)
    float force[kWarpChunk][3];
};

// Layer-0 gradient, kVec channels per lane as kVec / 2 pairs in the packed instructions of sm_100a.  Waits on its coefficient
// rows (8 KB per edge from L2) at 2.8 warps per scheduler, 0.41 instructions per cycle.  One-float form / pairs, 128 channels:
// 5,000 receivers 286 / 243 us, 40 receivers 21 / 18 us.
template <int kVec>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
l0_reverse_pair_kernel(int num_nodes, int node0, int parts, const int* __restrict__ first, const int* __restrict__ sources,
                       const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype, int num_active,
                       SplineGrid grid, const float* __restrict__ table, const float* __restrict__ A0_adj, ForceOutputs out,
                       DensityScale density)
{
    constexpr int C = 32 * kVec, F = 4 * C, kPairs = kVec / 2;
    extern __shared__ float4 chunk_words[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * kWarpsPerBlock + warp;
    const int local = slot / parts;                         // receiver inside the tile
    if (local >= num_nodes) return;
    const int i = node0 + local;                            // graph-wide receiver index
    WarpPairChunk& s = reinterpret_cast<WarpPairChunk*>(chunk_words)[warp];
    const int k = lane * kVec;
    const int type_i = atype[i];
    const int2 range = edge_part(first, i, slot % parts, parts);
    const int begin = range.x, end = range.y;
    // with density scaling the stored adjoint refers to the scaled A0: dE/dA0_unscaled = adj / (1 + rho_i)
    const float scale = density.table != nullptr ? density.inv_scale[i] : 1.0f;
    const float density_coef = density.table != nullptr ? density.dot[i] * scale : 0.0f;
    f2 adj[16][kPairs];
    {
        const f2* in = reinterpret_cast<const f2*>(A0_adj + static_cast<size_t>(local) * 16 * C + k);
        const f2 both = f2_pack(scale, scale);
#pragma unroll
        for (int lm = 0; lm < 16; ++lm)
#pragma unroll
            for (int v = 0; v < kPairs; ++v) adj[lm][v] = f2_mul(in[lm * (C / 2) + v], both);
    }
    // per-lane partial sums over the edges this lane finishes (lane t owns edge t of every chunk)
    double rfx = 0.0, rfy = 0.0, rfz = 0.0;
    double vir[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int chunk = begin; chunk < end; chunk += kWarpChunk) {
        const int count = min(kWarpChunk, end - chunk);
        __syncwarp();
        if (lane < count) {
            const EdgeGeom g = geom[chunk + lane];
            const int j = sources[chunk + lane];
            int base = -1;
            if (g.r < grid.r_cut) {
                int interval;
                float x;
                spline_point(grid, g.r, interval, x);
                const int type_j = atype[j];
                base = ((type_i * num_active + type_j) * grid.intervals + interval) * 4 * F;
                s.misc[lane] = make_float4(x, g.ux, g.uy, g.uz);
                fill_pair_harmonics<true>(g, s.y[lane], s.g[lane]);
                s.len[lane] = g.r;
                s.dens[lane] = density.table != nullptr
                                   ? scalar_spline_derivative(density.table, (type_i * density.types + (density.types > 1 ? type_j : 0)) * grid.intervals + interval, x)
                                   : 0.0f;
            }
            s.index[lane] = make_int2(base, j);
        }
        __syncwarp();
        for (int t = 0; t < count; ++t) {
            const int base = s.index[t].x;
            if (base < 0) continue;
            const float4 m = s.misc[t];
            const float xx_ = m.x * m.x;
            const f2 x = f2_pack(m.x, m.x), xx = f2_pack(xx_, xx_), xxx = f2_pack(xx_ * m.x, xx_ * m.x);
            const f2 x2 = f2_add(x, x), xx3 = f2_pack(3.0f * xx_, 3.0f * xx_);
            const float* c = table + base + k;
            f2 radial = 0ull;
            float fx = 0.0f, fy = 0.0f, fz = 0.0f;
            // value and slope of the l-th radial function, and its share of the radial and the angular force
            auto one_l = [&](auto l_tag) {
                constexpr int l = decltype(l_tag)::value, n = 2 * l + 1;
                f2 c0[kPairs], c1[kPairs], c2[kPairs], c3[kPairs], y[n], ang[n];
                PairLoad<kPairs>::load(c + l * C, c0);
                PairLoad<kPairs>::load(c + F + l * C, c1);
                PairLoad<kPairs>::load(c + 2 * F + l * C, c2);
                PairLoad<kPairs>::load(c + 3 * F + l * C, c3);
                load_pair_harmonics<l>(s.y[t], y);
#pragma unroll
                for (int v = 0; v < kPairs; ++v) {
                    const f2 value = f2_fma(c3[v], xxx, f2_fma(c2[v], xx, f2_fma(c1[v], x, c0[v])));
                    const f2 slope = f2_fma(c3[v], xx3, f2_fma(c2[v], x2, c1[v]));
                    f2 ya = f2_mul(y[0], adj[l * l][v]);
#pragma unroll
                    for (int a = 1; a < n; ++a) ya = f2_fma(y[a], adj[l * l + a][v], ya);
                    radial = f2_fma(slope, ya, radial);
                    if constexpr (l > 0) {
#pragma unroll
                        for (int a = 0; a < n; ++a)
                            ang[a] = v == 0 ? f2_mul(value, adj[l * l + a][v]) : f2_fma(value, adj[l * l + a][v], ang[a]);
                    }
                }
                if constexpr (l > 0) add_angular_force<l>(s.g[t], ang, fx, fy, fz);
            };
            one_l(std::integral_constant<int, 0>{});
            one_l(std::integral_constant<int, 1>{});
            one_l(std::integral_constant<int, 2>{});
            one_l(std::integral_constant<int, 3>{});
            const float along = f2_sum(radial);
            const float total = warp_reduce3_transposed(fmaf(along, m.y, fx), fmaf(along, m.z, fy), fmaf(along, m.w, fz), lane);
            if ((lane & 7) == 0 && lane < 24) s.force[t][lane >> 3] = total;
        }
        __syncwarp();
        finish_warp_chunk(s, lane, chunk, count, density_coef, out, rfx, rfy, rfz, vir);
    }
    finish_warp_receiver(lane, i, out, rfx, rfy, rfz, vir);
}

// The same for 32 channels: one per lane, in single floats.
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
l0_reverse_warp_kernel(int num_nodes, int node0, int parts, const int* __restrict__ first, const int* __restrict__ sources,
                       const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype, int num_active,
                       SplineGrid grid, const float* __restrict__ table, const float* __restrict__ A0_adj, ForceOutputs out,
                       DensityScale density)
{
    constexpr int C = 32, F = 4 * C;
    __shared__ WarpChunk<true> chunks[kWarpsPerBlock];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * kWarpsPerBlock + warp;
    const int local = slot / parts;                         // receiver inside the tile
    if (local >= num_nodes) return;
    const int i = node0 + local;                            // graph-wide receiver index
    WarpChunk<true>& s = chunks[warp];
    const int type_i = atype[i];
    const int2 range = edge_part(first, i, slot % parts, parts);
    const int begin = range.x, end = range.y;
    float adj[16];
    {
        const float* in = A0_adj + static_cast<size_t>(local) * 16 * C + lane;
#pragma unroll
        for (int lm = 0; lm < 16; ++lm) adj[lm] = in[lm * C];
    }
    // with density scaling the stored adjoint refers to the scaled A0: dE/dA0_unscaled = adj / (1 + rho_i)
    float density_coef = 0.0f;
    if (density.table != nullptr) {
        const float scale = density.inv_scale[i];
        density_coef = density.dot[i] * scale;
#pragma unroll
        for (int lm = 0; lm < 16; ++lm) adj[lm] *= scale;
    }
    // per-lane partial sums over the edges this lane finishes (lane t owns edge t of every chunk)
    double rfx = 0.0, rfy = 0.0, rfz = 0.0;
    double vir[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int chunk = begin; chunk < end; chunk += kWarpChunk) {
        const int count = min(kWarpChunk, end - chunk);
        __syncwarp();
        fill_warp_chunk<true>(s, lane, chunk, count, sources, geom, atype, type_i, num_active, grid, F, density.table, density.types);
        __syncwarp();
        for (int t = 0; t < count; ++t) {
            const int base = s.index[t].x;
            if (base < 0) continue;
            const float4 m = s.misc[t];
            const float x = m.x, xx = x * x, xxx = xx * x, x2 = 2.0f * x, xx3 = 3.0f * xx;
            const float* c = table + base + lane;
            float y[16], ang[16];
            load16(s.y[t], y);
            float radial = 0.0f;
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const float c0 = c[l * C], c1 = c[F + l * C], c2 = c[2 * F + l * C], c3 = c[3 * F + l * C];
                const float R = cubic(c0, c1, c2, c3, x, xx, xxx), dR = cubic_derivative(c1, c2, c3, x2, xx3);
                float ya = 0.0f;
#pragma unroll
                for (int lm = l * l; lm < (l + 1) * (l + 1); ++lm) {
                    ya = fmaf(y[lm], adj[lm], ya);
                    ang[lm] = R * adj[lm];
                }
                radial = fmaf(dR, ya, radial);
            }
            float fx = radial * m.y, fy = radial * m.z, fz = radial * m.w;
            {
                float g[16];
                load16(s.gx[t], g);
#pragma unroll
                for (int q = 0; q < 16; ++q) fx = fmaf(ang[q], g[q], fx);
                load16(s.gy[t], g);
#pragma unroll
                for (int q = 0; q < 16; ++q) fy = fmaf(ang[q], g[q], fy);
                load16(s.gz[t], g);
#pragma unroll
                for (int q = 0; q < 16; ++q) fz = fmaf(ang[q], g[q], fz);
            }
            const float total = warp_reduce3_transposed(fx, fy, fz, lane);
            if ((lane & 7) == 0 && lane < 24) s.force[t][lane >> 3] = total;
        }
        __syncwarp();
        finish_warp_chunk(s, lane, chunk, count, density_coef, out, rfx, rfy, rfz, vir);
    }
    finish_warp_receiver(lane, i, out, rfx, rfy, rfz, vir);
}

}  // namespace sxb
