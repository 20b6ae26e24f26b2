// Layer 0 on the radial network's own functions.
//
// A radial function of a compact model is a linear map of the 64 outputs phi_h(r) of its network's last hidden layer, and a
// cubic spline is linear in its nodal values, so with the source's element factor and the receiver's mixing matrix folded in
// (G[type_i][type_j][l], 64 x C)
//     A0_i[lm] = sum_types B_i[type][lm] G[type_i][type][l],      B_i[type][lm][h] = sum_(j of type) phi_h(r_ij) Y_lm(r_ij)
// The edges then see 64 functions without an l instead of 4 C, 1 KB of coefficients per edge instead of 8 KB (C = 128), and the
// contraction with G is one linear per (type_i, l) on the tensor cores (K = 64 types).  The gradient runs the same linears
// backwards, Badj = A0_adj G^T, and f_ij = -sum_(lm, h) Badj_i[type_j][lm][h] (rhat phi_h' Y_lm + phi_h grad Y_lm).
// Reference statements of the same math: libsymmetrix/source/mace.cpp:1356-1403 and 1486-1559, compact_radial.cpp:291-366.
//
// 0e+1o, 5,000 atoms, three types, 128 channels, folded table / this (edges + linear): sums 172 / 42 + 43, gradient 243 / 105 + 48 us.
#pragma once

#include "edge_kernels_warp.cuh"

namespace sxb {

constexpr int kBasis = 64;          // functions: width of the network's last hidden layer
constexpr int kBasisRow = 64;       // float4 per table row [2][32 lanes]: (c0, c0', c1, c1') and (c2, c2', c3, c3') of functions 2 lane, 2 lane + 1

__device__ __forceinline__ float2 f2_unpack(f2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// The run of edges inside the cutoff that receiver i has from sources of `type`.
__device__ __forceinline__ int2 typed_run(const ActiveEdges& active, const int* __restrict__ first, int i, int type)
{
    const int* ends = active.ends + static_cast<size_t>(i) * active.types;
    return make_int2(type == 0 ? first[i] : ends[type - 1], ends[type]);
}

// Table row of an edge: unordered species pair of a model with a distance transform, one table otherwise.
__device__ __forceinline__ int basis_row(const SplineGrid& grid, float r, int type_i, int type_j, int pair_types, float& x)
{
    int interval, pair = 0;
    spline_point(grid, r, interval, x);
    if (pair_types > 1) {
        const int a = min(type_i, type_j), b = max(type_i, type_j);
        pair = a * (2 * pair_types - a - 1) / 2 + b;
    }
    return (pair * grid.intervals + interval) * kBasisRow;
}

// Sums.  A warp owns one (receiver, source type), whose active edges are one run of the receiver's list, and a lane two functions.
// Packed operands pair neighbouring components lm, so the harmonics are read from shared memory as they are.  Waits on its
// coefficient rows (0.40 instructions per cycle and scheduler); one-warp blocks, because runs differ in length: 54 -> 43 us.
struct alignas(16) MomentChunk {
    float4 y[32][5];      // 16 harmonics; the fifth word keeps the rows of neighbouring lanes on different banks
    float2 point[32];     // x = offset inside the spline interval, y = table row (int)
};

// B[local][lm][type * 64 + h]
__global__ void __launch_bounds__(32)
l0_moments_kernel(int node0, int types, const int* __restrict__ first, const EdgeGeom* __restrict__ geom,
                  const ActiveEdges active, int pair_types, SplineGrid grid, const float4* __restrict__ table, float* __restrict__ B, const float* __restrict__ inv_scale)
{
    __shared__ MomentChunk s;
    const int lane = threadIdx.x;
    const int local = blockIdx.x / types, type = blockIdx.x % types;
    const int i = node0 + local, type_i = active.atype[i];
    f2 acc[8][2];
#pragma unroll
    for (int p = 0; p < 8; ++p) acc[p][0] = acc[p][1] = 0ull;
    const float4* table_lane = table + lane;
    const int2 run = typed_run(active, first, i, type);
    for (int chunk = run.x; chunk < run.y; chunk += 32) {
        const int count = min(32, run.y - chunk);
        __syncwarp();
        if (lane < count) {
            const EdgeGeom g = geom[active.edges[chunk + lane]];
            float x;
            const int row = basis_row(grid, g.r, type_i, type, pair_types, x);
            s.point[lane] = make_float2(x, __int_as_float(row));
            harmonics16<false>(g.ux, g.uy, g.uz, 0.0f, reinterpret_cast<float*>(s.y[lane]), nullptr, nullptr, nullptr);
        }
        __syncwarp();
#pragma unroll 4
        for (int t = 0; t < count; ++t) {
            const float2 point = s.point[t];
            const ulonglong2* c = reinterpret_cast<const ulonglong2*>(table_lane + __float_as_int(point.y));
            const ulonglong2 c01 = c[0], c23 = c[32];
            const float xx_ = point.x * point.x, xxx_ = xx_ * point.x;
            const float2 value = f2_unpack(f2_fma(c23.y, f2_pack(xxx_, xxx_), f2_fma(c23.x, f2_pack(xx_, xx_), f2_fma(c01.y, f2_pack(point.x, point.x), c01.x))));
            const f2 v0 = f2_pack(value.x, value.x), v1 = f2_pack(value.y, value.y);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(&s.y[t][q]);
                acc[2 * q][0] = f2_fma(v0, y.x, acc[2 * q][0]);
                acc[2 * q][1] = f2_fma(v1, y.x, acc[2 * q][1]);
                acc[2 * q + 1][0] = f2_fma(v0, y.y, acc[2 * q + 1][0]);
                acc[2 * q + 1][1] = f2_fma(v1, y.y, acc[2 * q + 1][1]);
            }
        }
    }
    const float scale = inv_scale != nullptr ? inv_scale[i] : 1.0f;   // density scaling, mace.cpp:1562-1584, commutes with the linear
    const int width = kBasis * types;
    float2* out = reinterpret_cast<float2*>(B + static_cast<size_t>(local) * 16 * width + type * kBasis) + lane;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const float2 a = f2_unpack(acc[p][0]), b = f2_unpack(acc[p][1]);
        out[(2 * p) * (width / 2)] = make_float2(a.x * scale, b.x * scale);
        out[(2 * p + 1) * (width / 2)] = make_float2(a.y * scale, b.y * scale);
    }
}

// ---------------------------------------------------------------------------------------------
// Gradient.  For the edges of a run, F[e][lm] = sum_h phi_h(r_e) Badj[lm][h] and D[e][lm] with the slopes phi_h' are two small
// matrix products with the same right-hand side, 16 edges x 64 functions x 16 components: mma.sync in FP64, where every product of
// two floats is exact, the sums are rounded to float once.  (tcgen05 wants 128 rows and its operands written to shared or tensor
// memory first; here every lane computes the functions it feeds to the instruction, and Badj stays in its registers for the whole
// run.)  Three TF32 passes take 31 / 95 us at 1,080 / 5,000 receivers, this 31 / 105, but the TF32 unit truncates whenever it adds:
// sums of 64 products of random sign were off by 1.1e-7 (2-norm) and pulled towards zero by 5e-8, in FP32 by 7e-8 and nothing.
// The FP32 form, a warp carrying one edge and reducing over its lanes, took 172 instructions per edge and 130 us (5,000
// receivers).  A warp walks all runs of a receiver (few receivers: one run or part of one): a warp's chain of dependent loads,
// first the edges, then their coefficient rows, is what it waits for, 12 warps per SM; as warps of one run each 113 us (TF32).
//
// Fragments: lane = 4 g + t.  Rows g and g + 8 are edges; column t (t + 4) of step s is function 16 t + 2 s (16 t + 2 s + 1),
// so that a lane reads 16 consecutive adjoints of a component, and the table lists the functions in the order of the steps.
struct alignas(16) MomentGradChunk {
    float fd[32][40];     // F[16], D[16] per edge; rows of 40 words keep the pairs of four neighbouring rows on different banks
    float2 point[32];     // x = offset inside the spline interval, y = table row (int)
};

__device__ __forceinline__ void mma_f64(double (&d)[4], const double (&a)[4], double b0, double b1)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

__global__ void __launch_bounds__(32, 12)
l0_moments_reverse_kernel(int node0, int types, const int* __restrict__ first, const int* __restrict__ sources,
                          const EdgeGeom* __restrict__ geom, const ActiveEdges active, int pair_types, SplineGrid grid,
                          const float4* __restrict__ table, const float* __restrict__ Badj, ForceOutputs out, DensityScale density)
{
    __shared__ MomentGradChunk s;
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
    const int local = blockIdx.x, i = node0 + local, type_i = active.atype[i];
    // gridDim.y = 1: all runs of the receiver; otherwise part blockIdx.y / types of one run
    const bool whole = gridDim.y == 1;
    const int parts = whole ? 1 : gridDim.y / types, part = whole ? 0 : blockIdx.y / types;
    // with density scaling the stored adjoint refers to the scaled A0: dE/dA0_unscaled = adj / (1 + rho_i)
    const float scale = density.table != nullptr ? density.inv_scale[i] : 1.0f;
    const float density_coef = density.table != nullptr ? density.dot[i] * scale : 0.0f;
    double sums[kForceSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};   // receiver force, virial
    for (int type = whole ? 0 : blockIdx.y % types; type < types; type += whole ? 1 : types) {
        int2 run = typed_run(active, first, i, type);
        {   // this part, in whole steps of 16 edges
            const int steps = (run.y - run.x + 15) / 16, begin = run.x;
            run.x = begin + 16 * (steps * part / parts);
            run.y = min(run.y, begin + 16 * (steps * (part + 1) / parts));
        }
        if (run.x >= run.y) continue;
        double b[2][16];      // [components g, g + 8][function 16 t + j]
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float4* in = reinterpret_cast<const float4*>(Badj + (static_cast<size_t>(local) * 16 + 8 * n + g) * (kBasis * types) + type * kBasis + 16 * t);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float4 w = in[m];
                b[n][4 * m] = w.x * scale;
                b[n][4 * m + 1] = w.y * scale;
                b[n][4 * m + 2] = w.z * scale;
                b[n][4 * m + 3] = w.w * scale;
            }
        }
        for (int chunk = run.x; chunk < run.y; chunk += 32) {
            const int count = min(32, run.y - chunk);
            int e = 0, source = 0;
            EdgeGeom geo{};
            __syncwarp();
            if (lane < count) {
                e = active.edges[chunk + lane];
                geo = geom[e];
                source = sources[e];
                float x;
                const int row = basis_row(grid, geo.r, type_i, type, pair_types, x);
                s.point[lane] = make_float2(x, __int_as_float(row));
            }
            __syncwarp();
            for (int e0 = 0; e0 < count; e0 += 16) {
                const int row[2] = {min(e0 + g, count - 1), min(e0 + g + 8, count - 1)};
                const float4* c[2];
                float x[2], xx[2], xxx[2], xx3[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 point = s.point[row[r]];
                    c[r] = table + __float_as_int(point.y) + t;
                    x[r] = point.x;
                    xx[r] = x[r] * x[r];
                    xxx[r] = xx[r] * x[r];
                    xx3[r] = 3.0f * xx[r];
                }
                double F[2][4] = {}, D[2][4] = {};   // [components 0-7, 8-15]
#pragma unroll
                for (int step = 0; step < 8; ++step) {
                    double value[4], slope[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int r = q & 1;
                        const float4 w = c[r][4 * (2 * step + (q >> 1))];
                        value[q] = cubic(w.x, w.y, w.z, w.w, x[r], xx[r], xxx[r]);
                        slope[q] = cubic_derivative(w.y, w.z, w.w, 2.0f * x[r], xx3[r]);
                    }
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        mma_f64(F[n], value, b[n][2 * step], b[n][2 * step + 1]);
                        mma_f64(D[n], slope, b[n][2 * step], b[n][2 * step + 1]);
                    }
                }
                // a lane holds components 2 t, 2 t + 1 (+ 8) of its two edges
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (e0 + g + 8 * r >= count) continue;
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        float* o = s.fd[row[r]] + 8 * n + 2 * t;
                        *reinterpret_cast<float2*>(o) = make_float2(F[n][2 * r], F[n][2 * r + 1]);
                        *reinterpret_cast<float2*>(o + 16) = make_float2(D[n][2 * r], D[n][2 * r + 1]);
                    }
                }
            }
            __syncwarp();
            if (lane < count) {   // directed force dE/d(xyz_ij) = -(sum F grad Y + (sum D Y) rhat), scatter and virial
                float f[16], y[16], fx = 0.0f, fy = 0.0f, fz = 0.0f, along = 0.0f;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 w = *reinterpret_cast<const float4*>(s.fd[lane] + 4 * q);
                    f[4 * q] = w.x; f[4 * q + 1] = w.y; f[4 * q + 2] = w.z; f[4 * q + 3] = w.w;
                }
                add_gradient_force(f, geo.ux, geo.uy, geo.uz, geo.r, y, fx, fy, fz);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 w = *reinterpret_cast<const float4*>(s.fd[lane] + 16 + 4 * q);
                    along = fmaf(w.x, y[4 * q], fmaf(w.y, y[4 * q + 1], fmaf(w.z, y[4 * q + 2], fmaf(w.w, y[4 * q + 3], along))));
                }
                if (density.table != nullptr) {   // dE/d(xyz) += (A_adj . A) / (1 + rho) * s'(r) * rhat
                    int interval;
                    float x;
                    spline_point(grid, geo.r, interval, x);
                    along -= density_coef * scalar_spline_derivative(density.table, (type_i * density.types + (density.types > 1 ? type : 0)) * grid.intervals + interval, x);
                }
                const double ex = -static_cast<double>(fmaf(along, geo.ux, fx)), ey = -static_cast<double>(fmaf(along, geo.uy, fy)),
                             ez = -static_cast<double>(fmaf(along, geo.uz, fz));
                if (out.atom_forces != nullptr) {
                    atomicAdd(out.atom_forces + 3 * static_cast<size_t>(source), ex);
                    atomicAdd(out.atom_forces + 3 * static_cast<size_t>(source) + 1, ey);
                    atomicAdd(out.atom_forces + 3 * static_cast<size_t>(source) + 2, ez);
                }
                sums[0] -= ex; sums[1] -= ey; sums[2] -= ez;
                const double len = geo.r, rx = len * geo.ux, ry = len * geo.uy, rz = len * geo.uz;
                sums[3] += ex * rx; sums[4] += ex * ry; sums[5] += ex * rz;
                sums[6] += ey * rx; sums[7] += ey * ry; sums[8] += ey * rz;
                sums[9] += ez * rx; sums[10] += ez * ry; sums[11] += ez * rz;
                if (out.edge_forces != nullptr) {
                    double* ef = out.edge_forces + 3 * static_cast<size_t>(e);
                    if (out.accumulate_edge) { ef[0] += ex; ef[1] += ey; ef[2] += ez; }
                    else { ef[0] = ex; ef[1] = ey; ef[2] = ez; }
                }
            }
        }
    }
    if (out.atom_forces == nullptr) return;
    reduce_force_sums(sums, lane);
    if (lane & 7) return;
    double* target = lane == 0 ? out.atom_forces + 3 * static_cast<size_t>(i) : out.virial_slots + (i % kVirialSlots) * 9 + 3 * (lane / 8 - 1);
#pragma unroll
    for (int q = 0; q < 3; ++q) atomicAdd(target + q, sums[q]);
}

}  // namespace sxb
