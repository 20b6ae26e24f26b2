// Layer-1 gradient with the receiver's row adjoints in shared memory, on channel pairs.
//
// The one-channel-per-thread kernel of edge_kernels.cuh keeps the 88 row adjoints of a receiver in registers: three warps per
// scheduler, 456 instructions per (edge, warp), bound by issue and by the register ports of three-operand instructions.  Here
// the adjoints lie in shared memory (45 KB a receiver, 122 KB with 243 rows), a warp carries 64 channels as pairs in the
// packed instructions of sm_100a and kEdges edges of the receiver at a time, and every adjoint it reads feeds two operations
// per edge.  All paths of a structure fit one kernel, whatever their number of rows, so the source features, the edge state
// and the force reduction are paid once per edge instead of once per path set.  Rows without a coupling term are left out.
// Teams of kC / 64 warps share a receiver.  Register form / this, 128 channels: hidden 0e+1o, 5,000 atoms 1.003 / 0.898 ms;
// 0e+1o+2e, 20,000 atoms 10.47 (three launches) / 8.88 ms.  Other shapes (teams, blocks per SM, edges) against (2, 3, 2) for
// 0e+1o: (4, 2, 1) +7 %, (4, 1, 2) +16 %; against (6, 1, 1) for 0e+1o+2e: (4, 1, 2) 0 %, (8, 1, 1) +3 %.
// Now bound by the shared-memory data pipe (77 % of its wavefronts at twelve warps per SM).  The reproducible mode keeps the
// register form, which leaves its records faster (1,080 receivers: 0.295 against 0.469 ms).  Registers: 168 at 128 channels (24 bytes spilled),
// three blocks of four warps; at 64 channels the edge state, which does not shrink with the width, leaves room for four blocks
// of two warps, so a thread may have 248: 5,000 receivers 0.451 ms, with the 168 of six blocks that never fit 0.599 ms.
//
// Math and reference citations: see edge_kernels.cuh (layer 1 reverse).
#pragma once

#include "edge_kernels.cuh"

namespace sxb {

__device__ __forceinline__ f2 f2_pack(float lo, float hi)
{
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
// adds a channel pair to a row of global memory, 32 channels apart
__device__ __forceinline__ void f2_red_split(float* address, f2 v)
{
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    atomicAdd(address, lo);
    atomicAdd(address + 32, hi);
}

// Shared-memory edge state, active edges only.  Harmonics are stored as pairs (Y, Y), each l starting on 16 bytes: l = 0 at
// 0, 1 at 2..4, 2 at 6..10, 3 at 12..18.  Gradients lie as [component][x, y, z], each l starting on 16 bytes: l = 1 at 0, 2
// at 12, 3 at 28.
constexpr int kPairSlots = 20, kGradSlots = 52;
struct alignas(16) ActiveChunk {
    float2 y[kEdgeChunk][kPairSlots];
    float g[kEdgeChunk][kGradSlots];
    float4 misc[kEdgeChunk];      // x = offset inside the spline interval, yzw = unit direction
    int4 index[kEdgeChunk];       // x = first 16-byte word of (pair, interval) in the table, y = source, z = edge
    float2 len[kEdgeChunk];       // x = length, y = d/dr of the density spline (0 without density scaling)
    int count;
};

template <int kL>
__device__ __forceinline__ void load_pair_harmonics(const float2* __restrict__ row, f2* __restrict__ y)
{
    constexpr int offset = kL == 0 ? 0 : kL == 1 ? 2 : kL == 2 ? 6 : 12;
    const f2* p = reinterpret_cast<const f2*>(row) + offset;
#pragma unroll
    for (int a = 0; a + 1 < 2 * kL + 1; a += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + a);
        y[a] = v.x;
        y[a + 1] = v.y;
    }
    y[2 * kL] = p[2 * kL];
}

// f += sum over the components of l of ang * grad Y, both channels
template <int kL>
__device__ __forceinline__ void add_angular_force(const float* __restrict__ row, const f2* __restrict__ ang, float& fx, float& fy, float& fz)
{
    constexpr int offset = kL == 1 ? 0 : kL == 2 ? 12 : 28, n = 2 * kL + 1;
    float g[(3 * n + 3) / 4 * 4];
#pragma unroll
    for (int q = 0; q < (3 * n + 3) / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(row + offset + 4 * q);
        g[4 * q] = v.x; g[4 * q + 1] = v.y; g[4 * q + 2] = v.z; g[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int a = 0; a < n; ++a) {
        const float s = f2_sum(ang[a]);
        fx = fmaf(s, g[3 * a], fx);
        fy = fmaf(s, g[3 * a + 1], fy);
        fz = fmaf(s, g[3 * a + 2], fz);
    }
}

// Writes the harmonics and gradients of an edge in that layout.
__device__ __forceinline__ void fill_pair_harmonics(const EdgeGeom& g, float2* __restrict__ y, float* __restrict__ grad)
{
    float Y[16], gX[16], gY[16], gZ[16];
    harmonics16<true>(g.ux, g.uy, g.uz, 1.0f / g.r, Y, gX, gY, gZ);
#pragma unroll
    for (int lm = 0; lm < 16; ++lm) {
        const int l = lm < 1 ? 0 : lm < 4 ? 1 : lm < 9 ? 2 : 3, m = lm - l * l;
        y[(l == 0 ? 0 : l == 1 ? 2 : l == 2 ? 6 : 12) + m] = make_float2(Y[lm], Y[lm]);
        if (l > 0) {
            float* o = grad + (l == 1 ? 0 : l == 2 ? 12 : 28) + 3 * m;
            o[0] = gX[lm]; o[1] = gY[lm]; o[2] = gZ[lm];
        }
    }
}

// Fills the chunk with the active ones of the edges [begin, begin + count) of one receiver, count <= 64: the first two
// warps, one edge per lane, in edge order.  `words` 16-byte words per (pair, interval) of the table.
__device__ __forceinline__ void fill_active_chunk(ActiveChunk& s, int begin, int count, const int* __restrict__ sources,
                                                  const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype, int type_i,
                                                  int pair_types, const SplineGrid& grid, int words, const float* __restrict__ density_table,
                                                  int density_types, const ForceOutputs& out)
{
    const int t = threadIdx.x, lane = t & 31;
    if (t >= 64) return;
    const int e = begin + t;
    EdgeGeom g;
    g.r = grid.r_cut;
    if (t < count) g = geom[e];
    const bool active = g.r < grid.r_cut;
    const unsigned mine = __ballot_sync(0xffffffffu, active);
    unsigned before = 0;    // the second warp looks at the first one's edges itself
    if (t >= 32) before = __ballot_sync(0xffffffffu, geom[begin + lane < begin + count ? begin + lane : begin].r < grid.r_cut && lane < count);
    const int slot = __popc(before) + __popc(mine & ((1u << lane) - 1u));
    if (t == 63) s.count = __popc(before) + __popc(mine);
    if (!active) {
        if (t < count && out.edge_forces != nullptr && !out.accumulate_edge) {
            double* ef = out.edge_forces + 3 * static_cast<size_t>(e);
            ef[0] = ef[1] = ef[2] = 0.0;
        }
        return;
    }
    const int j = sources[e];
    int interval;
    float x;
    spline_point(grid, g.r, interval, x);
    int pair = 0;
    if (pair_types > 1) {   // unordered species pair of a model with a distance transform
        const int type_j = atype[j], a = min(type_i, type_j), b = max(type_i, type_j);
        pair = a * (2 * pair_types - a - 1) / 2 + b;
    }
    s.index[slot] = make_int4((pair * grid.intervals + interval) * words, j, e, 0);
    s.misc[slot] = make_float4(x, g.ux, g.uy, g.uz);
    fill_pair_harmonics(g, s.y[slot], s.g[slot]);
    s.len[slot] = make_float2(g.r, density_table != nullptr
        ? scalar_spline_derivative(density_table, (type_i * density_types + (density_types > 1 ? atype[j] : 0)) * grid.intervals + interval, x) : 0.0f);
}

constexpr int kForceSums = 12;   // receiver force, virial
// Finishes the chunk's edges, one per thread of the first two warps: adds the channel groups' partial forces up, pushes the
// force to the source atom and leaves the receiver force and the virial of the chunk in sums[warp].
template <int kGroups>
__device__ __forceinline__ void flush_active_chunk(const ActiveChunk& s, const float (*__restrict__ partial)[kGroups][3], double (*__restrict__ sums)[kForceSums],
                                                   const ForceOutputs& out, float density_coef)
{
    const int t = threadIdx.x;
    if (t >= 64) return;
    double v[kForceSums];
#pragma unroll
    for (int q = 0; q < kForceSums; ++q) v[q] = 0.0;
    if (t < s.count) {
        float px = 0.0f, py = 0.0f, pz = 0.0f;
#pragma unroll
        for (int w = 0; w < kGroups; ++w) {
            px += partial[t][w][0];
            py += partial[t][w][1];
            pz += partial[t][w][2];
        }
        const float4 u = s.misc[t];
        const float2 len = s.len[t];
        const float d = density_coef * len.y;   // density scaling: dE/d(xyz_ij) += (A_adj . A) / (1 + rho_i) * s'(r) * rhat
        const double ex = -static_cast<double>(px - d * u.y), ey = -static_cast<double>(py - d * u.z), ez = -static_cast<double>(pz - d * u.w);
        const int4 id = s.index[t];
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y), ex);
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y) + 1, ey);
        atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y) + 2, ez);
        v[0] = -ex; v[1] = -ey; v[2] = -ez;
        const double rx = static_cast<double>(len.x) * u.y, ry = static_cast<double>(len.x) * u.z, rz = static_cast<double>(len.x) * u.w;
        v[3] = ex * rx; v[4] = ex * ry; v[5] = ex * rz;
        v[6] = ey * rx; v[7] = ey * ry; v[8] = ey * rz;
        v[9] = ez * rx; v[10] = ez * ry; v[11] = ez * rz;
        if (out.edge_forces != nullptr) {
            double* ef = out.edge_forces + 3 * static_cast<size_t>(id.z);
            if (out.accumulate_edge) { ef[0] += ex; ef[1] += ey; ef[2] += ez; }
            else { ef[0] = ex; ef[1] = ey; ef[2] = ez; }
        }
    }
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1)
#pragma unroll
        for (int q = 0; q < kForceSums; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], offset);
    if ((t & 31) == 0)
#pragma unroll
        for (int q = 0; q < kForceSums; ++q) sums[t >> 5][q] += v[q];
}

#define EACH(...) { constexpr int e = 0; __VA_ARGS__ } if constexpr (kEdges > 1) { constexpr int e = kEdges > 1 ? 1 : 0; __VA_ARGS__ }
#define ADJ(row) (*reinterpret_cast<const f2*>(adj + (row) * kC))
#define RADIAL(p)                                                                                                   \
    f2 R[kEdges], dR[kEdges];                                                                                       \
    EACH({ const float4 lo = coef[e][(p) * kC], hi = coef[e][(p) * kC + 32];                                        \
           const float x = m[e].x, xx = x * x, xxx = xx * x, x2 = x + x, xx3 = 3.0f * xx;                           \
           R[e] = f2_pack(cubic(lo.x, lo.y, lo.z, lo.w, x, xx, xxx), cubic(hi.x, hi.y, hi.z, hi.w, x, xx, xxx));    \
           dR[e] = f2_pack(cubic_derivative(lo.y, lo.z, lo.w, x2, xx3), cubic_derivative(hi.y, hi.z, hi.w, x2, xx3)); })

#define SXB_SHARED_TRANSPOSE(term, row, lme) if ((row) % kShares == share) rows[(row) * kC + column] += cgc.cg[term] * dphi[lme];

constexpr std::size_t shared_rows_bytes(int rows, int channels) { return static_cast<std::size_t>(rows) * channels * sizeof(float); }
// Shared memory of a block with `channels` channels: row adjoints, edge state, partial forces and sums, and the kilobyte that
// the system keeps.  The edge state is the same at every width, so halving the channels does not double the blocks per SM.
constexpr std::size_t shared_block_bytes(int rows, int channels)
{
    return shared_rows_bytes(rows, channels) + sizeof(ActiveChunk) + kEdgeChunk * (channels / 64) * 3 * sizeof(float)
           + 2 * kForceSums * sizeof(double) + 1024;
}
constexpr std::size_t kSharedPerSM = 228 * 1024;

// threads of a block per 64 channels, in warps, and resident blocks of an SM: what the launch bounds ask for and what the part
// rule counts with
constexpr int kSharedTeamsS1 = 2, kSharedTeamsS2 = 6;
template <int kC>
constexpr int kSharedBlocksS1 = kC == 128 ? 3 : 4;
template <int kC>
constexpr int kSharedBlocksS2 = 1;
static_assert(kSharedBlocksS1<128> * shared_block_bytes(SXB_S1_NUM_ROWS, 128) <= kSharedPerSM, "0e+1o, 128 channels");
static_assert(kSharedBlocksS1<64> * shared_block_bytes(SXB_S1_NUM_ROWS, 64) <= kSharedPerSM, "0e+1o, 64 channels");
static_assert(kSharedBlocksS2<128> * shared_block_bytes(SXB_S2_NUM_ROWS, 128) <= kSharedPerSM, "0e+1o+2e, 128 channels");

#define SXB_DEFINE_L1_SHARED_KERNEL(NAME, TEAMS, EDGES)                                                             \
template <int kC>                                                                                                   \
__global__ void __launch_bounds__(kC / 2 * TEAMS, kSharedBlocks##NAME<kC>)                                          \
l1_reverse_shared_kernel_##NAME(int node0, const int* __restrict__ first, const int* __restrict__ sources,          \
                                const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype, SplineGrid grid,\
                                const float4* __restrict__ table, const float* __restrict__ H1,                     \
                                const float* __restrict__ dPhi1, const __grid_constant__ CouplingConstants cgc,     \
                                float* __restrict__ H1_adj, ForceOutputs out, DensityScale density, int pair_types) \
{                                                                                                                   \
    constexpr int NP = SXB_##NAME##_NUM_PATHS, NR = SXB_##NAME##_NUM_ROWS, NH = SXB_##NAME##_NUM_HIDDEN;            \
    constexpr int NE = SXB_##NAME##_NUM_LME, kEdges = EDGES, kGroups = kC / 64;                                     \
    extern __shared__ float4 rows4[];                                                                               \
    float* const rows = reinterpret_cast<float*>(rows4);   /* [NR][kC] row adjoints */                              \
    __shared__ ActiveChunk s;                                                                                       \
    __shared__ float partial[kEdgeChunk][kGroups][3];                                                               \
    __shared__ double sums[2][kForceSums];                                                                          \
    const int local = blockIdx.x, i = node0 + local;                                                                \
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp % kGroups, team = warp / kGroups;      \
    const int k = 64 * group + lane;                                                                                \
    const int2 range = edge_part(first, i, blockIdx.y, gridDim.y);                                                  \
    const int type_i = atype[i];                                                                                    \
    if (threadIdx.x < 2 * kForceSums) sums[threadIdx.x / kForceSums][threadIdx.x % kForceSums] = 0.0;               \
    /* with density scaling dPhi1 holds the adjoint of the scaled Phi1: divide by 1 + rho_i once more */            \
    const float scale = density.table != nullptr ? density.inv_scale[i] : 1.0f;                                     \
    const float density_coef = density.table != nullptr ? density.dot[i] * scale : 0.0f;                            \
    {                                                                                                               \
        const int kk = threadIdx.x % kC, share = threadIdx.x / kC, column = (kk & ~63) + 2 * (kk & 31) + ((kk >> 5) & 1);\
        constexpr int kShares = TEAMS / 2;                                                                          \
        const float* in = dPhi1 + static_cast<size_t>(local) * NE * kC + kk;                                        \
        for (int q = share; q < NR; q += kShares) rows[q * kC + column] = 0.0f;                                     \
        float dphi[NE];                                                                                             \
        _Pragma("unroll") for (int q = 0; q < NE; ++q) dphi[q] = in[q * kC] * scale;                                \
        SXB_##NAME##_TERMS(SXB_SHARED_TRANSPOSE)                                                                    \
    }                                                                                                               \
    const float* adj = rows + k + lane;                                                                             \
    const float4* table_k = table + k;                                                                              \
    for (int chunk = range.x; chunk < range.y; chunk += kEdgeChunk) {                                               \
        __syncthreads();                                                                                            \
        fill_active_chunk(s, chunk, min(kEdgeChunk, range.y - chunk), sources, geom, atype, type_i, pair_types, grid, NP * kC,\
                          density.table, density.types, out);                                                       \
        __syncthreads();                                                                                            \
        const int count = s.count;                                                                                  \
        for (int t = kEdges * team; t < count; t += kEdges * TEAMS) {                                               \
            const int slot[2] = {t, min(t + 1, count - 1)};                                                         \
            const float2* yrow[kEdges]; const float* grow[kEdges]; float4 m[kEdges]; const float4* coef[kEdges];    \
            size_t source_row[kEdges];                                                                              \
            f2 h[kEdges][NH], hadj[kEdges][NH], radial[kEdges];                                                     \
            float fx[kEdges], fy[kEdges], fz[kEdges];                                                               \
            EACH({ const int4 id = s.index[slot[e]]; yrow[e] = s.y[slot[e]]; grow[e] = s.g[slot[e]]; m[e] = s.misc[slot[e]];\
                   coef[e] = table_k + id.x; source_row[e] = static_cast<size_t>(id.y) * NH * kC + k;               \
                   fx[e] = fy[e] = fz[e] = 0.0f; })                                                                 \
            EACH(_Pragma("unroll") for (int b = 0; b < NH; ++b) h[e][b] = f2_pack(H1[source_row[e] + b * kC], H1[source_row[e] + b * kC + 32]);)\
            SXB_##NAME##_L1_REVERSE_EDGES_BODY                                                                      \
            EACH(if (e == 0 || t + 1 < count) {                                                                     \
                _Pragma("unroll") for (int b = 0; b < NH; ++b) f2_red_split(H1_adj + source_row[e] + b * kC, hadj[e][b]);\
            })                                                                                                      \
            EACH({ const float along = f2_sum(radial[e]);                                                           \
                   const float total = warp_reduce3_transposed(fmaf(along, m[e].y, fx[e]), fmaf(along, m[e].z, fy[e]), fmaf(along, m[e].w, fz[e]), lane);\
                   if ((lane & 7) == 0 && lane < 24) partial[slot[e]][group][lane >> 3] = total; })                 \
        }                                                                                                           \
        __syncthreads();                                                                                            \
        flush_active_chunk<kGroups>(s, partial, sums, out, density_coef);                                           \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    if (threadIdx.x < kForceSums) {                                                                                 \
        const double total = sums[0][threadIdx.x] + sums[1][threadIdx.x];                                           \
        if (threadIdx.x < 3) atomicAdd(out.atom_forces + 3 * static_cast<size_t>(i) + threadIdx.x, total);          \
        else atomicAdd(out.virial_slots + (i % kVirialSlots) * 9 + threadIdx.x - 3, total);                         \
    }                                                                                                               \
}

SXB_DEFINE_L1_SHARED_KERNEL(S1, 2, 2)
SXB_DEFINE_L1_SHARED_KERNEL(S2, 6, 1)

#undef EACH
#undef ADJ
#undef RADIAL

}  // namespace sxb
