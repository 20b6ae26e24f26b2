// Layer-1 gradient on channel pairs, the receiver's row adjoints in tensor memory.
//
// Per edge and channel the gradient multiplies every row adjoint of the receiver (76 rows with a coupling term for hidden 0e+1o,
// 187 for 0e+1o+2e) into two sums.  One channel per thread with the rows in registers is bound by issue and register ports.  On
// channel pairs, in the packed instructions of sm_100a, they don't fit the registers; in shared memory (two edges per read) they
// took a third of the wavefronts of a kernel that the shared-memory pipe bounded.  Tensor memory is read by a path of its own:
// every warp reaches the 32 lanes of its quarter, so the rows of its 64 channels lie there as pairs, two columns a row, shared by the
// warps of the same quarter, and come in batches of eight while the batch before is used.  The first batch of an edge is asked for
// along with its source row, not by the edge before: registers that a load has yet to fill are not carried round a loop, where a
// copy of them may be placed (5,000 atoms, asked for by the edge before / this: 128 channels 701 / 695 us, 64 channels 388 / 392,
// 0e+1o+2e 1,549 / 1,555).  Without the rows the registers suffice for 16 warps per SM at one edge each (0e+1o; 12 warps for
// 0e+1o+2e).  Rows in registers one channel a thread / pairs with rows in
// registers / rows in shared memory / this: 0e+1o, 5,000 atoms 1.00 / 0.94 / 0.90 / 0.70 ms; 0e+1o+2e, 20,000 atoms 10.5 / - / 8.9 / 6.6 ms.
// Now FMA pipe 56 %, data pipe of L1 59 %, issue 52 %.  Reading 16 columns takes a warp 83 cycles with 16 warps on it, 390 bytes a
// cycle and SM.  Other shapes measured: 16 channels x 4 edges a warp +13 % (every 32 bytes of another line cost a wavefront), L1
// prefetch of the next edge's coefficients +15 %.
// Rows without a coupling term are left out.  In the reproducible mode the same kernel leaves records: every sum belongs to one
// edge and has one order, whichever warp, chunk or part the edge falls to (1,080 receivers, register form / this: 293 / 180 us).
//
// Math and reference citations: see edge_kernels.cuh (layer 1 reverse).
#pragma once

#include "edge_kernels.cuh"
#include "part_rules.hpp"

namespace sxb {

constexpr int kPairStep = 32, kWarpChannels = 64;

__device__ __forceinline__ f2 f2_pack(float lo, float hi)
{
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
// adds a channel pair to a row of global memory
__device__ __forceinline__ void f2_red_split(float* address, f2 v)
{
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    atomicAdd(address, lo);
    atomicAdd(address + kPairStep, hi);
}

// leaves a channel pair in a row of global memory that is read once, by another kernel
__device__ __forceinline__ void f2_store_split(float* address, f2 v)
{
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    address[0] = lo;
    address[kPairStep] = hi;
}

// Harmonics in shared memory as pairs (Y, Y), each l starting on 16 bytes: l = 0 at 0, 1 at 2..4, 2 at 6..10, 3 at 12..18.
// Gradients (layer 0 only) as [component][x, y, z], each l starting on 16 bytes: l = 1 at 0, 2 at 12, 3 at 28.
constexpr int kPairSlots = 20, kGradSlots = 52;

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

// Writes the harmonics (and gradients) of an edge in that layout.
template <bool kGradient>
__device__ __forceinline__ void fill_pair_harmonics(const EdgeGeom& g, float2* __restrict__ y, float* __restrict__ grad)
{
    float Y[16], gX[16], gY[16], gZ[16];
    harmonics16<kGradient>(g.ux, g.uy, g.uz, kGradient ? 1.0f / g.r : 0.0f, Y, gX, gY, gZ);
#pragma unroll
    for (int lm = 0; lm < 16; ++lm) {
        const int l = lm < 1 ? 0 : lm < 4 ? 1 : lm < 9 ? 2 : 3, m = lm - l * l;
        y[(l == 0 ? 0 : l == 1 ? 2 : l == 2 ? 6 : 12) + m] = make_float2(Y[lm], Y[lm]);
        if (kGradient && l > 0) {
            float* o = grad + (l == 1 ? 0 : l == 2 ? 12 : 28) + 3 * m;
            o[0] = gX[lm]; o[1] = gY[lm]; o[2] = gZ[lm];
        }
    }
}

// Adds sum_lm F[lm] grad Y_lm of the edge along the unit vector u to f; y receives the harmonics.
__device__ __forceinline__ void add_gradient_force(const float (&F)[16], float ux, float uy, float uz, float length, float (&y)[16],
                                                   float& fx, float& fy, float& fz)
{
    float gx[16], gy[16], gz[16];
    harmonics16<true>(ux, uy, uz, 1.0f / length, y, gx, gy, gz);
#pragma unroll
    for (int lm = 1; lm < 16; ++lm) {
        fx = fmaf(F[lm], gx[lm], fx);
        fy = fmaf(F[lm], gy[lm], fy);
        fz = fmaf(F[lm], gz[lm], fz);
    }
}

constexpr int kForceSums = 12;   // receiver force, virial
// Sums over the warp by exchanges that halve what a lane keeps: 18 instead of 60.  Lanes 0, 8, 16 and 24 end with the totals of
// three values each, v[3 * lane / 8 ...), in v[0 .. 3).
__device__ __forceinline__ void reduce_force_sums(double (&v)[kForceSums], int lane)
{
    const bool upper = lane & 16, second = lane & 8;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const double keep = upper ? v[q + 6] : v[q], send = upper ? v[q] : v[q + 6];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double keep = second ? v[q + 3] : v[q], send = second ? v[q] : v[q + 3];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int offset = 4; offset > 0; offset >>= 1)
#pragma unroll
        for (int q = 0; q < 3; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], offset);
}

// The same for 16 floats; lane 2 n ends with the total of f[n], which is returned.
__device__ __forceinline__ float reduce16(float (&f)[16], int lane)
{
#pragma unroll
    for (int half = 8; half > 0; half >>= 1) {
        const bool upper = lane & (2 * half);
#pragma unroll
        for (int q = 0; q < half; ++q) {
            const float keep = upper ? f[q + half] : f[q], send = upper ? f[q] : f[q + half];
            f[q] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * half);
        }
    }
    return f[0] + __shfl_xor_sync(0xffffffffu, f[0], 1);
}

// State of a receiver's edges in shared memory.
constexpr int kPairChunk = 96;
struct alignas(16) ActiveChunk {
    float2 y[kPairChunk][kPairSlots];
    float4 misc[kPairChunk];      // x = offset inside the spline interval, yzw = unit direction
    int4 index[kPairChunk];       // x = first 16-byte word of (pair, interval) in the table, y = source, z = edge
    float2 len[kPairChunk];       // x = length, y = d/dr of the density spline (0 without density scaling)
};

// Fills the chunk with `count` edges of one receiver, one per thread, from its list of edges inside the cutoff.  `words` 16-byte
// words per (pair, interval) of the table.
__device__ __forceinline__ void fill_active_chunk(ActiveChunk& s, int thread, const int* __restrict__ edges, int count, const int* __restrict__ sources,
                                                  const EdgeGeom* __restrict__ geom, const unsigned char* __restrict__ atype, int type_i,
                                                  int pair_types, const SplineGrid& grid, int words, const float* __restrict__ density_table,
                                                  int density_types)
{
    if (thread >= count) return;
    const int slot = thread, e = edges[slot], j = sources[e];
    const EdgeGeom g = geom[e];
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
    fill_pair_harmonics<false>(g, s.y[slot], nullptr);
    s.len[slot] = make_float2(g.r, density_table != nullptr
        ? scalar_spline_derivative(density_table, (type_i * density_types + (density_types > 1 ? atype[j] : 0)) * grid.intervals + interval, x) : 0.0f);
}

// Sums over the channels of a group per edge: [0] the radial force, [lm] the adjoint of harmonic lm.  The rows of neighbouring
// edges start four banks apart.
template <int kGroups>
struct ChunkSums {
    float f[kPairChunk][16 * kGroups + 4];
};

// Finishes the chunk's edges, one per thread of the first three warps: forces from the channel sums, pushed to the source atom;
// leaves the receiver force and the virial of the chunk in totals[warp].  With records (reproducible mode) each edge's force goes
// to its place in out.edge_forces and nowhere else.
template <int kGroups, bool kRecords>
__device__ __forceinline__ void flush_active_chunk(const ActiveChunk& s, int count, const ChunkSums<kGroups>& sums, double (*__restrict__ totals)[kForceSums],
                                                   const ForceOutputs& out, float density_coef)
{
    const int t = threadIdx.x, lane = t & 31;
    if (t >= kPairChunk || (t & ~31) >= count) return;
    double v[kForceSums];
#pragma unroll
    for (int q = 0; q < kForceSums; ++q) v[q] = 0.0;
    if (t < count) {
        float F[16], y[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float4 w = *reinterpret_cast<const float4*>(sums.f[t] + 4 * q);
#pragma unroll
            for (int g = 1; g < kGroups; ++g) {
                const float4 more = *reinterpret_cast<const float4*>(sums.f[t] + 16 * g + 4 * q);
                w.x += more.x; w.y += more.y; w.z += more.z; w.w += more.w;
            }
            F[4 * q] = w.x; F[4 * q + 1] = w.y; F[4 * q + 2] = w.z; F[4 * q + 3] = w.w;
        }
        const float4 u = s.misc[t];
        const float2 len = s.len[t];
        const float along = F[0] - density_coef * len.y;   // density scaling: dE/d(xyz_ij) += (A_adj . A) / (1 + rho_i) * s'(r) * rhat
        float px = along * u.y, py = along * u.z, pz = along * u.w;
        add_gradient_force(F, u.y, u.z, u.w, len.x, y, px, py, pz);
        const double ex = -static_cast<double>(px), ey = -static_cast<double>(py), ez = -static_cast<double>(pz);
        const int4 id = s.index[t];
        if constexpr (!kRecords) {
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y), ex);
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y) + 1, ey);
            atomicAdd(out.atom_forces + 3 * static_cast<size_t>(id.y) + 2, ez);
        }
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
    if constexpr (kRecords) return;
    reduce_force_sums(v, lane);
    if ((lane & 7) == 0)
#pragma unroll
        for (int q = 0; q < 3; ++q) totals[t >> 5][3 * (lane >> 3) + q] += v[q];
}

// ---------------------------------------------------------------------------------------------
// Row adjoints in tensor memory, kRowBatch rows (16 columns of the 32 lanes of a warp's quarter) at a time.
constexpr int kRowBatch = 8;

__device__ __forceinline__ void load_row_batch(unsigned taddr, unsigned (&raw)[2 * kRowBatch])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(raw[0]), "=r"(raw[1]), "=r"(raw[2]), "=r"(raw[3]), "=r"(raw[4]), "=r"(raw[5]), "=r"(raw[6]), "=r"(raw[7]), "=r"(raw[8]),
          "=r"(raw[9]), "=r"(raw[10]), "=r"(raw[11]), "=r"(raw[12]), "=r"(raw[13]), "=r"(raw[14]), "=r"(raw[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void store_row_batch(unsigned taddr, const f2 (&rows)[kRowBatch])
{
    unsigned raw[2 * kRowBatch];
#pragma unroll
    for (int q = 0; q < kRowBatch; ++q) asm("mov.b64 {%0, %1}, %2;" : "=r"(raw[2 * q]), "=r"(raw[2 * q + 1]) : "l"(rows[q]));
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(raw[0]), "r"(raw[1]), "r"(raw[2]), "r"(raw[3]), "r"(raw[4]), "r"(raw[5]), "r"(raw[6]), "r"(raw[7]), "r"(raw[8]),
          "r"(raw[9]), "r"(raw[10]), "r"(raw[11]), "r"(raw[12]), "r"(raw[13]), "r"(raw[14]), "r"(raw[15])
        : "memory");
}
// The batch asked for has arrived: its rows as channel pairs.  The registers go through the wait, so that whatever reads them
// depends on it.
__device__ __forceinline__ void take_row_batch(unsigned (&raw)[2 * kRowBatch], f2 (&rows)[kRowBatch])
{
    asm volatile(
        "tcgen05.wait::ld.sync.aligned;"
        : "+r"(raw[0]), "+r"(raw[1]), "+r"(raw[2]), "+r"(raw[3]), "+r"(raw[4]), "+r"(raw[5]), "+r"(raw[6]), "+r"(raw[7]), "+r"(raw[8]),
          "+r"(raw[9]), "+r"(raw[10]), "+r"(raw[11]), "+r"(raw[12]), "+r"(raw[13]), "+r"(raw[14]), "+r"(raw[15])
        :: "memory");
#pragma unroll
    for (int q = 0; q < kRowBatch; ++q) asm("mov.b64 %0, {%1, %2};" : "=l"(rows[q]) : "r"(raw[2 * q]), "r"(raw[2 * q + 1]));
}

#define RADIAL(p)                                                                                                   \
    f2 R, dR;                                                                                                       \
    { const float4 lo = coef[(p) * kC], hi = coef[(p) * kC + kPairStep];                                            \
      const float x = m.x, xx = x * x, xxx = xx * x, x2 = x + x, xx3 = 3.0f * xx;                                   \
      R = f2_pack(cubic(lo.x, lo.y, lo.z, lo.w, x, xx, xxx), cubic(hi.x, hi.y, hi.z, hi.w, x, xx, xxx));            \
      dR = f2_pack(cubic_derivative(lo.y, lo.z, lo.w, x2, xx3), cubic_derivative(hi.y, hi.z, hi.w, x2, xx3)); }
#define DPHI(lme) f2_mul(f2_pack(in[(lme) * kC], in[(lme) * kC + kPairStep]), both)
#define TERM(slot, term, lme) v[slot] = f2_mul(f2_pack(cgc.cg[term], cgc.cg[term]), DPHI(lme));
#define TERM_ADD(slot, term, lme) v[slot] = f2_fma(f2_pack(cgc.cg[term], cgc.cg[term]), DPHI(lme), v[slot]);
#define STORE(batch) store_row_batch(row_column + 2 * kRowBatch * (batch), v);
/* takes batch b and asks for the next one; what has been asked for is taken before the edge ends, so that no outstanding load is
   carried round the loop */
#define ROWS(b)                                                                                                     \
    take_row_batch(raw, rows);                                                                                      \
    if constexpr ((b) + 1 < kBatches) load_row_batch(row_column + 2 * kRowBatch * ((b) + 1), raw);

// Shared memory of a block with `channels` channels: edge state and channel sums; totals and the kilobyte that the system keeps.
constexpr std::size_t pair_dynamic_bytes(int channels)
{
    return sizeof(ActiveChunk) + (channels == 128 ? sizeof(ChunkSums<2>) : sizeof(ChunkSums<1>));
}
constexpr std::size_t pair_block_bytes(int channels)
{
    return pair_dynamic_bytes(channels) + 3 * kForceSums * sizeof(double) + 1024;
}
constexpr std::size_t kSharedPerSM = 228 * 1024;

// warps of a block and columns of tensor memory it allocates: the SM's 512 columns hold the rows of two receivers (0e+1o) or one,
// the resident blocks that the part rule counts with (part_rules.hpp)
constexpr int kPairWarpsS1 = 8, kPairWarpsS2 = 12;
constexpr int kPairColumnsS1 = 256, kPairColumnsS2 = 512;
static_assert(2 * kRowBatch * SXB_S1_ROW_BATCHES <= kPairColumnsS1 && kPairBlocksS1 * kPairColumnsS1 <= 512, "tensor memory, 0e+1o");
static_assert(2 * kRowBatch * SXB_S2_ROW_BATCHES <= kPairColumnsS2 && kPairBlocksS2 * kPairColumnsS2 <= 512, "tensor memory, 0e+1o+2e");
static_assert(kPairBlocksS1 * pair_block_bytes(128) <= kSharedPerSM && kPairBlocksS2 * pair_block_bytes(128) <= kSharedPerSM, "shared memory");

#define SXB_DEFINE_L1_PAIR_KERNEL(NAME)                                                                                 \
template <int kC, bool kRecords = false>                                                                                \
__global__ void __launch_bounds__(32 * kPairWarps##NAME, kPairBlocks##NAME)                                             \
l1_reverse_pair_kernel_##NAME(int node0, const int* __restrict__ first, const int* __restrict__ sources,                \
                              const EdgeGeom* __restrict__ geom, const ActiveEdges active, SplineGrid grid,             \
                              const float4* __restrict__ table, const float* __restrict__ H1,                           \
                              const float* __restrict__ dPhi1, const __grid_constant__ CouplingConstants cgc,           \
                              float* __restrict__ H1_adj, ForceOutputs out, DensityScale density, int pair_types)       \
{                                                                                                                       \
    constexpr int NP = SXB_##NAME##_NUM_PATHS, NH = SXB_##NAME##_NUM_HIDDEN, NE = SXB_##NAME##_NUM_LME;                 \
    constexpr int kBatches = SXB_##NAME##_ROW_BATCHES, kGroups = kC / kWarpChannels, kTeams = kPairWarps##NAME / kGroups;\
    extern __shared__ float4 chunk_words[];                                                                             \
    ActiveChunk& s = *reinterpret_cast<ActiveChunk*>(chunk_words);                                                      \
    ChunkSums<kGroups>& channel_sums = *reinterpret_cast<ChunkSums<kGroups>*>(&s + 1);                                  \
    __shared__ double totals[3][kForceSums];                                                                            \
    __shared__ unsigned tmem_slot;                                                                                      \
    const int local = blockIdx.x, i = node0 + local;                                                                    \
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp % kGroups, team = warp / kGroups;          \
    const int k = kWarpChannels * group + lane;                                                                         \
    const int type_i = active.atype[i];                                                                                 \
    const int list_begin = first[i], listed = active.ends[static_cast<size_t>(i + 1) * active.types - 1] - list_begin;  \
    const int begin = list_begin + static_cast<int>(static_cast<long>(listed) * blockIdx.y / gridDim.y);                \
    const int total = list_begin + static_cast<int>(static_cast<long>(listed) * (blockIdx.y + 1) / gridDim.y) - begin;  \
    if (total == 0) return;                                                                                             \
    if (threadIdx.x < 3 * kForceSums) totals[threadIdx.x / kForceSums][threadIdx.x % kForceSums] = 0.0;                 \
    /* with density scaling dPhi1 holds the adjoint of the scaled Phi1: divide by 1 + rho_i once more */                \
    const float scale = density.table != nullptr ? density.inv_scale[i] : 1.0f;                                         \
    const float density_coef = density.table != nullptr ? density.dot[i] * scale : 0.0f;                                \
    /* as few chunks as hold the edges, of about equal length */                                                        \
    const int chunks = (total + kPairChunk - 1) / kPairChunk, length = (total + chunks - 1) / chunks;                   \
    if (warp == 0) {                                                                                                    \
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"                                \
                     ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(&tmem_slot))), "r"(static_cast<unsigned>(kPairColumns##NAME)) : "memory");\
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");                        \
    }                                                                                                                   \
    /* the first chunk's edge state by the last warps, while the first four write the row adjoints */                   \
    fill_active_chunk(s, 32 * kPairWarps##NAME - 1 - threadIdx.x, active.edges + begin, min(length, total), sources, geom, active.atype, type_i,\
                      pair_types, grid, NP * kC, density.table, density.types);                                         \
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");                                                    \
    __syncthreads();                                                                                                    \
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");                                                     \
    /* a warp reaches the 32 lanes of its quarter of the tensor memory: warps w, w + 4, ... share a copy of their channels' rows */\
    const unsigned row_column = tmem_slot + (static_cast<unsigned>((warp & 3) * 32) << 16);                             \
    if (warp < 4) {                                                                                                     \
        const float* in = dPhi1 + static_cast<size_t>(local) * NE * kC + k;                                             \
        const f2 both = f2_pack(scale, scale);                                                                          \
        f2 v[kRowBatch];                                                                                                \
        SXB_##NAME##_L1_ADJOINT_ROWS                                                                                    \
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");                                                    \
    }                                                                                                                   \
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");                                                    \
    __syncthreads();                                                                                                    \
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");                                                     \
    for (int chunk = 0; chunk < total; chunk += length) {                                                               \
        const int count = min(length, total - chunk);                                                                   \
        if (chunk > 0) {                                                                                                \
            __syncthreads();                                                                                            \
            fill_active_chunk(s, threadIdx.x, active.edges + begin + chunk, count, sources, geom, active.atype, type_i, pair_types, grid,\
                              NP * kC, density.table, density.types);                                                   \
            __syncthreads();                                                                                            \
        }                                                                                                               \
        for (int t = team; t < count; t += kTeams) {                                                                    \
            const int4 id = s.index[t];                                                                                 \
            const float2* yrow = s.y[t];                                                                                \
            float f[16];                                                                                                \
            unsigned raw[2 * kRowBatch];                                                                                \
            load_row_batch(row_column, raw);                                                                            \
            const float4 m = s.misc[t];                                                                                 \
            const float4* coef = table + id.x + k;                                                                      \
            const size_t source_row = static_cast<size_t>(id.y) * NH * kC + k;                                          \
            f2 h[NH], hadj[NH], radial, rows[kRowBatch];                                                                \
            _Pragma("unroll") for (int b = 0; b < NH; ++b) h[b] = f2_pack(H1[source_row + b * kC], H1[source_row + b * kC + kPairStep]);\
            SXB_##NAME##_L1_REVERSE_EDGE_BODY                                                                           \
            /* kRecords: nothing is accumulated atomically; per-edge records are left for fixed-order passes */         \
            float* adjoint = kRecords ? out.edge_source_adjoint + static_cast<size_t>(id.z) * NH * kC + k : H1_adj + source_row;\
            _Pragma("unroll") for (int b = 0; b < NH; ++b) {                                                            \
                if constexpr (kRecords) f2_store_split(adjoint + b * kC, hadj[b]);                                      \
                else f2_red_split(adjoint + b * kC, hadj[b]);                                                           \
            }                                                                                                           \
            f[0] = f2_sum(radial);                                                                                      \
            const float total_of = reduce16(f, lane);                                                                   \
            if ((lane & 1) == 0) channel_sums.f[t][16 * group + (lane >> 1)] = total_of;                                \
        }                                                                                                               \
        __syncthreads();                                                                                                \
        flush_active_chunk<kGroups, kRecords>(s, count, channel_sums, totals, out, density_coef);                       \
    }                                                                                                                   \
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");                                                    \
    __syncthreads();                                                                                                    \
    if (warp == 0)                                                                                                      \
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(static_cast<unsigned>(kPairColumns##NAME)) : "memory");\
    if (!kRecords && threadIdx.x < kForceSums) {                                                                        \
        const double sum = totals[0][threadIdx.x] + totals[1][threadIdx.x] + totals[2][threadIdx.x];                    \
        if (threadIdx.x < 3) atomicAdd(out.atom_forces + 3 * static_cast<size_t>(i) + threadIdx.x, sum);                \
        else atomicAdd(out.virial_slots + (i % kVirialSlots) * 9 + threadIdx.x - 3, sum);                               \
    }                                                                                                                   \
}

SXB_DEFINE_L1_PAIR_KERNEL(S1)
SXB_DEFINE_L1_PAIR_KERNEL(S2)

#undef RADIAL
#undef DPHI
#undef TERM
#undef TERM_ADD
#undef STORE
#undef ROWS

}  // namespace sxb
