// Layer-1 forward kernels for coupling structures whose row count does not fit one thread's
// registers (hidden irreps up to l = 2: 17 paths, 243 rows, 71 outputs).  The paths are split at
// generation time into sets with equal row counts; one kernel instance handles one set for all
// receivers: it evaluates only that set's radial functions, keeps only that set's row sums in
// registers and writes only the outputs that set feeds - every output component belongs to exactly
// one path, so the sets write disjoint parts of Phi1.
// Thread mapping, edge chunking and the math are those of edge_kernels.cuh (layer 1 forward,
// libsymmetrix/source/mace.cpp:2023-2083).  The cluster builds (kParts) index lme_of at run time in their store, which keeps it
// in local memory (48 to 160 bytes a thread); the three launches take 101 / 45 us at 1 / 8 parts for 40 receivers, 105 / 101 at
// 1 / 2 for 160.
#pragma once

#include "edge_kernels.cuh"

namespace sxb {

#define SXB_DEFINE_L1_SPLIT_KERNELS(NAME, G)                                                                         \
    template <int kC, bool kParts = false>                                                                           \
    __global__ void __launch_bounds__(kC)                                                                            \
    l1_forward_split_kernel_##NAME##_##G(int num_nodes, int node0, const int* __restrict__ first,                    \
                                         const int* __restrict__ sources, const EdgeGeom* __restrict__ geom,         \
                                         const unsigned char* __restrict__ atype, SplineGrid grid,                   \
                                         const float4* __restrict__ table4, const float* __restrict__ H1,            \
                                         const __grid_constant__ CouplingConstants cgc, float* __restrict__ Phi1,    \
                                         const float* __restrict__ inv_scale, int pair_types)                        \
    {                                                                                                                \
        constexpr int C = kC;                                                                                        \
        constexpr int NP = SXB_##NAME##_NUM_PATHS, NH = SXB_##NAME##_NUM_HIDDEN, NE = SXB_##NAME##_NUM_LME;          \
        constexpr int NPG = SXB_##NAME##_##G##_NUM_PATHS, NRG = SXB_##NAME##_##G##_NUM_ROWS;                         \
        constexpr int NEG = SXB_##NAME##_##G##_NUM_LME;                                                              \
        constexpr int path_of[NPG] = SXB_##NAME##_##G##_PATH_LIST;                                                   \
        constexpr int lme_of[NEG] = SXB_##NAME##_##G##_LME_LIST;                                                     \
        constexpr int F = NP * C;                                                                                    \
        __shared__ ChunkState<false> s;                                                                              \
        const int local = blockIdx.x, i = node0 + local;                                                             \
        const int k = threadIdx.x;                                                                                   \
        const int2 range = kParts ? edge_part(first, i, blockIdx.y, gridDim.y) : make_int2(first[i], first[i + 1]);  \
        const int begin = range.x, end = range.y;                                                                    \
        float acc[NRG];                                                                                              \
        _Pragma("unroll") for (int r_ = 0; r_ < NRG; ++r_) acc[r_] = 0.0f;                                           \
        for (int chunk = begin; chunk < end; chunk += kEdgeChunk) {                                                  \
            const int count = min(kEdgeChunk, end - chunk);                                                          \
            __syncthreads();                                                                                         \
            fill_chunk<false, false>(s, chunk, count, sources, geom, atype, atype[i], pair_types, grid, F);          \
            __syncthreads();                                                                                         \
            for (int t = 0; t < count; ++t) {                                                                        \
                const int2 id = s.index[t];                                                                          \
                if (id.x < 0) continue;                                                                              \
                const float x = s.misc[t].x, xx = x * x, xxx = xx * x;                                               \
                const float4* c4 = table4 + (id.x >> 2) + k;                                                         \
                float R[NPG];                                                                                        \
                _Pragma("unroll") for (int q = 0; q < NPG; ++q) {                                                    \
                    const float4 c = c4[path_of[q] * C];                                                             \
                    R[q] = cubic(c.x, c.y, c.z, c.w, x, xx, xxx);                                                    \
                }                                                                                                    \
                const float* hsrc = H1 + static_cast<size_t>(id.y) * NH * C + k;                                     \
                float h[NH];                                                                                         \
                _Pragma("unroll") for (int q = 0; q < NH; ++q)                                                       \
                    h[q] = ((SXB_##NAME##_##G##_SOURCE_MASK >> q) & 1u) ? hsrc[q * C] : 0.0f;                         \
                float y[16];                                                                                         \
                load16(s.y[t], y);                                                                                   \
                SXB_##NAME##_##G##_FORWARD_BODY                                                                      \
            }                                                                                                        \
        }                                                                                                            \
        float out_lme[NEG];                                                                                          \
        _Pragma("unroll") for (int q = 0; q < NEG; ++q) out_lme[q] = 0.0f;                                           \
        SXB_##NAME##_##G##_TERMS(SXB_TERM_FORWARD)                                                                   \
        const float scale = inv_scale != nullptr ? inv_scale[i] : 1.0f;                                              \
        float* out = Phi1 + static_cast<size_t>(local) * NE * C + k;                                                 \
        if constexpr (!kParts) {                                                                                     \
            _Pragma("unroll") for (int q = 0; q < NEG; ++q) out[lme_of[q] * C] = out_lme[q] * scale;                          \
        } else {                                                                                                     \
            extern __shared__ float part_rows[];                                                                     \
            _Pragma("unroll") for (int q = 0; q < NEG; ++q) part_rows[q * C + k] = out_lme[q];                        \
            cluster_sum_rows(part_rows, NEG, C, [&](int q, float sum) { out[lme_of[q] * C] = sum * scale; });                 \
        }                                                                                                            \
    }

SXB_DEFINE_L1_SPLIT_KERNELS(S2, G0)
SXB_DEFINE_L1_SPLIT_KERNELS(S2, G1)
SXB_DEFINE_L1_SPLIT_KERNELS(S2, G2)

}  // namespace sxb
