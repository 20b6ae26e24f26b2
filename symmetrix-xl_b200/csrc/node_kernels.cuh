// Node-local kernels of the force path: symmetric contraction (forward and gradient),
// channel-mixing linears, readout.  Reference statements: symmetric contraction
// libsymmetrix/source/mace.cpp:1639-1688 and 2461-2513 (polynomial
// multivariate_polynomial.cpp:322-353), linears mace.cpp:1691-1757, 2305-2378 and
// 2516-2588, readout mace.cpp:2622-2657 with the MLP of multilayer_perceptron.cpp:34-80.
#pragma once

#include <cstddef>

#include "common.cuh"
#include "row_map.hpp"
#include "generated/structures.h"

namespace sxb {

// ---------------------------------------------------------------------------------------------
// Symmetric contraction.  One thread per (node, two adjacent channels): the 16 inputs of the node sit in registers as
// channel pairs and the compiled structure is straight-line code on them (contraction_lines in gen_structures.py: monomials
// grouped by their first two factors).  Weights are laid out [element][term][channel].  A block covers consecutive nodes and
// 32 channels, half a warp per node; it first copies the [term][32] weight slice of its nodes' element to shared
// memory.  Bound by the FMA pipe in turn with the weight reads (gradient of M0: 0.42 instructions per cycle and scheduler, the
// math pipe its first stall).  5,000 nodes, 128 channels, hidden 0e+1o, one channel per thread with every monomial on
// its own / this form: M0 62 / 48, its gradient 118 / 62, M1 27 / 22, its gradient 36 / 27 us; 40 nodes: gradient of M0 27 / 15.

// Density-scaled models: dot[node] += sum over (lm, channels of this half warp) of A_adj * A, the quantity
// the reference forms per node before the density force (libsymmetrix/source/mace.cpp:1611-1614,
// 2430-2433).  Called by a whole warp; one atomic per half warp.
__device__ __forceinline__ void poly_accumulate_dot(const f2* g, const f2* x, float* __restrict__ dot, int node, bool valid)
{
    f2 both = 0ull;
#pragma unroll
    for (int q = 0; q < 16; ++q) both = f2_fma(g[q], x[q], both);
    float partial = f2_sum(both);
#pragma unroll
    for (int offset = 8; offset > 0; offset >>= 1) partial += __shfl_xor_sync(0xffffffffu, partial, offset);
    if ((threadIdx.x & 15) == 0 && valid) atomicAdd(dot + node, partial);
}

// Copies the [terms][32] weight slice of one element into shared memory (all threads of the block).
__device__ __forceinline__ void stage_poly_weights(float4* __restrict__ dst, const float* __restrict__ weights, int type,
                                                   int terms, int C, int k_base)
{
    const float* src = weights + static_cast<size_t>(type) * terms * C + k_base;
    for (int idx = threadIdx.x; idx < terms * 8; idx += blockDim.x)
        dst[idx] = *reinterpret_cast<const float4*>(src + static_cast<size_t>(idx >> 3) * C + 4 * (idx & 7));
    __syncthreads();
}

// Walks the nodes of one block, two per warp and pass, one run of equal elements after the other.  Receivers are sorted by
// element (the counting sort of Evaluator::install_graph), so most blocks are one run, and the count of equal elements is the
// length of the run.  CALL sees node, valid (false for the lanes of a node past the end, which repeat the
// last one), k (first channel of the pair) and w (weight pairs of a term at w[term * 16]).
#define SXB_POLY_WALK(NT, CALL)                                                                                     \
    extern __shared__ float4 w_s[];                                                                                 \
    const int block_node0 = blockIdx.x * nodes_per_block, block_end = min(block_node0 + nodes_per_block, num_nodes);\
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;                            \
    const int k = blockIdx.y * 32 + 2 * (lane & 15);                                                                \
    for (int begin = block_node0; begin < block_end;) {                                                             \
        const int type = element[begin];   /* the count is also the barrier behind which the old weights may go */  \
        const int end = begin + __syncthreads_count(begin + static_cast<int>(threadIdx.x) < block_end &&            \
                                                    element[min(begin + static_cast<int>(threadIdx.x), block_end - 1)] == type);\
        stage_poly_weights(w_s, weights, type, NT, C, blockIdx.y * 32);                                             \
        for (int node0 = begin + 2 * warp; node0 < end; node0 += 2 * warps) {                                       \
            const bool valid = node0 + (lane >> 4) < end;                                                           \
            const int node = valid ? node0 + (lane >> 4) : node0;                                                   \
            int at = lane & 15;                                                                                     \
            asm volatile("" : "+r"(at));   /* keeps the weight loads of all terms from being hoisted out of the loop */\
            const f2* w = reinterpret_cast<const f2*>(w_s) + at;                                                    \
            CALL;                                                                                                   \
        }                                                                                                           \
        begin = end;                                                                                                \
    }

#define W(t) w[(t) * 16]

// Warps per block and blocks per SM: two blocks of 8 warps; where the weight slice of a block takes more than half of the
// shared memory (hidden l = 2: 114 KB), one of 16.
#define SXB_DEFINE_POLY_KERNELS(NAME, WARPS)                                                                        \
    constexpr int kPolyWarps##NAME = WARPS;                                                                         \
    /* M0[node][LM][k] from A0[node][16][k] */                                                                      \
    __device__ __forceinline__ void m0_forward_node_##NAME(int node, bool valid, int C, int k, const float* __restrict__ A0,\
                                                           const f2* w, float* __restrict__ M0)             \
    {                                                                                                               \
        constexpr int NH = SXB_##NAME##_NUM_HIDDEN;                                                                 \
        f2 x[16], o[NH];                                                                                            \
        const float* in = A0 + static_cast<size_t>(node) * 16 * C + k;                                              \
        _Pragma("unroll") for (int q = 0; q < 16; ++q) x[q] = *reinterpret_cast<const f2*>(in + q * C);             \
        _Pragma("unroll") for (int q = 0; q < NH; ++q) o[q] = 0ull;                                                 \
        SXB_##NAME##_M0_FORWARD_BODY                                                                                \
        float* out = M0 + static_cast<size_t>(node) * NH * C + k;                                                   \
        if (valid) { _Pragma("unroll") for (int q = 0; q < NH; ++q) *reinterpret_cast<f2*>(out + q * C) = o[q]; }   \
    }                                                                                                               \
    __global__ void __launch_bounds__(32 * WARPS, 16 / WARPS)                                                       \
    m0_forward_kernel_##NAME(int num_nodes, int nodes_per_block, int C, const float* __restrict__ A0,               \
                             const unsigned char* __restrict__ element, const float* __restrict__ weights,          \
                             float* __restrict__ M0)                                                                \
    {                                                                                                               \
        SXB_POLY_WALK(SXB_##NAME##_M0_NUM_TERMS, m0_forward_node_##NAME(node, valid, C, k, A0, w, M0))          \
    }                                                                                                               \
    /* A0_adj[node][16][k] = sum_LM M0_adj[node][LM][k] dM0[LM]/dA0 */                                              \
    __device__ __forceinline__ void m0_reverse_node_##NAME(int node, bool valid, int C, int k, const float* __restrict__ A0,\
                                                           const f2* w, const float* __restrict__ M0_adj,   \
                                                           float* __restrict__ A0_adj, float* __restrict__ dot)     \
    {                                                                                                               \
        constexpr int NH = SXB_##NAME##_NUM_HIDDEN;                                                                 \
        f2 x[16], g[16], adj[NH];                                                                                   \
        const float* in = A0 + static_cast<size_t>(node) * 16 * C + k;                                              \
        _Pragma("unroll") for (int q = 0; q < 16; ++q) { x[q] = *reinterpret_cast<const f2*>(in + q * C); g[q] = 0ull; }\
        const float* ain = M0_adj + static_cast<size_t>(node) * NH * C + k;                                         \
        _Pragma("unroll") for (int q = 0; q < NH; ++q) adj[q] = *reinterpret_cast<const f2*>(ain + q * C);          \
        SXB_##NAME##_M0_REVERSE_BODY                                                                                \
        float* out = A0_adj + static_cast<size_t>(node) * 16 * C + k;                                               \
        if (valid) { _Pragma("unroll") for (int q = 0; q < 16; ++q) *reinterpret_cast<f2*>(out + q * C) = g[q]; }   \
        if (dot != nullptr) poly_accumulate_dot(g, x, dot, node, valid);                                            \
    }                                                                                                               \
    __global__ void __launch_bounds__(32 * WARPS, 16 / WARPS)                                                       \
    m0_reverse_kernel_##NAME(int num_nodes, int nodes_per_block, int C, const float* __restrict__ A0,               \
                             const unsigned char* __restrict__ element, const float* __restrict__ weights,          \
                             const float* __restrict__ M0_adj, float* __restrict__ A0_adj, float* __restrict__ dot) \
    {                                                                                                               \
        SXB_POLY_WALK(SXB_##NAME##_M0_NUM_TERMS, m0_reverse_node_##NAME(node, valid, C, k, A0, w, M0_adj, A0_adj, dot))\
    }                                                                                                               \
    /* M1[node][k] from A1[node][16][k] */                                                                          \
    __device__ __forceinline__ void m1_forward_node_##NAME(int node, bool valid, int C, int k, const float* __restrict__ A1,\
                                                           const f2* w, float* __restrict__ M1)             \
    {                                                                                                               \
        f2 x[16], o[1];                                                                                             \
        const float* in = A1 + static_cast<size_t>(node) * 16 * C + k;                                              \
        _Pragma("unroll") for (int q = 0; q < 16; ++q) x[q] = *reinterpret_cast<const f2*>(in + q * C);             \
        o[0] = 0ull;                                                                                                \
        SXB_##NAME##_M1_FORWARD_BODY                                                                                \
        if (valid) *reinterpret_cast<f2*>(M1 + static_cast<size_t>(node) * C + k) = o[0];                           \
    }                                                                                                               \
    __global__ void __launch_bounds__(32 * WARPS, 16 / WARPS)                                                       \
    m1_forward_kernel_##NAME(int num_nodes, int nodes_per_block, int C, const float* __restrict__ A1,               \
                             const unsigned char* __restrict__ element, const float* __restrict__ weights,          \
                             float* __restrict__ M1)                                                                \
    {                                                                                                               \
        SXB_POLY_WALK(SXB_##NAME##_M1_NUM_TERMS, m1_forward_node_##NAME(node, valid, C, k, A1, w, M1))          \
    }                                                                                                               \
    /* A1_adj[node][16][k] = M1_adj[node][k] dM1/dA1 */                                                             \
    __device__ __forceinline__ void m1_reverse_node_##NAME(int node, bool valid, int C, int k, const float* __restrict__ A1,\
                                                           const f2* w, const float* __restrict__ M1_adj,   \
                                                           float* __restrict__ A1_adj, float* __restrict__ dot)     \
    {                                                                                                               \
        f2 x[16], g[16], adj[1];                                                                                    \
        const float* in = A1 + static_cast<size_t>(node) * 16 * C + k;                                              \
        _Pragma("unroll") for (int q = 0; q < 16; ++q) { x[q] = *reinterpret_cast<const f2*>(in + q * C); g[q] = 0ull; }\
        adj[0] = *reinterpret_cast<const f2*>(M1_adj + static_cast<size_t>(node) * C + k);                          \
        SXB_##NAME##_M1_REVERSE_BODY                                                                                \
        float* out = A1_adj + static_cast<size_t>(node) * 16 * C + k;                                               \
        if (valid) { _Pragma("unroll") for (int q = 0; q < 16; ++q) *reinterpret_cast<f2*>(out + q * C) = g[q]; }   \
        if (dot != nullptr) poly_accumulate_dot(g, x, dot, node, valid);                                            \
    }                                                                                                               \
    __global__ void __launch_bounds__(32 * WARPS, 16 / WARPS)                                                       \
    m1_reverse_kernel_##NAME(int num_nodes, int nodes_per_block, int C, const float* __restrict__ A1,               \
                             const unsigned char* __restrict__ element, const float* __restrict__ weights,          \
                             const float* __restrict__ M1_adj, float* __restrict__ A1_adj, float* __restrict__ dot) \
    {                                                                                                               \
        SXB_POLY_WALK(SXB_##NAME##_M1_NUM_TERMS, m1_reverse_node_##NAME(node, valid, C, k, A1, w, M1_adj, A1_adj, dot))\
    }

SXB_DEFINE_POLY_KERNELS(S0, 8)
SXB_DEFINE_POLY_KERNELS(S1, 8)
SXB_DEFINE_POLY_KERNELS(S2, 16)
#undef W

// ---------------------------------------------------------------------------------------------
// Readout polynomial of a single-layer model: M1[node][k] = sum_t w[element][t][k] prod_q H1[node][idx_t,q][k]
// over monomials of degree 1 to 3 in the hidden components, read as data (reference:
// libsymmetrix/source/mace.cpp:2460-2482 with the polynomial input switched to H1, and its gradient
// 2485-2512, which adds to H1_adj).  One thread per (node, channel); the monomial list is short (the
// invariants of at most nine components), so it is walked from global memory.
constexpr int kMaxHidden = 9;

template <bool kReverse>
__global__ void __launch_bounds__(128) hidden_poly_kernel(int num_nodes, int C, int num_hidden, int num_terms,
                                                          const int4* __restrict__ terms, const float* __restrict__ H1,
                                                          const unsigned char* __restrict__ element,
                                                          const float* __restrict__ weights, float* __restrict__ M1,
                                                          const float* __restrict__ M1_adj, float* __restrict__ H1_adj)
{
    const long index = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= static_cast<long>(num_nodes) * C) return;
    const int node = static_cast<int>(index / C), k = static_cast<int>(index - static_cast<long>(node) * C);
    float x[kMaxHidden], g[kMaxHidden];
#pragma unroll
    for (int q = 0; q < kMaxHidden; ++q) {
        x[q] = q < num_hidden ? H1[(static_cast<size_t>(node) * num_hidden + q) * C + k] : 0.0f;
        g[q] = 0.0f;
    }
    const float* w = weights + static_cast<size_t>(element[node]) * num_terms * C + k;
    float value = 0.0f;
    for (int t = 0; t < num_terms; ++t) {
        const int4 m = terms[t];
        const float wt = w[static_cast<size_t>(t) * C];
        const float a = x[m.x], b = m.y >= 0 ? x[m.y] : 1.0f, c = m.z >= 0 ? x[m.z] : 1.0f;
        if (!kReverse) {
            value = fmaf(wt, a * b * c, value);
        } else {
            g[m.x] = fmaf(wt, b * c, g[m.x]);
            if (m.y >= 0) g[m.y] = fmaf(wt, a * c, g[m.y]);
            if (m.z >= 0) g[m.z] = fmaf(wt, a * b, g[m.z]);
        }
    }
    if (!kReverse) {
        M1[static_cast<size_t>(node) * C + k] = value;
    } else {
        const float adj = M1_adj[static_cast<size_t>(node) * C + k];
        for (int q = 0; q < num_hidden; ++q) H1_adj[(static_cast<size_t>(node) * num_hidden + q) * C + k] += adj * g[q];
    }
}

// ---------------------------------------------------------------------------------------------
// Channel-mixing linear as a tiled FP32 GEMM with structured rows.
//   C[row(g)][n] (+)= sum_k A[row(g)][k] * B[k][n]      (B stored [K][N], or [N][K] when transposed)
// Logical row g of a node tensor (node, component, channel): node = first_node + g / components,
// m = g % components, address = node*node_stride + offset + m*component_stride.
struct GemmArgs {
    const float* A;
    const float* B;
    float* C;
    const float* bias;      // optional [N], added when not accumulating
    RowMap a_rows, c_rows;
    int first_node;
    int M, N, K;            // M = logical rows
    int ldb;
    int b_transposed;       // 0: B[k*ldb + n], 1: B[n*ldb + k]
    int accumulate;         // 1: C += A B
};

__device__ __forceinline__ long row_address(const RowMap& map, int first_node, int g)
{
    const int node = first_node + g / map.components;
    const int m = g % map.components;
    return static_cast<long>(node) * map.node_stride + map.offset + static_cast<long>(m) * map.component_stride;
}

constexpr int kGemmBM = 64, kGemmBN = 64, kGemmBK = 16;

__global__ void __launch_bounds__(256) gemm_rows_kernel(const GemmArgs args)
{
    __shared__ float As[kGemmBK][kGemmBM + 4];
    __shared__ float Bs[kGemmBK][kGemmBN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
    const int row0 = blockIdx.x * kGemmBM, col0 = blockIdx.y * kGemmBN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    // loader mapping: A tile 64 rows x 16 k: thread -> (row = tid/4, k4 = (tid%4)*4)
    const int a_row = tid >> 2, a_k = (tid & 3) * 4;
    const bool a_valid = row0 + a_row < args.M;
    const float* a_ptr = a_valid ? args.A + row_address(args.a_rows, args.first_node, row0 + a_row) : nullptr;
    for (int k0 = 0; k0 < args.K; k0 += kGemmBK) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int kk = k0 + a_k + q;
            As[a_k + q][a_row] = (a_valid && kk < args.K) ? a_ptr[kk] : 0.0f;
        }
        if (!args.b_transposed) {
            // B tile 16 k x 64 n: thread -> (k = tid/16, n4 = (tid%16)*4)
            const int bk = tid >> 4, bn = (tid & 15) * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int kk = k0 + bk, nn = col0 + bn + q;
                Bs[bk][bn + q] = (kk < args.K && nn < args.N) ? args.B[static_cast<long>(kk) * args.ldb + nn] : 0.0f;
            }
        } else {
            // stored [N][K]: thread -> (n = tid/4, k4 = (tid%4)*4)
            const int bn = tid >> 2, bk = (tid & 3) * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int kk = k0 + bk + q, nn = col0 + bn;
                Bs[bk + q][bn] = (kk < args.K && nn < args.N) ? args.B[static_cast<long>(nn) * args.ldb + kk] : 0.0f;
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kGemmBK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int g = row0 + ty * 4 + i;
        if (g >= args.M) continue;
        float* c_ptr = args.C + row_address(args.c_rows, args.first_node, g);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = col0 + tx * 4 + j;
            if (n >= args.N) continue;
            float v = acc[i][j];
            if (args.accumulate) v += c_ptr[n];
            else if (args.bias != nullptr) v += args.bias[n];
            c_ptr[n] = v;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Readout: E_i = E0[element] + q . xs_i + MLP(H2_i), MLP [C, hidden, 1] with hidden activation
// s*z*sigmoid(z); also the adjoint of H2.  One warp per node.
__global__ void __launch_bounds__(256)
readout_kernel(int num_nodes, int C, int hidden, float act_scale, const float* __restrict__ M0, int num_hidden_lm,
               const float* __restrict__ H2, const unsigned char* __restrict__ element,
               const double* __restrict__ atomic_energies, const float* __restrict__ q,
               const float* __restrict__ W1 /*[hidden][C]*/, const float* __restrict__ W2 /*[hidden]*/,
               double* __restrict__ node_energies, float* __restrict__ H2_adj, double* __restrict__ energy_slots)
{
    const int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (node >= num_nodes) return;
    const float* xs = M0 + static_cast<size_t>(node) * num_hidden_lm * C;   // scalar block of M0
    const float* h2 = H2 + static_cast<size_t>(node) * C;
    float e1 = 0.0f;
    for (int k = lane; k < C; k += 32) e1 = fmaf(q[k], xs[k], e1);
    float e2 = 0.0f;
    float coeff[64];   // V2[h] * dact[h], hidden <= 64
    for (int h = 0; h < hidden; ++h) {
        float z = 0.0f;
        for (int k = lane; k < C; k += 32) z = fmaf(W1[h * C + k], h2[k], z);
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) z += __shfl_xor_sync(0xffffffffu, z, offset);
        const float sig = 1.0f / (1.0f + expf(-z));
        e2 = fmaf(W2[h], act_scale * z * sig, e2);
        coeff[h] = W2[h] * (act_scale * sig + act_scale * z * sig * (1.0f - sig));
    }
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) e1 += __shfl_xor_sync(0xffffffffu, e1, offset);
    for (int k = lane; k < C; k += 32) {
        float g = 0.0f;
        for (int h = 0; h < hidden; ++h) g = fmaf(coeff[h], W1[h * C + k], g);
        H2_adj[static_cast<size_t>(node) * C + k] = g;
    }
    if (lane == 0) {
        const double e = atomic_energies[element[node]] + static_cast<double>(e1) + static_cast<double>(e2);
        node_energies[node] = e;
        if (energy_slots != nullptr) atomicAdd(energy_slots + (node % kVirialSlots), e);
    }
}

// The same readout for the common head shape (16 hidden units, C a multiple of 32, at most 256): the 16
// pre-activations of a node are formed together, each lane holding its channels' partial sums, and
// summed over the warp by a butterfly that halves the number of live values at every step (16 shuffles
// instead of 80); lane L ends up with hidden unit L / 2.  No per-thread array is indexed at run time.  Returns the node's
// energy without E0 (in lane 0); g is the adjoint of H2, channels lane + 32 j.
template <int kChunks>   // C / 32
__device__ __forceinline__ double readout16_node(int lane, float act_scale, const float* __restrict__ xs, const float* __restrict__ h2,
                                                 const float* __restrict__ q, const float* __restrict__ W1 /*[16][C]*/,
                                                 const float* __restrict__ W2 /*[16]*/, float (&g)[kChunks])
{
    constexpr int C = 32 * kChunks, kHidden = 16;
    float hv[kChunks];
    float e1 = 0.0f;
#pragma unroll
    for (int j = 0; j < kChunks; ++j) {
        hv[j] = h2[lane + 32 * j];
        e1 = fmaf(q[lane + 32 * j], xs[lane + 32 * j], e1);
    }
    float v[kHidden];
#pragma unroll
    for (int h = 0; h < kHidden; ++h) {
        float z = 0.0f;
#pragma unroll
        for (int j = 0; j < kChunks; ++j) z = fmaf(W1[h * C + lane + 32 * j], hv[j], z);
        v[h] = z;
    }
#pragma unroll
    for (int offset = 16, live = kHidden; offset >= 2; offset >>= 1, live >>= 1) {
        const bool upper = (lane & offset) != 0;
        const int half = live / 2;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i < half) {
                const float send = upper ? v[i] : v[i + half];
                const float recv = __shfl_xor_sync(0xffffffffu, send, offset);
                v[i] = (upper ? v[i + half] : v[i]) + recv;
            }
        }
    }
    const float z = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);      // lanes 2h and 2h+1: hidden unit h
    const int unit = lane >> 1;
    const float sig = 1.0f / (1.0f + expf(-z));
    const float w2 = W2[unit];
    float e2 = (lane & 1) ? 0.0f : w2 * (act_scale * z * sig);
    const float coeff = w2 * (act_scale * sig + act_scale * z * sig * (1.0f - sig));
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        e1 += __shfl_xor_sync(0xffffffffu, e1, offset);
        e2 += __shfl_xor_sync(0xffffffffu, e2, offset);
    }
#pragma unroll
    for (int j = 0; j < kChunks; ++j) g[j] = 0.0f;
#pragma unroll
    for (int h = 0; h < kHidden; ++h) {
        const float c = __shfl_sync(0xffffffffu, coeff, 2 * h);
#pragma unroll
        for (int j = 0; j < kChunks; ++j) g[j] = fmaf(c, W1[h * C + lane + 32 * j], g[j]);
    }
    return static_cast<double>(e1) + static_cast<double>(e2);
}

template <int kChunks>
__global__ void __launch_bounds__(256)
readout16_kernel(int num_nodes, float act_scale, const float* __restrict__ M0, int num_hidden_lm,
                 const float* __restrict__ H2, const unsigned char* __restrict__ element,
                 const double* __restrict__ atomic_energies, const float* __restrict__ q,
                 const float* __restrict__ W1, const float* __restrict__ W2,
                 double* __restrict__ node_energies, float* __restrict__ H2_adj, double* __restrict__ energy_slots)
{
    constexpr int C = 32 * kChunks;
    const int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (node >= num_nodes) return;
    float g[kChunks];
    const double e = atomic_energies[element[node]]
                     + readout16_node<kChunks>(lane, act_scale, M0 + static_cast<size_t>(node) * num_hidden_lm * C, H2 + static_cast<size_t>(node) * C, q, W1, W2, g);
#pragma unroll
    for (int j = 0; j < kChunks; ++j) H2_adj[static_cast<size_t>(node) * C + lane + 32 * j] = g[j];
    if (lane == 0) {
        node_energies[node] = e;
        if (energy_slots != nullptr) atomicAdd(energy_slots + (node % kVirialSlots), e);
    }
}

// ---------------------------------------------------------------------------------------------
// Everything between A1 and its adjoint in one launch: contraction M1, H2 = x T_element + M1 W with x the scalar block of M0,
// readout, and their adjoints back to A1_adj and to the scalar block of M0_adj (readout weights + T_element H2_adj).  All of it is
// local to a node, and as five launches it lasts as long as five short dependent kernels (9 to 13 us each up to a thousand nodes).
// A block takes 512 / kC nodes; the linears run in FP32 on the vectors in shared memory, a thread per output column and part of
// the sum, the weights once per block.
struct NodeReadoutArgs {
    int num_nodes;
    float act_scale;
    const unsigned char* element;
    const float *A1, *M0, *m1_weights;             // [node][16][kC], [node][NH][kC], [element][term][kC]
    const float *W, *Wt, *T, *Tt;                  // [in][out], [out][in], the same per element
    const float *q, *W1, *W2;
    const double* atomic_energies;
    float *M1, *H2, *H2_adj, *M1_adj, *A1_adj, *M0_adj;
    int M0_adj_stride;                             // floats between the nodes' scalar blocks
    float* dot;
    double *node_energies, *energy_slots;
};

// Its vectors in shared memory, [channel][node] or [node][channel]; the partial sums are read in channel pairs.
template <int kC>
struct alignas(16) NodeReadoutShared {
    static constexpr int G = 512 / kC, kParts = 256 / kC;
    float m1[kC][G], xs[kC][G], adj_s[kC][G], h2[G][kC], sums[2][kParts][G][kC];
    unsigned char types[G];
};
template <int kC>
constexpr bool pairs_aligned()
{
    using S = NodeReadoutShared<kC>;
    return alignof(S) % sizeof(float2) == 0 && offsetof(S, sums) % sizeof(float2) == 0 && kC % 2 == 0;
}
static_assert(pairs_aligned<32>() && pairs_aligned<64>() && pairs_aligned<128>(), "float2 reads of the partial sums");

#define W(t) w[(t) * (kC / 2)]
#define SXB_DEFINE_NODE_READOUT(NAME)                                                                               \
template <int kC>                                                                                                   \
__global__ void __launch_bounds__(256, 2) node_readout_kernel_##NAME(const NodeReadoutArgs a)                       \
{                                                                                                                   \
    constexpr int NH = SXB_##NAME##_NUM_HIDDEN, NT = SXB_##NAME##_M1_NUM_TERMS, G = 512 / kC, kParts = 256 / kC;    \
    __shared__ NodeReadoutShared<kC> s;                                                                             \
    const int tid = threadIdx.x, base = blockIdx.x * G;                                                             \
    const int n = tid / (kC / 2), k = 2 * (tid % (kC / 2));             /* node and channel pair of the contractions */ \
    const bool valid = base + n < a.num_nodes;                                                                      \
    const size_t node = valid ? base + n : a.num_nodes - 1;             /* a place past the end repeats the last node */ \
    const int column = tid % kC, part = tid / kC;                       /* output and part of the sum of the linears */ \
    const int type = a.element[node];                                                                               \
    const f2* const w = reinterpret_cast<const f2*>(a.m1_weights + static_cast<size_t>(type) * NT * kC + k);        \
    const float* const in = a.A1 + node * 16 * kC + k;                                                              \
    {                                                                                                               \
        f2 x[16], o[1];                                                                                             \
        _Pragma("unroll") for (int r = 0; r < 16; ++r) x[r] = *reinterpret_cast<const f2*>(in + r * kC);            \
        o[0] = 0ull;                                                                                                \
        SXB_##NAME##_M1_FORWARD_BODY                                                                                \
        const float2 value = *reinterpret_cast<const float2*>(&o[0]);                                               \
        const float2 scalar = *reinterpret_cast<const float2*>(a.M0 + node * NH * kC + k);                          \
        s.m1[k][n] = value.x; s.m1[k + 1][n] = value.y;                                                             \
        s.xs[k][n] = scalar.x; s.xs[k + 1][n] = scalar.y;                                                           \
        if (valid) *reinterpret_cast<float2*>(a.M1 + node * kC + k) = value;                                        \
        if (k == 0) s.types[n] = static_cast<unsigned char>(type);                                                  \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    {                                                                                                               \
        float acc[G];                                                                                               \
        _Pragma("unroll") for (int r = 0; r < G; ++r) acc[r] = 0.0f;                                                \
        _Pragma("unroll 8") for (int c = part * (kC / kParts); c < (part + 1) * (kC / kParts); ++c) {               \
            const float wv = a.W[c * kC + column];                                                                  \
            _Pragma("unroll") for (int r = 0; r < G; ++r) acc[r] = fmaf(s.m1[c][r], wv, acc[r]);                    \
        }                                                                                                           \
        for (int r0 = 0; r0 < G;) {   /* runs of equal elements: one in most blocks, receivers are sorted by element */ \
            const int run = s.types[r0];                                                                            \
            int r1 = r0 + 1;                                                                                        \
            while (r1 < G && s.types[r1] == run) ++r1;                                                              \
            const float* const T = a.T + static_cast<size_t>(run) * kC * kC + column;                               \
            _Pragma("unroll 8") for (int c = part * (kC / kParts); c < (part + 1) * (kC / kParts); ++c) {           \
                const float tv = T[c * kC];                                                                         \
                _Pragma("unroll") for (int r = 0; r < G; ++r) acc[r] = fmaf(r >= r0 && r < r1 ? s.xs[c][r] : 0.0f, tv, acc[r]); \
            }                                                                                                       \
            r0 = r1;                                                                                                \
        }                                                                                                           \
        _Pragma("unroll") for (int r = 0; r < G; ++r) s.sums[0][part][r][column] = acc[r];                          \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    for (int idx = tid; idx < G * kC; idx += 256) {                                                                 \
        const int r = idx / kC, c = idx % kC;                                                                       \
        float total = 0.0f;                                                                                         \
        _Pragma("unroll") for (int p = 0; p < kParts; ++p) total += s.sums[0][p][r][c];                             \
        s.h2[r][c] = total;                                                                                         \
        if (base + r < a.num_nodes) a.H2[static_cast<size_t>(base + r) * kC + c] = total;                           \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    for (int r = tid >> 5; r < G; r += 8) {                                                                         \
        const int lane = tid & 31;                                                                                  \
        const size_t at = min(base + r, a.num_nodes - 1);                                                           \
        float g[kC / 32];                                                                                           \
        const double e = a.atomic_energies[s.types[r]]                                                              \
                         + readout16_node<kC / 32>(lane, a.act_scale, a.M0 + at * NH * kC, s.h2[r], a.q, a.W1, a.W2, g); \
        _Pragma("unroll") for (int c = 0; c < kC / 32; ++c) {                                                       \
            s.adj_s[lane + 32 * c][r] = g[c];                                                                       \
            if (base + r < a.num_nodes) a.H2_adj[at * kC + lane + 32 * c] = g[c];                                   \
        }                                                                                                           \
        if (lane == 0 && base + r < a.num_nodes) {                                                                  \
            a.node_energies[at] = e;                                                                                \
            if (a.energy_slots != nullptr) atomicAdd(a.energy_slots + (at % kVirialSlots), e);                      \
        }                                                                                                           \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    {                                                                                                               \
        float acc[G], skip[G];                                                                                      \
        _Pragma("unroll") for (int r = 0; r < G; ++r) acc[r] = skip[r] = 0.0f;                                      \
        _Pragma("unroll 8") for (int c = part * (kC / kParts); c < (part + 1) * (kC / kParts); ++c) {               \
            const float wv = a.Wt[c * kC + column];                                                                 \
            _Pragma("unroll") for (int r = 0; r < G; ++r) acc[r] = fmaf(s.adj_s[c][r], wv, acc[r]);                 \
        }                                                                                                           \
        for (int r0 = 0; r0 < G;) {                                                                                 \
            const int run = s.types[r0];                                                                            \
            int r1 = r0 + 1;                                                                                        \
            while (r1 < G && s.types[r1] == run) ++r1;                                                              \
            const float* const T = a.Tt + static_cast<size_t>(run) * kC * kC + column;                              \
            _Pragma("unroll 8") for (int c = part * (kC / kParts); c < (part + 1) * (kC / kParts); ++c) {           \
                const float tv = T[c * kC];                                                                         \
                _Pragma("unroll") for (int r = 0; r < G; ++r) skip[r] = fmaf(r >= r0 && r < r1 ? s.adj_s[c][r] : 0.0f, tv, skip[r]); \
            }                                                                                                       \
            r0 = r1;                                                                                                \
        }                                                                                                           \
        _Pragma("unroll") for (int r = 0; r < G; ++r) { s.sums[0][part][r][column] = acc[r]; s.sums[1][part][r][column] = skip[r]; } \
    }                                                                                                               \
    __syncthreads();                                                                                                \
    {                                                                                                               \
        f2 x[16], g[16], adj[1];                                                                                    \
        float2 m1_adj = make_float2(0.0f, 0.0f), m0_adj = *reinterpret_cast<const float2*>(a.q + k);                \
        _Pragma("unroll") for (int p = 0; p < kParts; ++p) {                                                        \
            const float2 u = *reinterpret_cast<const float2*>(&s.sums[0][p][n][k]), v = *reinterpret_cast<const float2*>(&s.sums[1][p][n][k]); \
            m1_adj.x += u.x; m1_adj.y += u.y; m0_adj.x += v.x; m0_adj.y += v.y;                                     \
        }                                                                                                           \
        if (valid) {                                                                                                \
            *reinterpret_cast<float2*>(a.M1_adj + node * kC + k) = m1_adj;                                          \
            *reinterpret_cast<float2*>(a.M0_adj + node * a.M0_adj_stride + k) = m0_adj;                             \
        }                                                                                                           \
        _Pragma("unroll") for (int r = 0; r < 16; ++r) { x[r] = *reinterpret_cast<const f2*>(in + r * kC); g[r] = 0ull; } \
        adj[0] = *reinterpret_cast<const f2*>(&m1_adj);                                                             \
        SXB_##NAME##_M1_REVERSE_BODY                                                                                \
        float* out = a.A1_adj + node * 16 * kC + k;                                                                 \
        if (valid) { _Pragma("unroll") for (int r = 0; r < 16; ++r) *reinterpret_cast<f2*>(out + r * kC) = g[r]; }  \
        if (a.dot != nullptr) poly_accumulate_dot(g, x, a.dot, static_cast<int>(node), valid);                      \
    }                                                                                                               \
}
SXB_DEFINE_NODE_READOUT(S0)
SXB_DEFINE_NODE_READOUT(S1)
SXB_DEFINE_NODE_READOUT(S2)
#undef W

// What an evaluation accumulates into, set to zero by one launch (a chain of four to six fills cost 1 to 2 us each, one after the
// other: 40 atoms 193 -> 186 us, 320 atoms of the 32-channel model 166 -> 159, 5,000 atoms the same).  Regions of 4-byte words whose first lies on 16 bytes; the blocks stride over each in turn, 16 bytes a thread.
constexpr int kMaxClears = 6;
struct ClearList {
    float* begin[kMaxClears];
    long words[kMaxClears];
    int count = 0;
    void add(void* region, std::size_t bytes)
    {
        begin[count] = static_cast<float*>(region);
        words[count++] = static_cast<long>(bytes / sizeof(float));
    }
};
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ ClearList list)
{
    const long thread = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x, threads = static_cast<long>(gridDim.x) * blockDim.x;
    for (int r = 0; r < list.count; ++r) {
        const long vectors = list.words[r] >> 2;
        for (long k = thread; k < vectors; k += threads)
            reinterpret_cast<float4*>(list.begin[r])[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (thread < (list.words[r] & 3)) list.begin[r][4 * vectors + thread] = 0.0f;
    }
}

// tensor[node][0][k] = values[k] for the first num_nodes nodes of a (node, component, channel) tensor.
__global__ void fill_scalar_block_kernel(int num_nodes, int C, long node_stride, const float* __restrict__ values,
                                         float* __restrict__ tensor)
{
    const long index = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= static_cast<long>(num_nodes) * C) return;
    const long node = index / C, k = index - node * C;
    tensor[node * node_stride + k] = values[k];
}

// tensor[node][:] += table[element[node]][:] over rows of row_floats values (element-dependent constants).
__global__ void add_element_rows_kernel(int num_nodes, int row_floats, const unsigned char* __restrict__ element,
                                        const float* __restrict__ table, float* __restrict__ tensor)
{
    const long index = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (index >= static_cast<long>(num_nodes) * row_floats) return;
    const long node = index / row_floats, k = index - node * row_floats;
    tensor[index] += table[static_cast<long>(element[node]) * row_floats + k];
}

// Closing kernel of an evaluation, one thread per output value: sums the energy / virial slots into
// totals[10] and writes node energies and node forces in the caller's node order.  When `host` is
// given the same values are also published straight into mapped pinned host memory, laid out
// [status word, totals[10], energies[num_receivers], forces[num_nodes][3]] (consecutive threads write
// consecutive words, so the writes cross the bus in full segments), and the caller needs no
// device-to-host copy.  Only the first `host_values` values go to the host (a caller that keeps the forces
// on the device asks for status and totals alone and saves the bus traffic).
__global__ void publish_results_kernel(int num_receivers, int num_nodes, const int* __restrict__ internal_of,
                                       const double* __restrict__ energy_slots, const double* __restrict__ virial_slots,
                                       const double* __restrict__ node_energies, const double* __restrict__ forces,
                                       const int* __restrict__ status, double* __restrict__ totals,
                                       double* __restrict__ energies_out, double* __restrict__ forces_out,
                                       double* __restrict__ host, long host_values)
{
    const long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long total = 11 + static_cast<long>(num_receivers) + 3 * static_cast<long>(num_nodes);
    if (idx >= total) return;
    double value;
    if (idx == 0) {
        value = static_cast<double>(status[0]);
    } else if (idx < 11) {
        const int t = static_cast<int>(idx) - 1;
        value = 0.0;
        for (int slot = 0; slot < kVirialSlots; ++slot) value += (t == 0) ? energy_slots[slot] : virial_slots[slot * 9 + (t - 1)];
        totals[t] = value;
    } else if (idx < 11 + num_receivers) {
        const long o = idx - 11;
        value = node_energies[internal_of[o]];
        energies_out[o] = value;
    } else {
        const long j = idx - 11 - num_receivers;
        const long o = j / 3, q = j % 3;
        value = forces[3 * static_cast<long>(internal_of[o]) + q];
        forces_out[j] = value;
    }
    if (host != nullptr && idx < host_values) host[idx] = value;
}

}  // namespace sxb
