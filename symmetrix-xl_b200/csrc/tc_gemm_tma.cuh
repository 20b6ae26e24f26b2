// Channel-mixing linears on the 5th-generation tensor cores, persistent operand-streaming form.
//   C[row(g)][n] (+)= sum_k A[row(g)][k] * Bt[n][k]         (three TF32 passes, FP32 accumulation)
// Same arithmetic as tc_gemm.cuh; what changes is how the work is fed:
//   * one CTA per SM walks a list of (row tile, column tile) work items, so barrier set-up, tensor
//     memory allocation and descriptor fetches are paid once, and the pipeline never drains between
//     tiles: operand stages and their mbarrier phases run on across tile boundaries;
//   * the A rows (node, component, channel-block addressing) are fetched by the TMA engine as boxes
//     of a rank-3 tensor [node][component][K] straight into the 128-byte-swizzled K-major layout,
//     two K chunks deep, and two more split ones;
//   * four warps split a tile, a row per thread, into its TF32 high part and residual and leave both in tensor memory, where
//     the MMAs take their A operand from.  With A in shared memory the three passes read 96 KB of operands per chunk of 32 K
//     on top of 80 KB of copies and splitting, which at 128 bytes a cycle takes longer than the MMAs (0.93 us a chunk);
//   * the tensor core truncates whenever it adds to its accumulator, so a chain of K / 8 x 3 additions ends low by about one
//     part in 10^7 for every six of them (K = 192: 2e-6 against 3e-7 for an FP32 sum).  Each chunk of 32 K therefore gets an
//     accumulator of its own (two of 128 columns in tensor memory), its eight small products before its four large ones, and
//     eight warps add the chunks up in registers, rounded to nearest: 1.5e-7; where a launch asks for it with what the truncations
//     take on average put back (kT3Truncated);
//   * the same warps leave tile i in shared memory, from where the TMA engine stores it, or adds it to the output, while they
//     sum up tile i + 1.
// A row tile holds floor(128 / components) whole nodes (128, 126, 125 or 126 rows); the remaining
// accumulator lanes are never stored.  A column tile is 128, 96, 64 or 32 columns wide, as the launch chooses.
// Thread roles: warps 0-3 split, warps 4-11 sums and epilogue, warp 12 lane 0 tcgen05.mma issue (warp 12 also
// owns the tensor-memory allocation), warp 13 lane 0 weight TMA, warp 14 lane 0 activation TMA.  The
// issuing thread is the narrow point of such a pipeline (every mbarrier or tcgen05 instruction costs
// it 60-300 cycles of latency), so it does nothing else: per K chunk it waits for the accumulator and for one more barrier -
// the weight copy and the 128 splitting threads arrive on the same one - issues the 12 MMAs and commits once; every other role
// learns from that one commit that the chunk's operands are free and its accumulator full.
// Every wait is bounded: on expiry the kernel raises bit 1 of the status word, every role leaves
// its loop, the producers wait (bounded) for their own copies in flight, the tensor memory is
// freed and the CTA returns.
#pragma once

#include "tc_gemm.cuh"

namespace sxb {

constexpr int kT3AStages = 2;                 // raw activation tiles in flight
constexpr int kT3SplitStages = 3;             // split activation tiles (high part and residual) in tensor memory
constexpr int kT3Stages = 4;                  // weight tiles (hi + lo)
constexpr int kT3Ring = 4;                    // barriers per chunk in flight
constexpr int kT3OperandBytes = 128 * 128;    // 128 rows x 32 floats
constexpr int kT3SmemBytes = (kT3AStages + 2 * kT3Stages + 4) * kT3OperandBytes + 512;   // with the output tile, 4 x 32 columns
constexpr int kT3Threads = 480;
constexpr int kT3Issue = 384;                 // the issuing thread, first of warp 12
constexpr int kT3Accumulators = 2;            // one per K chunk in turn, of up to 128 columns
constexpr int kT3SplitColumn = 128 * kT3Accumulators;
constexpr int kT3Columns = 512;               // allocated: accumulators, and 64 columns per split tile
static_assert(kT3SplitColumn + 64 * kT3SplitStages <= kT3Columns, "tensor memory");
static_assert(kT3AStages <= kT3Ring && kT3Stages <= kT3Ring && kT3SplitStages <= kT3Ring, "rings of barriers");

// What the truncations of a chunk take from its sum, on average, put back.  Only the four large products count; after each the unit
// drops half a last place of the partial sum s_j, 0.72 x 2^-24 of it over mantissas spread evenly in their logarithm, and the s_j
// make up (1 + 2 + 3 + 4) / 4 of the sum, whether the terms have one sign or random ones: 1.07e-7, nearly the last place of 1.
// (Sums of 128 products emulated in double: 2-norm of the error 1.3e-7 -> 0.8e-7, pull -1.07e-7 -> +0.15e-7; FP32 in a chain 2.0e-7.)
constexpr float kT3Truncated = 1.0f + 1.1920929e-7f;

struct alignas(64) Tc3Problem {
    CUtensorMap map_a;       // activations [node][component][K], box [nodes_per_tile][components][32]
    CUtensorMap map_hi;      // Bt_hi [N][K], box [n_tile][32]
    CUtensorMap map_lo;
    CUtensorMap map_c;       // output [node][component][N], box [nodes_per_tile][components][32]
    const float* bias;       // optional [N], added when not accumulating
    int K;                   // K % 32 == 0
    int accumulate;
    float chunk_scale;       // 1, or kT3Truncated
    int rows_per_tile, nodes_per_tile;
    int n_tile, n_tiles;     // 32, 64, 96 or 128; N % n_tile == 0
    int m_tiles;
    int tile_begin;          // first work item of this problem (items are m-major: m_tile * n_tiles + n)
};

constexpr int kT3MaxProblems = 16;
struct Tc3Batch {
    Tc3Problem problem[kT3MaxProblems];
    int count;
    int total_tiles;
};

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, unsigned long long* bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// Writes a box from shared memory, or adds it; rows beyond the tensor's extent are left out.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem_src, int x, int y, int z, bool add)
{
    if (add)
        asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                     ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                     ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z) : "memory");
}

// the four epilogue warps of one half of the columns
__device__ __forceinline__ bool half_barrier_all(int half, bool mine)
{
    int all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %2, 0;\n\t"
        "barrier.cta.red.and.pred q, %1, 128, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(all) : "r"(1 + half), "r"(mine ? 1 : 0) : "memory");
    return all != 0;
}
__device__ __forceinline__ void half_barrier(int half) { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); }

__device__ __forceinline__ void umma_commit(unsigned long long* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Work item -> problem, row tile, column tile.
struct Tc3Item {
    int problem, m_tile, n_index;
};
__device__ __forceinline__ Tc3Item tc3_locate(const Tc3Batch& batch, int item)
{
    int pi = 0;
    for (int q = 1; q < batch.count; ++q)
        if (item >= batch.problem[q].tile_begin) pi = q;
    const int local = item - batch.problem[pi].tile_begin;
    return {pi, local / batch.problem[pi].n_tiles, local % batch.problem[pi].n_tiles};
}

// D += A * B with A (128 rows x 8, one TF32 value per column) in tensor memory.
__device__ __forceinline__ void umma_tf32_ts(unsigned tmem_d, unsigned tmem_a, unsigned long long desc_b, unsigned idesc, unsigned accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 32 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_store32(unsigned taddr, const float (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
          "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]), "f"(v[19]),
          "f"(v[20]), "f"(v[21]), "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]), "f"(v[28]), "f"(v[29]),
          "f"(v[30]), "f"(v[31])
        : "memory");
}

// Nearest TF32 value of x (ties away from zero), a float whose low 13 mantissa bits are zero (the residual of an infinity or a NaN is NaN).
__device__ __forceinline__ float tf32_round(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }

__global__ void __launch_bounds__(kT3Threads, 1) tc_gemm_tma_kernel(const __grid_constant__ Tc3Batch batch, int* __restrict__ error_flag)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5;

    unsigned char* a_raw = smem;                                                    // [kT3AStages]
    unsigned char* b_buf = a_raw + kT3AStages * kT3OperandBytes;                    // [kT3Stages][hi, lo]
    unsigned char* c_tile = b_buf + 2 * kT3Stages * kT3OperandBytes;                // [4 column groups][128 rows][128 B]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(c_tile + 4 * kT3OperandBytes);
    unsigned long long* full_a = bars;                       // [2] activation TMA landed (transaction barrier)
    unsigned long long* free_a = full_a + kT3AStages;        // [2] 128 arrivals: the raw tile has been read
    unsigned long long* ready = free_a + kT3AStages;         // [4] weight TMA landed + 128 arrivals: the split tile is written
    unsigned long long* done = ready + kT3Ring;              // [4] tcgen05.commit: the chunk's products are in its accumulator
    unsigned long long* acc_empty = done + kT3Ring;          // [2] 256 arrivals: the accumulator has been read
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(acc_empty + kT3Accumulators);
    volatile int* failed = reinterpret_cast<volatile int*>(acc_empty + kT3Accumulators + 1);

    if (tid == kT3Issue) {
        for (int s = 0; s < kT3AStages; ++s) { mbar_init(&full_a[s], 1); mbar_init(&free_a[s], 128); }
        for (int s = 0; s < kT3Ring; ++s) { mbar_init(&ready[s], 129); mbar_init(&done[s], 1); }
        for (int s = 0; s < kT3Accumulators; ++s) mbar_init(&acc_empty[s], 256);
        *failed = (smem_u32(smem) & 1023u) ? 1 : 0;   // the swizzled layout needs a 1 KB aligned base
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kT3Issue / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(static_cast<unsigned>(kT3Columns)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = *tmem_slot;
    const int first_item = blockIdx.x, item_step = gridDim.x;
    // chunk kc (counted over all work items of this CTA) has left its operand stages and stands in its accumulator.  No role
    // waits here for a chunk that another could overtake by four: each of them feeds or drains the chunks in between.
    auto wait_done = [&](int kc) { return mbar_wait(&done[kc % kT3Ring], static_cast<unsigned>((kc / kT3Ring) & 1), failed); };

    if (warp < 4) {
        // ------------------------------------------------------------- split: high part and residual, a row per thread
        int kc = 0;   // chunks seen by this CTA so far, over all of its work items
        for (int item = first_item; item < batch.total_tiles && !*failed; item += item_step) {
            const Tc3Item it = tc3_locate(batch, item);
            const int chunks = batch.problem[it.problem].K / kTcChunk;
            for (int c = 0; c < chunks; ++c, ++kc) {
                const int sa = kc % kT3AStages;
                // lanes leave a wait one by one; what follows (tcgen05.st) is for whole warps
                if (!__all_sync(0xffffffffu, mbar_wait(&full_a[sa], static_cast<unsigned>((kc / kT3AStages) & 1), failed))) break;
                const unsigned char* src = a_raw + sa * kT3OperandBytes;
                float v[32];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 w = *reinterpret_cast<const float4*>(src + swizzled_offset(tid, q));
                    v[4 * q] = w.x; v[4 * q + 1] = w.y; v[4 * q + 2] = w.z; v[4 * q + 3] = w.w;
                }
                // split tile kc % 3 was last read by chunk kc - 3
                if (!__all_sync(0xffffffffu, kc < kT3SplitStages || wait_done(kc - kT3SplitStages))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned column = tmem_base + (static_cast<unsigned>(warp * 32) << 16) + static_cast<unsigned>(kT3SplitColumn + 64 * (kc % kT3SplitStages));
                // the high part rounded to nearest: the residual has either sign, so that what the tensor core truncates of it
                // has no systematic one
                float hi[32];
#pragma unroll
                for (int q = 0; q < 32; ++q) hi[q] = tf32_round(v[q]);
                tmem_store32(column, hi);
#pragma unroll
                for (int q = 0; q < 32; ++q) v[q] -= hi[q];
                tmem_store32(column + 32u, v);
                // only now have all of the loads returned: behind the loads alone, the arrival can overtake them while the tensor core
                // keeps shared memory busy, and the next tile lands on rows that are still being read
                mbar_arrive(&free_a[sa]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&ready[kc % kT3Ring]);
            }
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------- sums over chunks, epilogue
        // Two warps per quarter of the tensor-memory lanes; of the tile's 32-column groups one takes the even, the other the
        // odd ones.  A lane adds the chunks of its row up in registers.
        const int quarter = warp & 3, half = (warp - 4) >> 2, lane = tid & 31, row = 32 * quarter + lane;
        const bool elected = quarter == 0 && lane == 0;      // issues the stores of its half
        int kc = 0;
        bool ok = true;
        for (int item = first_item; item < batch.total_tiles && ok; item += item_step) {
            const Tc3Item it = tc3_locate(batch, item);
            const Tc3Problem& P = batch.problem[it.problem];
            const int n_tile = P.n_tile, chunks = P.K / kTcChunk;
            float acc[64];
#pragma unroll
            for (int q = 0; q < 64; ++q) acc[q] = 0.0f;
            for (int c = 0; c < chunks; ++c, ++kc) {
                const int b = kc % kT3Accumulators;
                ok = __all_sync(0xffffffffu, wait_done(kc));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int c0 = 64 * g + 32 * half;
                    if (c0 >= n_tile) continue;
                    unsigned v[32];
                    const unsigned taddr = tmem_base + (static_cast<unsigned>(quarter * 32) << 16) + static_cast<unsigned>(b * 128 + c0);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
                          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
                          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr)
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < 32; ++q) asm volatile("" : "+r"(v[q]));   // no use of a register before the wait
#pragma unroll
                    for (int q = 0; q < 32; ++q) acc[32 * g + q] = fmaf(__uint_as_float(v[q]), P.chunk_scale, acc[32 * g + q]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&acc_empty[b]);
            }
            // registers -> the half's column groups of the output tile -> TMA store (or add), which runs on while the next
            // tile is summed up
            if (elected) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the previous tile has been read
            __syncwarp();       // barriers and tensor-memory loads are for whole warps
            half_barrier(half);
            const int col0 = it.n_index * n_tile;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const int c0 = 64 * g + 32 * half;
                if (c0 >= n_tile) continue;
                unsigned char* tile = c_tile + (c0 >> 5) * kT3OperandBytes;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    float4 o = make_float4(acc[32 * g + 4 * q], acc[32 * g + 4 * q + 1], acc[32 * g + 4 * q + 2], acc[32 * g + 4 * q + 3]);
                    if (P.bias != nullptr) {
                        const float4 bv = *reinterpret_cast<const float4*>(P.bias + col0 + c0 + 4 * q);
                        o.x += bv.x; o.y += bv.y; o.z += bv.z; o.w += bv.w;
                    }
                    *reinterpret_cast<float4*>(tile + swizzled_offset(row, q)) = o;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            ok = half_barrier_all(half, ok);    // a warp that gave up takes the other three along
            if (ok && elected) {
                for (int c0 = 32 * half; c0 < n_tile; c0 += 64)
                    tma_store_3d(&P.map_c, c_tile + (c0 >> 5) * kT3OperandBytes, col0 + c0, 0, it.m_tile * P.nodes_per_tile, P.accumulate != 0);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            __syncwarp();
        }
        if (elected) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if (tid == kT3Issue) {
        // ------------------------------------------------------------- tcgen05.mma issue: two waits, 12 MMAs and a commit per chunk
        const unsigned b_addr = smem_u32(b_buf);
        int kc = 0;
        if (!*failed) {
            bool ok = true;
            for (int item = first_item; item < batch.total_tiles && ok; item += item_step) {
                const Tc3Item it = tc3_locate(batch, item);
                const int NT = batch.problem[it.problem].n_tile, chunks = batch.problem[it.problem].K / kTcChunk;
                // instruction descriptor: D = F32, A = B = TF32, both K-major, N = NT, M = 128
                const unsigned idesc = (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<unsigned>(NT >> 3) << 17) |
                                       (static_cast<unsigned>(kTcRows >> 4) << 24);
                for (int c = 0; c < chunks; ++c, ++kc) {
                    const int s = kc % kT3Stages, b = kc % kT3Accumulators;
                    // the accumulator has been read (chunk kc - 2); the weights landed and the split tile is written
                    if ((kc >= kT3Accumulators && !mbar_wait(&acc_empty[b], static_cast<unsigned>((kc / kT3Accumulators - 1) & 1), failed))
                        || !mbar_wait(&ready[kc % kT3Ring], static_cast<unsigned>((kc / kT3Ring) & 1), failed)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned tmem_d = tmem_base + static_cast<unsigned>(b * 128);
                    const unsigned a_hi = tmem_base + static_cast<unsigned>(kT3SplitColumn + 64 * (kc % kT3SplitStages)), a_lo = a_hi + 32u;
                    const unsigned long long db_hi = umma_desc(b_addr + (2 * s) * kT3OperandBytes);
                    const unsigned long long db_lo = umma_desc(b_addr + (2 * s + 1) * kT3OperandBytes);
                    // the small products first: every addition in the tensor core truncates
#pragma unroll
                    for (int ks = 0; ks < kTcChunk / 8; ++ks) {
                        const unsigned long long step = static_cast<unsigned long long>(ks * 2);   // 32 bytes along K
                        umma_tf32_ts(tmem_d, a_hi + 8u * ks, db_lo + step, idesc, ks > 0 ? 1u : 0u);
                        umma_tf32_ts(tmem_d, a_lo + 8u * ks, db_hi + step, idesc, 1u);
                    }
#pragma unroll
                    for (int ks = 0; ks < kTcChunk / 8; ++ks) {
                        const unsigned long long step = static_cast<unsigned long long>(ks * 2);
                        umma_tf32_ts(tmem_d, a_hi + 8u * ks, db_hi + step, idesc, 1u);
                    }
                    umma_commit(&done[kc % kT3Ring]);
                }
            }
        }
    } else if (tid == kT3Issue + 32) {
        // ------------------------------------------------------------- weight TMA
        int issued = 0;
        if (!*failed) {
            bool ok = true;
            for (int item = first_item; item < batch.total_tiles && ok; item += item_step) {
                const Tc3Item it = tc3_locate(batch, item);
                const Tc3Problem& P = batch.problem[it.problem];
                const unsigned bytes = 2u * static_cast<unsigned>(P.n_tile) * 128u;
                const int chunks = P.K / kTcChunk, n0 = it.n_index * P.n_tile;
                for (int c = 0; c < chunks; ++c) {
                    const int s = issued % kT3Stages;
                    if (issued >= kT3Stages && !wait_done(issued - kT3Stages)) { ok = false; break; }
                    unsigned char* hi = b_buf + (2 * s) * kT3OperandBytes;
                    const int k0 = c * kTcChunk;
                    unsigned long long* bar = &ready[issued % kT3Ring];
                    mbar_expect_tx(bar, bytes);
                    tma_load_2d(hi, &P.map_hi, bar, k0, n0);
                    tma_load_2d(hi + kT3OperandBytes, &P.map_lo, bar, k0, n0);
                    ++issued;
                }
            }
            // after a failure: let the copies still in flight land before the CTA exits
            if (*failed)
                for (int q = max(0, issued - kT3Stages); q < issued; ++q) {
                    int never = 0;
                    mbar_wait(&ready[q % kT3Ring], static_cast<unsigned>((q / kT3Ring) & 1), &never);
                }
        }
    } else if (tid == kT3Issue + 64) {
        // ------------------------------------------------------------- activation TMA
        int issued = 0;
        if (!*failed) {
            bool ok = true;
            for (int item = first_item; item < batch.total_tiles && ok; item += item_step) {
                const Tc3Item it = tc3_locate(batch, item);
                const Tc3Problem& P = batch.problem[it.problem];
                const unsigned bytes = static_cast<unsigned>(P.rows_per_tile) * 128u;
                const int chunks = P.K / kTcChunk, node0 = it.m_tile * P.nodes_per_tile;
                for (int c = 0; c < chunks; ++c) {
                    const int s = issued % kT3AStages, use = issued / kT3AStages;
                    if (use > 0 && !mbar_wait(&free_a[s], static_cast<unsigned>((use - 1) & 1), failed)) { ok = false; break; }
                    mbar_expect_tx(&full_a[s], bytes);
                    tma_load_3d(a_raw + s * kT3OperandBytes, &P.map_a, &full_a[s], c * kTcChunk, 0, node0);
                    ++issued;
                }
            }
            if (*failed)
                for (int q = max(0, issued - kT3AStages); q < issued; ++q) {
                    int never = 0;
                    mbar_wait(&full_a[q % kT3AStages], static_cast<unsigned>((q / kT3AStages) & 1), &never);
                }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *failed) atomicOr(error_flag, 2);
    if (warp == kT3Issue / 32) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<unsigned>(kT3Columns)) : "memory");
    }
}

}  // namespace sxb
