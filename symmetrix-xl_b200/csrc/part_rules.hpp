// How many parts the edge kernels deal a receiver's edges to (edge_part in edge_kernels.cuh).  Host arithmetic without CUDA.
//
// A receiver is a serial chain of its edges, so with fewer receivers than the chip holds blocks (or warps) a kernel lasts as
// long as one chain.  What a rule needs of its kernel is how many blocks or warps of it are resident on an SM, by registers
// (65,536), shared memory (228 KB) and blocks (32).  Times below: us a launch, B200, medium model (97 list edges a receiver)
// unless said otherwise.
#pragma once

#include <algorithm>
#include <cmath>

namespace sxb {

// Time of `units` receivers of `edges` list edges each in `parts` parts on `slots` resident blocks or warps, in edges: a part
// costs its edges plus `overhead` edges' worth of prologue, chunk fill and reductions.  Up to a few rounds of the chip the last
// round is counted whole (a chain in it takes as long as any other), beyond that half of it.
inline double parts_cost(long units, double slots, double edges, double overhead, int parts)
{
    const double rounds = static_cast<double>(units) * parts / slots;
    return (rounds < 4.0 ? std::ceil(rounds) : rounds + 0.5) * (edges / parts + overhead);
}

// The best of 1, step, step^2, ... `most` parts; more parts have to bring the cost below `gain` of what it was.
inline int edge_parts(long units, double slots, double edges, double overhead, double gain, int step, int most)
{
    int best = 1;
    for (int parts = step; parts <= most; parts *= step)
        if (parts_cost(units, slots, edges, overhead, parts) < gain * parts_cost(units, slots, edges, overhead, best)) best = parts;
    return best;
}

// Resident blocks of the layer-1 gradient on channel pairs: what its launch bounds ask for, 0e+1o and 0e+1o+2e.
constexpr int kPairBlocksS1 = 2, kPairBlocksS2 = 1;

struct PartRules {
    int num_sms, channels, shape;      // shape: 0 hidden 0e, 1 0e+1o, 2 0e+1o+2e
    double edges;                      // mean list edges of a receiver

    int block_warps() const { return std::max(1, channels / 32); }

    // Layer-0 sums: a build for one warp and one for the four warps of a block per receiver, and nothing between them.  Resident
    // warps 16, 32 and 40 at 128, 64 and 32 channels (128, 64 and 48 registers).  One / four, 128 channels: 40 receivers 46 / 20,
    // 1,080: 59 / 46, 2,160: 76 / 82, 2,560: 109 / 97, 5,000: 176 / 174, 7,200: 222 / 238; 64 channels, where a part costs more
    // beside its edges: 2,160: 72 / 64, 3,240: 77 / 85, 7,560: 137 / 166.
    int l0_forward(long receivers) const
    {
        const int resident = channels == 128 ? 16 : channels == 64 ? 32 : 40;
        return edge_parts(receivers, 1.0 * num_sms * resident, edges, channels == 64 ? 11.0 : 5.0, 0.9, 4, 4);
    }

    // Layer-0 gradient: resident warps 12, 16 and 20 at 128, 64 and 32 channels (168 registers; 54 and 39 KB a block of four).
    // 1 / 2 / 4 / 8 parts, 128 channels: 40 receivers 66 / 39 / 25 / 17, 600: 72 / 48 / 50 / 48, 2,160: 138 / 119 / 123 / 142,
    // 5,000: 243 / 248 / 271 / 312; 64 channels, 1,500: 68 / 68 / 64 / 70; 32 channels (hidden 0e, 58 edges), 1,080: 35 / 29 /
    // 31 / 33.
    int l0_reverse(long receivers) const
    {
        const int resident = channels == 128 ? 12 : channels == 64 ? 16 : 20;
        return edge_parts(receivers, 1.0 * num_sms * resident, edges, 4.0, 0.95, 2, 8);
    }

    // Layer 0 on the radial functions (edge_kernels_basis.cuh, two kernels more than on the folded table) or on the table: sums and
    // gradient together, us, table / functions, 128 channels, three types: 320 receivers 54 / 63, 500: 73 / 68, 720: 96 / 75, 1,260:
    // 137 / 97, 5,000: 415 / 220; 64 channels: 500: 56 / 63, 600: 66 / 67, 720: 70 / 70, 1,260: 106 / 92.  The work of the functions grows
    // with the types: 5,000 receivers with 4, 6 and 8 types 457 / 257, 464 / 345, 468 / 411, 20,000 with ten 1,731 / 1,675.
    bool layer0_on_basis(long receivers, int types) const { return types <= 10 && receivers >= (channels == 128 ? 150l : 230l) * types; }

    // Layer-0 gradient on the radial functions: a warp per receiver (1) when that fills the twelve resident warps of every SM,
    // otherwise one per (receiver, source type) and part of whole steps of 16 edges (a run has 15 to 45 edges in the medium model).
    int l0_moments_reverse(long receivers, int types) const
    {
        const long slots = 12l * num_sms;
        if (receivers >= slots) return 1;
        return types * static_cast<int>(std::max(1l, std::min(4l, slots / std::max(1l, receivers * types))));
    }

    // Layer-1 sums, whose parts meet in a cluster: as many as fill the chip once, at most five blocks on an SM (placing the
    // blocks of more clusters takes longer than the chains they shorten).  1 / 2 / 4 / 8 parts, 128 channels: 40 receivers 39 /
    // 35 / 23 / 18, 320: 51 / 64 / 64 / 70; 64 channels, 160: 39 / 37 / 27 / 31; hidden 0e (58 edges) at 32 channels, 160: 21 /
    // 17 / 13 / 15, 600: 21 / 27 / 27 / 31, at 128 channels, 160: 27 / 21 / 17 / 21.
    int l1_forward(long receivers) const
    {
        const long slots = static_cast<long>(num_sms) * std::min(5, (shape == 0 ? 32 : 16) / block_warps());
        int parts = 1;
        while (parts < 8 && receivers * parts * 2 <= slots) parts *= 2;
        return parts;
    }

    // Layer-1 gradient on channel pairs with the row adjoints in tensor memory (edge_kernels_pairs.cuh) at the common widths of
    // hidden l > 0, or one channel per thread with the adjoints in registers.
    bool l1_reverse_paired() const { return shape == 2 || (shape == 1 && (channels == 128 || channels == 64)); }

    // Parts of that gradient: on channel pairs, `resident` blocks of it on an SM.  A block has eight or twelve warps, a part costs more
    // beside its edges than with a few warps: no more blocks than fill the chip about twice.  1 / 2 / 4 / 8 parts, 128 channels: 40
    // receivers 38 / 25 / 23 / 23, 160: 50 / 44 / 44 / 50, 320: 72 / 66 / 70 / 87, 600: 111 / 109 / 119 / 154, 1,080: 173 / 179 / 204 /
    // 267, 5,000: 699 / 762 / 904 / 1,308; 64 channels, 40: 23 / 17 / 17 / 19, 320: 44 / 42 / 50 / 68, 1,080: 97 / 105 / 136 / 199;
    // 0e+1o+2e, 40: 56 / 35 / 37 / 38, 160: 85 / 80 / 83 / 103, 600: 220 / 236 / 275 / 359.
    int l1_reverse_pairs(long receivers, int resident) const
    {
        int parts = edge_parts(receivers, 1.0 * num_sms * resident, edges, 8.0, 0.95, 2, 8);
        while (parts > 1 && 1.0 * receivers * parts > 2.2 * num_sms * resident) parts /= 2;
        return parts;
    }

    // Either; with the adjoints in registers, hidden 0e: 128 registers and 26 KB a block, eight blocks of up to two
    // warps, four of four.  1 / 2 / 4 / 8 parts, 32 channels (58 edges), 40 receivers: 31 / 21 / 15 / 13, 600: 35 / 33 / 33 / 35,
    // 1,080: 37 / 39 / 45 / 56, 1,500: 60 / 54 / 60 / 72.  0e+1o (widths without a paired kernel): counted with 12 warps; its
    // records at 128 channels, 40: 68 / 39 / 29 / 27, 600: 201 / 177 / 176 / 199, 1,080: 293 / 293 / 308 / 353.
    int l1_reverse(long receivers) const
    {
        if (l1_reverse_paired()) return l1_reverse_pairs(receivers, shape == 2 ? kPairBlocksS2 : kPairBlocksS1);
        const int resident = shape == 0 ? std::min(8, 16 / block_warps()) : 12 / block_warps();
        return edge_parts(receivers, 1.0 * num_sms * std::max(1, resident), edges, 5.0, 0.95, 2, 8);
    }
};

// Warps that share a receiver's stencil in the neighbor search: as many as the chip holds at once, about half full.  The whole
// build in us with 1 / 2 / 4 / 8 / 16: 40 receivers 179 / 173 / 138 / 136 / 133, 120: 162 / 144 / 138 / 138 / 136, 320: 167 / 153 /
// 143 / 141 / 147, 1,080: 195 / 173 / 170 / 170 / 179, 2,160: 205 / 197 / 197 / 202 / 228, 5,000: 275 / 270 / 277 / 302 / 349,
// 20,480: 597 / 617 / 671 / 774 / 985.
inline int stencil_parts(long receivers, int num_sms)
{
    int parts = 1;
    while (parts < 8 && 2 * parts * receivers <= 32l * num_sms) parts *= 2;
    return parts;
}

}  // namespace sxb
