// Side metadata of a planned SpMV launch ("plan"): the rows of a compressed matrix cut into virtual rows of
// bounded length, sorted by length. It is derived from row_indices and deltas once per matrix and leaves the
// three MACKO buffers untouched (the reference has no such structure: its kernel walks one row per warp,
// src/macko_spmv/cuda/kernels.cuh:41-60).
//
// A virtual row is a run of stored elements of one row: the whole row when it is short, else a segment
// [a0 + j*S, a0 + (j+1)*S) of it, a0 = the row's first element rounded down to a multiple of 8, so that every
// segment but the first starts on an 8-element unit. For each one the plan keeps where it starts, how long it
// is, the column sum in front of it (sum of delta + 1 over the row's elements before the segment: what the
// decode needs to continue in the middle of a row) and where its result goes.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace macko {

// x in shared memory is framed by zeros
constexpr int kXPadFront = 32;       // fp16 slots in front of x[0] (64 bytes: keeps x 16B-aligned)
constexpr int kXPadBack = 160;       // fp16 slots after x[cols-1]  (> 8 * 16 + 8)

constexpr int kPlanLenBits = 12;                         // a virtual row holds fewer than 4096 stored elements
constexpr int kPlanMaxSegment = 3840;                    // largest segment length (a multiple of 256)
constexpr int kPlanBuckets = 64;                         // length classes: 64-element sub-steps spanned, 0..60
constexpr unsigned kPlanPartialBit = 0x80000000u;        // destination word: a partial-sum slot, not a row of y

// Pointers into a plan buffer, as the SpMV kernel sees it.
struct PlanView {
    const uint2 *desc;      // sorted: {first stored element, length | column sum in front << kPlanLenBits}
    const unsigned *out;    // sorted: row of y, or kPlanPartialBit | natural index of the segment
    const unsigned *vrow;   // natural order: row of each virtual row
    float *partial;         // natural order: fp32 sums of the segments of rows cut into several
    const int *seg_first;   // [rows + 1] natural index of the first virtual row of each row
    const unsigned *split_list;   // rows cut into several segments (in no particular order)
    int n_split;
    int n_virtual;
};

// Byte offsets of the sections of a plan buffer for a matrix of `rows` rows and `padded` stored elements cut
// into segments of `seg` elements. Pure arithmetic, shared by the builder and the launcher.
struct PlanLayout {
    long long v_max;        // upper bound of the number of virtual rows
    long long header, seg_first, split_list, desc, out, vrow, partial, tmp_begin, tmp_pk, tmp_out, block_hist, total;
};

inline PlanLayout plan_layout(long long rows, long long padded, int seg)
{
    auto up = [](long long b) { return (b + 255) & ~255LL; };
    PlanLayout l{};
    // every row gives at least one virtual row; a row of n elements starting at offset o (< 8) inside its first
    // unit gives ceil((o + n) / seg) <= 1 + (n + 7) / seg
    l.v_max = rows + (padded + 8 * rows) / seg + 1;
    const long long blocks = (l.v_max + 1023) / 1024;
    long long at = 0;
    l.header = at;      at = up(at + 64);
    l.seg_first = at;   at = up(at + 4 * (rows + 1));
    l.split_list = at;  at = up(at + 4 * (rows + 1));
    l.desc = at;        at = up(at + 8 * l.v_max);
    l.out = at;         at = up(at + 4 * l.v_max);
    l.vrow = at;        at = up(at + 4 * l.v_max);
    l.partial = at;     at = up(at + 4 * l.v_max);
    l.tmp_begin = at;   at = up(at + 4 * l.v_max);
    l.tmp_pk = at;      at = up(at + 4 * l.v_max);
    l.tmp_out = at;     at = up(at + 4 * l.v_max);
    l.block_hist = at;  at = up(at + 4 * (blocks + 1) * kPlanBuckets);
    l.total = at;
    return l;
}

// Virtual rows that a planned launch walks at once: four per resident warp, with 32 warps on an SM while two CTAs hold x
// in its shared memory, else 16. The number of SMs is that of a B200 and not asked for: macko_spmv_plan_bytes has to
// agree with the builder and may be called where no device is.
constexpr long long kPlanTwoCtaCols = (227 * 1024 / 2 - 1024) / 2 - kXPadFront - kXPadBack;   // 57408: what launch_variant works out
inline long long plan_groups(long long cols) { return 148LL * 4 * (cols <= kPlanTwoCtaCols ? 32 : 16); }

// Segment length where the caller names none. A group of lanes gets a share of padded / plan_groups elements: a
// segment a little longer than the share leaves one long segment per group and the short rows to even the ends out,
// a much longer one leaves groups without work while others walk it, a much shorter one costs a hand-over and a
// partial sum each time. Above about 1088 elements per group a fixed 1536 is as good as any choice. Skewed matrices of
// mean density 0.2 (B200, graph of products, us, this rule / always 1536): 4879x7688 (share 474) 13.8 / 19.5,
// 12000x4096 (617) 14.5 / 19.9, 16000x4096 (822) 16.8 / 20.7, 4096x16384 (858) 20.9 / 23.7, 9000x9000 (1032)
// 20.6 / 22.5. With one CTA per SM (shares of twice the size; this rule / the segment for 32 warps / always 1536):
// 300x100000 (794) 23.7 / 32.0 / 25.8, 400x65536 (684) 14.8 / 18.7 / 18.0.
inline int plan_default_segment(long long padded, long long cols)
{
    const long long share = padded / plan_groups(cols);
    if (share > 1088) return 1536;
    const long long seg = (share + 16 + 255) / 256 * 256;
    return (int)(seg < 512 ? 512 : seg);
}

// When a plan of cut rows is recommended: either a group's share is kPlanMinShare elements or more, or the lanes that walk
// the longest row in the default launch take kPlanMinChain sub-steps or more over it (0.2 us each, whatever the rest of
// the chip does). Smaller matrices without such a row are done before the balance pays for the hand-overs and the second
// kernel. Default launch / plan (us) by share and sub-steps, B200, graph of products of rotating matrices:
//   neither     skewed, mean density 0.2: 5504x3200 (221, 25) 9.7 / 10.9, 2000x8192 (210, 32) 10.8 / 12.3, 3000x8192 (314, 32)
//               11.9 / 13.4, 3000x9000 (345, 35) 12.5 / 13.7; 4096x8192, 20 dense rows among d = 0.1 (224, 32) 11.4 / 10.9
//   long row    skewed: 1200x11008 (168, 43) 13.5 / 12.4, 2400x11008 (335, 43) 14.6 / 14.1, 2048x13184 (344, 51) 15.8 / 14.6, 1400x16384
//               (298, 64) 18.1 / 15.1, 400x65536 (684, 256) 58.9 / 14.8; dense rows among empty or sparse ones: 20 of 512x65536
//               (138, 256) 58.7 / 11.6, 200 of 900x30000 (316, 117) 30.3 / 17.1, 20 of 20000x4096 (313, 64) 18.1 / 10.7
//   large       skewed: 20000x1500 (373, 23) 14.0 / 11.6, 5000x6000 (381, 23) 14.4 / 13.2, 6000x5000 (380, 39) 14.4 / 12.6, but
//               3500x8500 (377, 33) 12.9 / 13.8 and 3072x18304 20.7 / 22.3: the share alone does not tell these apart
constexpr long long kPlanMinShare = 365;
constexpr long long kPlanMinChain = 40;

// Length class of a virtual row: 64-element sub-steps between the unit its first element sits in and its end.
__host__ __device__ inline int plan_length_class(int begin, int len)
{
    return ((begin & 7) + len + 63) >> 6;
}

}  // namespace macko
