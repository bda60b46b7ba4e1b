// GPU compressor producing MACKO buffers bit-identical to the reference host encoder
// `compress_rows_cpu` (src/macko_spmv/cuda/cpu_compressor.cuh:6-73).
//
// The reference walks every row with a running zero counter. The same output follows from a
// closed form that parallelises: a true non-zero at column c whose previous non-zero of the
// row (or -1) is at c0 has gap g = c - c0 - 1; it emits floor(g/16) pads, sitting on columns
// c0+16, c0+32, ... (value = the +-0 found there, delta 15), then itself with delta g mod 16.
// Zeros after the last non-zero of a row emit nothing. NaNs are stored as 0x7fff, -0.0 counts
// as zero (cpu_compressor.cuh:26-27,36).
//
// Phase 1 (count):  one warp per row -> stored elements per row -> prefix sum = row_indices.
// Phase 2 (emit):   one warp per row -> values and packed deltas in one pass.
// A warp reads 256 columns per step (one 128-bit load per lane, aligned on the matrix
// allocation, not on the row, so odd column counts still use vector loads).
//
// The reference's int8 encoder (src/macko_spmv/cuda/cpu_compressor.cuh:75-117) differs in two ways: a value is
// one signed byte, and trailing pads stay: a run of t zeros at the end of a row (or a whole empty row, t = cols)
// still emits floor(t / 16) pads (value 0, delta 15). Both encoders are instantiations of the same two kernels.
#include "common.cuh"

namespace macko {
namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kThreads = kWarpsPerCta * 32;
constexpr int kColsPerLane = 8;
constexpr int kColsPerStep = 32 * kColsPerLane;
constexpr int kUnroll = 4;        // steps whose loads are in flight together

// Warps of the emit kernel that had to refuse a store because row_indices pointed beyond the padded count they
// were given: non-zero means that the outputs of that call are incomplete.
// Per device, read and cleared by macko_compress_overflow().
static __device__ unsigned g_compress_overflow;

// Bit i set <=> element g0 + i lies inside the row [lo, hi).
__device__ __forceinline__ unsigned row_bits(unsigned g0, unsigned lo, unsigned hi)
{
    const unsigned a = g0 >= lo ? 0u : min(lo - g0, 8u), b = g0 >= hi ? 0u : min(hi - g0, 8u);
    return ((1u << b) - 1u) & ~((1u << a) - 1u);
}

// The 8 elements of a lane as they come from memory: 16-bit values (fp16 or bf16 bits) or int8 bytes.
template <bool I8> struct Raw { using Element = unsigned short; using Vec = uint4; };
template <> struct Raw<true> { using Element = unsigned char; using Vec = uint2; };

// Elements [g0, g0 + 8), known to lie in the allocation and to be aligned.
template <bool I8>
__device__ __forceinline__ typename Raw<I8>::Vec load8_inside(const typename Raw<I8>::Element *dense, unsigned g0)
{
    return __ldg(reinterpret_cast<const typename Raw<I8>::Vec *>(dense + g0));
}
// Loads elements [g0, g0 + 8) of the matrix; what lies outside the row [row_lo, row_hi) may hold anything and is
// cleared by clear_outside(). g0 is a multiple of 8 on the vector path, so the load is aligned on the allocation.
template <bool I8>
__device__ __forceinline__ typename Raw<I8>::Vec load8(const typename Raw<I8>::Element *dense, unsigned g0, unsigned row_lo,
                                                       unsigned row_hi, unsigned total, bool vec_ok)
{
    using Vec = typename Raw<I8>::Vec;
    Vec v{};
    if (g0 < row_hi) {
        if (vec_ok && g0 + 8u <= total) {
            v = __ldg(reinterpret_cast<const Vec *>(dense + g0));
        } else {
            unsigned *w = reinterpret_cast<unsigned *>(&v);
            constexpr int kPerWord = I8 ? 4 : 2;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (g0 + j >= row_lo && g0 + j < row_hi)
                    w[j / kPerWord] |= (unsigned)__ldg(dense + g0 + j) << ((32 / kPerWord) * (j % kPerWord));
        }
    }
    return v;
}

// The 8 elements as four words of two 16-bit fields (int8 bytes zero-extended).
template <bool I8>
__device__ __forceinline__ void words_of(const typename Raw<I8>::Vec &v, unsigned (&w)[4])
{
    if constexpr (I8) {
        w[0] = __byte_perm(v.x, 0u, 0x4140); w[1] = __byte_perm(v.x, 0u, 0x4342);
        w[2] = __byte_perm(v.y, 0u, 0x4140); w[3] = __byte_perm(v.y, 0u, 0x4342);
    } else {
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
}
// Zeroes the fields whose element (g0 + index) lies outside the row: the first and the last lanes of a row.
__device__ __forceinline__ void clear_outside(unsigned (&w)[4], unsigned g0, unsigned row_lo, unsigned row_hi)
{
    if (g0 < row_lo || g0 + 8u > row_hi) {
        const unsigned in = row_bits(g0, row_lo, row_hi);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            w[j] &= (((in >> (2 * j)) & 1u) * 0xffffu) | (((in >> (2 * j + 1)) & 1u) * 0xffff0000u);
    }
}

// Non-zero fields of the four words, bits out of order (for counting): +-0 is the only field whose low 15 bits
// are zero, and adding 0x7fff to them carries into bit 15 of the field exactly when they are not. An int8 byte
// is zero-extended and never touches bit 15.
__device__ __forceinline__ unsigned nonzero_fields(const unsigned (&w)[4])
{
    unsigned f = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) f |= (((w[j] & 0x7fff7fffu) + 0x7fff7fffu) >> (6 - 2 * j)) & (0x80008000u >> (6 - 2 * j));
    return f;
}
// The same in order: bit i set <=> element i is not zero.
__device__ __forceinline__ unsigned ordered_bits(unsigned fields)
{
    return ((fields >> 9) & 0x55u) | ((fields >> 24) & 0xaau);
}

// Column (row-relative) of the last non-zero strictly before this lane's 8 columns.
__device__ __forceinline__ int prev_nonzero_before_lane(unsigned any, int lane, int my_last_col, int carry)
{
    const unsigned lower = any & ((1u << lane) - 1u);
    const int src = lower ? 31 - __clz(lower) : lane;
    const int got = __shfl_sync(0xffffffffu, my_last_col, src);
    return lower ? got : carry;
}

// Stored elements of every row: its non-zeros plus floor(gap / 16) pads for every run of zeros in front of one
// (int8: also for the run at the end of the row). 16 zeros in a row cover a whole aligned group of 8 columns, so in
// a step in which every lane has seen a non-zero only the run in front of the step can reach 16, and it does not
// when the last lane of the step before has seen one too: such a short step only adds up its non-zeros (7 of 8
// steps of an iid mask of density 0.5); the others look at the gaps.
// Bound by HBM and the loads in flight: 11008x4096 at density 0.5 (90 MB) in 21.5 us (4.2 TB/s); 26.8 us when every
// step looked at the gaps and every load was guarded.
constexpr int kCarryInLast = -0x7fffffff;
template <bool I8>
__global__ void __launch_bounds__(kThreads)
count_rows_kernel(const typename Raw<I8>::Element *__restrict__ dense, int rows, int cols, bool vec_ok, int rows_per_warp, int *__restrict__ counts)
{
    asm volatile("griddepcontrol.launch_dependents;");
    const int lane = threadIdx.x & 31;
    const unsigned first_row = (blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5)) * (unsigned)rows_per_warp;
#pragma unroll 1
    for (unsigned row = first_row; row < min(first_row + (unsigned)rows_per_warp, (unsigned)rows); ++row) {
        // element indices fit 32 bits: the entry points refuse matrices of 2^31 elements or more, and a walk ends
        // less than 2048 elements behind its row
        const unsigned total = (unsigned)rows * (unsigned)cols;
        const unsigned row_lo = row * (unsigned)cols;
        const unsigned row_hi = row_lo + (unsigned)cols;
        // The first step starts at the 8-element boundary at or below the row start.
        const unsigned first = vec_ok ? (row_lo & ~7u) : row_lo;
        int count = 0;          // stored elements seen by this lane
        int carry = -1;         // column of the last non-zero seen so far in this row, unless the last step was a short one:
        unsigned last = 0u;     // then it is the last of lane 31's `last` fields, whose first column is `last_c0`
        int last_c0 = 0;
        bool ends_dense = true; // at most 7 zeros lie between the last non-zero (the row's start) and the next step
        for (unsigned group0 = first; group0 < row_hi; group0 += (unsigned)(kUnroll * kColsPerStep)) {
            // all loads of kUnroll steps are issued before the first one is consumed
            typename Raw<I8>::Vec v[kUnroll];
            const bool inner = vec_ok && group0 >= row_lo && group0 + (unsigned)(kUnroll * kColsPerStep) <= row_hi;   // warp-uniform
            if (inner) {
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) v[u] = load8_inside<I8>(dense, group0 + (unsigned)(u * kColsPerStep + lane * kColsPerLane));
            } else {
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
                    v[u] = load8<I8>(dense, group0 + (unsigned)(u * kColsPerStep + lane * kColsPerLane), row_lo, row_hi, total, vec_ok);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const unsigned step0 = group0 + (unsigned)(u * kColsPerStep), g0 = step0 + (unsigned)(lane * kColsPerLane);
                if (!inner && step0 >= row_hi) break;   // warp-uniform
                unsigned w[4];
                words_of<I8>(v[u], w);
                if (!inner) clear_outside(w, g0, row_lo, row_hi);
                const unsigned fields = nonzero_fields(w);
                count += __popc(fields);
                const unsigned any = __ballot_sync(0xffffffffu, fields != 0u);
                const int step_c0 = (int)(step0 - row_lo);   // may be negative on the first step
                if (any == 0xffffffffu && ends_dense) {
                    last = fields;
                    last_c0 = step_c0 + 31 * kColsPerLane;
                    carry = kCarryInLast;
                    continue;
                }
                if (carry == kCarryInLast) carry = last_c0 + 31 - __clz(ordered_bits(__shfl_sync(0xffffffffu, last, 31)));
                ends_dense = (int)any < 0;   // lane 31
                if (any == 0u) continue;
                const int c0 = step_c0 + lane * kColsPerLane;
                const unsigned nz = ordered_bits(fields);
                const int my_last = c0 + (31 - __clz(nz | 1u));
                const int prev = prev_nonzero_before_lane(any, lane, my_last, carry);
                if (nz) count += (c0 + (__ffs(nz) - 1) - prev - 1) >> 4;
                carry = __shfl_sync(0xffffffffu, my_last, 31 - __clz(any));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
        if constexpr (I8) {
            if (carry == kCarryInLast) carry = last_c0 + 31 - __clz(ordered_bits(__shfl_sync(0xffffffffu, last, 31)));
            count += (cols - 1 - carry) >> 4;
        }
        if (lane == 0) counts[row + 1] = count;
    }
}

// ---- emit: values and packed deltas in one pass ----------------------------------------------------------
// A warp walks its row, 16 columns per lane and step. What a step stores is appended to a ring in shared memory,
// one 32-bit entry per stored element (value bits, column mod 16 << 16) at ring slot (output slot mod 1024), so that
// an element costs one store and the ring never moves. The delta of an element is (column - column of the stored
// element in front of it - 1) mod 16, for pads as well, and is formed for 8 elements at once when they leave.
// Whenever 512 slots are waiting, each lane takes two groups of 8: the values leave as one vector store, their 8
// deltas packed into one 32-bit store. The first and the last group of a row may be shared with the neighbouring rows
// (rows start at arbitrary slots): their values leave one by one and their nibbles are merged into the word with
// atomicOr, which is why the caller clears `deltas` before the launch. Pads: only a lane's first non-zero of a step can
// have pads in front of it (later ones are less than 16 columns apart). The run in front of the first non-zero of the
// whole step can be as long as the row and is written by the warp together, 512 pads at a time; the others (at most 31
// per step) by their lane. The warp of the last row also clears values[n, P).
// Bound by instruction issue (70 % of the slots at 32 warps per SM): 11008x4096 at density 0.5 takes 41.5 us (146 MB)
// with 31.7 M warp instructions, against 66 us and 58 M with 8 columns per lane, separate 2-byte and 1-byte ring stores
// and the deltas counted element by element. Five CTAs per SM instead of four cost registers that spill (45.9 us).
// int8 values, whole call: 11008x4096 at density 0.5 84 us, 32000x4096 at 0.1 202 us; 156 and 423 us with one delta per
// byte in scratch memory and a packing kernel.
// Output slots are unsigned: with a padded count close to 2^31 the slots that a row counts up to (row_indices that do not
// belong to the matrix) and the last step of the clearing loop lie beyond it, and are refused there, not taken for negative ones.
constexpr int kEmitCols = 16;   // columns per lane and step: a warp takes 512 columns
constexpr int kRing = 1024;     // slots; a power of two. At most 511 wait, and a step or a batch of pads adds at most 512.
constexpr int kFlush = 512;     // slots that leave together: two groups of 8 per lane

struct EmitRing {
    unsigned *e;        // the ring: value | (column mod 16) << 16
    unsigned out;       // next output slot (warp-uniform)
    unsigned flushed;   // output slots below this have left; a multiple of 8 (warp-uniform)
    unsigned own_lo;    // first output slot that belongs to this row
    bool refused;
};

// Writes out slots [r.flushed, r.flushed + n), n <= 512, a group of 8 per lane at a time; n % 8 != 0 only for the last ones of a row.
template <bool I8>
__device__ __forceinline__ void ring_flush(EmitRing &r, typename Raw<I8>::Element *__restrict__ values,
                                           unsigned *__restrict__ deltas32, unsigned n, unsigned limit, bool vec_v, int lane)
{
    __syncwarp();
    for (unsigned at = 8u * (unsigned)lane; at < n; at += 256u) {
        const unsigned slot0 = r.flushed + at;
        const int lo = max((int)(r.own_lo - slot0), 0), hi = (int)min(n - at, 8u);   // the entries of the group that are this row's
        const uint4 a = *reinterpret_cast<const uint4 *>(r.e + (slot0 & (kRing - 1)));
        const uint4 b = *reinterpret_cast<const uint4 *>(r.e + (slot0 & (kRing - 1)) + 4);
        const unsigned before = r.e[(slot0 - 1u) & (kRing - 1)];
        const unsigned e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        unsigned col[2];   // 4 nibbles each: (column mod 16) of the entries
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const unsigned t = (__byte_perm(e[4 * j], e[4 * j + 1], 0x7632) & 0x000f000fu) + ((__byte_perm(e[4 * j + 2], e[4 * j + 3], 0x7632) & 0x000f000fu) << 8);
            col[j] = t | (t >> 12);
        }
        const unsigned now = __byte_perm(col[0], col[1], 0x5410);
        // nibble-wise now - previous - 1 = now + ~previous (ring entries of another row hold anything, and are masked out)
        const unsigned not_prev = ~((now << 4) | ((before >> 16) & 15u));
        const unsigned packed = ((now & 0x77777777u) + (not_prev & 0x77777777u)) ^ ((now ^ not_prev) & 0x88888888u);
        if (lo <= 0 && hi == 8 && slot0 + 8u <= limit) {
            if constexpr (I8) {
                uint2 o;
                o.x = __byte_perm(__byte_perm(e[0], e[1], 0x0040), __byte_perm(e[2], e[3], 0x0040), 0x5410);
                o.y = __byte_perm(__byte_perm(e[4], e[5], 0x0040), __byte_perm(e[6], e[7], 0x0040), 0x5410);
                if (vec_v) {
                    *reinterpret_cast<uint2 *>(values + slot0) = o;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) values[slot0 + j] = (unsigned char)e[j];
                }
            } else {
                if (vec_v) {
                    *reinterpret_cast<uint4 *>(values + slot0) =
                        make_uint4(__byte_perm(e[0], e[1], 0x5410), __byte_perm(e[2], e[3], 0x5410),
                                   __byte_perm(e[4], e[5], 0x5410), __byte_perm(e[6], e[7], 0x5410));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) values[slot0 + j] = (unsigned short)e[j];
                }
            }
            deltas32[slot0 >> 3] = packed;
        } else if (lo < hi) {
            unsigned mask = 0xffffffffu << (4 * lo);
            if (hi < 8) mask &= ~(0xffffffffu << (4 * hi));
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= lo && j < hi) {
                    if (slot0 + (unsigned)j < limit) {
                        values[slot0 + j] = (typename Raw<I8>::Element)e[j];
                    } else {
                        mask &= ~(0xfu << (4 * j));
                        r.refused = true;
                    }
                }
            }
            if ((packed & mask) != 0u && slot0 < limit) atomicOr(deltas32 + (slot0 >> 3), packed & mask);
        }
    }
    r.flushed += n;
    __syncwarp();
}

// Clears the deltas. The emit kernel is its programmatic dependent: its CTAs move in, read their row offsets and fetch their first
// columns while this runs, and wait for it before they write.
__global__ void __launch_bounds__(256) clear_deltas_kernel(unsigned *__restrict__ deltas32, unsigned words)
{
    asm volatile("griddepcontrol.launch_dependents;");
    const unsigned stride = gridDim.x * 256u, i0 = blockIdx.x * 256u + threadIdx.x;
    const unsigned vecs = (reinterpret_cast<uintptr_t>(deltas32) & 15) == 0 ? words >> 2 : 0u;
    for (unsigned i = i0; i < vecs; i += stride) reinterpret_cast<uint4 *>(deltas32)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (unsigned i = (vecs << 2) + i0; i < words; i += stride) deltas32[i] = 0u;
}

// `nan_add`: what lifts the bits (without sign) of every NaN of the value type to 0x8000 and above, in both halves
// of a word: 0x7fff minus the bits of +infinity. Every NaN is stored as 0x7fff (what the reference's float round
// trip makes of it, cpu_compressor.cuh:26,36). Not used with int8 values.
template <bool I8>
__global__ void __launch_bounds__(kThreads, 4)
emit_rows_kernel(const typename Raw<I8>::Element *__restrict__ dense, int rows, int cols, bool vec_ok,
                 const int *__restrict__ row_indices, typename Raw<I8>::Element *__restrict__ values,
                 unsigned *__restrict__ deltas32, int slots, unsigned nan_add, bool vec_v)
{
    __shared__ __align__(16) unsigned ring_s[(kWarpsPerCta + 1) * kRing];
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (row >= rows) return;
    // element indices fit 32 bits: the entry points refuse matrices of 2^31 elements or more, and a walk ends
    // less than 2048 elements behind its row
    const unsigned total = (unsigned)rows * (unsigned)cols;
    const unsigned row_lo = (unsigned)row * (unsigned)cols;
    const unsigned row_hi = row_lo + (unsigned)cols;
    const unsigned first = vec_ok ? (row_lo & ~15u) : row_lo;

    EmitRing ring;
    // the rings start at a multiple of their size, so that a wrapped offset is merged into the address with an OR
    const unsigned ring_all = (unsigned)__cvta_generic_to_shared(ring_s);
    const unsigned ring_base = ((ring_all + 4u * kRing - 1u) & ~(4u * kRing - 1u)) + (threadIdx.x >> 5) * 4u * kRing;
    ring.e = ring_s + ((ring_base - ring_all) >> 2);
    const unsigned limit = (unsigned)slots;
    const unsigned out0 = (unsigned)min(max(row_indices[row], 0), slots);   // a corrupt offset cannot leave the buffers
    ring.out = out0;
    ring.flushed = out0 & ~7u;
    ring.own_lo = out0;
    ring.refused = row_indices[row] != (int)out0;
    // columns mod 16 are counted from the allocation (only differences matter): the one in front of the row
    if (lane == 0) ring.e[(out0 - 1u) & (kRing - 1)] = ((row_lo - 1u - first) & 15u) << 16;
    __syncwarp();
    int carry = -1;   // column of the last non-zero seen so far in this row

    // n pads on columns after + 16, after + 32, ... by the whole warp, each with the +-0 it sits on
    auto append_pads = [&](int after, int n) {
        for (int b0 = 0; b0 < n; b0 += kFlush) {
            const int now = min(kFlush, n - b0);
            for (int i = lane; i < now; i += 32)
                ring.e[(ring.out + (unsigned)i) & (kRing - 1)] = (unsigned)__ldg(dense + row_lo + (unsigned)(after + 16 * (b0 + i + 1))) | (((row_lo - first + (unsigned)after) & 15u) << 16);
            ring.out += (unsigned)now;
            if (ring.out - ring.flushed >= (unsigned)kFlush) ring_flush<I8>(ring, values, deltas32, kFlush, limit, vec_v, lane);
        }
    };

    typename Raw<I8>::Vec v[2], v_next[2];
    auto fetch = [&](unsigned step0, typename Raw<I8>::Vec (&f)[2]) {
        const unsigned g0 = step0 + (unsigned)(lane * kEmitCols);
        if (vec_ok && step0 + 32u * kEmitCols <= row_hi) {   // warp-uniform
            f[0] = load8_inside<I8>(dense, g0);
            f[1] = load8_inside<I8>(dense, g0 + 8u);
        } else {
            f[0] = load8<I8>(dense, g0, row_lo, row_hi, total, vec_ok);
            f[1] = load8<I8>(dense, g0 + 8u, row_lo, row_hi, total, vec_ok);
        }
    };
    fetch(first, v_next);
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the deltas are cleared
#pragma unroll 1
    for (unsigned step0 = first; step0 < row_hi; step0 += 32u * kEmitCols) {
        const unsigned g0 = step0 + (unsigned)(lane * kEmitCols);
        v[0] = v_next[0];
        v[1] = v_next[1];
        fetch(step0 + 32u * kEmitCols, v_next);   // in flight while this step is worked on
        unsigned w[2][4];
        words_of<I8>(v[0], w[0]);
        words_of<I8>(v[1], w[1]);
        if (step0 < row_lo || step0 + 32u * kEmitCols > row_hi) {   // warp-uniform
            clear_outside(w[0], g0, row_lo, row_hi);
            clear_outside(w[1], g0 + 8u, row_lo, row_hi);
        }
        const unsigned nz = ordered_bits(nonzero_fields(w[0])) | (ordered_bits(nonzero_fields(w[1])) << 8);
        const unsigned any = __ballot_sync(0xffffffffu, nz != 0u);
        if (any == 0u) continue;   // warp-uniform
        if constexpr (!I8) {
            unsigned nans = 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j) nans |= (w[j >> 2][j & 3] & 0x7fff7fffu) + nan_add;
            if (nans & 0x80008000u) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    unsigned &x = w[j >> 2][j & 3];
                    const unsigned h = (x & 0x7fff7fffu) + nan_add;
                    if (h & 0x00008000u) x = (x & 0xffff0000u) | 0x7fffu;
                    if (h & 0x80000000u) x = (x & 0x0000ffffu) | 0x7fff0000u;
                }
            }
        }
        const int c0 = (int)(g0 - row_lo);   // column of element 0; may be negative on the first step
        const int i_first = __ffs(nz) - 1;   // -1 when the lane has no non-zero
        const int my_last = c0 + (31 - __clz(nz | 1u));
        const int prev = prev_nonzero_before_lane(any, lane, my_last, carry);
        const int gap = c0 + i_first - prev - 1;   // zeros in front of the lane's first non-zero
        int npad = nz ? gap >> 4 : 0;
        int mine = __popc(nz);
        const bool pads = __any_sync(0xffffffffu, npad > 0);
        if (pads) {
            // those in front of the step's first non-zero: the zeros behind `carry`, by the whole warp
            const int leader = __ffs(any) - 1;
            append_pads(carry, __shfl_sync(0xffffffffu, npad, leader));
            if (lane == leader) npad = 0;
            mine += npad;
        }
        carry = __shfl_sync(0xffffffffu, my_last, 31 - __clz(any));

        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            asm("{.reg .pred p; .reg .b32 t; shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff; @p add.s32 %0, %0, t;}" : "+r"(incl) : "r"(o));
        unsigned k = ring.out + (unsigned)(incl - mine);
        if (pads) {
            for (int q = 1; q <= npad; ++q, ++k)   // a gap of 16 or more zeros inside the step
                ring.e[k & (kRing - 1)] = (unsigned)__ldg(dense + row_lo + (unsigned)(prev + 16 * q)) | (((row_lo - first + (unsigned)prev) & 15u) << 16);
        }
        unsigned at = 4u * k;   // byte offset of the next entry, before the wrap
#pragma unroll
        for (int i = 0; i < kEmitCols; ++i) {
            const unsigned x = w[i >> 3][(i >> 1) & 3];
            // predicated, not branched over
            asm volatile("{.reg .pred p; .reg .b32 a; setp.ne.u32 p, %1, 0; and.b32 a, %0, %4; or.b32 a, a, %3; @p st.shared.u32 [a], %2; @p add.u32 %0, %0, 4;}"
                         : "+r"(at)
                         : "r"(x & ((i & 1) ? 0x7fff0000u : 0x7fffu)), "r"(__byte_perm(x, (unsigned)i, (i & 1) ? 0x5432 : 0x5410)), "r"(ring_base),
                           "n"(4 * kRing - 1) : "memory");
        }
        ring.out += (unsigned)__shfl_sync(0xffffffffu, incl, 31);
        if (ring.out - ring.flushed >= (unsigned)kFlush) ring_flush<I8>(ring, values, deltas32, kFlush, limit, vec_v, lane);
    }
    if constexpr (I8) append_pads(carry, (cols - 1 - carry) >> 4);   // the int8 format keeps the pads inside the zeros at the end of a row
    ring_flush<I8>(ring, values, deltas32, ring.out - ring.flushed, limit, vec_v, lane);
    if (row == rows - 1) {
        // everything from n = row_indices[rows] to the padded count is zero (the deltas already are)
        const int n = row_indices[rows];
        if (n < 0 || n > slots) ring.refused = true;   // row_indices and P do not belong together
        for (unsigned i = (unsigned)max(n, 0) + (unsigned)lane; i < limit; i += 32u) values[i] = 0;
    }
    if (__any_sync(0xffffffffu, ring.refused) && lane == 0) atomicAdd(&g_compress_overflow, 1u);
}

// In-place inclusive prefix sum over counts[1..rows]; counts[0] = 0. One CTA; a warp takes 512 consecutive entries per
// iteration (four 16-byte loads per lane, all in flight together), the CTA 16384: the iterations are a serial chain of
// loads, shuffles and barriers, and most matrices need only one.
// Launched as a programmatic dependent: its CTA is in place when the last counts are written. With `total` (host memory that
// the device can write) the sum goes there as well, for a host that waits for it without a copy.
__global__ void __launch_bounds__(1024) scan_rows_kernel(int *__restrict__ ri, int rows, int *total)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ int warp_sums[32];
    __shared__ int carry_s;
    constexpr int kVecs = 4, kPerWarp = 128 * kVecs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(ri) & 15) == 0;
    const long long n = (long long)rows + 1;   // entry 0 counts as zero, so that the vectors start at the allocation
    if (tid == 0) carry_s = 0;
    __syncthreads();
    for (long long base = 0; base < n; base += 32 * kPerWarp) {
        int v[kVecs][4];
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const long long i = base + warp * kPerWarp + k * 128 + lane * 4;
            if (vec_ok && i + 4 <= n) {
                const int4 t = *reinterpret_cast<const int4 *>(ri + i);
                v[k][0] = t.x; v[k][1] = t.y; v[k][2] = t.z; v[k][3] = t.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[k][j] = i + j < n ? ri[i + j] : 0;
            }
            if (i == 0) v[k][0] = 0;
        }
        int before = 0;   // sum of the warp's earlier vectors
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
#pragma unroll
            for (int j = 1; j < 4; ++j) v[k][j] += v[k][j - 1];
            int incl = v[k][3];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int add = before + incl - v[k][3];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[k][j] += add;
            before += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) warp_sums[warp] = before;
        __syncthreads();
        int sum = warp_sums[lane];   // every warp scans the 32 sums itself
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += t;
        }
        const int in_front = carry_s + (warp ? __shfl_sync(0xffffffffu, sum, (warp + 31) & 31) : 0);
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
            const long long i = base + warp * kPerWarp + k * 128 + lane * 4;
            if (vec_ok && i + 4 <= n) {
                *reinterpret_cast<int4 *>(ri + i) = make_int4(v[k][0] + in_front, v[k][1] + in_front, v[k][2] + in_front, v[k][3] + in_front);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (i + j < n) ri[i + j] = v[k][j] + in_front;
            }
        }
        __syncthreads();
        if (tid == 31) carry_s += sum;
        __syncthreads();
    }
    if (total != nullptr && tid == 0) *reinterpret_cast<volatile int *>(total) = carry_s;
}

// Largest padded count of macko_compress_emit_static (part of its contract).
constexpr long long kStaticCapacity = 16ll << 20;

int check_dense(const void *dense, int64_t rows, int64_t cols, uintptr_t element_bytes = 2)
{
    if (rows < 0 || cols < 0) return fail(MACKO_ERR_INVALID_ARGUMENT, "negative size (rows=%lld cols=%lld)", (long long)rows, (long long)cols);
    if (rows > 0 && cols > 0 && rows > ((1LL << 31) - 1) / cols)
        return fail(MACKO_ERR_SIZE_OVERFLOW, "rows*cols = %lld*%lld does not fit 31 bits", (long long)rows, (long long)cols);
    if (rows >= (1LL << 31) - 1) return fail(MACKO_ERR_SIZE_OVERFLOW, "too many rows");
    if (rows * cols > 0 && !dense) return fail(MACKO_ERR_INVALID_ARGUMENT, "null dense matrix");
    if (!aligned(dense, element_bytes)) return fail(MACKO_ERR_MISALIGNED, "dense must be aligned to its element size");
    return MACKO_OK;
}

int launch_error(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return MACKO_OK;
}


}  // namespace

int launch_row_scan(int *counts, int rows, cudaStream_t stream, int *total)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(1024);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, scan_rows_kernel, counts, rows, total);
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "row scan launch: %s", cudaGetErrorString(e));
    return launch_error("row scan launch");
}

}  // namespace macko

// Rows that a warp of the counting kernel takes one after the other: as many as make one round of the warps that the GPU holds
// at a time (48 on each of 148 SMs), so that no second round runs mostly empty.
static int count_rows_per_warp(int64_t rows)
{
    const int64_t n = (rows + 148 * 48 - 1) / (148 * 48);
    return (int)(n < 1 ? 1 : n > 8 ? 8 : n);
}

template <bool I8>
static int compress_count_typed(const void *dense, int64_t rows, int64_t cols, int32_t *row_indices, int32_t *total, void *stream)
{
    using namespace macko;
    using Element = typename Raw<I8>::Element;
    int st = check_dense(dense, rows, cols, sizeof(Element));
    if (st != MACKO_OK) return st;
    if (!row_indices) return fail(MACKO_ERR_INVALID_ARGUMENT, "null row_indices");
    if (!aligned(row_indices, 4)) return fail(MACKO_ERR_MISALIGNED, "row_indices must be 4-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (rows > 0) {
        const int per_warp = count_rows_per_warp(rows);
        const unsigned grid = (unsigned)((rows + kWarpsPerCta * per_warp - 1) / (kWarpsPerCta * per_warp));
        count_rows_kernel<I8><<<grid, kThreads, 0, s>>>(static_cast<const Element *>(dense), (int)rows, (int)cols,
                                                        aligned(dense, 8 * sizeof(Element)), per_warp, row_indices);
        st = launch_error("compress count launch");
        if (st != MACKO_OK) return st;
    }
    return launch_row_scan(row_indices, (int)rows, s, total);
}

// Checks and launch shared by the emit entry points.
template <bool I8>
static int compress_emit_typed(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                               int64_t padded_count, void *values, void *deltas, void *stream, unsigned infinity_bits)
{
    using namespace macko;
    using Element = typename Raw<I8>::Element;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Boundary groups of neighbouring rows merge their nibbles into one word: the deltas start at zero.
    if (rows == 0) {
        cudaError_t e = cudaMemsetAsync(deltas, 0, (size_t)padded_count / 2, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(values, 0, (size_t)padded_count * sizeof(Element), s);
        if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "clearing the outputs: %s", cudaGetErrorString(e));
        return MACKO_OK;
    }
    const unsigned words = (unsigned)(padded_count >> 3);   // a multiple of 8 stored elements: whole words
    clear_deltas_kernel<<<(unsigned)((words + 4095u) / 4096u < 592u ? (words + 4095u) / 4096u : 592u), 256, 0, s>>>(static_cast<unsigned *>(deltas), words);
    const int st = launch_error("clearing the deltas");
    if (st != MACKO_OK) return st;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((rows + kWarpsPerCta - 1) / kWarpsPerCta));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, emit_rows_kernel<I8>,
        static_cast<const Element *>(dense), (int)rows, (int)cols, aligned(dense, 8 * sizeof(Element)), row_indices,
        static_cast<Element *>(values), static_cast<unsigned *>(deltas), (int)padded_count,
        (0x7fffu - infinity_bits) * 0x10001u, aligned(values, 8 * sizeof(Element)));
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "compress emit launch: %s", cudaGetErrorString(e));
    return launch_error("compress emit launch");
}

template <bool I8>
static int compress_emit_workspace(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                                   int64_t padded_count, void *values, void *deltas,
                                   void *workspace, int64_t workspace_bytes, void *stream, unsigned infinity_bits)
{
    using namespace macko;
    int st = check_dense(dense, rows, cols, I8 ? 1 : 2);
    if (st != MACKO_OK) return st;
    if (!row_indices) return fail(MACKO_ERR_INVALID_ARGUMENT, "null row_indices");
    if (padded_count < 0 || padded_count % 8 != 0 || padded_count >= (1LL << 31))
        return fail(MACKO_ERR_INVALID_ARGUMENT, "padded_count %lld must be a non-negative multiple of 8 below 2^31", (long long)padded_count);
    if (padded_count == 0) return MACKO_OK;
    if (!values || !deltas || !workspace) return fail(MACKO_ERR_INVALID_ARGUMENT, "null output or workspace");
    if (!aligned(values, I8 ? 1 : 2) || !aligned(deltas, 4) || !aligned(workspace, 8))
        return fail(MACKO_ERR_MISALIGNED, "16-bit values need 2-, deltas 4-, workspace 8-byte alignment");
    // The kernel needs no workspace any more; its size is still checked: callers size it once for every entry point.
    if (workspace_bytes < macko_compress_workspace_bytes(padded_count))
        return fail(MACKO_ERR_WORKSPACE, "workspace has %lld bytes, %lld needed", (long long)workspace_bytes,
                    (long long)macko_compress_workspace_bytes(padded_count));
    return compress_emit_typed<I8>(dense, rows, cols, row_indices, padded_count, values, deltas, stream, infinity_bits);
}

extern "C" {

int macko_compress_count(const void *dense, int64_t rows, int64_t cols, int32_t *row_indices, void *stream)
{
    return compress_count_typed<false>(dense, rows, cols, row_indices, nullptr, stream);
}

int macko_compress_count_total(const void *dense, int64_t rows, int64_t cols, int32_t value_bytes, int32_t *row_indices,
                               int32_t *total, void *stream)
{
    using namespace macko;
    if (value_bytes != 1 && value_bytes != 2) return fail(MACKO_ERR_INVALID_ARGUMENT, "value_bytes must be 1 or 2 (got %d)", value_bytes);
    if (!total) return fail(MACKO_ERR_INVALID_ARGUMENT, "null total");
    if (!aligned(total, 4)) return fail(MACKO_ERR_MISALIGNED, "total must be 4-byte aligned");
    void *device_total = nullptr;
    const cudaError_t e = cudaHostGetDevicePointer(&device_total, total, 0);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(MACKO_ERR_INVALID_ARGUMENT, "total is not host memory that the device can write: %s", cudaGetErrorString(e));
    }
    return value_bytes == 1 ? compress_count_typed<true>(dense, rows, cols, row_indices, static_cast<int32_t *>(device_total), stream)
                            : compress_count_typed<false>(dense, rows, cols, row_indices, static_cast<int32_t *>(device_total), stream);
}

int64_t macko_compress_workspace_bytes(int64_t padded_count) { return padded_count < 0 ? 0 : padded_count; }

int macko_compress_emit(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                        int64_t padded_count, void *values, void *deltas,
                        void *workspace, int64_t workspace_bytes, void *stream)
{
    return compress_emit_workspace<false>(dense, rows, cols, row_indices, padded_count, values, deltas, workspace,
                                          workspace_bytes, stream, 0x7c00u);
}

int macko_compress_emit_bf16(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                             int64_t padded_count, void *values, void *deltas,
                             void *workspace, int64_t workspace_bytes, void *stream)
{
    return compress_emit_workspace<false>(dense, rows, cols, row_indices, padded_count, values, deltas, workspace,
                                          workspace_bytes, stream, 0x7f80u);
}

int macko_compress_count_int8(const void *dense, int64_t rows, int64_t cols, int32_t *row_indices, void *stream)
{
    return compress_count_typed<true>(dense, rows, cols, row_indices, nullptr, stream);
}

int macko_compress_emit_int8(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                             int64_t padded_count, void *values, void *deltas,
                             void *workspace, int64_t workspace_bytes, void *stream)
{
    return compress_emit_workspace<true>(dense, rows, cols, row_indices, padded_count, values, deltas, workspace,
                                         workspace_bytes, stream, 0u);
}

int macko_compress_overflow(uint32_t *count, void *stream)
{
    using namespace macko;
    if (!count) return fail(MACKO_ERR_INVALID_ARGUMENT, "null count");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned seen = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&seen, g_compress_overflow, sizeof(seen), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && seen != 0) {
        const unsigned zero = 0;
        e = cudaMemcpyToSymbolAsync(g_compress_overflow, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "reading the compressor's overflow word: %s", cudaGetErrorString(e));
    *count = seen;
    return MACKO_OK;
}

int64_t macko_compress_static_capacity(void) { return macko::kStaticCapacity; }

int macko_compress_emit_static(const void *dense, int64_t rows, int64_t cols, const int32_t *row_indices,
                               int64_t padded_count, void *values, void *deltas, void *stream)
{
    using namespace macko;
    int st = check_dense(dense, rows, cols);
    if (st != MACKO_OK) return st;
    if (!row_indices) return fail(MACKO_ERR_INVALID_ARGUMENT, "null row_indices");
    if (padded_count < 0 || padded_count % 8 != 0)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "padded_count %lld must be a non-negative multiple of 8", (long long)padded_count);
    if (padded_count > kStaticCapacity)
        return fail(MACKO_ERR_WORKSPACE,
                    "padded_count %lld exceeds the built-in scratch of %lld stored elements (no longer used, still the limit of "
                    "this entry point); use macko_compress_emit with a caller-provided workspace",
                    (long long)padded_count, (long long)kStaticCapacity);
    if (padded_count == 0) return MACKO_OK;
    if (!values || !deltas) return fail(MACKO_ERR_INVALID_ARGUMENT, "null output");
    if (!aligned(values, 2) || !aligned(deltas, 4))
        return fail(MACKO_ERR_MISALIGNED, "values needs 2-, deltas 4-byte alignment");
    return compress_emit_typed<false>(dense, rows, cols, row_indices, padded_count, values, deltas, stream, 0x7c00u);
}
}
