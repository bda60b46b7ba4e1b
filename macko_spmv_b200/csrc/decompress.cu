// MACKO -> dense fp16 on the GPU.
//
// The reference has no decompressor; a dense copy is what a product with many right-hand sides wants
// (a tensor-core GEMM on the dense matrix beats streaming the compressed matrix once per few vectors),
// and it is the inverse used to check the compressor. Semantics follow the format as the reference SpMV
// reads it (src/macko_spmv/cuda/kernels.cuh:86-108): element k of a row sits at column
// (sum of the deltas of elements 0..k) + k; stored non-zeros are written with their stored bits and
// everything else (pads included, whatever their sign bit) is +0.
#include "common.cuh"

namespace macko {
namespace {

// Zero the deltas and the 16-bit values of one 8-element unit outside element range [lo, hi).
__device__ __forceinline__ void keep_elements(uint4 &v, unsigned &w, int lo, int hi)
{
    const int l = min(max(lo, 0), 8), h = min(max(hi, 0), 8);
    unsigned m = l >= 8 ? 0u : (0xffffffffu << (4 * l));
    if (h < 8) m &= ~(0xffffffffu << (4 * h));
    w &= m;
    unsigned *vw = reinterpret_cast<unsigned *>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        vw[j] &= (((m >> (8 * j)) & 1u) * 0xffffu) | (((m >> (8 * j + 4)) & 1u) * 0xffff0000u);
}

constexpr int kWarps = 8;        // warps (rows in flight) per CTA
constexpr int kWin = 1024;       // fp16 slots of a warp's window of the dense row (a multiple of 256)

// One warp per row, no barrier wider than the warp. The row is assembled window by window in shared memory (zeros,
// then the stored elements scattered to their columns) and leaves as one bulk copy, which costs the load/store pipe
// nothing, while the warp clears and fills a second window; every byte of the dense matrix is written exactly once
// and no clearing pass is needed. Windows start on 128-byte lines of the matrix; the up to 7 slots at either end of a
// row that share 16 bytes with a neighbouring row go one by one. A step decodes 256 stored elements, 8 per lane: the column
// offsets of a unit come from byte-wise prefix sums of its deltas (as in the product kernel: byte j of `ce` / `co`
// is twice the column of element 2j / 2j+1 relative to the unit's base, and the top byte of `co` plus 2 is twice the
// columns the unit advances), the units' bases from a warp scan. A step that reaches beyond the window stays in
// registers: what lies inside is stored, the window leaves, and the rest goes to the next one. Pads and everything
// else that is +-0 stay +0. The loads of the next step are issued before a step is scattered, and the second-level cache is asked for
// the stream four steps ahead: with one step of loads alone a warp waits for memory in every step (4096x11008 at density 0.5 33.1 us
// without; at density 0.2 it matters less: a call of 11003x4093 24.6 us without, 23.7..24.3 with it). More loads in flight take
// registers that the fifth CTA needs.
// Bound by the load/store pipe (a 2-byte shared store of 32 elements takes 3.8 passes: random columns, random banks) and
// close behind it HBM: 11003x4093 at density 0.2 (113 MB) in 21.5 us = 5.2 TB/s, 4096x11008 at 0.5 (146 MB) in 29.3 us
// = 5.0 TB/s; a CTA per row takes 32.8 and 31.8 us. With the window flushed and cleared by the same 16-byte loads and
// stores instead of a bulk copy 22.7 and 32.5 us; with six CTAs per SM instead of five 23.3 and 30.3 us.
// Element positions are unsigned in both kernels: a walk looks up to 2048 elements ahead of a count that may come close
// to 2^31, where a signed position turns negative and passes for one inside the row.
__global__ void __launch_bounds__(kWarps * 32, 5)
decompress_rows_kernel(const uint4 *__restrict__ values, const unsigned *__restrict__ deltas,
                       const int *__restrict__ ri, int rows, int cols, int stored,
                       unsigned short *__restrict__ dense, bool vec_ok)
{
    __shared__ __align__(16) unsigned short window_s[kWarps][2][kWin];
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * kWarps + (int)(threadIdx.x >> 5);
    if (row >= rows) return;
    unsigned short *window = window_s[threadIdx.x >> 5][0], *other = window_s[threadIdx.x >> 5][1];
    // offsets clamped into [0, stored]: a corrupt row_indices cannot send loads outside the buffers
    const unsigned begin = (unsigned)min(max(__ldg(ri + row), 0), stored);
    const unsigned end = (unsigned)min(max(__ldg(ri + row + 1), 0), stored);
    auto clear = [&]() {
#pragma unroll
        for (int c = lane; c < kWin / 8; c += 32) reinterpret_cast<uint4 *>(window)[c] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
    };
    clear();
    const long long row0 = row * (long long)cols;
    const int lo = vec_ok ? (int)(row0 & 63) : 0;   // the row takes slots [lo, hi) from the line that holds its start
    const int hi = lo + cols;
    unsigned short *out = dense + (row0 - lo);
    int start = 0;                          // first slot of the window
    int col2 = 2 * lo - 2 * (int)(begin & 7u);    // byte offset in the window of the column in front of the next step
    auto flush = [&]() {
        const int a = max(lo, start), b = min(hi, start + kWin);               // the row's slots in this window
        const int a8 = vec_ok ? (a + 7) & ~7 : b, b8 = vec_ok ? b & ~7 : b;    // the whole 16-byte chunks among them
        if (a8 < b8) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out + a8),
                             "r"((unsigned)__cvta_generic_to_shared(window + (a8 - start))), "r"(2 * (b8 - a8)) : "memory");
            }
            if (a + lane < a8) out[a + lane] = window[a + lane - start];
            if (b8 + lane < b) out[b8 + lane] = window[b8 + lane - start];
        } else {
            __syncwarp();
            for (int e = a + lane; e < b; e += 32) out[e] = window[e - start];
        }
        // the other window is free once its copy has been read
        if (lane == 0) asm volatile("cp.async.bulk.commit_group; cp.async.bulk.wait_group.read 1;" ::: "memory");
        unsigned short *t = window;
        window = other;
        other = t;
        start += kWin;
        col2 -= 2 * kWin;
        __syncwarp();
        clear();
    };
    auto fetch = [&](unsigned first, uint4 &v, unsigned &w) {
        v = make_uint4(0u, 0u, 0u, 0u);
        w = 0u;
        if (first < end) {
            v = __ldcs(values + (first >> 3));
            w = __ldcs(deltas + (first >> 3));
        }
    };
    // Asks the second-level cache for `steps` steps of 256 stored elements from `from` on: lanes [0, 4 * steps) the lines of the values,
    // the next `steps` those of the deltas.
    auto prefetch = [&](unsigned from, unsigned steps) {
        const unsigned l = (unsigned)lane;
        const bool value_line = l < 4u * steps;
        const unsigned e = from + (value_line ? 64u * l : 256u * (l - 4u * steps));
        if (l < 5u * steps && e < end)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(value_line ? reinterpret_cast<const char *>(values) + 2 * (size_t)e : reinterpret_cast<const char *>(deltas) + (e >> 1)));
    };
    unsigned first = (begin & ~7u) + (unsigned)(lane * 8);   // first element of the lane's unit
    uint4 v;
    unsigned w;
    fetch(first, v, w);
    const bool far = end > begin + 768u;   // shorter rows are over before it helps: 16000x1001 d = 0.7 15.0 us with it, 14.6 without
    if (far) prefetch((begin & ~7u) + 256u, 3u);
    for (unsigned pos = begin & ~7u; pos < end && start < hi; pos += 256u, first += 256u) {
        uint4 v_next;
        unsigned w_next;
        fetch(first + 256u, v_next, w_next);
        if (far) prefetch(pos + 1024u, 1u);
        if (first < begin || (first < end && first + 8u > end)) keep_elements(v, w, (int)(begin - first), (int)(end - first));
        const unsigned ev = w & 0x0f0f0f0fu, od = (w >> 4) & 0x0f0f0f0fu;
        const unsigned pe = ev * 0x02020202u + 0x0c080400u, po = od * 0x02020202u;
        const unsigned ce = po * 256u + pe, co = pe + po + 0x02020202u;
        const int mine = first < end ? (int)(co >> 24) + 2 : 0;   // twice the columns this unit advances
        int inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
            asm("{.reg .pred p; .reg .b32 t; shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff; @p add.s32 %0, %0, t;}" : "+r"(inc) : "r"(o));
        const int total = __shfl_sync(0xffffffffu, inc, 31);
        int at = col2 + inc - mine;   // byte offset in the window of the unit's base column
        const unsigned vw[4] = {v.x, v.y, v.z, v.w};
        for (;;) {
            const unsigned window_addr = (unsigned)__cvta_generic_to_shared(window);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned be = (unsigned)__dp4a(ce, 1u << (8 * j), (unsigned)at);
                const unsigned bo = (unsigned)__dp4a(co, 1u << (8 * j), (unsigned)at);
                // predicated, not branched over; offsets in front of the window (already stored) are huge as unsigned numbers
                asm volatile("{.reg .pred p, q; .reg .b16 l, h; mov.b32 {l, h}, %4; setp.ne.u32 p, %5, 0; setp.ne.u32 q, %6, 0;"
                             "setp.lt.and.u32 p, %0, %7, p; setp.lt.and.u32 q, %2, %7, q; @p st.shared.u16 [%1], l; @q st.shared.u16 [%3], h;}"
                             ::"r"(be), "r"(window_addr + be), "r"(bo), "r"(window_addr + bo), "r"(vw[j]), "r"(vw[j] & 0x7fffu), "r"(vw[j] & 0x7fff0000u),
                               "n"(2 * kWin) : "memory");
            }
            if (col2 + total <= 2 * kWin) break;
            flush();
            at -= 2 * kWin;
            if (start >= hi) break;   // only deltas that no compressor can produce reach beyond the row
        }
        col2 += total;
        v = v_next;
        w = w_next;
    }
    while (start < hi) flush();   // the last elements and the zeros behind them
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

constexpr int kRowThreads = 256;   // threads of a CTA of the row kernel: 256 units (2048 stored elements) per pass

// One CTA per row; the whole dense row is assembled in shared memory (zeroed once, re-zeroed while it is
// flushed). A pass takes 256 consecutive 8-element units of the row, one per thread: the 8 column offsets of a
// unit come from byte-wise prefix sums of its deltas (as in the product kernel: byte j of `ce` / `co` is twice
// the column of element 2j / 2j+1 relative to the unit's base, and the top byte of `co` plus 2 is twice the
// columns the unit advances), the units' bases from a scan over the CTA. Stored non-zeros are written to their
// columns with 2-byte shared stores; pads and everything else stay +0. The row leaves with 16-byte stores.
// `off` = (row * cols) mod 8 slots of the buffer lie in front of the row so that aligned chunks of the buffer are
// aligned chunks of the dense matrix.
__global__ void __launch_bounds__(kRowThreads)
decompress_row_cta_kernel(const uint4 *__restrict__ values, const unsigned *__restrict__ deltas,
                          const int *__restrict__ ri, int rows, int cols, int stored,
                          unsigned short *__restrict__ dense, bool vec_ok)
{
    extern __shared__ __align__(16) unsigned short rowbuf[];   // cols + 16 slots
    __shared__ unsigned warp_total[2][kRowThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int buf_chunks = (cols + 16) >> 3;
    for (int c = tid; c < buf_chunks; c += kRowThreads) reinterpret_cast<uint4 *>(rowbuf)[c] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const unsigned row_bytes = 2u * (unsigned)cols;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        // offsets clamped into [0, stored]: a corrupt row_indices cannot send loads outside the buffers
        const unsigned begin = (unsigned)min(max(__ldg(ri + row), 0), stored);
        const unsigned end = (unsigned)min(max(__ldg(ri + row + 1), 0), stored);
        const long long row0 = row * (long long)cols;
        const int off = vec_ok ? (int)(row0 & 7) : 0;
        unsigned char *base = reinterpret_cast<unsigned char *>(rowbuf + off);
        // twice the column in front of the unit that holds `begin`: its leading elements belong to the row before
        int col2 = -2 * (int)(begin & 7u);
        int parity = 0;
        for (unsigned pos = begin & ~7u; pos < end; pos += kRowThreads * 8u, parity ^= 1) {
            const unsigned first = pos + (unsigned)(tid * 8);
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            unsigned w = 0u;
            const bool active = first < end;
            if (active) {
                v = __ldg(values + (first >> 3));
                w = __ldg(deltas + (first >> 3));
                // a unit that straddles an end of the row: drop what lies outside
                if (first < begin || first + 8u > end) keep_elements(v, w, (int)(begin - first), (int)(end - first));
            }
            const unsigned ev = w & 0x0f0f0f0fu, od = (w >> 4) & 0x0f0f0f0fu;
            const unsigned pe = ev * 0x02020202u + 0x0c080400u, po = od * 0x02020202u;
            const unsigned ce = po * 256u + pe, co = pe + po + 0x02020202u;
            const unsigned mine = active ? (co >> 24) + 2u : 0u;   // twice the columns this unit advances
            unsigned inc = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            if (lane == 31) warp_total[parity][warp] = inc;
            __syncthreads();
            unsigned before = 0u, all = 0u;
#pragma unroll
            for (int k = 0; k < kRowThreads / 32; ++k) {
                const unsigned t = warp_total[parity][k];
                if (k < warp) before += t;
                all += t;
            }
            const int a0 = col2 + (int)(before + inc - mine);   // twice the unit's base column
            col2 += (int)all;
            const unsigned *vw = reinterpret_cast<const unsigned *>(&v);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned lo16 = vw[j] & 0xffffu, hi16 = vw[j] >> 16;
                const unsigned be = (unsigned)(a0 + (int)((ce >> (8 * j)) & 0xffu));
                const unsigned bo = (unsigned)(a0 + (int)((co >> (8 * j)) & 0xffu));
                // +-0 (pads, masked elements) is not stored; offsets of malformed input stay inside the row
                if ((lo16 & 0x7fffu) != 0u && be < row_bytes) *reinterpret_cast<unsigned short *>(base + be) = (unsigned short)lo16;
                if ((hi16 & 0x7fffu) != 0u && bo < row_bytes) *reinterpret_cast<unsigned short *>(base + bo) = (unsigned short)hi16;
            }
        }
        __syncthreads();
        // flush the row and leave the buffer zeroed for the next one
        const int n_chunks = (off + cols + 7) >> 3;
        unsigned short *out = dense + (row0 - off);
        for (int c = tid; c < n_chunks; c += kRowThreads) {
            const uint4 q = reinterpret_cast<const uint4 *>(rowbuf)[c];
            reinterpret_cast<uint4 *>(rowbuf)[c] = make_uint4(0u, 0u, 0u, 0u);
            const int e0 = 8 * c;
            if (vec_ok && e0 >= off && e0 + 8 <= off + cols) {
                reinterpret_cast<uint4 *>(out)[c] = q;
            } else {
                const unsigned short *qh = reinterpret_cast<const unsigned short *>(&q);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (e0 + j >= off && e0 + j < off + cols) out[e0 + j] = qh[j];
            }
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace macko

extern "C" int macko_decompress_fp16(const void *values, const void *deltas, const int32_t *row_indices,
                                     int64_t rows, int64_t cols, int64_t padded_count, void *dense, void *stream)
{
    using namespace macko;
    if (rows < 0 || cols < 0 || padded_count < 0 || padded_count % 8 != 0)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "bad sizes (rows=%lld cols=%lld P=%lld)", (long long)rows,
                    (long long)cols, (long long)padded_count);
    if (rows >= (1LL << 31) - 64 || cols >= (1LL << 30) || padded_count >= (1LL << 31))
        return fail(MACKO_ERR_SIZE_OVERFLOW, "rows=%lld cols=%lld P=%lld exceed 31-bit indexing", (long long)rows,
                    (long long)cols, (long long)padded_count);
    if (rows == 0 || cols == 0) return MACKO_OK;
    if (!row_indices || !dense) return fail(MACKO_ERR_INVALID_ARGUMENT, "null row_indices or dense");
    if (padded_count > 0 && (!values || !deltas)) return fail(MACKO_ERR_INVALID_ARGUMENT, "null values or deltas");
    if (!aligned(values, 16) || !aligned(deltas, 4) || !aligned(row_indices, 4) || !aligned(dense, 2))
        return fail(MACKO_ERR_MISALIGNED, "values need 16-, deltas and row_indices 4-, dense 2-byte alignment");
    const DeviceInfo *dev = nullptr;
    int st = current_device_info(&dev);
    if (st != MACKO_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t row_smem = ((size_t)cols + 16) * sizeof(unsigned short);
    cudaError_t e;
    // CTAs of the kernel that holds a whole row in shared memory (0: the row does not fit)
    long long per_sm = (long long)((size_t)dev->max_smem_optin / (row_smem + 1024));
    if (per_sm > 2048 / kRowThreads) per_sm = 2048 / kRowThreads;
    // A CTA per row where a warp per row would leave three quarters of the warps idle that the CTAs bring; and for long rows,
    // of which a warp that starts late holds up the end, wherever that measured faster: a second wave of the warp
    // kernel (40 rows per SM at a time) that is mostly empty, few rows, or little to decode. The counts come from a grid, not
    // from a model: 1200..10000 rows, 1500..15000 columns, densities 0.1, 0.3, 0.6, 0.9; the pick is within 5 % of the faster
    // kernel on 291 of its 296 points and at most 10 % behind on the others. Measured (B200, us, CTA per
    // row / warp per row): few rows 1024x16384 d = 0.5 16.9 / 24.1, 512x49152 36.6 / 62.8; second wave 6600x10000 d = 0.3
    // 39.6 / 48.4, 8000x12000 56.5 / 61.3, 6600x8192 36.3 / 39.0; little to decode 5200x10000 d = 0.1 24.9 / 27.1, 3600x15000
    // 25.1 / 28.3. On the other side of the lines: 4400x8192 d = 0.6 33.1 / 27.0, 6600x5000 33.0 / 27.1, 10000x8192
    // 69.6 / 60.4, 4400x10000 d = 0.3 28.8 / 25.4, 4096x4096 d = 0.5 18.9 / 13.2, 11008x4096 44.8 / 31.7.
    const long long at_once = 40LL * dev->sm_count;
    const bool few_rows = rows < 2LL * dev->sm_count * per_sm;
    const bool late_wave = rows > at_once && (rows + at_once - 1) / at_once * at_once * 100 > 135 * rows;
    const bool sparse = 4 * padded_count < rows * cols;
    const bool long_rows = per_sm >= 4 && (cols >= 16384 || (cols >= 8192 && late_wave) || (cols >= 9216 && sparse) ||
                                           (cols >= 9216 && rows < 18LL * dev->sm_count) || (cols >= 10240 && rows < 27LL * dev->sm_count));
    if (per_sm > 0 && (few_rows || long_rows)) {
        // a CTA per row with the row in shared memory; as many CTAs per SM as threads and shared memory allow
        if (row_smem > 48 * 1024) {
            e = cudaFuncSetAttribute(decompress_row_cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)row_smem);
            if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        }
        long long grid = (long long)dev->sm_count * per_sm;
        if (grid > rows) grid = rows;
        decompress_row_cta_kernel<<<(unsigned)grid, kRowThreads, row_smem, s>>>(
            static_cast<const uint4 *>(values), static_cast<const unsigned *>(deltas), row_indices, (int)rows, (int)cols,
            (int)padded_count, static_cast<unsigned short *>(dense), aligned(dense, 16));
    } else {
        decompress_rows_kernel<<<(unsigned)((rows + kWarps - 1) / kWarps), kWarps * 32, 0, s>>>(
            static_cast<const uint4 *>(values), static_cast<const unsigned *>(deltas), row_indices, (int)rows, (int)cols,
            (int)padded_count, static_cast<unsigned short *>(dense), aligned(dense, 16));
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "decompress launch: %s", cudaGetErrorString(e));
    return MACKO_OK;
}
