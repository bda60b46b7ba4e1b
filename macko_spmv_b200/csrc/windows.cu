// Products with several right-hand sides over column windows (see windows.cuh), for matrices whose windows were built once.
//
// The product of a few vectors is bound by the shared-memory gathers of x: every stored element fetches the 16 bytes
// that eight interleaved vectors hold in its column, and a warp's 32 fetches of 16 bytes take four passes of the load/store
// pipe when no two lanes of a quarter-warp meet in a bank, about twelve with random columns in one copy of x (spmv.cu, BV = 8).
// Here every lane has its own banks: a column takes 128 bytes of shared memory, eight copies of its 16 bytes, and lane l reads
// copy l mod 8. One SM then holds some 1400 columns, so a CTA (one per SM) works on one window of the columns and a share of the
// rows; the sums of a row over the windows are added by a second small kernel, in window order, so y is reproducible.
//
// Measured (B200, graph of products of rotating matrices, us, one kernel for all columns / windows): 8 vectors, 11008x4096 d = 0.5
// 41.2 / 25.1, 4096x11008 d = 0.5 43.5 / 24.1, 16384x4096 d = 0.9 107.3 / 51.3, 4096x4096 d = 0.3 14.8 / 10.2, skewed 8192x28672 325 /
// 113; 4 vectors, 11008x4096 27.9 / 20.5, 32000x4096 d = 0.5 69.0 / 47.9. What bounds it: the four passes of a 16-byte gather, 32 of
// about 44 passes of the load/store pipe per 8 x 32 elements, then the walk of the few blocks of rows that a warp gets.
#include "common.cuh"
#include "unit.cuh"
#include "windows.cuh"

namespace macko {
namespace {

constexpr int kThreads = 1024;       // one CTA per SM: x takes its shared memory
constexpr int kWarps = kThreads / 32;
constexpr int L = 8;                 // lanes per row; a warp walks a block of four rows side by side
constexpr int K = 32 / L;
constexpr int STEP = kGroup * L;     // stored elements of a row per sub-step
constexpr int D = 2;                 // sub-steps in flight: more cost registers that the accumulators need (11008x4096
                                     // d = 0.5, 8 vectors: 24.6 us with two, 26.0 with four)

// ---- windows of a matrix -----------------------------------------------------------------------------------------------
// One warp per row walks its deltas once, 256 elements per step; the lane whose unit is the first of a window writes the
// section. Corrupt input is clamped: every section is written, none reaches beyond the row.
constexpr int kSteps = 4;
__global__ void __launch_bounds__(256)
window_sections_kernel(const unsigned *__restrict__ deltas32, const int *__restrict__ ri, int rows, int stored, int windows, int width,
                       uint2 *__restrict__ sections)
{
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const unsigned begin = (unsigned)min(max(__ldg(ri + row), 0), stored);
    const unsigned end = (unsigned)min(max(__ldg(ri + row + 1), (int)begin), stored);
    uint2 *mine = sections + row;   // window w at mine[w * rows]
    if (lane == 0) mine[0] = make_uint2(begin, (unsigned)kWindowFront);
    int col = 0;        // columns used up by the row's elements in front of the step
    int last = 0;       // window of the last unit in front of it
    for (unsigned group = begin & ~7u; group < end; group += 256u * kSteps) {
        unsigned w[kSteps];   // the loads of several steps are in flight together
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const unsigned k0 = group + 256u * (unsigned)u + 8u * (unsigned)lane;
            w[u] = k0 < end ? __ldg(deltas32 + (k0 >> 3)) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const unsigned base = group + 256u * (unsigned)u, k0 = base + 8u * (unsigned)lane;
            if (base >= end) break;   // warp-uniform
            const bool live = k0 < end;
            // columns of the unit: its deltas and one per element, without those of the neighbouring rows
            const unsigned lo = k0 < begin ? min(begin - k0, 8u) : 0u, hi = live ? min(end - k0, 8u) : 0u;
            const unsigned mine_w = lo < hi ? w[u] & (0xffffffffu << (4u * lo)) & (0xffffffffu >> (4u * (8u - hi))) : 0u;
            const int sum = (int)__dp4a((mine_w & 0x0f0f0f0fu) + ((mine_w >> 4) & 0x0f0f0f0fu), 0x01010101u, lo < hi ? hi - lo : 0u);
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int front = col + incl - sum;   // columns used up in front of the unit
            // window of the unit; the row's first unit is in the first one whatever its elements say
            const int win = k0 <= begin ? 0 : min((front + (int)(w[u] & 15u)) / width, windows - 1);
            int before = __shfl_up_sync(0xffffffffu, win, 1);
            if (lane == 0) before = last;
            if (live)
                for (int q = before + 1; q <= win; ++q)
                    mine[(size_t)q * rows] = make_uint2(k0, (unsigned)min(max(front - q * width + kWindowFront, 0), (1 << kWindowColBits) - 1));
            last = __shfl_sync(0xffffffffu, win, 31 - __clz(__ballot_sync(0xffffffffu, live)));
            col += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    for (int q = last + 1 + lane; q < windows; q += 32) mine[(size_t)q * rows] = make_uint2(end, (unsigned)kWindowFront);
    __threadfence_block();
    __syncwarp();
    for (int q = lane; q < windows; q += 32) {
        const unsigned first = *reinterpret_cast<volatile unsigned *>(&mine[(size_t)q * rows].x);
        const unsigned next = q + 1 < windows ? *reinterpret_cast<volatile unsigned *>(&mine[(size_t)(q + 1) * rows].x) : end;
        mine[(size_t)q * rows].y |= (next - first) << kWindowColBits;
    }
}

// ---- product -----------------------------------------------------------------------------------------------------------
// The sums of BV accumulators over the L lanes of a row: lane i of the group ends with the sum of vector i mod BV. Each of the
// first log2(BV) exchanges halves the vectors that a lane still carries, so 8 x 8 sums take 7 shuffles and not 24.
template <int BV>
__device__ __forceinline__ float group_sums(float (&a)[BV], int lane)
{
    int n = BV;
#pragma unroll
    for (int o = BV / 2; o > 0; o >>= 1) {
        const bool up = lane & o;
        n >>= 1;
#pragma unroll
        for (int i = 0; i < BV / 2; ++i) {
            if (i < n) {
                const float keep = up ? a[i + n] : a[i], send = up ? a[i] : a[i + n];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
#pragma unroll
    for (int o = BV; o < L; o <<= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    return a[0];
}

// CTA b: window b mod W, group of BV vectors (b / W) mod G, share b / (W * G) of the rows. Every warp takes a contiguous range
// of blocks of four rows and walks the rows of a block in step: they reach their ends together, so that the sums, the stores
// and the next block's set-up run once per block for all four (rows that differ in length wait for the longest; a walk in
// which every group fetched its own next row, as in spmv.cu, took 27.0 us instead of 24.6). The next block's section is
// fetched while this one is walked, and its first units while this one's sums are formed: a unit's registers take the unit D sub-steps on
// as soon as it has been worked on, so a warp always has D of them in flight (8 vectors, all units of an iteration at its top /
// like this: 32000x4096 d = 0.5 58.1 / 55.5 us, 2048x2048 7.8 / 7.0, 11008x4096 25.0 / 24.5; 16384x1024 9.0 / 9.2). The first units of the
// first block are in flight while x is staged and, for an immutable matrix, before the wait for the kernel in front.
template <int BV>
__global__ void __launch_bounds__(kThreads, 1)
windows_kernel(const uint4 *__restrict__ values, const unsigned *__restrict__ deltas, const uint2 *__restrict__ sections,
               const __half *__restrict__ x, float *__restrict__ partial, __half *__restrict__ y, int rows, int cols, int stored,
               int windows, int width, int groups, int shares, int batch, float alpha, float beta, int immutable)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, lig = lane & (L - 1);
    asm volatile("griddepcontrol.launch_dependents;");
    if (!immutable) asm volatile("griddepcontrol.wait;" ::: "memory");

    const int win = blockIdx.x % windows, rest = blockIdx.x / windows;
    const int grp = rest % groups, share = rest / groups;
    const unsigned n_blocks = ((unsigned)rows + K - 1) / K, n_warps = (unsigned)shares * kWarps, warp_id = (unsigned)share * kWarps + (tid >> 5);
    unsigned block = (unsigned)((unsigned long long)n_blocks * warp_id / n_warps);
    const unsigned block_hi = (unsigned)((unsigned long long)n_blocks * (warp_id + 1) / n_warps);

    const int col0 = win * width, here = max(min(width, cols - col0), 0);   // columns of this window
    const unsigned smem0 = (unsigned)__cvta_generic_to_shared(smem);
    auto stage_x = [&]() {
        // a thread takes a column: its BV values, written to the copies in an order that keeps neighbouring columns of a
        // store on different banks. Columns in front of the window and behind the matrix are zero.
#pragma unroll 1
        for (int c = tid - kWindowFront; c < here + kWindowHalo; c += kThreads) {
            unsigned q[4] = {0u, 0u, 0u, 0u};
            if (c >= 0 && col0 + c < cols) {
                const __half *xc = x + (size_t)grp * BV * cols + col0 + c;
#pragma unroll
                for (int b = 0; b < BV; ++b)
                    if (grp * BV + b < batch) q[b >> 1] |= (unsigned)ldg_fresh_u16(xc + (size_t)b * cols) << (16 * (b & 1));
                if (BV == 4) { q[2] = q[0]; q[3] = q[1]; }
            }
            const unsigned at = smem0 + (unsigned)(c + kWindowFront) * (unsigned)kWindowColBytes;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(at + 16u * (unsigned)((k + lane) & 7)), "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]) : "memory");
        }
        __syncthreads();
    };

    uint2 section = make_uint2(0u, 0u);
    auto fetch_section = [&]() {
        const unsigned row = block * K + (unsigned)(lane / L);
        section = make_uint2(0u, 0u);
        if (block < block_hi && row < (unsigned)rows) section = ldg_fresh_v2(sections + (size_t)win * rows + row);
    };
    fetch_section();
    // byte address of the lane's copy; offsets into x are kept doubled (bytes of fp16), as the prefix sums come, and a column
    // is 64 of those units wide
    const int x_base = (int)smem0 + (BV == 4 ? 8 * (lane & 15) : 16 * (lane & 7));
    const unsigned lane_const = (unsigned)(2 * lig);
    const unsigned a_max = (unsigned)(2 * (kWindowFront + here));
    // where the rows of the block stand: first unit of the next sub-step, elements left from there, their columns
    unsigned run = 0u, pos = 0u;
    int rem = 0, lo = 0, left = 0;
    bool masks = false;
    auto take_block = [&]() {
        const unsigned begin = min(section.x, (unsigned)stored), end = min(begin + (section.y >> kWindowColBits), (unsigned)stored);
        // twice the column in front of the row's next unit, less 14 per lane below in the group (see spmv.cu)
        run = lane_const + 2u * (section.y & ((1u << kWindowColBits) - 1u)) - 2u * (begin & (unsigned)(kGroup - 1));
        pos = (begin & ~(unsigned)(kGroup - 1)) + (unsigned)(kGroup * lig);
        rem = (int)(end - pos);
        lo = (int)(begin - pos);   // elements of the row before in the lane's first unit
        left = (int)__reduce_max_sync(0xffffffffu, end - (begin & ~(unsigned)(kGroup - 1)));
        masks = __any_sync(0xffffffffu, ((begin | end) & (unsigned)(kGroup - 1)) != 0u);   // not in a window inside the rows
        ++block;
        fetch_section();
    };
    uint4 v[D];
    unsigned w[D];
    auto load_unit = [&](int s, int step) {
        v[s] = make_uint4(0u, 0u, 0u, 0u);
        w[s] = 0u;
        if (step * STEP < rem) {
            v[s] = ldg_stream_v4(values + (pos >> 3) + step * L);
            w[s] = ldg_stream_u32(deltas + (pos >> 3) + step * L);
        }
    };
    const bool any_rows = block < block_hi;
    take_block();
#pragma unroll
    for (int s = 0; s < D; ++s) load_unit(s, s);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    stage_x();
    if (!any_rows) return;
    for (;;) {
        float acc[BV];
#pragma unroll
        for (int b = 0; b < BV; ++b) acc[b] = 0.f;
        do {
            // byte-wise prefix sums of the deltas and one scan over the group for two sub-steps, as in spmv.cu
            unsigned ce[D], co[D];
#pragma unroll
            for (int s = 0; s < D; ++s) {
                if (masks) {
                    const int r = rem - s * STEP;
                    if (__any_sync(0xffffffffu, (r > 0 && r < kGroup) || (s == 0 && lo > 0))) mask_unit(v[s], w[s], s == 0 ? lo : 0, r);
                }
                const unsigned ev = w[s] & 0x0f0f0f0fu, od = (w[s] >> 4) & 0x0f0f0f0fu;
                const unsigned pe = ev * 0x02020202u + 0x0c080400u, po = od * 0x02020202u;
                ce[s] = po * 256u + pe;
                co[s] = pe + po + 0x02020202u;
            }
            const unsigned t = (co[0] >> 24) | ((co[1] >> 8) & 0x00ff0000u);
            unsigned inc = t;
#pragma unroll
            for (int o = 1; o < L; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, inc, o, L);
                if (lig >= o) inc += u;
            }
            const unsigned g = __shfl_sync(0xffffffffu, inc, L - 1, L);
            const unsigned ex = inc - t;
#pragma unroll
            for (int s = 0; s < D; ++s) {
                if (s > 0 && left <= s * STEP) break;   // no row of the block reaches that far
                const unsigned sel = s ? 0x0100u : 0x0001u;
                const unsigned a0 = min(__dp2a_lo(ex, sel, run) + (unsigned)(2 * L * s), a_max);   // keeps malformed input inside the staged x
                run = __dp2a_lo(g, sel, run);
                const unsigned *vw = reinterpret_cast<const unsigned *>(&v[s]);
                const int ab = x_base + (int)a0 * (kWindowColBytes / 2);
                auto element_pair = [&](auto jt) {
                    constexpr int J = decltype(jt)::value;
                    unsigned xe[BV / 2], xo[BV / 2];
                    lds_vec<BV>((unsigned)add_byte<J, kWindowColBytes / 2>(ce[s], ab), xe);
                    lds_vec<BV>((unsigned)add_byte<J, kWindowColBytes / 2>(co[s], ab), xo);
#pragma unroll
                    for (int b = 0; b < BV; b += 2) {
                        acc[b] = fma_hh<0, 0>(acc[b], vw[J], xe[b / 2]);
                        acc[b + 1] = fma_hh<0, 1>(acc[b + 1], vw[J], xe[b / 2]);
                        acc[b] = fma_hh<1, 0>(acc[b], vw[J], xo[b / 2]);
                        acc[b + 1] = fma_hh<1, 1>(acc[b + 1], vw[J], xo[b / 2]);
                    }
                };
                element_pair(Int<0>{});
                element_pair(Int<1>{});
                element_pair(Int<2>{});
                element_pair(Int<3>{});
                load_unit(s, s + D);   // the unit D sub-steps on takes its place
            }
            lo = 0;
            run += (unsigned)(2 * L * D);
            pos += (unsigned)(D * STEP);
            rem -= D * STEP;
            left -= D * STEP;
        } while (left > 0);
        const unsigned row = (block - 1u) * K + (unsigned)(lane / L);
        const bool more = block < block_hi;
        if (more) {   // the first units of the next block are on their way while this one is added up
            take_block();
#pragma unroll
            for (int s = 0; s < D; ++s) load_unit(s, s);
        }
        const float total = group_sums<BV>(acc, lane);
        if (row < (unsigned)rows && lig < BV) {
            if (windows > 1) {
                partial[((size_t)(grp * windows + win) * rows + row) * BV + lig] = total;
            } else if (grp * BV + lig < batch) {
                __half *out = y + (size_t)(grp * BV + lig) * rows + row;
                float r = alpha * total;
                if (beta != 0.f) r += beta * __half2float(*out);
                *out = __float2half_rn(r);
            }
        }
        if (!more) break;
    }
}

// y = fp16(alpha * (sum over the windows, in their order) + beta * y). A CTA takes 256 / BV rows of a group of BV vectors: the
// partial sums are read as they lie ([row][vector]) and turned in shared memory, so that y is written in runs of rows.
template <int BV>
__global__ void __launch_bounds__(256)
windows_sum_kernel(const float *__restrict__ partial, __half *__restrict__ y, int rows, int windows, int batch, float alpha, float beta)
{
    constexpr int R = 256 / BV;
    __shared__ float turn[BV][R + 1];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int grp = blockIdx.y, r0 = blockIdx.x * R;
    const float *p = partial + ((size_t)grp * windows * rows + r0) * BV + threadIdx.x;
    float sum = 0.f;
    if (r0 + (int)threadIdx.x / BV < rows) {
#pragma unroll 4
        for (int w = 0; w < windows; ++w) sum += __ldcg(p + (size_t)w * rows * BV);
    }
    turn[threadIdx.x % BV][threadIdx.x / BV] = sum;
    __syncthreads();
    const int b = threadIdx.x / R, row = r0 + threadIdx.x % R;
    if (row < rows && grp * BV + b < batch) {
        __half *out = y + (size_t)(grp * BV + b) * rows + row;
        float r = alpha * turn[b][threadIdx.x % R];
        if (beta != 0.f) r += beta * __half2float(*out);
        *out = __float2half_rn(r);
    }
}

// Vectors that share a pass: 8, or 4 where that is all there are.
int vectors_per_pass(int64_t batch) { return batch > 4 ? 8 : 4; }

template <int BV>
int launch_windows(const void *values, const void *deltas, const void *sections, int rows, int cols, int stored, const void *x, void *y,
                   int batch, float alpha, float beta, void *workspace, uint32_t flags, cudaStream_t stream, const DeviceInfo &dev)
{
    const WindowLayout layout = window_layout(rows, cols, stored);
    const int windows = layout.count, width = layout.width, groups = (batch + BV - 1) / BV;
    const long long columns = (long long)windows * groups, n_blocks = ((long long)rows + K - 1) / K;
    long long shares = dev.sm_count / columns;   // CTAs that share the rows of a window and a group of vectors
    if (shares > n_blocks) shares = n_blocks;
    if (shares < 1) shares = 1;
    const size_t smem = (size_t)(kWindowFront + width + kWindowHalo) * kWindowColBytes;
    if (smem > (size_t)dev.max_smem_optin)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "the launch needs %lld bytes of shared memory, the device offers %d", (long long)smem, dev.max_smem_optin);
    auto kernel = windows_kernel<BV>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   // on every call: every device
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(columns * shares));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kernel, static_cast<const uint4 *>(values), static_cast<const unsigned *>(deltas), static_cast<const uint2 *>(sections),
                           static_cast<const __half *>(x), static_cast<float *>(workspace), static_cast<__half *>(y), rows, cols, stored, windows, width,
                           groups, (int)shares, batch, alpha, beta, (flags & MACKO_SPMV_MATRIX_IMMUTABLE) ? 1 : 0);
    if (e == cudaSuccess && windows > 1) {
        cfg.gridDim = dim3((unsigned)((rows + 256 / BV - 1) / (256 / BV)), (unsigned)groups);
        cfg.blockDim = dim3(256);
        cfg.dynamicSmemBytes = 0;
        e = cudaLaunchKernelEx(&cfg, windows_sum_kernel<BV>, static_cast<const float *>(workspace), static_cast<__half *>(y), rows, windows, batch, alpha, beta);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "windowed product launch: %s", cudaGetErrorString(e));
    return MACKO_OK;
}

constexpr int64_t kMaxBatch = 65535 * 4;   // groups are a grid dimension of the second kernel

int check_sizes(int64_t rows, int64_t cols, int64_t padded_count)
{
    if (rows < 0 || cols < 0 || padded_count < 0)
        return fail(MACKO_ERR_INVALID_ARGUMENT, "negative size (rows=%lld cols=%lld P=%lld)", (long long)rows, (long long)cols, (long long)padded_count);
    if (rows >= (1LL << 30) || cols >= (1LL << 24) || padded_count >= (1LL << 31))
        return fail(MACKO_ERR_SIZE_OVERFLOW, "rows=%lld cols=%lld P=%lld are beyond what windows can index", (long long)rows, (long long)cols, (long long)padded_count);
    return MACKO_OK;
}

}  // namespace
}  // namespace macko

extern "C" {

int64_t macko_spmm_windows_bytes(int64_t rows, int64_t cols, int64_t padded_count)
{
    using namespace macko;
    if (check_sizes(rows, cols, padded_count) != MACKO_OK) return -1;
    return rows * window_layout(rows, cols, padded_count).count * (int64_t)sizeof(uint2);
}

int macko_spmm_windows(const void *deltas, const int32_t *row_indices, int64_t rows, int64_t cols, int64_t padded_count,
                       void *windows, int64_t windows_bytes, void *stream)
{
    using namespace macko;
    const int st = check_sizes(rows, cols, padded_count);
    if (st != MACKO_OK) return st;
    if (rows == 0) return MACKO_OK;
    if (!windows || !row_indices || (padded_count > 0 && !deltas)) return fail(MACKO_ERR_INVALID_ARGUMENT, "null windows, row_indices or deltas");
    if (!aligned(windows, 8) || !aligned(deltas, 4) || !aligned(row_indices, 4))
        return fail(MACKO_ERR_MISALIGNED, "windows need 8-, deltas and row_indices 4-byte alignment");
    if (windows_bytes < macko_spmm_windows_bytes(rows, cols, padded_count))
        return fail(MACKO_ERR_WORKSPACE, "windows buffer has %lld bytes, %lld needed", (long long)windows_bytes, (long long)macko_spmm_windows_bytes(rows, cols, padded_count));
    const WindowLayout layout = window_layout(rows, cols, padded_count);
    window_sections_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const unsigned *>(deltas), row_indices, (int)rows, (int)padded_count, layout.count, layout.width, static_cast<uint2 *>(windows));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(MACKO_ERR_CUDA, "windows launch: %s", cudaGetErrorString(e));
    return MACKO_OK;
}

int64_t macko_spmm_windowed_workspace_bytes(int64_t rows, int64_t cols, int64_t padded_count, int64_t batch)
{
    using namespace macko;
    if (check_sizes(rows, cols, padded_count) != MACKO_OK || batch < 0 || batch > kMaxBatch) return -1;
    const int windows = window_layout(rows, cols, padded_count).count, bv = vectors_per_pass(batch);
    return windows > 1 ? (batch + bv - 1) / bv * bv * rows * windows * (int64_t)sizeof(float) : 0;
}

int macko_spmm_fp16_windowed(const void *values, const void *deltas, const int32_t *row_indices, int64_t rows, int64_t cols,
                             int64_t padded_count, const void *windows, int64_t windows_bytes, const void *x, void *y, int64_t batch,
                             float alpha, float beta, void *workspace, int64_t workspace_bytes, uint32_t flags, void *stream)
{
    using namespace macko;
    if (batch < 0 || batch > kMaxBatch) return fail(MACKO_ERR_INVALID_ARGUMENT, "batch %lld outside 0..%lld", (long long)batch, (long long)kMaxBatch);
    if (flags & ~(uint32_t)MACKO_SPMV_MATRIX_IMMUTABLE) return fail(MACKO_ERR_INVALID_ARGUMENT, "unknown flag bits 0x%x", flags);
    if (batch == 0) return MACKO_OK;   // nothing to read or write: x and y may be null
    int st = check_sizes(rows, cols, padded_count);
    if (st == MACKO_OK) st = check_product_args(values, deltas, row_indices, rows, cols, padded_count, x, y);
    if (st != MACKO_OK) return st;
    if (rows == 0) return MACKO_OK;
    if (!windows) return fail(MACKO_ERR_INVALID_ARGUMENT, "null windows");
    if (!aligned(windows, 8)) return fail(MACKO_ERR_MISALIGNED, "windows must be 8-byte aligned");
    if (windows_bytes < macko_spmm_windows_bytes(rows, cols, padded_count))
        return fail(MACKO_ERR_WORKSPACE, "windows buffer has %lld bytes, %lld needed", (long long)windows_bytes, (long long)macko_spmm_windows_bytes(rows, cols, padded_count));
    const int64_t need = macko_spmm_windowed_workspace_bytes(rows, cols, padded_count, batch);
    if (need > 0 && (!workspace || workspace_bytes < need))
        return fail(MACKO_ERR_WORKSPACE, "workspace has %lld bytes, %lld needed", (long long)(workspace ? workspace_bytes : 0), (long long)need);
    if (!aligned(workspace, 4)) return fail(MACKO_ERR_MISALIGNED, "workspace must be 4-byte aligned");
    const DeviceInfo *dev = nullptr;
    st = current_device_info(&dev);
    if (st != MACKO_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return vectors_per_pass(batch) == 8
        ? launch_windows<8>(values, deltas, windows, (int)rows, (int)cols, (int)padded_count, x, y, (int)batch, alpha, beta, workspace, flags, s, *dev)
        : launch_windows<4>(values, deltas, windows, (int)rows, (int)cols, (int)padded_count, x, y, (int)batch, alpha, beta, workspace, flags, s, *dev);
}
}
