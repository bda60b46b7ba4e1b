// Column windows of a compressed matrix: where the stored elements of every row enter each window of columns. Side metadata
// for the multi-vector product (windows.cu), derived once per matrix from row_indices and deltas; the three MACKO buffers
// stay what the format defines (the reference has no counterpart, it multiplies one vector at a time,
// c_benchmarking/utils.cuh:299).
//
// A unit (8 stored elements, aligned in the buffers) belongs as a whole to the window in which its first element lies, so
// that only the first and the last unit of a row are ever masked. The elements of a window's last unit may reach up to
// 127 columns beyond it: a CTA stages that many more columns of x behind its window.
#pragma once

#include <cstdint>

namespace macko {

constexpr int kWindowFront = 16;     // zero columns in front of a window: a unit may start up to 15 columns before its first element
constexpr int kWindowHalo = 128;     // columns of x behind it (8 elements, 16 columns each)
constexpr int kWindowColBytes = 128; // shared memory per column: 8 vectors x fp16 x 8 copies (or 4 x 16)
// Columns of a window at most. 227 KB would hold 1664, but beyond 195 KB of shared memory the SM keeps only 28 KB for the
// first-level cache, through which the 40 KB of matrix data that its 1024 threads keep in flight have to pass: 8 vectors,
// 4096x11008 d = 0.5 23.8 us in 8 windows, 31.6 in 7 of 1576 columns; 5000x6000 19.8 in 5, 26.5 in 4 of 1504.
constexpr int kWindowMax = 1408;
constexpr int kWindowSms = 148;      // of a B200; not asked for, the layout has to be the same where no device is
constexpr int kWindowWarps = 32;     // per SM, each with a block of four rows at a time

struct WindowLayout { int count, width; };

// How the columns are cut. All windows get the same number of SMs, and every warp of a window the same number of blocks of four
// rows or one more, so with few blocks per warp the last round may be mostly empty: among the six smallest numbers of
// windows the one with the lowest cost is taken, which is the mean of a warp's average and largest number of blocks, times
// the 64-element sub-steps of a section and 1.5 for its set-up and the half-filled last one, and 0.3 per window for
// the partial sums. 8 vectors, us, chosen / fewest windows: 4096x11008 d = 0.5 23.6 (9) / 23.8 (8), 5000x6000 19.0 (7) /
// 19.8 (5), 2048x2048 8.2 (4) / 10.4 (2), 4096x4096 d = 0.7 15.5 (4) / 16.4 (3), 300x4096 6.8 (8) / 9.4 (3); more windows than
// chosen: 11008x4096 24.6 (3) / 26.3 (4), 8192x8192 d = 0.7 41.0 (6) / 45.4 (7), 12288x4096 25.8 (3) / 27.2 (4).
inline WindowLayout window_layout(long long rows, long long cols, long long padded)
{
    const long long least = cols > kWindowMax ? (cols + kWindowMax - 1) / kWindowMax : 1;
    const long long blocks = (rows + 3) / 4;
    const double row = rows > 0 ? (double)padded / (double)rows : 0.0;   // stored elements
    long long best = least;
    double lowest = 0.0;
    for (long long w = least; w < least + 6; ++w) {
        const long long warps = (w < kWindowSms ? kWindowSms / w : 1) * kWindowWarps;
        const double per_warp = (double)blocks / (double)warps, most = (double)((blocks + warps - 1) / warps);
        const double cost = 0.5 * (per_warp + most) * (row / (64.0 * (double)w) + 1.5) + 0.3 * (double)w;
        if (w == least || cost < lowest) {
            lowest = cost;
            best = w;
        }
    }
    const long long width = ((cols + best - 1) / best + 7) / 8 * 8;
    return {(int)best, (int)(width < 8 ? 8 : width)};
}

// Section of a row inside a window, [window][row]: the first stored element, and elements << kWindowColBits | column in front
// of that element, counted from kWindowFront columns before the window. A well-formed row gives 1..143 for it
// (kWindowFront in the first window).
constexpr int kWindowColBits = 8;

}  // namespace macko
