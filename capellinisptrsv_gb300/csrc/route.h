// Which kernel solves a level-ordered view when the caller leaves the choice to
// the library: rules on sizes, row lengths, precision and right-hand sides
// (host-only logic, tested without the CUDA runtime).
#pragma once

namespace capsp {

enum SolveKernel { kSolveRows = 0, kSolveChain = 1, kSolveStream = 2 };

// Rows per level up to which the chain kernel is the faster one.  Measured on
// GB300 in FP64, chain against row kernel: 8 rows per level (1,048,576 Zipf rows)
// 28.3 against 100.9 ms, 13 (2,003 rows) 29 against 137 us, 115 (40,000 rows of
// 3-12 dependencies) 162 against 460 us, 146 (38,261 rows of 3-10) 146 against 336
// us, 200 (20,000 rows of 1-5) 57 against 92 us, 377 (60,000 rows of 1-7) 171
// against 147 us.
constexpr long long kChainLevelRows = 256;
// ... and off-diagonal entries per level, as one SM walks them all.  Time of the row
// kernel / time of the chain kernel on 150 levels (rows per level, mean entries: 1, 4,
// 16 and 32 right-hand sides):
//   FP64  200 x 24  1.35 1.04 1.11 1.48    150 x 34  1.37 1.07 1.24 1.74
//         256 x 14  1.25 1.39 1.28 1.92    240 x 21  1.42 1.51 1.48 2.20
//         240 x 24  1.00 0.83 0.90 1.25    180 x 34  1.19 0.91 1.06 1.50
//         256 x 26  0.96 0.93 0.94 1.65    256 x 34  0.86 0.60 0.73 1.05
//   FP32  256 x 34  1.97 1.33 1.51 2.39    240 x 48  1.37 1.02 1.30 2.21
//         256 x 48  1.09 0.79 1.01 1.77
constexpr long long kChainLevelEntries64 = 5120, kChainLevelEntries32 = 11520;

// Rows per level below which the row kernels give every row a warp
constexpr long long kDeepRows = 32;

// Rows per level from which the stream kernel is the faster one whatever the
// number of right-hand sides (auto_kernel)
constexpr long long kStreamAnyRows = 12288;
// ... and the longest row it takes: a lane walks its row 8 or 12 entries at a
// time, so longer ones are for the mixed row kernel's warps.  (Banded matrices
// have some of 40 to 110 entries in their transposes, where few columns precede.)
constexpr int kStreamLongest = 128;
// ... and the share of rows (1 / this) in groups that the mixed row kernel would give
// a warp per row, with fewer than 8 right-hand sides.  A warp sums a row as a tree, a
// lane one entry after the other; where such rows are the norm that shows (12,800 rows
// per level, 33-60 entries, 2-norm of the error against more than 64 bits: FP64 2.6e-17,
// in a lane 4.6e-17; FP32 1.4e-8, 2.4e-8), where they are few it is lost in the rest
// (a seventh or a sixth of the rows: 1.02 to 1.06 times the error).  The trees cost
// time: 12,288 rows per level, 26 entries on average, FP64, row kernels / stream kernel
// 203 / 61 us (1 RHS) and 151 / 65 us (4); 6,000 rows of 33, FP32, 4 RHS 154 / 77 us; 1,500
// rows of 64 195 / 194 us.  With 8 and more the row kernels use a lane too.
constexpr long long kStreamHeavyShare = 6;
constexpr int kHeavyEntries = 32;  // stored entries per row of such a group, on average

struct ViewShape {
    long long n = 0, levels = 0, entries = 0;  // rows, levels, off-diagonal entries
    int longest = 0;                           // off-diagonal entries of the longest row
    long long heavy = 0;                       // rows in heavy groups, as grouped for `cols`
    bool chain = false;                        // a launch plan of the chain kernel exists
    bool f64 = true;
};

// whether the levels are narrow enough for the chain kernel
inline bool chain_levels(long long n, long long levels, long long entries, bool f64)
{
    return n <= kChainLevelRows * levels && entries <= (f64 ? kChainLevelEntries64 : kChainLevelEntries32) * levels;
}

// `cols`: right-hand sides, rounded up to the lanes or lane slots they take.
//
// The chain kernel comes first wherever it has a plan.  Of the others, the row
// kernels follow a chain of dependencies faster, the stream kernel gets through
// more rows.  Measured on GB300, time of the row kernel / time of the stream
// kernel:
//   1 RHS: FP64 0.87 at 5.9k rows per level, 1.03 at 12k, 1.25 at 14k, 1.36 at 47k;
//          FP32 0.92, -, 1.40, 1.42
//   2 RHS: FP64 0.91 at 5.9k, 1.47 at 14k, 1.74 at 47k; FP32 1.00, 1.51, 1.86
//   4 and more, FP32: 1.04 to 3.0 from 700 rows per level on
//   4 and more, FP64: by the rows' length.  5 to 8 entries on average (12 fit a
//          lane, 8 a lane of the row kernel): 1.05 to 1.24 from 700 rows per level
//          on.  Shorter: 1.03 at 4.6k row-columns per level, 0.96 at 11k, 1.17 at
//          23k, 1.10 to 1.49 above.  Longer: 0.94 at 6k, 1.10 at 12k.
inline SolveKernel auto_kernel(const ViewShape &s, int cols)
{
    if (s.chain)
        return kSolveChain;
    if (s.longest > kStreamLongest || s.levels < 1 || (cols < 8 && kStreamHeavyShare * s.heavy > s.n))
        return kSolveRows;
    const long long rows = s.n / s.levels;  // per level
    if (rows >= kStreamAnyRows)
        return kSolveStream;
    if (rows < kChainLevelRows || cols == 1)
        return kSolveRows;
    if (cols == 2)
        return rows >= 8192 ? kSolveStream : kSolveRows;
    if (!s.f64)
        return kSolveStream;
    if (s.entries > 8 * s.n)
        return rows * cols >= 10240 ? kSolveStream : kSolveRows;
    return s.entries > 5 * s.n || rows * cols >= 16384 ? kSolveStream : kSolveRows;
}

}  // namespace capsp
