// CPU check of the rules that choose a solve's kernel (capsp::auto_kernel): the
// lines between the chain, stream and row kernels, from either side, and that no
// shape is claimed by two of them.
#include "route.h"

#include <cstdio>

using namespace capsp;

#define CHECK(c)                                          \
    do {                                                  \
        if (!(c)) {                                       \
            std::printf("FAIL line %d: %s\n", __LINE__, #c); \
            return 1;                                     \
        }                                                 \
    } while (0)

static ViewShape shape(long long rows, long long levels, long long mean, int longest, bool f64)
{
    ViewShape s;
    s.n = rows * levels;
    s.levels = levels;
    s.entries = mean * s.n;
    s.longest = longest;
    s.f64 = f64;
    s.chain = chain_levels(s.n, s.levels, s.entries, f64);  // as where the plan fits
    return s;
}

int main()
{
    for (int f64 = 0; f64 < 2; ++f64)
        for (int cols = 1; cols <= 32; cols *= 2)
            for (long long mean = 1; mean <= 12; ++mean) {
                // around the chain kernel's line: the chain kernel up to and with it, whatever else would hold
                CHECK(auto_kernel(shape(255, 100, mean, 12, f64), cols) == kSolveChain);
                CHECK(auto_kernel(shape(256, 100, mean, 12, f64), cols) == kSolveChain);
                CHECK(auto_kernel(shape(257, 100, mean, 12, f64), cols) != kSolveChain);
                // a matrix without a plan there never takes it
                ViewShape s = shape(256, 100, mean, 12, f64);
                s.chain = false;
                CHECK(auto_kernel(s, cols) != kSolveChain);
                // wide levels: stream for any number of right-hand sides
                CHECK(auto_kernel(shape(12288, 3, mean, 12, f64), cols) == kSolveStream);
                CHECK(auto_kernel(shape(12287, 3, mean, 12, f64), 1) == kSolveRows);
                // rows longer than a lane walks
                CHECK(auto_kernel(shape(20000, 3, mean, 129, f64), cols) == kSolveRows);
            }
    CHECK(!chain_levels(25601, 100, 0, true) && chain_levels(25600, 100, 0, true));
    // entries per level, by precision
    CHECK(chain_levels(20000, 100, 512000, true) && !chain_levels(20000, 100, 512001, true));
    CHECK(chain_levels(20000, 100, 1152000, false) && !chain_levels(20000, 100, 1152001, false));
    // two right-hand sides, and FP64 by row-columns per level
    CHECK(auto_kernel(shape(8191, 3, 4, 12, true), 2) == kSolveRows);
    CHECK(auto_kernel(shape(8192, 3, 4, 12, true), 2) == kSolveStream);
    CHECK(auto_kernel(shape(4095, 3, 4, 12, true), 4) == kSolveRows);
    CHECK(auto_kernel(shape(4096, 3, 4, 12, true), 4) == kSolveStream);
    CHECK(auto_kernel(shape(4095, 3, 6, 12, true), 4) == kSolveStream);
    CHECK(auto_kernel(shape(300, 3, 4, 12, false), 4) == kSolveStream);
    CHECK(auto_kernel(shape(300, 3, 4, 12, false), 2) == kSolveRows);
    // rows that the mixed row kernel would sum as trees: a few of them, or more, with
    // fewer than 8 right-hand sides and with 8
    for (int cols = 1; cols <= 32; cols *= 2) {
        ViewShape s = shape(12800, 4, 40, 60, true);
        s.heavy = s.n / 6;
        CHECK(auto_kernel(s, cols) == kSolveStream);
        s.heavy = s.n / 6 + 1;
        CHECK(auto_kernel(s, cols) == (cols < 8 ? kSolveRows : kSolveStream));
    }
    std::printf("routes ok\n");
    return 0;
}
