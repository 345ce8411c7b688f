// mph_shapes.h - launch shapes that follow from a case's size and its device
// (host arithmetic without CUDA calls).
#pragma once

#include <algorithm>

namespace mph {

// The penalty operator's blocks (k_penalty.cu): rows a block, threads a row,
// whether a phase's iterations run in one cooperative kernel, and whether that
// kernel may take its form with one block an SM.
struct PenShape {
    int rows, w;
    bool resident, alone;
};

// pair, single: blocks that the device holds at once of the resident kernel's
// form with two blocks an SM and of the one with a block an SM (0: none);
// fits(rows): a block of that many rows fits the kernel's threads and shared
// memory.
//
// Resident (up to 155,648 particles on 152 SMs): up to `threads` threads a
// block, the rows spread evenly over at most two blocks an SM (the choice does
// not depend on what a step's blocks stage, so that staged and gathering runs
// keep one order of sums).  As long as the rows fit, one block an SM: half the
// blocks at a crossing and twice the registers.  A step of 33,600 particles in
// 3-D 2.44 -> 2.03 ms, 57,000 2.61 -> 2.42, 71,000 3.03 -> 2.75; 2-D the same
// either way.  (One block of up to 1024 threads an SM beyond 77,824 particles,
// with the registers of two: no difference.)
//
// Beyond, and for lists too long for shared memory, 256 rows a block in the
// per-iteration kernels (a row's share of the staged neighbours falls with the
// block), or fewer and several threads a row where the blocks would not reach
// every SM.
template <typename F>
inline PenShape pen_shape_for(int N, int min_rows, int threads, int pair, int single, F&& fits)
{
    auto spread = [N](int blocks) { return ((N + blocks - 1) / blocks + 31) / 32 * 32; };
    int rows = std::max(min_rows, pair > 0 ? spread(pair) : 0);
    if (single > 0) {
        const int one = spread(single);
        if (one > rows && fits(one)) rows = one;
    }
    const long long blocks = ((long long)N + rows - 1) / rows;
    if (fits(rows) && (blocks <= pair || blocks <= single)) return {rows, threads / rows, true, blocks <= single};
    if (N > 152 * 512) return {256, 1, false, false};
    if (N > 152 * 192) return {128, 2, false, false};
    return {64, 4, false, false};
}

}  // namespace mph
