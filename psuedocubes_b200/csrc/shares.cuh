// How the work of the fused matcher is divided among its CTAs (plain arithmetic, on host and device).
//
// A block's work is its v rows and a fixed cost in rows.  A CTA works through shares: its first is its own number, further
// ones are claimed in ascending order.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define PC_BOTH __host__ __device__ __forceinline__
#else
#define PC_BOTH inline
#endif

// With pairs, shares are whole blocks: the first `pairs` of them two each, the others one.  Without, share i is the part
// [work i / n, work (i + 1) / n) of all work in block order.
struct Shares {
    uint32_t n, pairs;
};

// Few blocks (below 16 per CTA): one even part per CTA, so that the CTAs finish together whatever the blocks' sizes.
//
// More blocks, none above an eighth of a CTA's fair part: whole blocks, the last ones claimed singly.  The CTAs end within
// a block of each other, which costs less than the second building of each block that a cut divides.
//
// More blocks, one of them larger: a share of whole blocks could outlast everything else, so the work is cut into even
// parts again, as many for every CTA, but none below the fixed cost of 16 blocks, of which a cut adds one.  (2,518 blocks of
// eight windows and one of 9.6e5 or 9.7e6 rows, 148 CTAs: 2.81 and 3.09 ms, in whole blocks 6.40 and 40.9; without the
// large block, whole, 2.71.)
PC_BOTH Shares divide_work(uint64_t work, uint64_t largest, uint64_t nblocks, uint32_t grid, uint32_t block_cost) {
    if (nblocks < 16 * (uint64_t)grid) return {grid, 0};
    if (largest <= work / (8 * (uint64_t)grid)) {
        const uint32_t pairs = (uint32_t)((nblocks - 2 * (uint64_t)grid) / 2);
        return {(uint32_t)nblocks - pairs, pairs};
    }
    const uint64_t each = work / (16 * (uint64_t)block_cost * grid);
    return {grid * (uint32_t)(each < 1 ? 1 : each < 16 ? each : 16), 0};
}

// Rows [row, end) of a block, whose rows start at `start` in the work, that lie in [at, at_end) of it.
PC_BOTH void cut_rows(uint64_t start, uint64_t at, uint64_t at_end, uint32_t &row, uint32_t &end) {
    if (at_end < start + end) end = at_end > start ? (uint32_t)(at_end - start) : 0;
    if (at > start + row) row = at - start < end ? (uint32_t)(at - start) : end;
}
