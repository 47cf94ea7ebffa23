// How the matcher's warps claim the seeds [0, total) of a launch.
//
// A block takes the next of `blocks` rows when it starts, and its warp w the
// seed row + blocks * w: neighbouring seeds (of one hub, often) start in
// different blocks.  The seeds behind the rows are claimed one at a time.  A
// warp that finds no more of those takes a row whose block has not started, and
// all of its seeds: no seed belongs to a block that has not started, so that
// whatever part of the grid is resident finishes the launch (another handle's
// kernels may hold the rest of the device for as long).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CGB_HD __host__ __device__
#else
#define CGB_HD
#endif

namespace cgb {

// Where a warp's next seed comes from: its block's row, a row it took alone, the
// counter, the counter after a wait, nowhere.
enum : uint32_t { kSeedFirst = 0, kSeedRow = 1, kSeedNext = 2, kSeedLater = 3, kSeedNone = 4 };

// The next seed of a warp, or `total` (then `from` is kSeedLater or kSeedNone).
// A warp whose block's row holds no seed for it looks for others only later
// (`patient`), after a wait for the blocks that are about to start.
// counter[0]: seeds claimed behind the rows; counter[1]: rows taken.  add(i, n):
// atomic addition to counter[i]; peek(i): its value, perhaps an old one.
template <class Add, class Peek>
CGB_HD inline uint32_t seed_claim(uint32_t& from, uint32_t& row, uint32_t block_row, uint32_t w, uint32_t total,
                                  uint32_t blocks, uint32_t warps, bool patient, Add add, Peek peek) {
    const uint32_t rows_end = blocks * warps;
    uint32_t seed = total;
    if (from == kSeedFirst) {
        from = kSeedNext;
        if (block_row < blocks) seed = block_row + blocks * w;
        if (seed < total) return seed;
        if (patient) from = kSeedLater;
    }
    while (from <= kSeedNext) {
        if (from == kSeedRow) {
            seed = row;
            row += blocks;
            if (seed < rows_end && seed < total) return seed;
        }
        from = kSeedNext;
        if (rows_end < total) {
            seed = rows_end + add(0, 1);
            if (seed < total) return seed;
        }
        from = kSeedNone;
        if (peek(1) < blocks && (row = add(1, 1)) < blocks) from = kSeedRow;
    }
    return total;
}

}  // namespace cgb
