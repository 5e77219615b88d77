// q4k_runs.cuh - which super-blocks of a plane a CTA of q4k_tc5.cu takes (plain C++: tests/test_q4k_runs.py compiles it for the host).
#pragma once
#include <cstdint>
#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace q4k_runs {

constexpr uint32_t kTileRows = 128;

// A plane is tiles of 128 rows, a tile's K range ppt pairs of super-blocks (weight boxes); the pairs of tile t are t ppt .. (t + 1) ppt.
// The pieces of a cut are pairs, half tiles or tiles in that order, and CTA c takes base of them, one more when c < extra.
// Whatever the cut, a tile has at most two CTAs (runs of pairs are as long as a tile or longer).  The longer runs come first, where c x pieces / grid
// spread them over the grid: 2048 x 25856, 20 tokens 18.8 -> 16.2 us, 1536 x 24320, 28 tokens 16.4 -> 14.0, 5120 x 25600, 16 tokens 29.5 -> 28.1.
enum Cut : uint32_t { kPairs, kHalves, kTiles };
struct Runs {
    uint32_t cut, grid, base, extra;
};

// Where CTA c's run starts.  (c x pieces / grid is also two 64-bit divisions in every thread: 0.1 to 0.4 us, 1024 x 8128, 31 tokens 8.33 -> 7.92.)
__host__ __device__ __forceinline__ uint32_t start(const Runs& r, uint32_t c, uint32_t ppt) {
    const uint32_t i = c * r.base + (c < r.extra ? c : r.extra);
    if (r.cut == kPairs) return i;
    if (r.cut == kTiles) return i * ppt;
    return (i >> 1) * ppt + (i & 1u) * (ppt >> 1);
}

// Half tiles where the plane has at most half a tile per SM (also of an odd number of pairs: 9728 x 6528, 9 tokens 31.6 us whole, 19.5 in halves), whole
// tiles up to one per SM.  From there runs or whole tiles by the busiest CTA's estimate: 1.5 us per pair, 1.3 per tile that it touches
// (its accumulator is drained while nothing is produced), 0.5 for runs.  4608 x 19968, 10 tokens: whole tiles 32.2 us, runs 22.7;
// 1536 x 25856, 20 tokens: 15.9, 17.3; 5120 x 25600, 16 tokens: half tiles in turn 30.1, runs 29.8.
inline Runs pick(uint32_t tiles, uint32_t ppt, uint32_t sms) {
    Cut cut = kTiles;
    uint32_t grid = tiles;
    if (2u * tiles <= sms && ppt >= 2u) {
        cut = kHalves;
        grid = 2u * tiles;
    } else if (tiles > sms) {
        const uint32_t whole = (tiles + sms - 1u) / sms;
        const uint64_t run = ((uint64_t)tiles * ppt + sms - 1u) / sms;
        const float by_tiles = (1.5f * (float)ppt + 1.3f) * (float)whole, by_pairs = 1.5f * (float)run + 1.3f * (float)(whole + 1u) + 0.5f;
        cut = by_tiles <= by_pairs ? kTiles : kPairs;
        grid = sms;
    }
    const uint64_t pieces = (uint64_t)tiles * (cut == kPairs ? ppt : cut == kHalves ? 2u : 1u);
    return Runs{cut, grid, (uint32_t)(pieces / grid), (uint32_t)(pieces % grid)};
}

}  // namespace q4k_runs
