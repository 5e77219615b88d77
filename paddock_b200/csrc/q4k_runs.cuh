// q4k_runs.cuh - which super-blocks of a plane a CTA of q4k_tc5.cu takes (plain C++: tests/test_q4k_runs.py compiles it for the host).
#pragma once
#include <cstdint>
#include <initializer_list>
#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace q4k_runs {

constexpr uint32_t kTileRows = 128;
constexpr uint32_t kZeroCtas = 32;     // CTAs of the kernel in front that zero y, beside one per token column
inline uint32_t token_columns(uint32_t batch) { return batch <= 16u ? 16u : 32u; }

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

// The cut with the shortest estimate, in us, of the busiest CTA: 1.3 per pair and 0.2 per tile that it touches (its accumulator is drained while nothing
// is produced); and where the grid leaves the kernel in front (a CTA per SM) no room, its CTAs start that much
// later: 0.02 per CTA too many, 0.04 with 32 token columns.  Fitted to 434 shapes of 9 ... 32 tokens (K = 1024 ... 16384, N = 512 ... 27648): 0.2 % over
// the best cut on average, 11 % at worst.  us, tiles / halves / pairs:
//   4608 x 19968, 10 tokens    32.2 / 28.0 / 21.5     runs of pairs balance whatever the tiles are
//   2048 x 25856, 20 tokens    18.3 / 15.7 / 16.2     halves touch two tiles at most, runs three
//   1024 x 23040, 10 tokens    11.6 / 10.3 / 10.3
//   9728 x 6528, 9 tokens      31.6 / 19.5            at most half a tile per SM: halves fill the chip
//   1536 x 9216, 25 tokens      9.2 /  9.8            but not where a pair saved is less than the later start
// Between half a tile and a tile per SM a cut saves the busiest CTA nothing.
inline Runs pick(uint32_t tiles, uint32_t ppt, uint32_t sms, uint32_t columns, float* estimate = nullptr) {
    const uint32_t ahead = kZeroCtas + columns;
    Runs best{};
    float best_cost = 0.0f;
    for (uint32_t cut : {kTiles, kHalves, kPairs}) {
        if (cut == kHalves && (ppt < 2u || (2u * tiles > sms && tiles < sms))) continue;
        if (cut == kPairs && tiles < sms) continue;      // a run would be shorter than a tile
        const uint64_t pieces = (uint64_t)tiles * (cut == kPairs ? ppt : cut == kHalves ? 2u : 1u);
        const uint32_t grid = pieces < sms ? (uint32_t)pieces : sms;
        const uint32_t most = (uint32_t)((pieces + grid - 1u) / grid);
        const uint32_t pairs = cut == kPairs ? most : cut == kTiles ? most * ppt : most / 2u * ppt + (most & 1u) * ((ppt + 1u) / 2u);
        const uint32_t touched = cut == kPairs ? (most + ppt - 2u) / ppt + 1u : cut == kTiles ? most : most / 2u + 1u;
        const float cost = 1.3f * (float)pairs + 0.2f * (float)touched +
                           (grid + ahead > sms ? (float)(grid + ahead - sms) * (columns > 16u ? 0.04f : 0.02f) : 0.0f);
        if (best.grid != 0u && cost >= best_cost) continue;
        best_cost = cost;
        best = Runs{cut, grid, (uint32_t)(pieces / grid), (uint32_t)(pieces % grid)};
    }
    if (estimate != nullptr) *estimate = best_cost;
    return best;
}

// What a launch of up to 32 tokens takes, in us: within 3 % (rms) over the same shapes.
inline float launch_us(uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t sms) {
    const uint32_t ppt = in_dim >> 9 != 0u ? in_dim >> 9 : 1u;
    float busiest = 0.0f;
    (void)pick((out_dim - 1u) / kTileRows + 1u, ppt, sms, token_columns(batch), &busiest);
    return 4.3f + 1.13f * busiest;
}

}  // namespace q4k_runs
