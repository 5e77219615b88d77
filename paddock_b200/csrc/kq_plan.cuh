// kq_plan.cuh - shared-memory layout and split plan of kq_batch.cu (plain C++: tests/test_kq_plan.py compiles it for the host).
#pragma once
#include <cstddef>
#include <cstdint>
#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace kq {

enum Fmt : int { kQ4K = 0, kQ40 = 1, kQ5K = 2, kQ6K = 3, kQ80 = 4 };

constexpr uint32_t kRows = 16;           // rows of a tile
constexpr uint32_t kWarps = 16;          // of a CTA, whatever its column tiles (NT: tiles of 8 tokens, one or two)
constexpr uint32_t kMaxSplit = 8;        // portable cluster size
constexpr uint32_t kMaxStages = 6;
constexpr uint32_t kSmemMax = 232448;    // 227 KB
constexpr uint32_t kBox0 = kRows * 128u;

template <int F>
struct Fmts {
    static constexpr uint32_t kUnit = F == kQ80 ? 256u : F == kQ6K ? 192u : F == kQ5K ? 160u : 128u;   // data bytes of 256 weights
    static constexpr uint32_t kBox1 = kRows * (kUnit - 128u);                         // the high bits' box, or the second half's
    static constexpr uint32_t kBlocks = F == kQ6K ? 16u : 8u;
    static constexpr uint32_t kRec = F == kQ80 ? 16u : 24u, kRecs = kRows * kRec;     // scale records, of a row and of a tile
    static constexpr uint32_t kStage = kBox0 + kBox1 + kRecs;
};

// Shared memory: ring ([warp][stage] boxes, then second boxes, then records), the activation image, the partial tiles,
// the barriers.  When a round's weights are consumed its ring takes the partial sums that other CTAs send.
struct Layout {
    uint32_t off_box1, off_rec, off_b, pitch, off_step, off_xs, off_red, off_bar, total;
};
template <int F, uint32_t NT>
__host__ __device__ __forceinline__ Layout layout(uint32_t stages, uint32_t batch, uint32_t ku, uint32_t tiles) {
    using T = Fmts<F>;
    Layout l;
    const uint32_t n = kWarps * stages;
    l.off_box1 = n * kBox0;
    l.off_rec = l.off_box1 + n * T::kBox1;
    l.off_b = l.off_rec + n * T::kRecs;
    l.pitch = ku * 1024u + 64u;            // the odd 64 bytes put two tokens' rows on distinct banks
    l.off_step = l.off_b + batch * l.pitch;
    l.off_xs = l.off_step + ((ku * batch * 4u + 15u) & ~15u);
    l.off_red = l.off_xs + ku * batch * T::kBlocks * 4u;
    l.off_bar = l.off_red + (tiles + kWarps) * kRows * NT * 8u * 4u;
    l.total = l.off_bar + n * 8u + 16u;
    return l;
}

struct Plan {
    uint32_t split, clusters, rounds, round_tiles, ku, stages;
    size_t smem;
    float cost;      // the estimate that chose it, in units of one super-block's time in a warp
};

// S and the number of rounds by an estimate in units of one super-block's time in a warp: the longest warp's units and three
// more per round (the ring fills, the partials meet), one 48th per token and unit of K for the activation image that every CTA
// builds, and for a split the start of a cluster and the partial tiles that cross it (cluster sizes that are no power of two
// divide rows and SMs unevenly).  Fitted to 1480 random shapes of all formats on a B200 (K = 1024 ... 17408, N = 512 ... 27648, 2 ... 16
// tokens, every split): within 1.2 % of the best split on average, 16 % at worst.  (Without the terms for the image and
// the partials, and with a penalty for two stages, 4.4 %: Q6_K, K = 3328, N = 4096, 16 tokens 22.3 us at S = 3, 14.4 at S = 4.)
template <int F, uint32_t NT>
bool make_plan(Plan& best, const uint32_t* cap, uint32_t in_dim, uint32_t out_dim, uint32_t batch) {
    constexpr uint32_t kTilesMax = kSmemMax / (kRows * NT * 8u * 4u);      // no layout holds partials of more
    const uint32_t n_unit = in_dim >> 8, n_tiles = (out_dim + kRows - 1u) / kRows;
    float best_cost = 0.0f;
    best.split = 0u;
    for (uint32_t s = 1; s <= kMaxSplit && s <= n_unit; ++s) {
        if (cap[s] == 0u) continue;
        const uint32_t ku = (n_unit + s - 1u) / s, clusters = cap[s] < n_tiles ? cap[s] : n_tiles;
        const uint32_t per = (n_tiles + clusters - 1u) / clusters;
        // one tile a round at two stages has to fit (the first test keeps the sizes below within 32 bits)
        if (ku > 1024u || layout<F, NT>(2u, batch, ku, 1u).total > kSmemMax) continue;
        for (uint32_t rounds = (per + kTilesMax - 1u) / kTilesMax; rounds <= per; ++rounds) {
            const uint32_t rt = (per + rounds - 1u) / rounds;
            uint32_t d = kMaxStages;
            while (d >= 2u && layout<F, NT>(d, batch, ku, rt).total > kSmemMax) --d;
            // what the other CTAs send fits the ring
            if (s * batch * ((rt * kRows + s - 1u) / s) * 4u > kWarps * d * Fmts<F>::kStage) d = 0u;
            if (d < 2u) continue;
            const uint32_t units = (rt * ku + kWarps - 1u) / kWarps;
            const float cross = s > 1u ? 1.0f + (float)(batch * rt) / 128.0f + ((s & (s - 1u)) != 0u ? 0.5f : 0.0f) : 0.0f;
            const float cost = (float)rounds * (float)(units + 3u) + (float)(batch * ku) / 48.0f + cross;
            if (best.split == 0u || cost < best_cost) {
                best_cost = cost;
                best = Plan{s, clusters, rounds, rt, ku, d, layout<F, NT>(d, batch, ku, rt).total, cost};
            }
            break;     // more rounds only cost more
        }
    }
    return best.split != 0u;
}

}  // namespace kq
