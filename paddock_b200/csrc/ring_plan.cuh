// ring_plan.cuh - how gemv_ring.cu cuts a decode GEMV: warps, teams, CTAs of a cluster, stages, and where the register-staged kernels
// are faster (plain C++: tests/test_ring_plan.py compiles it for the host).
#pragma once
#include <cstddef>
#include <cstdint>

namespace ring {

constexpr uint32_t kMaxWarps = 12;                      // with 168 registers a thread
constexpr uint32_t kManyWarps = 20, kMaxTeams = 10;     // with 96: instances spill 8 bytes (Q6_K) to 92
constexpr uint32_t kMaxDepth = 4;
constexpr uint32_t kRedBufs = 8;                        // of a team
constexpr uint32_t kSmemMax = 232448;  // 227 KB per CTA on sm_100
constexpr uint32_t kBoxBytes = 2048;   // 16 rows x 128 bytes

struct RingPlan {
    uint32_t W;          // warps of a team
    uint32_t teams;      // teams of a CTA: tile i of the CTA is team i % teams'
    uint32_t D;          // stages per warp
    uint32_t split;      // CTAs of a cluster, which share tiles and split the pairs of a row
    uint32_t clusters;
    uint32_t invariant;  // W >= pairs of a row's part: a warp's pair never changes
    uint32_t k_part;     // elements of a row that a CTA's activations cover, at most
    uint32_t off_xmeta, off_red, off_recv, off_bar, off_rec, off_data, smem_bytes;
};

constexpr uint32_t kMaxSplit = 8;      // portable cluster size

// What the plan has to know of a format.  A unit is 256 weights of a row: kDataBytes packed, of which kDataBoxes boxes of 128 bytes
// and one of kHighBytes, a scale record of kRecBytes; sums over kBlock elements of x.  kMany: the instance of many warps exists.
// kStepCost, kManyCost, kRegsCost, kOddCost: prices of make_plan.
struct Q4KPlane {
    static constexpr uint32_t kDataBytes = 128, kRecBytes = 24, kDataBoxes = 1, kHighBytes = 0, kBlock = 32;
    static constexpr bool kMany = true;
    static constexpr float kStepCost = 0.048f, kManyCost = 0.052f, kRegsCost = 0.90f, kOddCost = 0.3f;
};
struct Q40Plane {
    static constexpr uint32_t kDataBytes = 128, kRecBytes = 24, kDataBoxes = 1, kHighBytes = 0, kBlock = 32;
    static constexpr bool kMany = true;
    static constexpr float kStepCost = 0.048f, kManyCost = 0.052f, kRegsCost = 0.83f, kOddCost = 0.3f;
};
struct Q80Plane {
    static constexpr uint32_t kDataBytes = 256, kRecBytes = 16, kDataBoxes = 2, kHighBytes = 0, kBlock = 32;
    static constexpr bool kMany = false;       // two boxes a unit leave no room for the stages
    static constexpr float kStepCost = 0.120f, kManyCost = 0.0f, kRegsCost = 1.91f, kOddCost = 0.0f;
};
struct Q5KPlane {
    static constexpr uint32_t kDataBytes = 160, kRecBytes = 24, kDataBoxes = 1, kHighBytes = 32, kBlock = 32;
    static constexpr bool kMany = true;
    static constexpr float kStepCost = 0.127f, kManyCost = 0.087f, kRegsCost = 1.55f, kOddCost = 0.0f;
};
struct Q6KPlane {
    static constexpr uint32_t kDataBytes = 192, kRecBytes = 24, kDataBoxes = 1, kHighBytes = 64, kBlock = 16;
    static constexpr bool kMany = true;
    static constexpr float kStepCost = 0.127f, kManyCost = 0.087f, kRegsCost = 1.49f, kOddCost = 0.0f;
};

// What a CTA keeps in shared memory; false when fewer than two stages per warp fit.
template <class F>
bool ring_layout(RingPlan& p, uint32_t in_dim, uint32_t out_dim) {
    constexpr uint32_t kData = 2u * (F::kDataBoxes * kBoxBytes + 16u * F::kHighBytes), kRec = 32u * F::kRecBytes;
    const uint32_t n = p.W * p.teams, pairs = ((in_dim + 511u) / 512u + p.split - 1u) / p.split;
    const uint64_t tiles = ((out_dim + 15u) / 16u + p.clusters - 1u) / p.clusters;
    const uint64_t recv = p.split > 1u ? (uint64_t)p.split * ((tiles * 16u + p.split - 1u) / p.split) * 4u : 0u;
    if (pairs > 512u || recv > kSmemMax) return false;
    p.invariant = p.W >= pairs ? 1u : 0u;
    p.k_part = pairs * 512u;
    p.off_xmeta = 2u * p.k_part + 32u;
    p.off_red = p.off_xmeta + (p.k_part / F::kBlock) * 8u;
    p.off_recv = p.off_red + kRedBufs * n * 64u;
    p.off_bar = (p.off_recv + (uint32_t)recv + 7u) & ~7u;
    p.off_rec = (p.off_bar + (n * kMaxDepth + 2u * kRedBufs * p.teams + 1u) * 8u + 127u) & ~127u;
    for (p.D = kMaxDepth; p.D >= 2u; --p.D) {
        p.off_data = (p.off_rec + n * p.D * kRec + 1023u) & ~1023u;  // swizzled boxes start on 1 KB
        p.smem_bytes = p.off_data + n * p.D * kData;
        if (p.smem_bytes <= kSmemMax) return true;
    }
    return false;
}

// The split with the shortest estimate, in us; false where the register-staged kernel (gemv_i8.cu, gemv_q6k.cu) has a shorter one.
//   one team     1.19 + steps (1.035 + kStepCost W): a step is a pair of a tile, and the longer the more warps share the SM; 0.5 more where a warp
//                meets more than one pair of a row: the CTA builds the limbs together, and B is read again at every step
//   many warps   2.36 + steps (0.65 + kManyCost warps) + 1.61 per tile of a team (its fold)
//   the stream   1.26 + 22 ns per KB of the CTA; the shorter of it and the above counts 4.4 % on top of the longer
//   split        1.45 more for two CTAs, 2.18 for more
//   odd rows     kOddCost more (the lanes copy the records; 4-bit planes, where the register kernel is close)
//   registers    1.43 + rounds of 64 rows per SM x K / 1024 x kRegsCost, up to 1.32 times that when its four slots are full
//                (fitted before calls with peers had an instance of their own, which made it 2 to 8 % faster on short rows)
// Fitted to every split of 973 shapes (K = 1280 ... 17408, N = 520 ... 25600, all formats).  Over every plan of 599 other random shapes
// (K = 1280 ... 17408, N = 512 ... 27648): 1.9 % over the best plan or the register kernel on average, 26 % at worst (Q4_K 9728 x 4864: 12.0 us, 9.5 with
// four warps x five teams); without the terms for more pairs a warp and for odd rows 2.3 %, 42 % (Q4_K 6912 x 520: 4.8 us, 3.4 in a cluster of four).
// Measured (us; register kernel -> here): Q6_K 17152 x 1024 25.2 -> 8.1 (four CTAs), 9472 x 2560 15.6 -> 9.8, 5120 x 25600 23.5 -> 20.1; Q8_0
// 5376 x 6016 11.7 -> 7.6, 17152 x 520 29.3 -> 5.3; Q4_K 9472 x 1024 12.0 -> 5.1; and the other way round Q4_K 1792 x 9792 6.1 -> 4.6, Q4_0 2816 x 4352
// 4.3 -> 3.7.  Q4_K 5120 x 25600: one team of ten 17.6, two of ten 17.3, four of five 14.8; 4096 x 25600: eight 14.5, six teams of three 13.0.
// Q4_0 5120 x 25600 stays on registers (16.2 us) though four teams of five take 15.3: a price that moves it makes other planes slower.
template <class F>
bool make_plan(uint32_t in_dim, uint32_t out_dim, const uint32_t* cap, RingPlan& best) {
    const uint32_t all = (in_dim + 511u) / 512u, n_tiles = (out_dim + 15u) / 16u, slots = 4u * cap[1];
    constexpr float kPairKb = (float)(2u * (F::kDataBoxes * kBoxBytes + 16u * F::kHighBytes) + 32u * F::kRecBytes) / 1000.0f;
    float best_cost = 0.0f;
    bool found = false;
    for (uint32_t s = 1; s <= kMaxSplit && s <= all; ++s) {
        if (cap[s] == 0u || s == 5u || s == 7u || (s > 1u && n_tiles > 3u * cap[1])) continue;    // wide planes fill the chip unsplit
        const uint32_t np = (all + s - 1u) / s, clusters = cap[s] < n_tiles ? cap[s] : n_tiles, per = (n_tiles + clusters - 1u) / clusters;
        const float fixed = (s == 1u ? 0.0f : s == 2u ? 1.45f : 2.18f) + ((in_dim & 511u) != 0u ? F::kOddCost : 0.0f);
        const float stream = 1.26f + (float)((uint64_t)per * np) * kPairKb * 0.022f;
        for (uint32_t rounds = 1; rounds <= 5u && rounds <= np; ++rounds) {
            const uint32_t W = (np + rounds - 1u) / rounds;
            if (W > kManyWarps) continue;
            const uint32_t most = kManyWarps / W, teams[5] = {1u, 2u, kMaxWarps / W, most / 2u, most};
            for (uint32_t i = 0; i < 5u; ++i) {
                const uint32_t T = teams[i] < kMaxTeams ? teams[i] : kMaxTeams, n = W * T, folds = T != 0u ? (per + T - 1u) / T : 0u;
                if (T == 0u || n > kManyWarps || (i > 0u && T <= teams[i - 1u])) continue;
                const bool many = T > 1u || n > kMaxWarps;
                if (many && !F::kMany) continue;
                const float steps = (float)(folds * rounds);
                const float work = many ? 2.36f + steps * (0.65f + F::kManyCost * (float)n) + 1.61f * (float)folds
                                        : 1.19f + steps * (1.035f + F::kStepCost * (float)n);
                const float cost = fixed + (work > stream ? work + 0.044f * stream : stream + 0.044f * work) + (rounds > 1u && !many ? 0.5f : 0.0f);
                if (found && cost >= best_cost) continue;
                RingPlan p{};
                p.W = W; p.teams = T; p.split = s; p.clusters = clusters;
                if (!ring_layout<F>(p, in_dim, out_dim)) continue;
                best_cost = cost;
                best = p;
                found = true;
            }
        }
    }
    const float fill = n_tiles < slots ? (float)n_tiles / (float)slots : 1.0f;
    const float regs = 1.43f + (float)((n_tiles + slots - 1u) / slots) * (float)in_dim / 1024.0f * F::kRegsCost * (1.0f + 0.32f * fill);
    return found && best_cost <= regs;
}

}  // namespace ring
