// moe_grouped.cuh - the grouped expert GEMM of moe_tc5.cu: block-scaled tcgen05 over expert-contiguous positions.
//
// Positions come in groups of eight tokens; a group is 32 operand columns (four NVFP4 term rows per token), row
// term * 8 + token of the group's 32 rows.  A 32-token block is four groups, an 8-token block one.  Consecutive groups of
// one expert share a tile: the weight tile is brought into shared memory once for all of them, and the MMA's N is the number
// of live groups x 32, so neither the padding of an expert's last block nor a second block of the same expert costs another
// pass over the weights.  (One tile per 32-token block: at 1024 tokens and 4 of 128 experts half of the experts spill a few
// tokens into a second block, whose tile reads all of the expert's weights again for them.)
#pragma once
#include "nvf4_tc5.cuh"

namespace moe_gemm {

using namespace nvf4tc5;

enum Kind : uint32_t { kPlain = 0u, kScatter = 1u, kGated = 2u };   // the kernel of the first two is one (Args::scatter)

struct Args {
    const uint8_t* w_sf[2];      // tiled UE4M3 weight scales per plane
    const float* scale2[2];      // per-plane factor (device memory), or per expert when scale2_per_expert
    const float* bias[2];        // [expert][out_dim] or null
    float* out[2];               // plain: [positions][out_dim] per plane; scatter: part [(row, slot)][out_dim]; gated: out[0]
    const uint8_t* x_sf;         // [quad records][slab][2048]: the record of a run's groups 4q .. 4q + 3 sits at the first one's block
    const float* xstep;          // [positions]
    const uint32_t* block_expert;
    const uint32_t* sorted_row;
    const uint32_t* sorted_slot;  // scatter only
    const float* topk_w;          // scatter only
    uint32_t in_dim, out_dim, max_blocks, n_planes, n_active, scatter, ahead, scale2_per_expert, block_shift;  // 2: 32-token blocks, 0: 8
    float alpha, limit, up_add;   // gated only
    unsigned int* err_word;
};

// The ring leaves 16 KB of an SM's shared memory: the kernels in front and behind are dependent launches, and a CTA of theirs
// that finds no room here starts when this one has left (a ring of 216 KB cost a block of one token 0.4 us).  The ring of LONG runs
// takes it all: three stages of two slabs.
constexpr uint32_t kRing = 196u * 1024u, kRingLong = 216u * 1024u, kMaxSlots = 10u;
constexpr uint32_t kMaxBlocks = 1024;  // block_expert[] and the tile table are kept in shared memory
constexpr size_t kTableBytes = kMaxBlocks * 8u;   // experts, tiles, groups by block, live groups

// W groups per tile at most, NA weight tiles of 128 rows under one B.  NA = 2 (gate and up): one pair of accumulators.  NA = 1:
// two accumulators, the next tile's MMAs run under this one's epilogue.  A stage of the ring is KS slabs (256 elements) of the
// weight tiles, the groups and their scale records; a stage's hand-off costs the issuing warp about as long as half a slab (its
// busy cycles per slab of four groups: 530 in stages of two slabs, 615 in stages of one, 660 with the second scale cell of six groups).
template <uint32_t W, uint32_t NA, bool LONG>
struct Geo {
    static constexpr uint32_t kS = NA == 1u && W <= (LONG ? 4u : 2u) ? 2u : 1u;
    static constexpr uint32_t kN = W * 32u, kGroupBytes = 32u * BKB, kQuads = (W + 3u) / 4u;
    // a stage: weight boxes [tile][slab], groups [slab][group], weight records [tile][slab], activation records [quad][slab]
    static constexpr uint32_t kOffB = kS * NA * kABytes, kOffSfa = kOffB + kS * W * kGroupBytes;
    static constexpr uint32_t kOffSfb = kOffSfa + kS * NA * kSfBytes, kSlot = kOffSfb + kS * kQuads * kSfBytes;
    static constexpr uint32_t kFit = (LONG ? kRingLong : kRing) / kSlot, kSlots = kFit < kMaxSlots ? kFit : kMaxSlots;
    // tensor memory: two accumulators, then the scale cells of a slab; copies and MMAs of one thread execute in order, two
    // sets or more let a slab's copies run under the MMAs of the one before
    static constexpr uint32_t kSfStep = 4u * kQuads, kSfSlab = NA * 16u + 4u * kSfStep, kSfCol0 = 2u * kN;
    static constexpr uint32_t kRoom = (kTmemCols - kSfCol0) / kSfSlab, kSets = kRoom < kSlots * kS ? kRoom : kSlots * kS;
    static_assert(kSets >= 2u && kSlots >= 3u && kSlot % 1024u == 0u, "tensor memory, shared memory, alignment");
};

struct Ctl {
    uint64_t full[kMaxSlots], empty[kMaxSlots], tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
    int abort_flag;
    uint32_t starts[kMaxBlocks / 32u], counts[kMaxBlocks / 32u], widths[kMaxBlocks / 32u];   // of 32 blocks each, for the tile table
};

// tile word: first group | live groups << 13
__device__ __forceinline__ uint32_t tile_group(uint32_t t) { return t & 0x1FFFu; }
__device__ __forceinline__ uint32_t tile_ng(uint32_t t) { return t >> 13; }

// The routing tables past the first-level cache.  With `ahead` they are read before this kernel's own griddepcontrol.wait: the
// kernel in front began only when the one that wrote them was complete (it waits before it lets this one in), so L2 has them, but
// nothing clears a line that an earlier launch left in this SM's first level before that wait.
__device__ __forceinline__ uint32_t table_word(const uint32_t* p) { return __ldcg(p); }

// Groups of the tile that starts at block b, 0 where none does; r: blocks of the run from b on (counted up to MAXG + 1), from_first:
// blocks of the run before b, live / next_live: live groups of b and of the block behind it.  A run = the consecutive blocks of one
// expert.  Every four groups are a tile; with MAXG = 6 the last one takes a rest of up to six (a rest of one or two groups is not
// worth a pass over the weights).  Tiles start at a scale record's first group: an MMA takes its scales from an even tensor-memory
// column, an odd one is a misaligned address.
template <uint32_t MAXG>
__device__ __forceinline__ uint32_t tile_groups(uint32_t shift, uint32_t from_first, uint32_t r, uint32_t live, uint32_t next_live) {
    static_assert(MAXG == 4u || MAXG == 6u, "tiles start at whole records");
    if (shift == 0u) return (from_first & 3u) != 0u || (MAXG > 4u && from_first && r <= MAXG - 4u) ? 0u : r <= MAXG ? r : 4u;
    if (MAXG > 4u && from_first && r == 1u && live <= MAXG - 4u) return 0u;
    if (MAXG > 4u && r == 2u && next_live <= MAXG - 4u) return 4u + next_live;
    return r > 1u ? 4u : live;
}

// The tile table of a call, the whole CTA; a warp takes 32 blocks at a time.  (One warp for all of them took 0.33 us per 32 blocks, all
// of it in front of the first MMA where nothing hides it: down at K = 512, N = 384, 32 experts, 12800 pairs on 430 blocks 24.9 us, in
// this form 20.8.)
template <uint32_t MAXG>
__device__ __forceinline__ uint32_t build_tiles(const Args& a, uint32_t* s_expert, uint16_t* s_tile, uint8_t* s_ng, uint8_t* s_live,
                                                Ctl* sh, uint32_t& widest) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5, nb = a.max_blocks, shift = a.block_shift;
    const uint32_t chunks = (nb + 31u) >> 5;
    for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) {
        const uint32_t e = table_word(a.block_expert + b);
        s_expert[b] = e;
        if (shift && e != PDK_MOE_PAD) {   // a 32-token block's padding is at its end
            uint32_t live = 1;
#pragma unroll
            for (uint32_t g = 1; g < 4u; ++g) live += table_word(a.sorted_row + b * 32u + g * 8u) != PDK_MOE_PAD;
            s_live[b] = (uint8_t)live;
        }
    }
    __syncthreads();
    auto expert_at = [&](uint32_t b) { return b < nb ? s_expert[b] : PDK_MOE_PAD; };
    for (uint32_t c = warp; c < chunks; c += nwarp) {
        const uint32_t b = c * 32u + lane;
        const uint32_t starts = __ballot_sync(0xffffffffu, b == 0u || expert_at(b) != expert_at(b - 1u));
        if (lane == 0u) sh->starts[c] = starts;
    }
    __syncthreads();
    auto groups_at = [&](uint32_t c) {
        const uint32_t b = c * 32u + lane, e = expert_at(b);
        if (e == PDK_MOE_PAD) return 0u;
        uint32_t q = c, mine = sh->starts[c] & (0xffffffffu >> (31u - lane));
        while (mine == 0u) mine = sh->starts[--q];     // bit 0 of the first word is set
        const uint32_t from_first = b - (q * 32u + 31u - __clz(mine));
        uint32_t r = 1;
        while (r <= MAXG && expert_at(b + r) == e) ++r;
        const uint32_t live = shift ? s_live[b] : 1u, next_live = shift && r > 1u ? s_live[b + 1u] : 1u;
        return tile_groups<MAXG>(shift, from_first, r, live, next_live);
    };
    for (uint32_t c = warp; c < chunks; c += nwarp) {
        const uint32_t ng = groups_at(c), tiles = __ballot_sync(0xffffffffu, ng != 0u), most = __reduce_max_sync(0xffffffffu, ng);
        if (c * 32u + lane < nb) s_ng[c * 32u + lane] = (uint8_t)ng;
        if (lane == 0u) { sh->counts[c] = __popc(tiles); sh->widths[c] = most; }
    }
    __syncthreads();
    const uint32_t count = lane < chunks ? sh->counts[lane] : 0u;
    widest = __reduce_max_sync(0xffffffffu, lane < chunks ? sh->widths[lane] : 0u);
    for (uint32_t c = warp; c < chunks; c += nwarp) {
        const uint32_t b = c * 32u + lane, ng = b < nb ? s_ng[b] : 0u, before = __reduce_add_sync(0xffffffffu, lane < c ? count : 0u);
        const uint32_t tiles = __ballot_sync(0xffffffffu, ng != 0u);
        if (ng) s_tile[before + __popc(tiles & ((1u << lane) - 1u))] = (uint16_t)((b << shift) | (ng << 13));
    }
    return __reduce_add_sync(0xffffffffu, count);
}

// The same for calls of up to 32 blocks: every warp for itself, from global memory straight into a table of its own, so
// nothing waits for another warp (1.1 us of a call of one token's).
template <uint32_t MAXG>
__device__ __forceinline__ uint32_t build_tiles_warp(const Args& a, uint32_t* s_expert, uint16_t* s_tile, uint32_t& widest, bool& once) {
    const uint32_t lane = threadIdx.x & 31u, shift = a.block_shift;
    const uint32_t e = lane < a.max_blocks ? table_word(a.block_expert + lane) : PDK_MOE_PAD;
    const bool used = e != PDK_MOE_PAD;
    uint32_t live = 1;
    if (shift && used) {
#pragma unroll
        for (uint32_t g = 1; g < 4u; ++g) live += table_word(a.sorted_row + lane * 32u + g * 8u) != PDK_MOE_PAD;
    }
    const uint32_t prev = __shfl_up_sync(0xffffffffu, e, 1);
    const uint32_t starts = __ballot_sync(0xffffffffu, lane == 0u || e != prev);
    const uint32_t first = 31u - __clz(starts & (0xffffffffu >> (31u - lane)));
    const uint32_t later = lane == 31u ? 0u : starts >> (lane + 1u);               // runs that start behind this block
    const uint32_t r = later ? (uint32_t)__ffs(later) : 32u - lane;                // blocks of the run from here on
    const uint32_t next_live = __shfl_down_sync(0xffffffffu, live, 1);
    const uint32_t ng = used ? tile_groups<MAXG>(shift, lane - first, r, live, next_live) : 0u;
    const uint32_t tiles = __ballot_sync(0xffffffffu, ng != 0u);
    s_expert[lane] = e;
    if (ng) s_tile[__popc(tiles & ((1u << lane) - 1u))] = (uint16_t)((lane << shift) | (ng << 13));
    widest = __reduce_max_sync(0xffffffffu, ng);
    once = __popc(tiles) == __popc(starts & __ballot_sync(0xffffffffu, used));
    __syncwarp();
    return __popc(tiles);
}

// One 256-element K slab of a tile: `steps` MMAs of 64 elements, each preceded by the copies of its scale cells - the weight
// tile's, and NB cells of the activations: none when another weight tile under the same B has brought them.  The block has only
// the copies that a tile of this width needs: a predicated-off copy takes the issuing warp as long as one that runs, and so does
// a branch between two such blocks (either one: 13 instead of 11.6 us for gate and up of one token, 4 experts of 2880 x 2880).
#define PDK_GRP_STEP(J, PRED, CPB0, CPB1)                                                                              \
    "setp.gt.and.u32 ej, %9, " #J ", e;\n\t"                                                                           \
    "add.u64 a, %1, " #J "*2;\n\tadd.u64 b, %2, " #J "*2;\n\tadd.u32 sa, %5, " #J "*4;\n\tadd.u32 sb, %6, " #J "*%10;\n\t" \
    "add.u64 ca, %7, " #J "*32;\n\tadd.u64 cb, %8, " #J "*32;\n\t"                                                     \
    "@ej tcgen05.cp.cta_group::1.32x128b.warpx4 [sa], ca;\n\t" CPB0 CPB1                                               \
    "@ej tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], a, b, %3, [sa], [sb], " PRED ";\n\t"
#define PDK_GRP_CELL "@ej tcgen05.cp.cta_group::1.32x128b.warpx4 [sb], cb;\n\t"
#define PDK_GRP_CELL2 "add.u32 sc, sb, 4;\n\tadd.u64 cc, cb, %11;\n\t@ej tcgen05.cp.cta_group::1.32x128b.warpx4 [sc], cc;\n\t"
#define PDK_GRP_SLAB(CPB0, CPB1)                                                                                       \
    asm volatile("{\n\t.reg .pred e, p, q, ej;\n\t.reg .b64 a, b, ca, cb, cc;\n\t.reg .b32 sa, sb, sc;\n\t"             \
                 "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t"                     \
                 PDK_GRP_STEP(0, "p", CPB0, CPB1) PDK_GRP_STEP(1, "q", CPB0, CPB1)                                     \
                 PDK_GRP_STEP(2, "q", CPB0, CPB1) PDK_GRP_STEP(3, "q", CPB0, CPB1) "}" ::"r"(d_tmem),                  \
                 "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc_first), "r"(sfa_t), "r"(sfb_t), "l"(cell_a),            \
                 "l"(cell_b), "r"(steps), "n"(SBSTEP), "n"(QUAD)                                                       \
                 : "memory")
template <uint32_t NB, uint32_t SBSTEP, uint32_t QUAD>
__device__ __forceinline__ void slab_group(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc_first,
                                           uint32_t sfa_t, uint32_t sfb_t, uint32_t sfa_smem, uint32_t sfb_smem, uint32_t steps) {
    const uint64_t cell = ((uint64_t)1u << 16) | ((uint64_t)8u << 32);
    const uint64_t cell_a = (uint64_t)((sfa_smem >> 4) & 0x3FFFu) | cell, cell_b = (uint64_t)((sfb_smem >> 4) & 0x3FFFu) | cell;
    if constexpr (NB == 0u) { PDK_GRP_SLAB("", ""); }
    else if constexpr (NB == 1u) { PDK_GRP_SLAB(PDK_GRP_CELL, ""); }
    else { PDK_GRP_SLAB(PDK_GRP_CELL, PDK_GRP_CELL2); }
}
#undef PDK_GRP_STEP
#undef PDK_GRP_CELL
#undef PDK_GRP_CELL2
#undef PDK_GRP_SLAB

// A value that all lanes hold, as the compiler cannot know of one that comes from memory: a warp-wide reduction leaves it in a
// uniform register.  Descriptors, tensor-memory addresses and the branches around TMA and tcgen05 instructions depend on it.
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_or_sync(0xffffffffu, v); }

// tc5::mbar_wait with the part that is rarely run out of line.  Two GEMMs and a preparation take turns on the instruction cache of
// an SM; what a kernel runs once per launch is fetched from L2 each time.
static __device__ __noinline__ bool wait_longer(uint64_t* bar, uint32_t parity, volatile int* abort_flag, unsigned int* err,
                                                unsigned int code, unsigned int detail) {
    return tc5::mbar_wait(bar, parity, tc5::WaitCtx{abort_flag, err}, code, detail);
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, const tc5::WaitCtx& ctx, unsigned int code, unsigned int detail) {
    return tc5::mbar_try_wait(bar, parity) || wait_longer(bar, parity, ctx.abort_flag, ctx.err, code, detail);
}

__device__ __forceinline__ uint64_t l2_policy_normal() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void bulk_load_hint_elect(void* smem_dst, const void* gmem, uint32_t bytes, uint64_t* bar, uint64_t policy) {
    asm volatile(TC5_ELECT
                 "@e cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n\t}" ::"r"(
                     tc5::smem_u32(smem_dst)),
                 "l"(gmem), "r"(bytes), "r"(tc5::smem_u32(bar)), "l"(policy)
                 : "memory");
}

// What a tile index means: the groups, the weight plane (the first of two, where a tile has both) and the row tile.
template <uint32_t NA>
struct TileAt {
    uint32_t word, plane, rt;
    __device__ __forceinline__ TileAt(const uint16_t* s_tile, uint32_t tile, uint32_t per_chunk, uint32_t row_tiles) {
        const uint32_t rem = tile % per_chunk;
        word = uniform(s_tile[tile / per_chunk]);
        plane = NA == 1u ? rem / row_tiles : 0u;
        rt = NA == 1u ? rem % row_tiles : rem;
    }
};

// Roles: warp 0 brings the weights (TMA boxes, bulk copies of their scale records), warp 1 issues the MMAs, warp 2 brings the
// groups' term rows and their records, the others are the epilogue (lane quarter = warp % 4; the warps of a quarter take the
// groups in turn).  Tensor memory is addressed from column 0, where an allocation of all 512 columns starts.
// The code is kept short - one group per turn of the epilogue's loop, one kernel for raw rows and for down: what a launch runs is
// fetched into the instruction cache anew when another large kernel ran in between (with the epilogue unrolled over a tile's
// groups a block of one token took 38.2 us instead of 34.8, 512 tokens with 8 of 128 experts of 2048 x 768 180 instead of 166).
template <uint32_t W, uint32_t NA, uint32_t KIND, uint32_t EPI, bool WG, bool LONG>
__device__ __forceinline__ void roles(const CUtensorMap& tmap_w0, const CUtensorMap& tmap_w1, const CUtensorMap& tmap_x, const Args& a,
                                      uint8_t* rings, Ctl* sh, const uint32_t* s_expert, const uint16_t* s_tile, uint32_t tiles, bool once) {
    using G = Geo<W, NA, LONG>;
    constexpr uint32_t kBufs = NA == 2u ? 1u : 2u;
    const uint32_t warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31u;
    const uint32_t row_tiles = (a.out_dim + BM - 1u) / BM;
    const uint32_t per_chunk = NA == 2u ? row_tiles : a.n_planes * row_tiles;
    const uint32_t n_mma = a.in_dim >> 6;                 // 64-element MMA steps (in_dim % 64 == 0)
    const uint32_t num_kb = (n_mma + 3u) >> 2;            // 256-element slabs, the last may be partial
    const uint32_t n_tiles = tiles * per_chunk;
    const tc5::WaitCtx ctx{&sh->abort_flag, a.err_word};

    if (warp == 0) {
        // ------------------------------------------------------------ weights (whole warp, one lane issues)
        // Weights that a small call reads once leave L2 first, so the rows that the launches around this one hand on stay there (128
        // experts of 2880 x 2880, 1 / 4 / 8 tokens: 27.3 / 54.5 / 84.3 -> 26.0 / 50.9 / 80.4 us a block; over 24 shapes of up to 32
        // blocks 1.006 to 1.08 times faster, 1.04 on average).  Calls of most experts keep the normal policy: 60 tokens of that block
        // take 1.04 times as long with the other (the rest of a 256-byte line that the next slab wants has left by then), though of
        // 16 shapes with 37 to 160 blocks most would gain 1 to 6 %.
        const uint64_t policy = once ? tc5::l2_policy_evict_first() : l2_policy_normal();
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const TileAt<NA> t(s_tile, tile, per_chunk, row_tiles);
            const uint32_t expert = uniform(s_expert[tile_group(t.word) >> a.block_shift]);
            const CUtensorMap* tw = t.plane ? &tmap_w1 : &tmap_w0;
            const int32_t row = (int32_t)(expert * a.out_dim + t.rt * BM);
            const size_t sf0 = ((size_t)expert * row_tiles + t.rt) * num_kb * kSfBytes;
            const uint8_t* wsf = a.w_sf[t.plane] + sf0;
            for (uint32_t kb0 = 0; kb0 < num_kb; kb0 += G::kS) {
                ok = __all_sync(0xffffffffu, wait_for(&sh->empty[stage], phase ^ 1u, ctx, tc5::kErrEmptyWait, stage));
                if (!ok) break;
                uint8_t* st = rings + stage * G::kSlot;
                uint64_t* full = &sh->full[stage];
                const uint32_t nsl = min(G::kS, num_kb - kb0);
                const size_t kb_sf = (size_t)kb0 * kSfBytes;
                tc5::mbar_arrive_expect_tx_elect(full, nsl * NA * (kABytes + (WG ? 0u : kSfBytes)));
#pragma unroll
                for (uint32_t u = 0; u < G::kS; ++u)
                    if (u < nsl) {
                        const int32_t x = (int32_t)((kb0 + u) * BKB);
                        tc5::tma_load_2d_hint_elect(st + u * kABytes, tw, full, x, row, policy);
                        if (NA == 2u) tc5::tma_load_2d_hint_elect(st + (G::kS + u) * kABytes, &tmap_w1, full, x, row, policy);
                    }
                if (!WG) {
                    bulk_load_hint_elect(st + G::kOffSfa, wsf + kb_sf, nsl * kSfBytes, full, policy);
                    if (NA == 2u) bulk_load_hint_elect(st + G::kOffSfa + G::kS * kSfBytes, a.w_sf[1] + sf0 + kb_sf, nsl * kSfBytes, full, policy);
                } else {
                    // cell j of slab u: byte l*16 + c*4 + b = scale[rt*128 + c*32 + l][(kb0+u)*16 + j*4 + b]
                    const uint32_t sf_row = a.in_dim >> 4;
                    const uint32_t dst0 = tc5::smem_u32(st + G::kOffSfa) + lane * 16u;
#pragma unroll
                    for (uint32_t u = 0; u < G::kS; ++u)
                        if (u < nsl)
#pragma unroll
                            for (uint32_t j = 0; j < 4u; ++j) {
                                const uint32_t off = (kb0 + u) * 16u + j * 4u;
#pragma unroll
                                for (uint32_t c = 0; c < 4u; ++c) {
                                    const uint32_t r = t.rt * BM + c * 32u + lane;
                                    const uint32_t size = (r < a.out_dim && off < sf_row) ? 4u : 0u;
                                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                                                     dst0 + u * kSfBytes + j * 512u + c * 4u),
                                                 "l"(a.w_sf[t.plane] + (size ? (size_t)r * sf_row + off : 0u)), "r"(size)
                                                 : "memory");
                                }
                            }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc5::smem_u32(full)) : "memory");
                }
                if (++stage == G::kSlots) { stage = 0; phase ^= 1u; }
            }
        }
        if (!ok && lane == 0)
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
    } else if (warp == 2) {
        // ------------------------------------------------------------ activations (whole warp, one lane issues)
        if (a.ahead) pdk_pdl_wait_then_launch();
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const uint32_t word = uniform(s_tile[tile / per_chunk]), g0 = tile_group(word), ng = tile_ng(word), nq = (ng + 3u) >> 2;
            const size_t rec_bytes = (size_t)num_kb * kSfBytes;
            const uint8_t* xsf = a.x_sf + (size_t)(g0 >> a.block_shift) * rec_bytes;
            for (uint32_t kb0 = 0; kb0 < num_kb; kb0 += G::kS) {
                ok = __all_sync(0xffffffffu, wait_for(&sh->empty[stage], phase ^ 1u, ctx, tc5::kErrEmptyWait, stage));
                if (!ok) break;
                uint8_t* st = rings + stage * G::kSlot;
                uint64_t* full = &sh->full[stage];
                const uint32_t nsl = min(G::kS, num_kb - kb0);
                const size_t kb_sf = (size_t)kb0 * kSfBytes;
                tc5::mbar_arrive_expect_tx_elect(full, nsl * (ng * G::kGroupBytes + nq * kSfBytes));
#pragma unroll
                for (uint32_t u = 0; u < G::kS; ++u)
#pragma unroll
                    for (uint32_t g = 0; g < W; ++g)
                        if (u < nsl && g < ng)
                            tc5::tma_load_2d_elect(st + G::kOffB + (u * W + g) * G::kGroupBytes, &tmap_x, full,
                                                   (int32_t)((kb0 + u) * BKB), (int32_t)((g0 + g) * 32u));
                tc5::bulk_load_elect(st + G::kOffSfb, xsf + kb_sf, nsl * kSfBytes, full);
                // the second record: four groups on, four blocks of 8 tokens or one of 32
                if (G::kQuads > 1u && nq > 1u)
                    tc5::bulk_load_elect(st + G::kOffSfb + G::kS * kSfBytes, xsf + (4u >> a.block_shift) * rec_bytes + kb_sf,
                                         nsl * kSfBytes, full);
                if (++stage == G::kSlots) { stage = 0; phase ^= 1u; }
            }
        }
        if (!ok && lane == 0)
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
        uint32_t stage = 0, phase = 0, iter = 0, set = 0;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const TileAt<NA> t(s_tile, tile, per_chunk, row_tiles);
            const uint32_t ng = W == 1u ? 1u : tile_ng(t.word);
            const uint32_t buf = kBufs == 2u ? iter & 1u : 0u, aphase = kBufs == 2u ? (iter >> 1) & 1u : iter & 1u;
            // e2m1 x e2m1 (format code 1 in the mxf4 encoding), UE4M3 scales, scale ids 0
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((ng * 4u) << 17) | ((BM >> 4) << 24);
            ok = __all_sync(0xffffffffu, wait_for(&sh->tmem_empty[buf], aphase ^ 1u, ctx, tc5::kErrTmemEmptyWait, buf));
            if (!ok) break;
            ++iter;
            tc5::fence_after_sync();
            const uint32_t d_tmem = buf * G::kN;
            for (uint32_t kb0 = 0; kb0 < num_kb; kb0 += G::kS) {
                ok = __all_sync(0xffffffffu, wait_for(&sh->full[stage], phase, ctx, tc5::kErrFullWait, stage));
                if (!ok) break;
                tc5::fence_after_sync();
                if (WG) fence_proxy_async_smem();  // the gathered cells were written through the generic proxy
                const uint32_t s_addr = tc5::smem_u32(rings + stage * G::kSlot), nsl = min(G::kS, num_kb - kb0);
#pragma unroll
                for (uint32_t u = 0; u < G::kS; ++u) {
                    if (u >= nsl) break;
                    const uint32_t kb = kb0 + u, steps = min(4u, n_mma - kb * 4u);
                    const uint32_t sf_t = G::kSfCol0 + set * G::kSfSlab, sfb_t = sf_t + NA * 16u;
                    const uint32_t sfa = s_addr + G::kOffSfa + u * kSfBytes, sfb = s_addr + G::kOffSfb + u * kSfBytes;
                    const uint64_t b_desc = tc5::smem_desc_sw128(s_addr + G::kOffB + u * W * G::kGroupBytes);
                    const uint64_t a_desc = tc5::smem_desc_sw128(s_addr + u * kABytes);
                    // (a tile of up to four groups in a launch of wider ones copies a second cell all the same; no MMA reads it)
                    slab_group<G::kQuads, G::kSfStep, G::kS * 128u>(d_tmem, a_desc, b_desc, idesc, kb != 0u, sf_t, sfb_t, sfa, sfb, steps);
                    if (NA == 2u)
                        slab_group<0u, G::kSfStep, 0u>(d_tmem + G::kN, tc5::smem_desc_sw128(s_addr + (G::kS + u) * kABytes), b_desc,
                                                       idesc, kb != 0u, sf_t + 16u, sfb_t, sfa + G::kS * kSfBytes, sfb, steps);
                    if (++set == G::kSets) set = 0;
                }
                tc5::mma_commit_elect(&sh->empty[stage]);
                if (++stage == G::kSlots) { stage = 0; phase ^= 1u; }
            }
            if (ok) tc5::mma_commit_elect(&sh->tmem_full[buf]);
        }
    } else {
        // ------------------------------------------------------------ epilogue (one group at a time: the loop stays small)
        constexpr uint32_t kShare = EPI / 4u;
        const uint32_t quarter = warp & 3u, share = (warp - 3u) >> 2;
        if (a.ahead) pdk_pdl_wait();
        uint32_t iter = 0;
        bool ok = true;
        for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const TileAt<NA> t(s_tile, tile, per_chunk, row_tiles);
            const uint32_t g0 = tile_group(t.word), ng = W == 1u ? 1u : tile_ng(t.word);
            const uint32_t expert = s_expert[g0 >> a.block_shift];
            const uint32_t buf = kBufs == 2u ? iter & 1u : 0u, aphase = kBufs == 2u ? (iter >> 1) & 1u : iter & 1u;
            ++iter;
            // lane j * 8 + i: routing data of token i of this warp's j-th group, broadcast below
            const uint32_t my_g = min(share + kShare * (lane >> 3), ng - 1u);
            const uint32_t my_pos = (g0 + my_g) * 8u + (lane & 7u);
            const uint32_t my_src = a.sorted_row[my_pos];
            uint32_t my_row = my_pos;  // output row: position, or the (token, slot) pair
            float my_wgt = 1.0f;       // routing weight when scattering
            if (KIND != kGated && a.scatter && my_src != PDK_MOE_PAD) {
                my_row = my_src * a.n_active + a.sorted_slot[my_pos];
                my_wgt = a.topk_w[my_row];
            }
            const float my_step = a.xstep[my_pos];
            const uint32_t n = t.rt * BM + quarter * 32u + lane;
            float scale2[NA], bias[NA];
#pragma unroll
            for (uint32_t s = 0; s < NA; ++s) {
                const uint32_t p = NA == 2u ? s : t.plane;
                scale2[s] = a.scale2[p][a.scale2_per_expert ? expert : 0u];
                bias[s] = (n < a.out_dim && a.bias[p]) ? a.bias[p][(size_t)expert * a.out_dim + n] : 0.0f;
            }
            const uint32_t live = __ballot_sync(0xffffffffu, my_src != PDK_MOE_PAD);
            float* out = a.out[t.plane];
            ok = __all_sync(0xffffffffu, wait_for(&sh->tmem_full[buf], aphase, ctx, tc5::kErrTmemFullWait, buf));
            if (!ok) break;
            tc5::fence_after_sync();
#pragma unroll 1
            for (uint32_t g = share, from = 0; g < ng; g += kShare, from += 8u) {
                // tensor-memory lane = weight row; columns of a group = term * 8 + token
                float v[NA][8];
                uint32_t r[NA][32];
#pragma unroll
                for (uint32_t s = 0; s < NA; ++s)
                    tc5::tmem_ld_32x32(((quarter * 32u) << 16) + (buf + s) * G::kN + g * 32u, r[s]);
                tc5::tmem_ld_wait();
                if (g + kShare >= ng) {   // the last of this warp's share: the accumulators are in registers
                    tc5::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc5::mbar_arrive(&sh->tmem_empty[buf]);
                }
#pragma unroll
                for (uint32_t s = 0; s < NA; ++s)
#pragma unroll
                    for (uint32_t i = 0; i < 8u; ++i)
                        v[s][i] = fmaf(__uint_as_float(r[s][24u + i]), 0.000244140625f,
                                       fmaf(__uint_as_float(r[s][16u + i]), 0.00390625f,
                                            fmaf(__uint_as_float(r[s][8u + i]), 0.0625f, __uint_as_float(r[s][i]))));
                // Padding is computed too and the store is predicated: with a branch around each row a tile of 32 tokens held the
                // epilogue for 2500 cycles, and with short K it is what a tile costs (this form 1800).  The gated unit costs more a row,
                // and a group of a decode step has one or two tokens: it may stop at two points.
                const uint32_t rows = KIND == kGated ? 32u - __clz((live >> from) & 0xFFu) : 8u;
#pragma unroll
                for (uint32_t i = 0; i < 8u; ++i) {
                    if (KIND == kGated && (i == 2u || i == 4u) && rows <= i) break;
                    const bool is_live = (live >> (from + i)) & 1u;
                    const uint32_t row = __shfl_sync(0xffffffffu, my_row, from + i);
                    const float step = __shfl_sync(0xffffffffu, my_step, from + i);
                    const float wgt = KIND != kGated ? __shfl_sync(0xffffffffu, my_wgt, from + i) : 1.0f;
                    float y;
                    if (KIND == kGated) {
                        const float xg = fminf(fmaf(v[0][i], step * scale2[0], bias[0]), a.limit);
                        const float yu = fminf(fmaxf(fmaf(v[NA - 1u][i], step * scale2[NA - 1u], bias[NA - 1u]), -a.limit), a.limit);
                        y = (xg / (1.0f + __expf(-a.alpha * xg))) * (yu + a.up_add);
                    } else {
                        y = fmaf(v[0][i], step * scale2[0] * wgt, bias[0] * wgt);   // (acc * scale2 * step + bias) * routing weight
                    }
                    if (is_live && n < a.out_dim) out[(size_t)row * a.out_dim + n] = y;
                }
            }
            if (share >= ng && lane == 0) tc5::mbar_arrive(&sh->tmem_empty[buf]);   // a tile of fewer groups than shares
        }
    }
}

// MAXG: the most groups of a tile, 4 or 6 (build_tiles); the launch takes the geometry of the widest tile that it has.
template <uint32_t MAXG, uint32_t NA, uint32_t KIND, uint32_t EPI, bool WG, bool LONG>
__global__ void __launch_bounds__(96u + 32u * EPI, 1)
grouped_kernel(const __grid_constant__ CUtensorMap tmap_w0, const __grid_constant__ CUtensorMap tmap_w1,
               const __grid_constant__ CUtensorMap tmap_x, const Args a) {
    static_assert(EPI % 4u == 0u && (KIND == kGated) == (NA == 2u), "whole sets of four lane quarters; gate and up, or one plane");
    static_assert(MAXG <= EPI, "a warp's lanes hold the routing data of four groups: EPI / 4 shares of up to four");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* rings = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    Ctl* sh = reinterpret_cast<Ctl*>(rings + (LONG ? kRingLong : kRing));
    uint32_t* s_expert = reinterpret_cast<uint32_t*>(sh + 1);
    uint16_t* s_tile = reinterpret_cast<uint16_t*>(s_expert + kMaxBlocks);
    const uint32_t warp = threadIdx.x >> 5;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kMaxSlots; ++s) {
            tc5::mbar_init(&sh->full[s], WG ? 34 : 2);  // both producers' expect_tx arrivals (+ 32 lanes' cp.async arrivals)
            tc5::mbar_init(&sh->empty[s], 1);
        }
        for (uint32_t b = 0; b < 2u; ++b) {
            tc5::mbar_init(&sh->tmem_full[b], 1);
            tc5::mbar_init(&sh->tmem_empty[b], EPI);
        }
        sh->abort_flag = 0;
        tc5::mbar_fence_init();
        tc5::tma_prefetch_desc(&tmap_w0);
        tc5::tma_prefetch_desc(&tmap_w1);
        tc5::tma_prefetch_desc(&tmap_x);
    }
    if (warp == 1) {
        tc5::tmem_alloc(&sh->tmem_base, kTmemCols);
        tc5::tmem_relinquish();
    }
    // dependent launch: barriers and tensor memory are set up while the previous kernel drains.  ahead: the routing tables are
    // older than the kernel in front, so the tiles are laid out and the first weights requested under that kernel as well; only
    // what reads its rows, or writes where it may still read, waits for it.
    if (!a.ahead) pdk_pdl_wait_then_launch();
    uint32_t n, widest;
    bool once = false;   // every expert has one tile per row tile
    if (a.max_blocks <= 32u) {
        s_expert += 64u * warp;
        s_tile = reinterpret_cast<uint16_t*>(s_expert + 32u);
        n = build_tiles_warp<MAXG>(a, s_expert, s_tile, widest, once);
    } else {
        uint8_t* s_ng = reinterpret_cast<uint8_t*>(s_tile + kMaxBlocks);
        n = build_tiles<MAXG>(a, s_expert, s_tile, s_ng, s_ng + kMaxBlocks, sh, widest);
    }
    tc5::fence_before_sync();
    __syncthreads();
    tc5::fence_after_sync();
    if (WG || widest <= 1u) roles<1u, NA, KIND, EPI, WG, LONG>(tmap_w0, tmap_w1, tmap_x, a, rings, sh, s_expert, s_tile, n, once);
    else if (widest <= 2u) roles<2u, NA, KIND, EPI, false, LONG>(tmap_w0, tmap_w1, tmap_x, a, rings, sh, s_expert, s_tile, n, once);
    else if (widest <= 4u) roles<4u, NA, KIND, EPI, false, LONG>(tmap_w0, tmap_w1, tmap_x, a, rings, sh, s_expert, s_tile, n, once);
    else if (MAXG > 4u) roles<MAXG, NA, KIND, EPI, false, LONG>(tmap_w0, tmap_w1, tmap_x, a, rings, sh, s_expert, s_tile, n, once);

    tc5::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc5::fence_after_sync();
        tc5::tmem_dealloc(sh->tmem_base, kTmemCols);
    }
}

template <uint32_t MAXG, uint32_t NA, uint32_t KIND, uint32_t EPI, bool WG = false, bool LONG = false>
int launch(const CUtensorMap& tw0, const CUtensorMap& tw1, const CUtensorMap& tx, const Args& a, cudaStream_t st) {
    constexpr size_t smem = (size_t)(LONG ? kRingLong : kRing) + sizeof(Ctl) + kTableBytes + 1024u;
    static_assert(smem <= 227u * 1024u, "shared memory of an SM");
    auto kern = grouped_kernel<MAXG, NA, KIND, EPI, WG, LONG>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const uint32_t row_tiles = (a.out_dim + BM - 1u) / BM;
    const uint32_t per_chunk = NA == 2u ? row_tiles : a.n_planes * row_tiles;
    const uint64_t n_tiles = (uint64_t)a.max_blocks * per_chunk;
    uint32_t grid = (uint32_t)pdk_sm_count();
    if (grid > n_tiles) grid = (uint32_t)n_tiles;
    return pdk_launch_pdl(kern, dim3(grid), dim3(96u + 32u * EPI), smem, st, tw0, tw1, tx, a);
}

}  // namespace moe_gemm
