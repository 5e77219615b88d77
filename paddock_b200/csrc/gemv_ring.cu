// gemv_ring.cu - single-token decode GEMV for Q4_K, Q5_K, Q6_K, Q4_0 and Q8_0 planes with the weights staged
// in shared memory by TMA, every warp running its own ring.
//
// The arithmetic is that of gemv_i8.cu (integer dot products on mma m16n8k32, activations as two
// int8 limbs of a 15-bit block floating point, block-diagonal B operand, f32 scale fold); what
// differs is how the bytes reach the SM.  A decode GEMV reads every weight once, so its time is
// the time HBM needs, provided enough bytes are in flight: about 7 MB over the chip.  Loads
// issued from registers cap that at (threads x registers spent on staging); here every warp keeps
// D tiled TMA copies outstanding into its own shared-memory stages, 150-190 KB per SM whatever
// the warps hold in registers, and requests them at kernel start, before the wait on the previous
// kernel in the stream (programmatic dependent launch).
//
//   * A CTA (one per SM) owns a contiguous range of 16-row tiles, its teams of W warps take them in turn, and warp w of a team
//     takes pairs w, w + W, ... of a tile (pair = two units, unit = 256 weights of a row; the last pair of an odd row is
//     half zeros).  On narrow planes of long rows a cluster of CTAs shares the tiles and splits the pairs, and the sums meet in
//     distributed shared memory.  Per (tile, pair) the warp's elected lane issues
//     2-D TMA copies of the 16 rows x 128 bytes of packed weights of each unit (two for Q8_0's 256 bytes; a second box for the high bits of
//     Q5_K and Q6_K) and one of the rows' scale records.  The planes stay in the byte layout the repack slots write
//     (super-block local: the engine concatenates planes at super-block offsets); the tensor maps
//     describe them as [rows][row bytes].
//   * The weight boxes are written with the 128-byte swizzle, which puts the 16-byte chunks that
//     the eight rows of one mma fragment load touch into eight different bank groups: fragment
//     loads are conflict free, and the shared-memory port carries each byte twice (in and out).
//   * A warp is the only reader of its stages: it waits on its own mbarrier, moves the fragments
//     to registers, and re-arms the stage itself after the mma sequence has consumed them.  No
//     producer warp, no cross-warp hand-shake in the weight path, so a warp that falls behind
//     delays nobody's loads.  When W equals the pairs of a row (one team) a warp meets
//     the same slice of the activations in every tile and keeps its B operand in registers.
//   * Per tile each warp leaves 16 partial row sums in one of the team's kRedBufs shared buffers and arrives
//     on the buffer's mbarrier without waiting; warp (tile mod W) of the team adds the W partials in warp order
//     once they are all there - it looks once per iteration - and stores y (or, row sharded, the
//     band into every rank's y).
//
// Every wait is bounded (tc5::mbar_wait): a wait that runs out records a code in the device
// error word and raises the CTA's abort flag; every warp then stops computing, and before it
// leaves waits (bounded again) for the copies it still has in flight.
#include <cstdlib>

#include "cluster_caps.cuh"
#include "gemv_i8_traits.cuh"
#include "ring_plan.cuh"
#include "tc5.cuh"

namespace {

using namespace gemv_i8;

using namespace ring;
static_assert(kMaxSplit == kPdkMaxCluster, "cluster_caps.cuh asks for these sizes");

enum : unsigned int { kErrRingFull = 0x11, kErrRingFold = 0x13, kErrRingDrain = 0x14, kErrRingFree = 0x15 };

// ---------------------------------------------------------------------------
// Ring traits: how a unit of a tile is read back from its boxes.  Stage, fold and kUnsignedA come
// from the shared traits.  The mma scheme differs from gemv_i8.cu's: one mma carries both
// activation limbs.  Its 32 k-slots are 8 weights of each of four blocks (lane t: block
// blk(p, t), slots 4t..4t+3 and 16+4t..16+4t+3), its eight columns are (block, limb) pairs, and
// column 2b + l is non-zero only in block b's slots.  Four mmas (j = 0..3) finish four blocks,
// two passes the unit's eight: 8 mmas per unit, and lane (g, t) ends up holding the high- and
// low-limb sums of blocks blk(0, t) and blk(1, t) for rows g and g + 8, which it folds with
// their scales.
// ---------------------------------------------------------------------------
// Physical offset of 16-byte chunk c of row r in a box written with the 128-byte swizzle.
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }
__device__ __forceinline__ uint32_t word4(const uint4& v, uint32_t i) { return i == 0u ? v.x : i == 1u ? v.y : i == 2u ? v.z : v.w; }

// load_ring arguments: `box` = the unit's first data box, o0 / o1 = swz(g, 2t) / swz(g, 2t + 1)
// (rows g + 8 lie 1024 bytes further), `rec` = row g's record of the unit (row g + 8: 8 box rows on).
struct RQ4K : Q4K, Q4KPlane {
    using Q4KPlane::kDataBytes, Q4KPlane::kRecBytes;
    static constexpr uint32_t kPasses = 2, kSub = 4;
    // pass p of lane t feeds block 2t + p: the low (p = 0) or high nibbles of ggml group t, whose
    // first 16 bytes (chunk 2t) sit in k-slots 4t.. and whose second 16 (chunk 2t+1) in slots 16+4t..
    __device__ static __forceinline__ uint32_t blk(uint32_t p, uint32_t t) { return 2u * t + p; }
    __device__ static __forceinline__ void a_pass(const Stage& s, uint32_t p, uint32_t j, uint32_t& a0, uint32_t& a1,
                                                  uint32_t& a2, uint32_t& a3) {
        const uint32_t mask = p ? 0xF0F0F0F0u : 0x0F0F0F0Fu;  // high nibbles stay in place: 16 x code, shifted back after
        a0 = word4(s.q[0], j) & mask;
        a1 = word4(s.q[2], j) & mask;
        a2 = word4(s.q[1], j) & mask;
        a3 = word4(s.q[3], j) & mask;
    }
    __device__ static __forceinline__ void load_ring(Stage& s, const uint8_t* box, const uint8_t*, const uint8_t* rec, uint32_t rec8,
                                                     uint32_t o0, uint32_t o1, uint32_t, uint32_t t) {
        s.q[0] = *reinterpret_cast<const uint4*>(box + o0);
        s.q[1] = *reinterpret_cast<const uint4*>(box + o1);
        s.q[2] = *reinterpret_cast<const uint4*>(box + o0 + 1024u);
        s.q[3] = *reinterpret_cast<const uint4*>(box + o1 + 1024u);
        const uint8_t* r1 = rec + rec8;
        s.dd[0] = *reinterpret_cast<const uint32_t*>(rec);
        s.dd[1] = *reinterpret_cast<const uint32_t*>(r1);
        s.sm[0] = (uint32_t)*reinterpret_cast<const uint16_t*>(rec + 4u + 2u * t) |
                  ((uint32_t)*reinterpret_cast<const uint16_t*>(rec + 12u + 2u * t) << 16);
        s.sm[1] = (uint32_t)*reinterpret_cast<const uint16_t*>(r1 + 4u + 2u * t) |
                  ((uint32_t)*reinterpret_cast<const uint16_t*>(r1 + 12u + 2u * t) << 16);
    }
};

struct RQ40 : Q40, Q40Plane {
    using Q40Plane::kDataBytes, Q40Plane::kRecBytes;
    static constexpr uint32_t kPasses = 2, kSub = 4;
    __device__ static __forceinline__ uint32_t blk(uint32_t p, uint32_t t) { return 2u * t + p; }
    __device__ static __forceinline__ void a_pass(const Stage& s, uint32_t p, uint32_t j, uint32_t& a0, uint32_t& a1,
                                                  uint32_t& a2, uint32_t& a3) {
        const uint32_t mask = p ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
        a0 = word4(s.q[0], j) & mask;
        a1 = word4(s.q[2], j) & mask;
        a2 = word4(s.q[1], j) & mask;
        a3 = word4(s.q[3], j) & mask;
    }
    __device__ static __forceinline__ void load_ring(Stage& s, const uint8_t* box, const uint8_t*, const uint8_t* rec, uint32_t rec8,
                                                     uint32_t o0, uint32_t o1, uint32_t, uint32_t t) {
        s.q[0] = *reinterpret_cast<const uint4*>(box + o0);
        s.q[1] = *reinterpret_cast<const uint4*>(box + o1);
        s.q[2] = *reinterpret_cast<const uint4*>(box + o0 + 1024u);
        s.q[3] = *reinterpret_cast<const uint4*>(box + o1 + 1024u);
        s.dd[0] = *reinterpret_cast<const uint32_t*>(rec + 4u * t);
        s.dd[1] = *reinterpret_cast<const uint32_t*>(rec + rec8 + 4u * t);
    }
};

struct RQ80 : Q80, Q80Plane {     // boxes: blocks 0..3 | blocks 4..7 of the unit
    using Q80Plane::kDataBytes, Q80Plane::kRecBytes;
    static constexpr uint32_t kPasses = 2, kSub = 4;
    // pass p of lane t feeds block t + 4p: box p holds blocks 4p..4p+3, chunk 2t its block t's first
    // 16 bytes (k-slots 4t..), chunk 2t+1 the second 16 (slots 16+4t..)
    __device__ static __forceinline__ uint32_t blk(uint32_t p, uint32_t t) { return t + 4u * p; }
    __device__ static __forceinline__ void a_pass(const Stage& s, uint32_t p, uint32_t j, uint32_t& a0, uint32_t& a1,
                                                  uint32_t& a2, uint32_t& a3) {
        a0 = word4(s.q[2u * p], j);
        a1 = word4(s.q[4u + 2u * p], j);
        a2 = word4(s.q[2u * p + 1u], j);
        a3 = word4(s.q[5u + 2u * p], j);
    }
    __device__ static __forceinline__ void load_ring(Stage& s, const uint8_t* box, const uint8_t*, const uint8_t* rec, uint32_t rec8,
                                                     uint32_t o0, uint32_t o1, uint32_t, uint32_t t) {
        s.q[0] = *reinterpret_cast<const uint4*>(box + o0);
        s.q[1] = *reinterpret_cast<const uint4*>(box + o1);
        s.q[2] = *reinterpret_cast<const uint4*>(box + kBoxBytes + o0);
        s.q[3] = *reinterpret_cast<const uint4*>(box + kBoxBytes + o1);
        s.q[4] = *reinterpret_cast<const uint4*>(box + o0 + 1024u);
        s.q[5] = *reinterpret_cast<const uint4*>(box + o1 + 1024u);
        s.q[6] = *reinterpret_cast<const uint4*>(box + kBoxBytes + o0 + 1024u);
        s.q[7] = *reinterpret_cast<const uint4*>(box + kBoxBytes + o1 + 1024u);
        const uint8_t* r0 = rec + 2u * t;  // f16 d[t] | d[t + 4] << 16
        s.dd[0] = (uint32_t)*reinterpret_cast<const uint16_t*>(r0) | ((uint32_t)*reinterpret_cast<const uint16_t*>(r0 + 8u) << 16);
        s.dd[1] = (uint32_t)*reinterpret_cast<const uint16_t*>(r0 + rec8) |
                  ((uint32_t)*reinterpret_cast<const uint16_t*>(r0 + rec8 + 8u) << 16);
    }
};

// Q5_K: the Q4_K nibbles and record, and 32 bytes whose bit b is bit 4 of block b's codes.  Lane t's blocks 2t and 2t + 1 take
// two bits of every byte.
struct RQ5K : Q4K, Q5KPlane {
    using Q5KPlane::kDataBytes, Q5KPlane::kRecBytes;
    static constexpr uint32_t kPasses = 2, kSub = 4;
    static constexpr int kHiShift = 0;
    struct Stage : Q4K::Stage {
        uint4 h[4];   // rows g, g + 8: the high-bit bytes, shifted so that block 2t's bit is bit 0
    };
    __device__ static __forceinline__ uint32_t blk(uint32_t p, uint32_t t) { return 2u * t + p; }
    __device__ static __forceinline__ void a_pass(const Stage& s, uint32_t p, uint32_t j, uint32_t& a0, uint32_t& a1,
                                                  uint32_t& a2, uint32_t& a3) {
        auto code = [p](uint32_t w, uint32_t h) {
            return p ? ((w >> 4) & 0x0F0F0F0Fu) | ((h << 3) & 0x10101010u) : (w & 0x0F0F0F0Fu) | ((h << 4) & 0x10101010u);
        };
        a0 = code(word4(s.q[0], j), word4(s.h[0], j));
        a1 = code(word4(s.q[2], j), word4(s.h[2], j));
        a2 = code(word4(s.q[1], j), word4(s.h[1], j));
        a3 = code(word4(s.q[3], j), word4(s.h[3], j));
    }
    __device__ static __forceinline__ void load_ring(Stage& s, const uint8_t* box, const uint8_t* high, const uint8_t* rec, uint32_t rec8,
                                                     uint32_t o0, uint32_t o1, uint32_t g, uint32_t t) {
        RQ4K::load_ring(s, box, nullptr, rec, rec8, o0, o1, g, t);
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            const uint4 v = *reinterpret_cast<const uint4*>(high + (g + (i >> 1) * 8u) * 32u + (i & 1u) * 16u);
            s.h[i] = make_uint4(v.x >> (2u * t), v.y >> (2u * t), v.z >> (2u * t), v.w >> (2u * t));
        }
    }
};

// Q6_K: sixteen blocks of 16 weights, so four passes of two mmas.  Lane t holds, of the 128-weight half t / 2, the blocks at
// elements 16 (t & 1) + 32 p (p = pass): low nibbles of two 16-byte chunks of ql for p = 0, 1, high nibbles for p = 2, 3,
// and bits 2p, 2p + 1 of one chunk of qh.  Codes stay unsigned; the -32 goes through the 16-element sums of the activations.
struct RQ6K : Q6KPlane {
    static constexpr uint32_t kPasses = 4, kSub = 2;
    static constexpr bool kUnsignedA = true;
    static constexpr int kHiShift = 0;
    struct Stage {
        uint4 q[4];      // row g: ql chunks of p = 0, 2 and of p = 1, 3; row g + 8 likewise
        uint4 h[2];      // qh chunk of rows g, g + 8
        uint32_t d[2];   // f16 d of the two rows (low half)
        uint2 sc[2];     // the half's eight int8 scales, for this lane's blocks: bytes 2 p of the eight, shifted by t & 1
    };
    __device__ static __forceinline__ uint32_t blk(uint32_t p, uint32_t t) { return 8u * (t >> 1) + 2u * p + (t & 1u); }
    __device__ static __forceinline__ void a_pass(const Stage& s, uint32_t p, uint32_t j, uint32_t& a0, uint32_t& a1,
                                                  uint32_t& a2, uint32_t& a3) {
        auto code = [p](uint32_t w, uint32_t h) {
            const uint32_t lo = (p >> 1) ? (w >> 4) & 0x0F0F0F0Fu : w & 0x0F0F0F0Fu;
            return lo | ((p == 0u ? h << 4 : p == 1u ? h << 2 : p == 2u ? h : h >> 2) & 0x30303030u);
        };
        const uint32_t c = p & 1u;
        a0 = code(word4(s.q[c], j), word4(s.h[0], j));
        a1 = code(word4(s.q[2u + c], j), word4(s.h[1], j));
        a2 = code(word4(s.q[c], 2u + j), word4(s.h[0], 2u + j));
        a3 = code(word4(s.q[2u + c], 2u + j), word4(s.h[1], 2u + j));
    }
    __device__ static __forceinline__ void load_ring(Stage& s, const uint8_t* box, const uint8_t* high, const uint8_t* rec, uint32_t rec8,
                                                     uint32_t, uint32_t, uint32_t g, uint32_t t) {
        const uint32_t c0 = 4u * (t >> 1) + (t & 1u);
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            s.q[2u * h] = *reinterpret_cast<const uint4*>(box + h * 1024u + swz(g, c0));
            s.q[2u * h + 1u] = *reinterpret_cast<const uint4*>(box + h * 1024u + swz(g, c0 + 2u));
            // 64-byte rows under the 64-byte swizzle: chunk index xor bits 1..2 of the row
            s.h[h] = *reinterpret_cast<const uint4*>(high + (g + h * 8u) * 64u + ((t ^ ((g >> 1) & 3u)) << 4));
            const uint8_t* r = rec + h * rec8;
            s.d[h] = *reinterpret_cast<const uint32_t*>(r);
            const uint32_t w0 = *reinterpret_cast<const uint32_t*>(r + 4u + 8u * (t >> 1)), w1 = *reinterpret_cast<const uint32_t*>(r + 8u + 8u * (t >> 1));
            s.sc[h] = make_uint2(w0 >> (8u * (t & 1u)), w1 >> (8u * (t & 1u)));
        }
    }
    __device__ static __forceinline__ void fold(const Stage& s, const int (&c)[4][4], const float2 (&xm)[4], float& acc_g, float& acc_g8) {
        float v[2] = {0.0f, 0.0f};
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h)
#pragma unroll
            for (uint32_t p = 0; p < 4u; ++p) {
                const uint32_t w = (p >> 1) ? s.sc[h].y : s.sc[h].x;
                const float f = fmaf((float)(c[p][2u * h] * 256 + c[p][2u * h + 1u]), xm[p].x, -32.0f * xm[p].y);
                v[h] = fmaf((float)(int8_t)((w >> (16u * (p & 1u))) & 0xffu), f, v[h]);
            }
        acc_g = fmaf(__half2float(__ushort_as_half((unsigned short)s.d[0])), v[0], acc_g);
        acc_g8 = fmaf(__half2float(__ushort_as_half((unsigned short)s.d[1])), v[1], acc_g8);
    }
};

__device__ __forceinline__ void cp_async8_fill(uint32_t dst, const void* src, bool valid) {     // zeros where not valid
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid ? 8u : 0u) : "memory");
}

// MANY: up to kManyWarps warps in one or more teams, the units of a pair one after the other; else one team of up to kMaxWarps.
// ODD: the last pair of a row is one unit and zeros; 24-byte records of such a row are not a multiple of 16 bytes, and the lanes copy them.
// SPLIT: a cluster of pl.split CTAs shares its tiles and splits the pairs of a row.  (As template arguments: what an instance
// does not need costs it 0.1 to 0.25 of its 3 to 5 us where there are few tiles.)
template <class F, bool MANY, bool ODD, bool SPLIT>
__global__ void __launch_bounds__((MANY ? kManyWarps : kMaxWarps) * 32u, 1)
gemv_ring_kernel(const __grid_constant__ CUtensorMap dmap, const __grid_constant__ CUtensorMap rmap, const __grid_constant__ CUtensorMap hmap,
                 const uint8_t* __restrict__ recs, const float* __restrict__ bias, const float* __restrict__ x, float* __restrict__ y,
                 uint32_t in_dim, uint32_t out_dim, const int8_t* __restrict__ xq, const float* __restrict__ xq_scale, const PeerOut peers,
                 const RingPlan pl, unsigned int* __restrict__ err) {
    using Stage = typename F::Stage;
    constexpr uint32_t kUnitData = F::kDataBoxes * kBoxBytes, kUnitHigh = 16u * F::kHighBytes;   // one unit's boxes
    constexpr uint32_t kRecRow = 2u * F::kRecBytes;                 // a pair's records of one row
    constexpr uint32_t kStageHigh = 2u * kUnitData, kStageData = kStageHigh + 2u * kUnitHigh, kStageRec = 16u * kRecRow;
    constexpr uint32_t kPasses = F::kPasses, kSub = F::kSub;
    constexpr bool RECS_ASYNC = ODD && F::kRecBytes % 16u != 0u;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t k_part = ODD || SPLIT ? pl.k_part : in_dim;
    uint8_t* xs_hi = smem;
    uint8_t* xs_lo = smem + k_part;
    uint8_t* zeros = smem + 2u * (size_t)k_part;
    float2* xmeta = reinterpret_cast<float2*>(smem + pl.off_xmeta);
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t W = pl.W, D = pl.D;
    uint32_t warp = tid >> 5, team = 0u;
    const uint32_t cta_warp = warp, teams = MANY ? pl.teams : 1u;
    if (MANY)
        for (; warp >= W; warp -= W) ++team;
    float* red = reinterpret_cast<float*>(smem + pl.off_red) + team * kRedBufs * (W * 16u);
    float* recv = reinterpret_cast<float*>(smem + pl.off_recv);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + pl.off_bar);  // [warp][kMaxDepth], then per team the fold barriers
    uint64_t* red_full = full + W * teams * kMaxDepth + 2u * team * kRedBufs;
    uint64_t* red_free = red_full + kRedBufs;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(full + W * teams * kMaxDepth + 2u * teams * kRedBufs);

    const uint32_t split = SPLIT ? pl.split : 1u, rank = SPLIT ? blockIdx.x % split : 0u, cl = SPLIT ? blockIdx.x / split : blockIdx.x;
    const uint32_t all_pairs = (ODD ? in_dim + 511u : in_dim) >> 9;
    const uint32_t p_lo = SPLIT ? rank * all_pairs / split : 0u, n_pair = (SPLIT ? (rank + 1u) * all_pairs / split : all_pairs) - p_lo;
    const uint32_t n_tiles = (out_dim + 15u) >> 4, n_cl = SPLIT ? pl.clusters : gridDim.x;
    const uint32_t tile_lo = (uint32_t)((uint64_t)cl * n_tiles / n_cl);
    const uint32_t tile_hi = (uint32_t)((uint64_t)(cl + 1u) * n_tiles / n_cl);
    const uint32_t cta_tiles = tile_hi - tile_lo;
    // the team's tiles team, team + teams, ..., and this warp's pairs of a tile: warp, warp + W, ... below n_pair
    const uint32_t my_tiles = MANY ? (team < cta_tiles ? (cta_tiles - team + teams - 1u) / teams : 0u) : cta_tiles;
    const uint32_t my_pairs = warp < n_pair ? (n_pair - warp + W - 1u) / W : 0u;
    const uint32_t total = my_tiles * my_pairs;

    uint64_t* my_full = full + cta_warp * kMaxDepth;
    uint8_t* my_data = smem + pl.off_data + (size_t)cta_warp * D * kStageData;
    uint8_t* my_rec = smem + pl.off_rec + (size_t)cta_warp * D * kStageRec;
    const size_t rec_pitch = (size_t)(in_dim >> 8) * F::kRecBytes;

    // (tile, pair) number i of this warp -> stage i % D; issue = arm the barrier, then the copies.
    // Called by the whole (converged) warp: one elected lane issues, so addresses and the
    // tensor-map pointers stay in uniform registers.  What lies beyond a row's end is filled with zeros.
    const uint64_t stream_once = tc5::l2_policy_evict_first();   // a plane is read once per launch
    auto issue = [&](uint32_t stage, uint32_t tl, uint32_t pr) {
        uint64_t* bar = my_full + stage;
        const uint32_t gp = p_lo + pr;
        tc5::mbar_arrive_expect_tx_elect(bar, kStageData + (RECS_ASYNC ? 0u : kStageRec));
        const int32_t row = (int32_t)((tile_lo + tl) * 16u);
        uint8_t* st = my_data + stage * kStageData;
#pragma unroll
        for (uint32_t u = 0; u < 2u; ++u) {
#pragma unroll
            for (uint32_t b = 0; b < F::kDataBoxes; ++b)
                tc5::tma_load_2d_hint_elect(st + u * kUnitData + b * kBoxBytes, &dmap, bar, (int32_t)((gp * 2u + u) * F::kDataBytes + b * 128u), row,
                                            stream_once);
            if constexpr (F::kHighBytes != 0u)
                tc5::tma_load_2d_hint_elect(st + kStageHigh + u * kUnitHigh, &hmap, bar, (int32_t)((gp * 2u + u) * F::kDataBytes + 128u), row, stream_once);
        }
        if constexpr (!RECS_ASYNC) {
            tc5::tma_load_2d_hint_elect(my_rec + stage * kStageRec, &rmap, bar, (int32_t)(gp * kRecRow), row, stream_once);
        } else {
            constexpr uint32_t kPieces = kRecRow / 8u;      // of a row
            const uint32_t dst = tc5::smem_u32(my_rec + stage * kStageRec), last = out_dim - 1u;
#pragma unroll
            for (uint32_t i = 0; i < kPieces / 2u; ++i) {
                const uint32_t c = i * 32u + lane, r = c / kPieces, off = gp * kRecRow + (c - r * kPieces) * 8u;
                const bool valid = off < rec_pitch;
                cp_async8_fill(dst + c * 8u, recs + (size_t)min((uint32_t)row + r, last) * rec_pitch + (valid ? off : 0u), valid);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc5::smem_u32(bar)) : "memory");
        }
    };

    // ---- prologue: every warp arms its own barriers and requests its first D stages; only then
    // does the CTA meet (shared barriers of the tile fold) and wait for the previous kernel
    if (lane == 0u) {
        for (uint32_t s = 0; s < D; ++s) tc5::mbar_init(my_full + s, RECS_ASYNC ? 33u : 1u);
        tc5::mbar_fence_init();
    }
    __syncwarp();
    uint32_t i_tl = team, i_pr = warp, issued = 0;  // issue cursor
    auto issue_next = [&]() {
        issue(issued % D, i_tl, i_pr);
        ++issued;
        i_pr += W;
        if (i_pr >= n_pair) { i_pr = warp; i_tl += teams; }
    };
    // the first stage of every warp goes out alone: it is what the first iteration waits for, and
    // it arrives sooner when the chip's first burst is a quarter of the ring
    if (total > 0u) issue_next();
    if (warp == 0u && lane == 0u) {
        for (uint32_t b = 0; b < kRedBufs; ++b) {
            tc5::mbar_init(&red_full[b], W);
            tc5::mbar_init(&red_free[b], 1u);
        }
        if (team == 0u) *abort_flag = 0;
        tc5::mbar_fence_init();
    }
    if (tid < 8u) reinterpret_cast<uint32_t*>(zeros)[tid] = 0u;
    // The CTA meets once, here, where it would wait for the previous kernel anyway: the fold
    // barriers and the zero line are shared, everything after is per warp (invariant plans of one team).
    // A cluster meets too: its CTAs store into one another's shared memory later.
    if constexpr (SPLIT) {
        __syncwarp();
        tc5::cluster_sync();
    } else {
        __syncthreads();
    }
    // Programmatic dependent launch: the next kernel of the stream may start its prologue (its own
    // first requests: weights never depend on this kernel) as soon as this one's CTAs have all started.
    pdk_pdl_launch_dependents();
    pdk_pdl_wait();  // x (and y's previous contents) belong to the previous kernel until here
    uint32_t peer_step = 0u;
    const bool peer_deferred = peers.n != 0u && peers.signal == 2u && blockIdx.x == 0u && tid == 0u;
    if (peer_deferred) peer_step = peer_post_previous(peers);
    const bool invariant = pl.invariant != 0u;
    const uint32_t x0 = p_lo * 64u, x_groups = in_dim >> 3;     // groups of 8 elements before this part, of a row
    // what lies beyond the row's end counts as zero; the load itself is unconditional, so that two of them are in flight at once
    auto load8 = [&](uint32_t grp, float (&v)[8]) { limb_load8(x, xq, xq_scale, ODD ? min(x0 + grp, x_groups - 1u) : x0 + grp, v); };
    auto store8 = [&](float (&v)[8], uint32_t grp) {
        if (ODD && x0 + grp >= x_groups) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        }
        limb_store8<F::kBlock>(v, grp, xs_hi, xs_lo, xmeta);
    };
    if (invariant) {
        // A warp only ever meets its own pair's 512 activations: it builds their limbs itself (the first team for all).  The
        // loads of x go out before the rest of the ring is requested, so they do not queue behind it.
        const uint32_t g0 = warp * 64u + lane;   // groups of 8 elements: this lane's two
        float v0[8], v1[8];
        load8(g0, v0);
        load8(g0 + 32u, v1);
        while (issued < D && issued < total) issue_next();
        if ((!MANY || team == 0u) && (!(MANY || SPLIT) || warp < n_pair)) {      // one team, no split: every warp has its pair
            store8(v0, g0);
            store8(v1, g0 + 32u);
        }
        if (MANY) __syncthreads();
        else __syncwarp();
    } else {
        const uint32_t groups = n_pair * 64u;
        for (uint32_t grp = tid; grp < groups; grp += W * teams * 32u) {
            float v[8];
            load8(grp, v);
            store8(v, grp);
        }
        while (issued < D && issued < total) issue_next();
        __syncthreads();
    }
    const tc5::WaitCtx ctx{abort_flag, err};

    const uint32_t g = lane >> 2, t = lane & 3u;
    // B operand of this lane: columns 2b, 2b + 1 are the high and low limb of local block b, so
    // lane (g, t) feeds limb g & 1 of block blk(p, t) when g >> 1 == t, and zeros otherwise.
    const bool role = (g >> 1) == t;
    const uint8_t* my_limb = (g & 1u) ? xs_lo : xs_hi;
    // Where a thread has registers for it, both units of a pair side by side (independent accumulator chains), and
    // with an invariant pair B stays in registers; else one unit after the other.
    constexpr uint32_t kSide = MANY ? 1u : 2u;
    uint32_t vb[kSide][kPasses][2u * kSub];  // [unit][pass]: words 0.. -> b0 of mma j, words kSub.. -> b1
    float2 xm[kSide][kPasses];               // {step, sum} of the blocks this lane folds
    auto load_b = [&](uint32_t first) {
#pragma unroll
        for (uint32_t i = 0; i < kSide; ++i) {
            const uint32_t u = first + i;
#pragma unroll
            for (uint32_t p = 0; p < kPasses; ++p) {
                const uint8_t* src = role ? my_limb + u * 256u + F::blk(p, t) * F::kBlock : zeros;
#pragma unroll
                for (uint32_t c = 0; c < kSub / 2u; ++c) {
                    const uint4 a = *reinterpret_cast<const uint4*>(src + 16u * c);
                    vb[i][p][4u * c] = a.x; vb[i][p][4u * c + 1u] = a.y; vb[i][p][4u * c + 2u] = a.z; vb[i][p][4u * c + 3u] = a.w;
                }
                xm[i][p] = xmeta[u * (256u / F::kBlock) + F::blk(p, t)];
            }
        }
    };
    if (!MANY && invariant && warp < n_pair) load_b(2u * warp);

    // per-lane offsets inside a stage
    const uint32_t o0 = swz(g, 2u * t), o1 = swz(g, 2u * t + 1u);
    const uint32_t rec_g = g * kRecRow, rec8 = 8u * kRecRow;

    // ---- tile fold.  Per tile each warp of the team leaves 16 partial row sums in buffer tl % kRedBufs (tl counts the team's
    // tiles) and arrives on the buffer's barrier (fire and forget).  The tile belongs to the team's warp tl % W, which
    // looks at the barrier once per later iteration and, when all W warps have arrived, adds the
    // partials in warp order, stores y and hands the buffer back; it blocks only before taking on
    // another tile, before it would wait for that very buffer, and at the end.  A buffer is written again (tile tl + kRedBufs)
    // only after its fold.  With K split, the sum goes to the CTA of the cluster that adds up the row.
    constexpr uint32_t kNone = 0xffffffffu;
    uint32_t pend = kNone;  // the team's tile this warp still has to fold
    bool alive = true;
    const uint32_t rows = cta_tiles * 16u, rpo = SPLIT ? (rows + split - 1u) / split : 0u;   // rows per owner
    auto put = [&](uint32_t row, float v) {
        if (bias) v += bias[row];
        if (peers.n == 0u) {
            y[row] = v;
            return;
        }
#pragma unroll
        for (uint32_t p = 0; p < 8u; ++p)  // constant indices: the pointers stay in the parameter bank
            if (p < peers.n) peers.ptr[p][peers.row0 + row] = v;
    };
    auto fold_tile = [&](uint32_t tl_f) {
        const uint32_t rbf = tl_f % kRedBufs;
        const float* rbuf = red + (size_t)rbf * (W * 16u);
        const uint32_t r = (team + tl_f * teams) * 16u + lane, row = tile_lo * 16u + r;
        float v = 0.0f;
        if (lane < 16u)
            for (uint32_t w = 0; w < W; ++w) v += rbuf[w * 16u + lane];
        __syncwarp();
        if (lane == 0u) tc5::mbar_arrive(&red_free[rbf]);
        if constexpr (SPLIT) {
            if (lane < 16u) {
                const uint32_t owner = r / rpo;
                tc5::st_cluster(tc5::cluster_addr(tc5::smem_u32(recv), owner) + (rank * rpo + r - owner * rpo) * 4u, v);
            }
            return;
        }
        if (lane < 16u && row < out_dim) put(row, v);
    };
    auto poll_fold = [&](bool block) {
        if (pend == kNone || !alive) return;
        const uint32_t rbf = pend % kRedBufs, ph = (pend / kRedBufs) & 1u;
        bool done;
        if (block) {
            alive = __all_sync(0xffffffffu, tc5::mbar_wait(&red_full[rbf], ph, ctx, kErrRingFold, rbf));
            done = alive;
        } else {
            done = __all_sync(0xffffffffu, tc5::mbar_try_wait(&red_full[rbf], ph));
        }
        if (done) {
            fold_tile(pend);
            pend = kNone;
        }
    };

    uint32_t stage = 0, phase = 0;       // consume cursor
    uint32_t rb = 0, rb_phase = 0, owner = 0;
    for (uint32_t tl = 0; tl < my_tiles; ++tl) {
        float acc_g = 0.0f, acc_g8 = 0.0f;
        for (uint32_t pr = warp; pr < n_pair; pr += W) {
            if (alive) alive = __all_sync(0xffffffffu, tc5::mbar_wait(my_full + stage, phase, ctx, kErrRingFull, stage));
            if (alive) {
                const uint8_t* sd = my_data + stage * kStageData;
                const uint8_t* sr = my_rec + stage * kStageRec + rec_g;
                // [unit][pass], {hi, lo} of row g, {hi, lo} of row g + 8
#pragma unroll
                for (uint32_t i0 = 0; i0 < 2u; i0 += kSide) {
                    Stage st[kSide];
#pragma unroll
                    for (uint32_t i = 0; i < kSide; ++i)
                        F::load_ring(st[i], sd + (i0 + i) * kUnitData, sd + kStageHigh + (i0 + i) * kUnitHigh, sr + (i0 + i) * F::kRecBytes, rec8, o0,
                                     o1, g, t);
                    if (MANY || !invariant) load_b(2u * pr + i0);
                    int c[kSide][kPasses][4] = {};
#pragma unroll
                    for (uint32_t j = 0; j < kSub; ++j) {
#pragma unroll
                        for (uint32_t i = 0; i < kSide; ++i) {
#pragma unroll
                            for (uint32_t p = 0; p < kPasses; ++p) {
                                uint32_t a0, a1, a2, a3;
                                F::a_pass(st[i], p, j, a0, a1, a2, a3);
                                if constexpr (F::kUnsignedA) mma_u8s8_nv(c[i][p], a0, a1, a2, a3, vb[i][p][j], vb[i][p][kSub + j]);
                                else mma_s8_nv(c[i][p], a0, a1, a2, a3, vb[i][p][j], vb[i][p][kSub + j]);
                            }
                        }
                    }
#pragma unroll
                    for (uint32_t i = 0; i < kSide; ++i) {
                        const float2 (&m)[kPasses] = xm[i];
                        if constexpr (kPasses == 4u) {
                            F::fold(st[i], c[i], m, acc_g, acc_g8);
                        } else {
                            float f[4];
                            f[0] = (float)(c[i][0][0] * 256 + c[i][0][1]) * m[0].x;
                            f[1] = (float)((c[i][1][0] * 256 + c[i][1][1]) >> F::kHiShift) * m[1].x;
                            f[2] = (float)(c[i][0][2] * 256 + c[i][0][3]) * m[0].x;
                            f[3] = (float)((c[i][1][2] * 256 + c[i][1][3]) >> F::kHiShift) * m[1].x;
                            F::fold(st[i], f, m[0].y, m[1].y, acc_g, acc_g8);
                        }
                    }
                }
                // Every register the stage's loads filled has been consumed by now, so those loads
                // are complete: the stage can take its next copy.
                __syncwarp();
                if (issued < total) issue_next();
            }
            if (++stage == D) { stage = 0; phase ^= 1u; }
        }
        float a = acc_g, b = acc_g8;
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        b += __shfl_xor_sync(0xffffffffu, b, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        b += __shfl_xor_sync(0xffffffffu, b, 2);
        float* rbuf = red + (size_t)rb * (W * 16u);
        if (alive && tl >= kRedBufs) {
            if (pend + kRedBufs == tl) poll_fold(true);   // the buffer waits for this warp's own fold
            if (alive)
                alive = __all_sync(0xffffffffu, tc5::mbar_wait(&red_free[rb], rb_phase ^ 1u, ctx, kErrRingFree, rb));
        }
        if (alive) {
            if (t == 0u) {
                rbuf[warp * 16u + g] = a;
                rbuf[warp * 16u + g + 8u] = b;
            }
            __syncwarp();
            if (lane == 0u) tc5::mbar_arrive(&red_full[rb]);  // release: the partials above are visible to the folding warp
        }
        if (owner == warp) {
            poll_fold(true);   // the previous tile of this warp, if it is still waiting (W tiles ago)
            pend = tl;
        }
        poll_fold(false);
        if (++owner == W) owner = 0;
        if (++rb == kRedBufs) { rb = 0; rb_phase ^= 1u; }
    }
    poll_fold(true);
    if constexpr (SPLIT) {
        __syncwarp();
        tc5::cluster_sync();     // every CTA's sums are here
        const uint32_t at = rank * rpo, row0 = tile_lo * 16u + at;
        const uint32_t mine = min(min(rpo, rows - min(rows, at)), out_dim - min(out_dim, row0));
        auto sum = [&](uint32_t r) {
            float v = 0.0f;
            for (uint32_t s = 0; s < split; ++s) v += recv[s * rpo + r];
            return v;
        };
        // with the peers' store in the one loop, calls without peers took 0.04 to 0.1 us longer (Q6_K 12032 x 832 5.46 -> 5.54)
        if (peers.n == 0u) {
            for (uint32_t r = tid; r < mine; r += W * teams * 32u) y[row0 + r] = bias ? sum(r) + bias[row0 + r] : sum(r);
        } else {
            for (uint32_t r = tid; r < mine; r += W * teams * 32u) put(row0 + r, sum(r));
        }
    }
    if (peers.n != 0u && peers.signal == 1u) {   // uniform over the grid
        __syncthreads();
        if (tid == 0u) peer_signal(peers, err);
    }
    if (peer_deferred) peer_check_previous(peers, peer_step, err);
    if (!alive) {
        // a wait ran out somewhere in the CTA: the copies this warp still has in flight must land
        // before its shared memory can go to another CTA.  At most D are outstanding, one per stage.
        const unsigned long long t0 = tc5::globaltimer_ns();
        for (uint32_t s = 0; s < D && s < issued; ++s) {
            // the last copy into stage s is number n = the largest n < issued with n % D == s
            const uint32_t n = issued - 1u - ((issued - 1u - s) % D);
            while (!tc5::mbar_try_wait(my_full + s, (n / D) & 1u)) {
                if (tc5::globaltimer_ns() - t0 > tc5::kWaitBudgetNs) {
                    if (lane == 0u) tc5::report(err, kErrRingDrain, s);
                    break;
                }
            }
        }
    }
}

// PDK_GEMV_REGS=1 sends every call to the register-staged kernel (A/B switch, read once).
bool force_regs() {
    static const bool v = [] {
        const char* e = getenv("PDK_GEMV_REGS");
        return e && e[0] == '1';
    }();
    return v;
}

// Tensor maps of the planes a thread used last (weights stay where they are, so a decode loop
// encodes each plane's maps once): [rows][row bytes] uint8, data boxes 128 x 16 swizzled, record
// boxes of a unit pair's records x 16 dense.
struct MapEntry {
    const void *data, *recs;
    uint32_t in_dim, out_dim, format;     // format: data bytes and record bytes of a unit
    CUtensorMap dmap, hmap, rmap;
};
// whether a row's records can be described by a tensor map
template <class F>
bool recs_by_tma(uint32_t in_dim) { return ((in_dim >> 8) * F::kRecBytes) % 16u == 0u; }

template <class F>
int plane_maps(const void* data, const void* recs, uint32_t in_dim, uint32_t out_dim, const MapEntry** out) {
    constexpr int kEntries = 16;
    constexpr uint32_t kFormat = F::kDataBytes << 8 | F::kRecBytes;
    thread_local MapEntry cache[kEntries];
    thread_local int next = 0, used = 0;
    for (int i = 0; i < used; ++i) {
        const MapEntry& e = cache[i];
        if (e.data == data && e.recs == recs && e.in_dim == in_dim && e.out_dim == out_dim && e.format == kFormat) {
            *out = &e;
            return 0;
        }
    }
    MapEntry& e = cache[next];
    const uint32_t n_unit = in_dim >> 8;
    const uint64_t pitch = (uint64_t)n_unit * F::kDataBytes;
    int rc = pdk_make_tmap_2d(&e.dmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1u, data, pitch, out_dim, pitch, 128u, 16u);
    e.hmap = e.rmap = e.dmap;
    if (rc == 0 && F::kHighBytes == 32u) rc = pdk_make_tmap_2d_dense(&e.hmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1u, data, pitch, out_dim, pitch, 32u, 16u);
    if (rc == 0 && F::kHighBytes == 64u) rc = pdk_make_tmap_2d_sw64(&e.hmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1u, data, pitch, out_dim, pitch, 64u, 16u);
    if (rc == 0 && recs_by_tma<F>(in_dim))
        rc = pdk_make_tmap_2d_dense(&e.rmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1u, recs, (uint64_t)n_unit * F::kRecBytes,
                                    out_dim, (uint64_t)n_unit * F::kRecBytes, 2u * F::kRecBytes, 16u);
    if (rc != 0) {
        e.data = nullptr;
        return rc;
    }
    e.data = data; e.recs = recs; e.in_dim = in_dim; e.out_dim = out_dim; e.format = kFormat;
    *out = &e;
    next = (next + 1) % kEntries;
    if (used < kEntries) ++used;
    return 0;
}

template <class F, bool MANY, bool ODD, bool SPLIT>
int launch_plan(const MapEntry& m, const void* recs, const float* bias, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                cudaStream_t st, const int8_t* xq, const float* xq_scale, const PeerOut& po, const RingPlan& pl) {
    auto kern = gemv_ring_kernel<F, MANY, ODD, SPLIT>;
    static bool attr_set[64] = {false};  // per device, per instance
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    unsigned int* err = pdk_error_word();
    if (err == nullptr) return (int)cudaErrorUnknown;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.split * pl.clusters);
    cfg.blockDim = dim3(pl.W * pl.teams * 32u);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdk_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = pl.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kern, m.dmap, m.rmap, m.hmap, (const uint8_t*)recs, bias, x, y, in_dim, out_dim, xq, xq_scale, po, pl, err);
    return e == cudaSuccess ? pdk_launch_status() : (int)e;
}

// The plan of a shape on the current device: 0, a cudaError_t, or -1 where there is none or the register-staged kernel is faster.
template <class F>
int shape_plan(uint32_t in_dim, uint32_t out_dim, const RingPlan** plan) {
    if (in_dim <= 1024u || (in_dim & 255u) != 0u || out_dim > 0x40000000u) return -1;
    // clusters of s CTAs that are resident at once: one CTA per SM, whatever the instance
    static PdkClusterCaps table;
    const uint32_t* cap = nullptr;
    if (int rc = pdk_cluster_caps(table, (const void*)gemv_ring_kernel<F, false, false, true>, kMaxWarps * 32u, kSmemMax, &cap)) return rc;
    // the plans of the shapes a thread met last
    struct Known { const uint32_t* cap; uint32_t in_dim, out_dim, ok; RingPlan plan; };
    constexpr uint32_t kKnown = 32;
    thread_local Known known[kKnown] = {};
    Known& k = known[(in_dim / 256u * 7u + out_dim / 8u) % kKnown];
    if (k.cap != cap || k.in_dim != in_dim || k.out_dim != out_dim) {
        k = Known{cap, in_dim, out_dim, 0u, RingPlan{}};
        k.ok = make_plan<F>(in_dim, out_dim, cap, k.plan) ? 1u : 0u;
    }
    *plan = &k.plan;
    return k.ok != 0u ? 0 : -1;
}

// -1: outside the plan (rows of up to four units: Q6_K 1024 x 618 2.2 us on registers, 2.5 here; planes that do not start on
// 16 bytes, activations too long), or the register-staged kernel is faster.
template <class F>
int launch_ring(const void* data, const void* recs, const float* bias, const float* x, float* y, uint32_t in_dim,
                uint32_t out_dim, cudaStream_t st, const int8_t* xq = nullptr, const float* xq_scale = nullptr,
                const PeerOut* peers = nullptr) {
    if (force_regs()) return -1;
    const bool tma = recs_by_tma<F>(in_dim);
    if (!pdk_aligned(recs, tma ? 16 : 8)) return -1;
    const RingPlan* plan = nullptr;
    if (int rc = shape_plan<F>(in_dim, out_dim, &plan)) return rc;
    const RingPlan& pl = *plan;
    const MapEntry* maps = nullptr;
    if (plane_maps<F>(data, recs, in_dim, out_dim, &maps) != 0) return -1;
    PeerOut po{};
    if (peers) po = *peers;
#define PDK_RING(M, O, S) return launch_plan<F, M, O, S>(*maps, recs, bias, x, y, in_dim, out_dim, st, xq, xq_scale, po, pl)
    const bool odd = (in_dim & 511u) != 0u;
    if constexpr (F::kMany) {
        if (pl.teams > 1u || pl.W > kMaxWarps) {
            if (pl.split > 1u) { if (odd) PDK_RING(true, true, true); else PDK_RING(true, false, true); }
            if (odd) PDK_RING(true, true, false); else PDK_RING(true, false, false);
        }
    }
    if (pl.split > 1u) { if (odd) PDK_RING(false, true, true); else PDK_RING(false, false, true); }
    if (odd) PDK_RING(false, true, false);
    PDK_RING(false, false, false);
#undef PDK_RING
}


// ---------------------------------------------------------------------------
// Q8_0 with 2..8 tokens on the same ring: the tokens are the mma's eight columns.
//
// Plans with one unit pair per warp only (W == K / 512, K = 2048, 2560 .. 5632): warp w meets the same
// 512 activations of every token in every tile, so its B operand - two int8 limbs of the 15-bit
// block floating point, per (token, 32-block) power-of-two steps - is built once from x and stays
// in 64 registers.  Per 32-weight block: one ldmatrix.x4 takes the 16 rows x 32 int8 out of the
// swizzled box (conflict free: the eight rows of a matrix sit in eight different bank groups),
// one mma per limb gives the integer tile [16 rows][8 tokens], and lane (g, t) folds its four
// entries with d[row][block] * step[token][block] in f32.  Weights leave HBM once for all tokens.
// ---------------------------------------------------------------------------
constexpr uint32_t kBatchRedBufs = 4;

struct BatchPlan {
    uint32_t W, D;
    uint32_t off_steps, off_red, off_bar, off_rec, off_data, smem_bytes;
};

enum : unsigned int { kErrBatchFull = 0x18, kErrBatchFold = 0x19, kErrBatchFree = 0x1a, kErrBatchDrain = 0x1b };

__device__ __forceinline__ void ldmatrix_x4(uint32_t saddr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(saddr));
}

__global__ void __launch_bounds__(kMaxWarps * 32u, 1)
gemm_ring_q8_kernel(const __grid_constant__ CUtensorMap dmap, const __grid_constant__ CUtensorMap rmap,
                    const float* __restrict__ bias, const float* __restrict__ x, float* __restrict__ y, uint32_t in_dim,
                    uint32_t out_dim, uint32_t batch, const BatchPlan pl, unsigned int* __restrict__ err,
                    const uint32_t last_pass) {
    constexpr uint32_t kUnitData = 2u * kBoxBytes;             // a unit's two boxes (blocks 0..3 | 4..7)
    constexpr uint32_t kRecRow = 2u * Q80::kRecBytes;          // a pair's records of one row
    constexpr uint32_t kStageData = 2u * kUnitData, kStageRec = 16u * kRecRow;
    extern __shared__ __align__(1024) uint8_t smem[];
    float* steps = reinterpret_cast<float*>(smem + pl.off_steps);   // [W][16 blocks][8 tokens]
    float* red = reinterpret_cast<float*>(smem + pl.off_red);       // [kBatchRedBufs][W][16 rows][8 tokens]
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + pl.off_bar);
    uint64_t* red_full = full + kMaxWarps * kMaxDepth;
    uint64_t* red_free = red_full + kBatchRedBufs;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(red_free + kBatchRedBufs);

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t W = pl.W, D = pl.D;
    const uint32_t n_tiles = (out_dim + 15u) >> 4;
    const uint32_t tile_lo = (uint32_t)((uint64_t)blockIdx.x * n_tiles / gridDim.x);
    const uint32_t tile_hi = (uint32_t)((uint64_t)(blockIdx.x + 1u) * n_tiles / gridDim.x);
    const uint32_t my_tiles = tile_hi - tile_lo;

    uint64_t* my_full = full + warp * kMaxDepth;
    uint8_t* my_data = smem + pl.off_data + (size_t)warp * D * kStageData;
    uint8_t* my_rec = smem + pl.off_rec + (size_t)warp * D * kStageRec;

    // The call's last pass over the plane loads it evict-first (nothing reads it again); an earlier pass
    // of a call with more than eight tokens leaves what fits in L2 to the pass that follows.
    const uint64_t stream_once = tc5::l2_policy_evict_first();
    auto issue = [&](uint32_t stage, uint32_t tl) {
        uint64_t* bar = my_full + stage;
        tc5::mbar_arrive_expect_tx_elect(bar, kStageData + kStageRec);
        const int32_t row = (int32_t)((tile_lo + tl) * 16u);
        if (last_pass) {
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b)
                tc5::tma_load_2d_hint_elect(my_data + stage * kStageData + b * kBoxBytes, &dmap, bar,
                                            (int32_t)(warp * 2u * Q80::kDataBytes + b * 128u), row, stream_once);
            tc5::tma_load_2d_hint_elect(my_rec + stage * kStageRec, &rmap, bar, (int32_t)(warp * kRecRow), row, stream_once);
        } else {
#pragma unroll
            for (uint32_t b = 0; b < 4u; ++b)
                tc5::tma_load_2d_elect(my_data + stage * kStageData + b * kBoxBytes, &dmap, bar,
                                       (int32_t)(warp * 2u * Q80::kDataBytes + b * 128u), row);
            tc5::tma_load_2d_elect(my_rec + stage * kStageRec, &rmap, bar, (int32_t)(warp * kRecRow), row);
        }
    };

    if (lane == 0u) {
        for (uint32_t s = 0; s < D; ++s) tc5::mbar_init(my_full + s, 1u);
        tc5::mbar_fence_init();
    }
    __syncwarp();
    uint32_t issued = 0;
    if (my_tiles > 0u) { issue(0u, 0u); issued = 1u; }
    if (tid == 0u) {
        for (uint32_t b = 0; b < kBatchRedBufs; ++b) {
            tc5::mbar_init(&red_full[b], W);
            tc5::mbar_init(&red_free[b], 1u);
        }
        *abort_flag = 0;
        tc5::mbar_fence_init();
    }
    __syncthreads();
    pdk_pdl_launch_dependents();
    pdk_pdl_wait();   // x and y belong to the previous kernel until here

    // ---- B operand: token g, this warp's 16 blocks.  Lane (g, t) holds elements 4t..4t+3 and
    // 16+4t..16+4t+3 of each block, which is exactly its share of the mma's B fragment.
    const uint32_t g = lane >> 2, t = lane & 3u;
    uint32_t bh[16][2], bl[16][2];
    {
        const float* xt = x + (size_t)(g < batch ? g : 0u) * in_dim + warp * 512u + 4u * t;
        float* my_steps = steps + warp * 128u;
#pragma unroll
        for (uint32_t b = 0; b < 16u; ++b) {
            float4 v0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v1 = v0;
            if (g < batch) {
                v0 = *reinterpret_cast<const float4*>(xt + b * 32u);
                v1 = *reinterpret_cast<const float4*>(xt + b * 32u + 16u);
            }
            float amax = fmaxf(fmaxf(fmaxf(fabsf(v0.x), fabsf(v0.y)), fmaxf(fabsf(v0.z), fabsf(v0.w))),
                               fmaxf(fmaxf(fabsf(v1.x), fabsf(v1.y)), fmaxf(fabsf(v1.z), fabsf(v1.w))));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            // amax < 2^ex -> step 2^(ex-14): |q| <= 2^14, q = 256 * hi + lo with lo in [-128, 127]
            float step = 1.0f, inv = 0.0f;
            if (amax > 0.0f && amax < 3.0e38f) {
                const int ex = max((int)(__float_as_uint(amax) >> 23) - 126, -110);
                step = __uint_as_float((uint32_t)(ex + 113) << 23);
                inv = __uint_as_float((uint32_t)(141 - ex) << 23);
            }
            const int q0 = __float2int_rn(v0.x * inv), q1 = __float2int_rn(v0.y * inv), q2 = __float2int_rn(v0.z * inv),
                      q3 = __float2int_rn(v0.w * inv), q4 = __float2int_rn(v1.x * inv), q5 = __float2int_rn(v1.y * inv),
                      q6 = __float2int_rn(v1.z * inv), q7 = __float2int_rn(v1.w * inv);
            bl[b][0] = __byte_perm(__byte_perm(q0, q1, 0x0040), __byte_perm(q2, q3, 0x0040), 0x5410);
            bl[b][1] = __byte_perm(__byte_perm(q4, q5, 0x0040), __byte_perm(q6, q7, 0x0040), 0x5410);
            bh[b][0] = __byte_perm(__byte_perm(q0 + 128, q1 + 128, 0x0051), __byte_perm(q2 + 128, q3 + 128, 0x0051), 0x5410);
            bh[b][1] = __byte_perm(__byte_perm(q4 + 128, q5 + 128, 0x0051), __byte_perm(q6 + 128, q7 + 128, 0x0051), 0x5410);
            if (t == 0u) my_steps[b * 8u + g] = step;
        }
        __syncwarp();
    }
    while (issued < D && issued < my_tiles) { issue(issued % D, issued); ++issued; }
    const tc5::WaitCtx ctx{abort_flag, err};

    // ldmatrix row addresses: lane l supplies row (l & 7) + 8 * ((l >> 3) & 1) of k-half (l >> 4);
    // block bb of a unit = chunks 2 * (bb & 3) + k-half of box bb >> 2
    const uint32_t m_row = (lane & 7u) + ((lane >> 3) & 1u) * 8u, m_half = lane >> 4;
    uint32_t a_off[4];
#pragma unroll
    for (uint32_t c = 0; c < 4u; ++c) a_off[c] = swz(m_row, 2u * c + m_half);
    const float* my_steps = steps + warp * 128u + 2u * t;
    const uint32_t rec_g = g * kRecRow, rec8 = 8u * kRecRow;

    constexpr uint32_t kNone = 0xffffffffu;
    uint32_t pend = kNone;
    bool alive = true;
    auto fold_tile = [&](uint32_t tl_f) {
        const uint32_t rbf = tl_f % kBatchRedBufs;
        const float* rbuf = red + (size_t)rbf * (W * 128u);
        // lane -> row lane & 15, tokens 4 * (lane >> 4) .. + 3
        const uint32_t r = lane & 15u, c0 = (lane >> 4) * 4u;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t w = 0; w < W; ++w) {
            const float4 p = *reinterpret_cast<const float4*>(rbuf + w * 128u + r * 8u + c0);
            v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
        }
        __syncwarp();
        if (lane == 0u) tc5::mbar_arrive(&red_free[rbf]);
        const uint32_t row = (tile_lo + tl_f) * 16u + r;
        if (row < out_dim) {
            const float bv = bias ? bias[row] : 0.0f;
#pragma unroll
            for (uint32_t c = 0; c < 4u; ++c)
                if (c0 + c < batch) y[(size_t)(c0 + c) * out_dim + row] = v[c] + bv;
        }
    };
    auto poll_fold = [&](bool block) {
        if (pend == kNone || !alive) return;
        const uint32_t rbf = pend % kBatchRedBufs, ph = (pend / kBatchRedBufs) & 1u;
        bool done;
        if (block) {
            alive = __all_sync(0xffffffffu, tc5::mbar_wait(&red_full[rbf], ph, ctx, kErrBatchFold, rbf));
            done = alive;
        } else {
            done = __all_sync(0xffffffffu, tc5::mbar_try_wait(&red_full[rbf], ph));
        }
        if (done) {
            fold_tile(pend);
            pend = kNone;
        }
    };

    uint32_t stage = 0, phase = 0, rb = 0, rb_phase = 0, owner = 0;
    for (uint32_t tl = 0; tl < my_tiles; ++tl) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // (g, 2t) (g, 2t+1) (g+8, 2t) (g+8, 2t+1)
        if (alive) alive = __all_sync(0xffffffffu, tc5::mbar_wait(my_full + stage, phase, ctx, kErrBatchFull, stage));
        if (alive) {
            const uint32_t sd = tc5::smem_u32(my_data + stage * kStageData);
            const uint8_t* sr = my_rec + stage * kStageRec + rec_g;
#pragma unroll
            for (uint32_t i = 0; i < 2u; ++i) {
                const uint4 dg = *reinterpret_cast<const uint4*>(sr + i * Q80::kRecBytes);
                const uint4 dg8 = *reinterpret_cast<const uint4*>(sr + rec8 + i * Q80::kRecBytes);
#pragma unroll
                for (uint32_t bb = 0; bb < 8u; ++bb) {
                    const uint32_t b = i * 8u + bb;
                    uint32_t a0, a1, a2, a3;
                    ldmatrix_x4(sd + i * kUnitData + (bb >> 2) * kBoxBytes + a_off[bb & 3u], a0, a1, a2, a3);
                    int ch[4] = {0, 0, 0, 0}, cl[4] = {0, 0, 0, 0};
                    mma_s8_nv(ch, a0, a1, a2, a3, bh[b][0], bh[b][1]);
                    mma_s8_nv(cl, a0, a1, a2, a3, bl[b][0], bl[b][1]);
                    const float2 s = *reinterpret_cast<const float2*>(my_steps + b * 8u);
                    const uint32_t wg = word4(dg, bb >> 1), wg8 = word4(dg8, bb >> 1);
                    const __half2 hg = *reinterpret_cast<const __half2*>(&wg), hg8 = *reinterpret_cast<const __half2*>(&wg8);
                    const float d0 = (bb & 1u) ? __high2float(hg) : __low2float(hg);
                    const float d8 = (bb & 1u) ? __high2float(hg8) : __low2float(hg8);
                    acc[0] += (float)(ch[0] * 256 + cl[0]) * (d0 * s.x);
                    acc[1] += (float)(ch[1] * 256 + cl[1]) * (d0 * s.y);
                    acc[2] += (float)(ch[2] * 256 + cl[2]) * (d8 * s.x);
                    acc[3] += (float)(ch[3] * 256 + cl[3]) * (d8 * s.y);
                }
            }
            __syncwarp();
            if (issued < my_tiles) { issue(issued % D, issued); ++issued; }
        }
        if (++stage == D) { stage = 0; phase ^= 1u; }

        float* rbuf = red + (size_t)rb * (W * 128u);
        if (alive && tl >= kBatchRedBufs)
            alive = __all_sync(0xffffffffu, tc5::mbar_wait(&red_free[rb], rb_phase ^ 1u, ctx, kErrBatchFree, rb));
        if (alive) {
            *reinterpret_cast<float2*>(rbuf + warp * 128u + g * 8u + 2u * t) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(rbuf + warp * 128u + (g + 8u) * 8u + 2u * t) = make_float2(acc[2], acc[3]);
            __syncwarp();
            if (lane == 0u) tc5::mbar_arrive(&red_full[rb]);
        }
        if (owner == warp) {
            poll_fold(true);
            pend = tl;
        }
        poll_fold(false);
        if (++owner == W) owner = 0;
        if (++rb == kBatchRedBufs) { rb = 0; rb_phase ^= 1u; }
    }
    poll_fold(true);
    if (!alive) {
        const unsigned long long t0 = tc5::globaltimer_ns();
        for (uint32_t s = 0; s < D && s < issued; ++s) {
            const uint32_t n = issued - 1u - ((issued - 1u - s) % D);
            while (!tc5::mbar_try_wait(my_full + s, (n / D) & 1u)) {
                if (tc5::globaltimer_ns() - t0 > tc5::kWaitBudgetNs) {
                    if (lane == 0u) tc5::report(err, kErrBatchDrain, s);
                    break;
                }
            }
        }
    }
}

bool make_batch_plan(uint32_t in_dim, BatchPlan& p) {
    if (in_dim == 0u || (in_dim & 511u) != 0u) return false;
    const uint32_t W = in_dim >> 9;
    if (W < 4u || W > kMaxWarps) return false;
    constexpr uint32_t kStage = 4u * kBoxBytes + 32u * Q80::kRecBytes;
    p.W = W;
    p.off_steps = 0u;
    p.off_red = W * 512u;
    p.off_bar = p.off_red + kBatchRedBufs * W * 512u;
    p.off_rec = (p.off_bar + (kMaxWarps * kMaxDepth + 2u * kBatchRedBufs) * 8u + 16u + 127u) & ~127u;
    if (p.off_rec + 1024u + 2u * W * kStage > kSmemMax) return false;
    p.D = (kSmemMax - p.off_rec - 1024u) / (W * kStage);
    if (p.D > kMaxDepth) p.D = kMaxDepth;
    p.off_data = (p.off_rec + W * p.D * 32u * Q80::kRecBytes + 1023u) & ~1023u;
    p.smem_bytes = p.off_data + W * p.D * 4u * kBoxBytes;
    return p.smem_bytes <= kSmemMax && p.D >= 2u;
}


}  // namespace

// gemv_i8.cu: the register-staged kernel
int pdk_q4k_gemv_i8_regs(const void*, const void*, const float*, float*, uint32_t, uint32_t, cudaStream_t);
int pdk_q4_0_gemv_i8_regs(const void*, const void*, const float*, float*, uint32_t, uint32_t, cudaStream_t);
int pdk_q5k_gemv_i8_regs(const void*, const void*, const float*, float*, uint32_t, uint32_t, cudaStream_t);
int pdk_q6k_gemv_i8_regs(const void*, const void*, const float*, float*, uint32_t, uint32_t, cudaStream_t);
int pdk_q8_0_gemv_i8_regs(const void*, const void*, const float*, const float*, float*, uint32_t, uint32_t, cudaStream_t);
int pdk_q4k_gemv_i8_q8act_regs(const void*, const void*, const int8_t*, const float*, float*, uint32_t, uint32_t,
                               cudaStream_t);
int pdk_q4k_gemv_peers_regs(const void*, const void*, const float*, const gemv_i8::PeerOut*, uint32_t, uint32_t,
                            cudaStream_t);

// Decode GEMV entry points of the int8 tensor path.  Each returns 0 / a cudaError_t, or -1 when the
// shape is outside both kernels' plans (K not a multiple of 256, fewer than four units per row, or
// activations too long for shared memory) and the caller should take another route.  The ring
// kernel takes rows of five units and more where its plan's price is the lower one (ring_plan.cuh);
// the register-staged kernels take the rest.
int pdk_q4k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                    uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ4K>(data, scales, nullptr, x, y, in_dim, out_dim, st);
    return rc != -1 ? rc : pdk_q4k_gemv_i8_regs(data, scales, x, y, in_dim, out_dim, st);
}

int pdk_q4_0_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                     uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ40>(data, scales, nullptr, x, y, in_dim, out_dim, st);
    return rc != -1 ? rc : pdk_q4_0_gemv_i8_regs(data, scales, x, y, in_dim, out_dim, st);
}

int pdk_q5k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                    uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ5K>(data, scales, nullptr, x, y, in_dim, out_dim, st);
    return rc != -1 ? rc : pdk_q5k_gemv_i8_regs(data, scales, x, y, in_dim, out_dim, st);
}

int pdk_q6k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ6K>(data, scales, nullptr, x, y, in_dim, out_dim, st);
    return rc != -1 ? rc : pdk_q6k_gemv_i8_regs(data, scales, x, y, in_dim, out_dim, st);
}

int pdk_q8_0_gemv_i8(const void* data, const void* scale, const float* bias, const float* x, float* y,
                     uint32_t in_dim, uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ80>(data, scale, bias, x, y, in_dim, out_dim, st);
    return rc != -1 ? rc : pdk_q8_0_gemv_i8_regs(data, scale, bias, x, y, in_dim, out_dim, st);
}

// Q8_0 small batch: x f32 [batch][in_dim], y f32 [batch][out_dim]; tokens in groups of up to eight,
// one weight pass per group.  -1 when the shape is outside the plan (K / 512 warps, 4 .. 12).
int pdk_q8_0_gemm_i8(const void* data, const void* scale, const float* bias, const float* x, float* y, uint32_t in_dim,
                     uint32_t out_dim, uint32_t batch, cudaStream_t st) {
    if (force_regs() || !pdk_aligned(scale, 16)) return -1;
    BatchPlan pl;
    if (!make_batch_plan(in_dim, pl)) return -1;
    const MapEntry* maps = nullptr;
    if (plane_maps<RQ80>(data, scale, in_dim, out_dim, &maps) != 0) return -1;
    static bool attr_set[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(gemm_ring_q8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    unsigned int* err = pdk_error_word();
    if (err == nullptr) return (int)cudaErrorUnknown;
    const uint32_t n_tiles = (out_dim + 15u) / 16u;
    uint32_t grid = (uint32_t)pdk_sm_count();
    if (grid > n_tiles) grid = n_tiles;
    for (uint32_t t0 = 0; t0 < batch; t0 += 8u) {
        const uint32_t nb = batch - t0 < 8u ? batch - t0 : 8u;
        const int rc = pdk_launch_pdl(gemm_ring_q8_kernel, dim3(grid), dim3(pl.W * 32u), (size_t)pl.smem_bytes, st, maps->dmap,
                                      maps->rmap, bias, x + (size_t)t0 * in_dim, y + (size_t)t0 * out_dim, in_dim, out_dim,
                                      nb, pl, err, t0 + 8u >= batch ? 1u : 0u);
        if (rc != 0) return rc;
    }
    return 0;
}

// warps of a team, teams, CTAs of a cluster, stages of the ring kernel's plan for a one-token call on this device; all 0 = not its call
PDK_EXPORT int pdk_gemv_plan(uint32_t in_dim, uint32_t out_dim, uint32_t dtype, uint32_t* plan) {
    if (plan == nullptr || out_dim == 0u) return cudaErrorInvalidValue;
    const RingPlan* p = nullptr;
    int rc;
    switch (dtype) {
        case PDK_KQ_Q4K: rc = shape_plan<RQ4K>(in_dim, out_dim, &p); break;
        case PDK_KQ_Q4_0: rc = shape_plan<RQ40>(in_dim, out_dim, &p); break;
        case PDK_KQ_Q5K: rc = shape_plan<RQ5K>(in_dim, out_dim, &p); break;
        case PDK_KQ_Q6K: rc = shape_plan<RQ6K>(in_dim, out_dim, &p); break;
        case 8u: rc = shape_plan<RQ80>(in_dim, out_dim, &p); break;      // ggml's Q8_0
        default: return cudaErrorInvalidValue;
    }
    if (rc > 0) return rc;
    const bool on = rc == 0 && !force_regs();
    plan[0] = on ? p->W : 0u;
    plan[1] = on ? p->teams : 0u;
    plan[2] = on ? p->split : 0u;
    plan[3] = on ? p->D : 0u;
    return 0;
}

// Q4_K GEMV on int8 activations (xq int8 [in_dim], one f32 scale per 32): same kernels, the
// activation staging widens q * scale before it builds its limbs.
int pdk_q4k_gemv_i8_q8act(const void* data, const void* scales, const int8_t* xq, const float* xq_scale, float* y,
                          uint32_t in_dim, uint32_t out_dim, cudaStream_t st) {
    const int rc = launch_ring<RQ4K>(data, scales, nullptr, nullptr, y, in_dim, out_dim, st, xq, xq_scale);
    return rc != -1 ? rc : pdk_q4k_gemv_i8_q8act_regs(data, scales, xq, xq_scale, y, in_dim, out_dim, st);
}

namespace {
int shard_launch(const void* data, const void* scales, const void* x, const void* const* y_ptrs, const void* const* flag_ptrs,
                 void* ctr, uint32_t n_ranks, uint32_t rank, uint32_t row0, uint32_t step, uint32_t signal, uint32_t in_dim,
                 uint32_t out_dim, cudaStream_t st) {
    if (out_dim == 0) return 0;
    if (n_ranks == 0 || n_ranks > 8u || y_ptrs == nullptr) return cudaErrorInvalidValue;
    if (!pdk_aligned(data, 16) || !pdk_aligned(scales, 8) || !pdk_aligned(x, 16)) return cudaErrorInvalidValue;
    gemv_i8::PeerOut po{};
    for (uint32_t p = 0; p < n_ranks; ++p) {
        if (y_ptrs[p] == nullptr || !pdk_aligned(y_ptrs[p], 4)) return cudaErrorInvalidValue;
        po.ptr[p] = (float*)y_ptrs[p];
    }
    po.n = n_ranks;
    po.row0 = row0;
    if (signal != 0u) {
        if (flag_ptrs == nullptr || ctr == nullptr || rank >= n_ranks || !pdk_aligned(ctr, 4))
            return cudaErrorInvalidValue;
        for (uint32_t p = 0; p < n_ranks; ++p) {
            if (flag_ptrs[p] == nullptr || !pdk_aligned(flag_ptrs[p], 4)) return cudaErrorInvalidValue;
            po.flag[p] = (uint32_t*)flag_ptrs[p];
        }
        po.ctr = (uint32_t*)ctr;
        po.rank = rank;
        po.step = step;
        po.signal = signal;
    }
    int rc = launch_ring<RQ4K>(data, scales, nullptr, (const float*)x, nullptr, in_dim, out_dim, st, nullptr, nullptr, &po);
    if (rc == -1) rc = pdk_q4k_gemv_peers_regs(data, scales, (const float*)x, &po, in_dim, out_dim, st);
    return rc >= 0 ? rc : (int)cudaErrorNotSupported;
}

// One warp: lane p waits until flags[p] has reached the step (wrap-around safe), for at most
// budget_ns; a lane that gives up records kErrFlagWait << 8 | p in the device error word.  The
// step is `step`; or, when that is 0, one more than the count of waits kept in flags[8], which
// the kernel then advances; or, when it is 0x80000000 | r, the value of flags[r].
enum : unsigned int { kErrFlagWait = 0x16 };
__global__ void peer_flags_wait_kernel(uint32_t* flags, uint32_t n_ranks, uint32_t step, unsigned long long budget_ns,
                                       unsigned int* err) {
    pdk_pdl_launch_dependents();
    pdk_pdl_wait();   // ordered after the kernel before it in the stream (this rank's own band)
    const uint32_t p = threadIdx.x;
    const uint32_t target = (step & 0x80000000u) ? flags[step & 7u] : step != 0u ? step : flags[8] + 1u;
    __syncwarp();
    if (step == 0u && p == 0u) flags[8] = target;
    if (p >= n_ranks) return;
    const volatile uint32_t* f = flags + p;
    const unsigned long long t0 = tc5::globaltimer_ns();
    uint32_t spins = 0;
    while ((int32_t)(*f - target) < 0) {
        if ((++spins & 31u) == 0u && tc5::globaltimer_ns() - t0 > budget_ns) {
            tc5::report(err, kErrFlagWait, p);
            return;
        }
    }
    __threadfence_system();   // acquire: the bands stored before the flags are visible to what follows
}
__global__ void peer_flags_post_kernel(const gemv_i8::PeerOut po) {
    pdk_pdl_launch_dependents();
    pdk_pdl_wait();   // the launch this signals, peer stores included, is complete
    if (threadIdx.x != 0u) return;
    const uint32_t step = po.ctr[1];
    if (step == 0u) return;
    for (uint32_t p = 0; p < po.n; ++p) gemv_i8::st_relaxed_sys(po.flag[p] + po.rank, step);
}
}  // namespace

// No counterpart in the reference (its multi-GPU story is one process per GPU, replicas only):
// Q4_K decode GEMV of one rank's row band that writes its band straight into every rank's
// full-length y (y_ptrs[0..n_ranks), device pointers valid on this GPU: its own buffer and the
// peers' buffers mapped over NVLink) at rows row0 .. row0 + out_dim.  The exchange that an
// all-gather would do is the kernel's own stores.  This form signals nothing: the stores are
// complete when the kernel is, and the caller orders consumers after it (stream order locally,
// a barrier across ranks).  n_ranks <= 8.  Returns 801 for shapes outside the GEMV kernels' plans.
PDK_EXPORT int pdk_q4k_gemv_shard(const void* data, const void* scales, const void* x, const void* const* y_ptrs,
                                  uint32_t n_ranks, uint32_t row0, uint32_t in_dim, uint32_t out_dim, void* stream) {
    return shard_launch(data, scales, x, y_ptrs, nullptr, nullptr, n_ranks, 0u, row0, 0u, 0u, in_dim, out_dim,
                        (cudaStream_t)stream);
}

// The same with a completion signal, so that a step needs no host barrier: after its band is
// stored everywhere, rank `rank` stores the step number into word `rank` of every rank's flag
// array (flag_ptrs[p] = rank p's array, mapped like y_ptrs; 16 u32 words, zeroed once at set-up:
// words 0..7 the flags, word 8 the count of pdk_peer_flags_wait calls).  ctr = two zeroed u32
// words of this rank's own memory, not shared between streams: the kernel's CTAs count
// themselves out on word 0, word 1 counts the rank's signalled steps.  step != 0 names the step
// (it must grow from call to call); step == 0 takes word 1 plus one, which lets a captured
// launch be replayed.  A consumer of y on rank p runs pdk_peer_flags_wait on its own flag array
// first.  The band is written with plain stores: a rank must not start step s + 1 before its
// consumers of step s are done with y (the wait kernel in the same stream gives that order), or y
// is double buffered.
PDK_EXPORT int pdk_q4k_gemv_shard_sync(const void* data, const void* scales, const void* x, const void* const* y_ptrs,
                                       const void* const* flag_ptrs, void* ctr, uint32_t n_ranks, uint32_t rank,
                                       uint32_t row0, uint32_t step, uint32_t in_dim, uint32_t out_dim, void* stream) {
    return shard_launch(data, scales, x, y_ptrs, flag_ptrs, ctr, n_ranks, rank, row0, step, 1u, in_dim, out_dim,
                        (cudaStream_t)stream);
}

// The same for a loop that keeps THREE (or more) y buffers in rotation.  All buffers of the loop share
// ONE flag array per rank and one pair of counter words.  Nothing is signalled at the end of the
// kernel (the system-scope fence that takes costs an NVLink round trip per step); instead every launch
// stores, behind its griddepcontrol.wait - when the stream's previous kernel and its peer stores are
// complete - the number of the PREVIOUS launch into the flags, and checks before it ends (at most a
// second; 0x1c << 8 | rank in the error word for a rank that is late) that every rank's previous step has
// arrived here.  What sits between launch s and launch s + 1 in the stream may therefore read step s - 1
// of every rank: a peer can be one launch ahead and already store step s + 1, but its step s + 2 - the
// first to return to the buffer of s - 1 when there are three - cannot start before this rank's launch
// s + 1 has begun.  One launch per step, consecutive steps overlap like single-GPU launches do, and the
// arrival of every step is still observed on the device.  After the last launch pdk_peer_flags_post
// signals it and pdk_peer_flags_wait (step = 0x80000000 | rank) observes it.
PDK_EXPORT int pdk_q4k_gemv_shard_lagged(const void* data, const void* scales, const void* x, const void* const* y_ptrs,
                                         const void* const* flag_ptrs, void* ctr, uint32_t n_ranks, uint32_t rank,
                                         uint32_t row0, uint32_t step, uint32_t in_dim, uint32_t out_dim, void* stream) {
    return shard_launch(data, scales, x, y_ptrs, flag_ptrs, ctr, n_ranks, rank, row0, step, 2u, in_dim, out_dim,
                        (cudaStream_t)stream);
}

// Closes a pdk_q4k_gemv_shard_lagged loop: stores the number of the stream's last launch (ctr[1]) into
// word `rank` of every rank's flag array, behind the stream's previous kernel.
PDK_EXPORT int pdk_peer_flags_post(const void* const* flag_ptrs, void* ctr, uint32_t n_ranks, uint32_t rank, void* stream) {
    if (flag_ptrs == nullptr || ctr == nullptr || n_ranks == 0u || n_ranks > 8u || rank >= n_ranks) return cudaErrorInvalidValue;
    gemv_i8::PeerOut po{};
    for (uint32_t p = 0; p < n_ranks; ++p) {
        if (flag_ptrs[p] == nullptr || !pdk_aligned(flag_ptrs[p], 4)) return cudaErrorInvalidValue;
        po.flag[p] = (uint32_t*)flag_ptrs[p];
    }
    po.ctr = (uint32_t*)ctr;
    po.n = n_ranks;
    po.rank = rank;
    return pdk_launch_pdl(peer_flags_post_kernel, dim3(1), dim3(32), 0, (cudaStream_t)stream, po);
}

// Waits on the device (one small kernel in `stream`) until every one of the n_ranks <= 8 flag
// words of `flags` (this rank's own 16-word flag array) has reached the step: `step`, or, when
// that is 0, one more than the array's count of such waits (word 8), which the kernel advances;
// or, when it is 0x80000000 | r, the step rank r (the caller's own rank) signalled last: every
// rank has then caught up with this rank.
// The wait is bounded: after budget_us microseconds (1 .. 10,000,000) the kernel records
// 0x16 << 8 | rank-that-is-late in the device error word (pdk_device_error) and returns; the
// context stays usable.  What follows in the stream sees every rank's band of that step.
PDK_EXPORT int pdk_peer_flags_wait(void* flags, uint32_t n_ranks, uint32_t step, uint32_t budget_us, void* stream) {
    if (flags == nullptr || n_ranks == 0u || n_ranks > 8u || budget_us == 0u || budget_us > 10000000u ||
        !pdk_aligned(flags, 4))
        return cudaErrorInvalidValue;
    unsigned int* err = pdk_error_word();
    if (err == nullptr) return (int)cudaErrorUnknown;
    return pdk_launch_pdl(peer_flags_wait_kernel, dim3(1), dim3(32), 0, (cudaStream_t)stream, (uint32_t*)flags, n_ranks, step,
                          (unsigned long long)budget_us * 1000ull, err);
}
