// splitk_gemm.cu - the FP8 row-scaled and the NVFP4 GEMM wherever the 256 x 256 tiles of the pair
// kernels (fp8_gemm2.cu, nvf4_gemm2.cu) cannot fill the chip: decode widths, and short prompts through
// narrow planes.
//
//   fp8    y[t][n] = ( sum_k e4m3(X[t][k]) * e4m3(W[n][k]) ) * xs[t] * ws[n]
//   nvfp4  y[t][n] = scale2 * ( block-scaled e2m1 sum ) + bias[n]
//
// At decode widths the work is a stream of weights and the time is set by how many SMs pull on
// HBM and how soon they start.  One CTA per output tile leaves most of the chip idle for the
// planes a decode step meets (5120 x 5120: 20 tiles of 256 channels for 148 SMs, 18 us for a
// plane that HBM delivers in 4), so K is split as well: a tile is 128 channels x BN tokens, and a
// cluster of S CTAs shares it, each summing every S-th part of K.  The partial accumulators meet
// through distributed shared memory and are added in rank order: same sum whatever the timing, no
// scratch, no zeroing, no second launch.  Where K is short or the tokens are many the meeting costs more
// than the split saves: one CTA takes the tile and stores it from tensor memory (plan_split has the line).
//
// Two CTAs share an SM (about 100 KB of stages and at most half the tensor memory each): while one meets
// its cluster and stores, the other streams, and a CTA's start-up (barriers, tensor memory, first boxes)
// is hidden the same way.  A CTA owns one tile part and leaves; the hardware scheduler does the rest.  (One
// persistent CTA per SM with double-buffered accumulators measured slower: 11.7 against 9.6 us for one
// NVFP4 token through 5120 x 17408, 8.1 against 7.4 for seven FP8 tokens through 5120 x 5120.)
//
// Weights are the A operand (128 rows = 128 tensor-memory lanes), tokens the N dimension, so a
// decode batch costs N = 32 columns.  A stage is 128 bytes of K:
//   warp 0      producer: TMA boxes of W and X (128-byte swizzle); nvfp4: the weight scale record as
//               a bulk copy
//   warp 1      MMA issuer (four MMAs per stage, nvfp4 with their scale-cell copies)
//   warps 2..5  nvfp4: warp 2 + c brings token rows 32 c .. 32 c + 31's activation scales into cell order,
//               16 bytes per row and stage through registers (4-byte cp.async from the producer took four
//               times the L1 requests and bound the kernel from 64 tokens on); then the epilogue
#include "cluster_caps.cuh"
#include "nvf4_tc5.cuh"

namespace {

using tc5::cluster_addr;
using tc5::cluster_sync;
using tc5::st_cluster;

enum Kind : int { kFp8 = 0, kNvf4 = 1 };

constexpr uint32_t BM = 128, BKB = 128;
constexpr uint32_t kABytes = BM * BKB, kSfBytes = 2048;
constexpr uint32_t kMaxSplit = kPdkMaxCluster;
constexpr uint32_t kThreads = 192;
constexpr uint32_t kMaxStages = 5;
constexpr uint32_t kSmemHalf = 115712;  // what lets two CTAs share an SM: 228 KB / 2 - 1 KB reserved

template <int KIND, uint32_t BN>
struct Cfg {
    static constexpr uint32_t kBBytes = BN * BKB;
    static constexpr uint32_t kOffSfa = kABytes + kBBytes, kOffSfb = kOffSfa + kSfBytes;
    static constexpr uint32_t kStageBytes = KIND == kFp8 ? kABytes + kBBytes : kOffSfb + kSfBytes;
    static constexpr uint32_t kFit = (kSmemHalf - 256u) / kStageBytes;
    static constexpr uint32_t kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static constexpr uint32_t kTmemCols = KIND == kFp8 ? BN : 256u;   // nvfp4: 32 columns of scale cells per stage behind the accumulator
    static constexpr uint32_t kIdesc = KIND == kFp8 ? tc5::idesc_f32acc(0u, 0u, BM, BN)
                                                    : (1u << 7) | (1u << 10) | ((BN >> 3) << 17) | ((BM >> 4) << 24);
    static constexpr uint32_t kSmemBytes = kStages * kStageBytes + 256u;
    static_assert(KIND == kFp8 || BN + 32u * kStages <= 256u, "tensor memory of one of two CTAs");
    // the partial sums of a tile reuse the stages: S x BN tokens x ceil(128 / S) channels, rounded up to four
    static_assert(BN * (BM + 4u * kMaxSplit) * 4u <= kStages * kStageBytes, "partial sums fit the stages");
};

struct Shared {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_full;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Shared) <= 256u, "control block");

struct Args {
    const uint8_t* w_sf;       // nvfp4: tiled weight scale records
    const uint8_t* x_sf;       // nvfp4: row-major activation scales
    const float* w_scale;      // fp8: per channel
    const float* x_scale;      // fp8: per token
    const float* bias;         // nvfp4, optional
    float scale2;              // nvfp4
    void* y;
    uint32_t in_dim, out_dim, batch, num_kb;
    uint32_t tile_t0, tile_w0; // the launch's first token and channel tile
    uint32_t vec_store;        // y rows take 4-channel vector stores
    uint32_t sf_vec;           // nvfp4: x_sf is 16-byte aligned
    unsigned int* err;
};

// A store that may be past the batch.  Predicated, not branched around: with `if (i < left)` in front of it the compiler
// leaves a branch per store, about 50 cycles each, one microsecond for 32 tokens.
__device__ __forceinline__ void store_if(float* p, float v, bool on) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void store_if(__nv_bfloat16* p, __nv_bfloat16 v, bool on) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.b16 [%0], %1;\n\t}" ::"l"(p), "h"(__bfloat16_as_ushort(v)), "r"((uint32_t)on) : "memory");
}

template <typename TO>
__device__ __forceinline__ void store4(TO* p, const float (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(float* p, const float (&v)[4]) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    __stcs(reinterpret_cast<uint2*>(p), make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b)));
}
__device__ __forceinline__ float to_out(float v, float*) { return v; }
__device__ __forceinline__ __nv_bfloat16 to_out(float v, __nv_bfloat16*) { return __float2bfloat16_rn(v); }

template <int KIND, uint32_t BN, typename TO>
__global__ void __launch_bounds__(kThreads, 2)
splitk_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const Args a) {
    using C = Cfg<KIND, BN>;
    extern __shared__ __align__(1024) uint8_t smem[];
    Shared* sh = reinterpret_cast<Shared*>(smem + C::kStages * C::kStageBytes);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t split = gridDim.x, rank = blockIdx.x;   // the cluster spans x
    const uint32_t tw = a.tile_w0 + blockIdx.z, t0 = (a.tile_t0 + blockIdx.y) * BN, n0 = tw * BM, n_tok = min(BN, a.batch - t0);
    const uint32_t kb_lo = rank * a.num_kb / split, kb_hi = (rank + 1u) * a.num_kb / split;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < C::kStages; ++s) {
            tc5::mbar_init(&sh->full[s], KIND == kFp8 ? 1u : 1u + BN / 32u);   // the expected-bytes arrival (+ one per scale warp)
            tc5::mbar_init(&sh->empty[s], 1);
        }
        tc5::mbar_init(&sh->acc_full, 1);
        sh->abort_flag = 0;
        tc5::mbar_fence_init();
        tc5::tma_prefetch_desc(&tmap_w);
        tc5::tma_prefetch_desc(&tmap_x);
    }
    if (warp == 1) {
        tc5::tmem_alloc(&sh->tmem_base, C::kTmemCols);
        tc5::tmem_relinquish();
    }
    if constexpr (KIND == kNvf4) {
        // activation scale cells: the scale warps write the row groups a token tile has; the rest stay zero
        for (uint32_t i = threadIdx.x; i < C::kStages * (kSfBytes / 16u); i += kThreads)
            reinterpret_cast<uint4*>(smem + (i / (kSfBytes / 16u)) * C::kStageBytes + C::kOffSfb)[i % (kSfBytes / 16u)] =
                make_uint4(0u, 0u, 0u, 0u);
        nvf4tc5::fence_proxy_async_smem();
    }
    tc5::fence_before_sync();
    __syncthreads();
    tc5::fence_after_sync();
    const uint32_t tmem_base = sh->tmem_base;
    const tc5::WaitCtx ctx{&sh->abort_flag, a.err};
    pdk_pdl_launch_dependents();

    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------ producer (whole warp, one lane issues)
        const uint64_t stream_once = tc5::l2_policy_evict_first();
        const bool reused = gridDim.y > 1u;    // several token tiles read the same weights: keep them in L2
        auto issue_w = [&](uint32_t stage, uint32_t kb) {
            uint8_t* s = smem + stage * C::kStageBytes;
            tc5::mbar_arrive_expect_tx_elect(&sh->full[stage], kABytes + C::kBBytes + (KIND == kNvf4 ? kSfBytes : 0u));
            if (reused) tc5::tma_load_2d_elect(s, &tmap_w, &sh->full[stage], (int32_t)(kb * BKB), (int32_t)n0);
            else tc5::tma_load_2d_hint_elect(s, &tmap_w, &sh->full[stage], (int32_t)(kb * BKB), (int32_t)n0, stream_once);
            if constexpr (KIND == kNvf4)
                tc5::bulk_load_elect(s + C::kOffSfa, a.w_sf + ((size_t)tw * a.num_kb + kb) * kSfBytes, kSfBytes, &sh->full[stage]);
        };
        // weights depend on nothing the previous kernel in the stream writes: the first stages go out before the wait for it
        const uint32_t pre = min(kb_hi - kb_lo, C::kStages);
        for (uint32_t i = 0; i < pre; ++i) issue_w(i, kb_lo + i);
        pdk_pdl_wait();
        uint32_t stage = 0, phase = 0;
        for (uint32_t kb = kb_lo; kb < kb_hi; ++kb) {
            if (kb - kb_lo >= pre) {
                ok = __all_sync(0xffffffffu, tc5::mbar_wait(&sh->empty[stage], phase ^ 1u, ctx, tc5::kErrEmptyWait, stage));
                if (!ok) break;
                issue_w(stage, kb);
            }
            tc5::tma_load_2d_elect(smem + stage * C::kStageBytes + kABytes, &tmap_x, &sh->full[stage], (int32_t)(kb * BKB), (int32_t)t0);
            if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok && lane == 0)   // copies already issued still land in this CTA's shared memory
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
        uint32_t stage = 0, phase = 0;
        for (uint32_t kb = kb_lo; kb < kb_hi; ++kb) {
            ok = __all_sync(0xffffffffu, tc5::mbar_wait(&sh->full[stage], phase, ctx, tc5::kErrFullWait, stage));
            if (!ok) break;
            tc5::fence_after_sync();
            const uint32_t s_addr = tc5::smem_u32(smem + stage * C::kStageBytes);
            const uint64_t a_desc = tc5::smem_desc_sw128(s_addr), b_desc = tc5::smem_desc_sw128(s_addr + kABytes);
            if constexpr (KIND == kFp8) {
                tc5::mma_f8f6f4_x4_elect(tmem_base, a_desc, b_desc, C::kIdesc, kb != kb_lo);
            } else {
                const uint32_t sfa_t = tmem_base + BN + stage * 32u;
                nvf4tc5::slab_nvf4<true>(tmem_base, a_desc, b_desc, C::kIdesc, kb != kb_lo, sfa_t, sfa_t + 16u, s_addr + C::kOffSfa,
                                         s_addr + C::kOffSfb, 4u);
            }
            tc5::mma_commit_elect(&sh->empty[stage]);
            if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
        }
        if (ok) tc5::mma_commit_elect(&sh->acc_full);
        pdk_pdl_wait();
    } else {
        pdk_pdl_wait();   // activations, scales and y may still be in use by the previous kernel
        if (KIND == kNvf4 && warp - 2u < BN / 32u) {
            // word (j, l, c) of a stage's 2 KB record is xs[t0 + c*32 + l][kb*16 + 4j .. 4j+3]
            const uint32_t c = warp - 2u, t = t0 + c * 32u + lane, n_kb = kb_hi - kb_lo;
            const uint8_t* src = a.x_sf + (size_t)min(t, a.batch - 1u) * (a.in_dim >> 4) + kb_lo * 16u;
            const bool live = t < a.batch;
            auto load = [&](uint32_t i) {      // the row's 16 scales of stage i
                if (!live || i >= n_kb) return make_uint4(0u, 0u, 0u, 0u);
                if (a.sf_vec) return *reinterpret_cast<const uint4*>(src + i * 16u);
                const uint32_t* w = reinterpret_cast<const uint32_t*>(src + i * 16u);
                return make_uint4(w[0], w[1], w[2], w[3]);
            };
            constexpr uint32_t kAhead = 4;
            uint4 next[kAhead];
#pragma unroll
            for (uint32_t i = 0; i < kAhead; ++i) next[i] = load(i);
            uint32_t stage = 0, phase = 0;
            for (uint32_t k0 = 0; k0 < n_kb && ok; k0 += kAhead) {
                uint4 cur[kAhead];
#pragma unroll
                for (uint32_t i = 0; i < kAhead; ++i) {
                    cur[i] = next[i];
                    next[i] = load(k0 + kAhead + i);
                }
#pragma unroll
                for (uint32_t i = 0; i < kAhead; ++i) {
                    if (k0 + i >= n_kb || !ok) break;
                    if (k0 + i >= C::kStages)
                        ok = __all_sync(0xffffffffu, tc5::mbar_wait(&sh->empty[stage], phase ^ 1u, ctx, tc5::kErrEmptyWait, stage));
                    if (!ok) break;
                    uint32_t* d = reinterpret_cast<uint32_t*>(smem + stage * C::kStageBytes + C::kOffSfb) + lane * 4u + c;
                    d[0] = cur[i].x; d[128] = cur[i].y; d[256] = cur[i].z; d[384] = cur[i].w;
                    nvf4tc5::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0u) tc5::mbar_arrive(&sh->full[stage]);
                    if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
                }
            }
        }
        ok = tc5::mbar_wait(&sh->acc_full, 0u, ctx, tc5::kErrTmemFullWait, 0u);
        __syncwarp();
    }
    tc5::fence_before_sync();
    __syncthreads();
    // every CTA's stages are consumed from here on: they take the partial sums
    if (split > 1u) cluster_sync();
    tc5::fence_after_sync();

    // Rank r adds up and stores channels [r * cpr, (r + 1) * cpr) of the tile: each CTA leaves its partial sums in
    // the owner's buffer [rank][token][cpr channels].  A lane is a channel, so its owner and address are fixed and
    // its columns go out back to back (by token columns, the owner changing from store to store, 93 tokens over 8
    // CTAs took 12.3 us instead of 9.7).
    const uint32_t cpr = ((BM + split - 1u) / split + 3u) & ~3u;
    float* red = reinterpret_cast<float*>(smem);
    TO* y = reinterpret_cast<TO*>(a.y);
    if (split == 1u) {
        // The tile is whole: straight from tensor memory to y, 32 neighbouring channels per store.  By way of the partial
        // sums' buffer below it took NVFP4, K = 1024, N = 5120 4.5 us instead of 3.2 at 32 tokens, 8.8 instead of 5.2 at 200.
        if (warp >= 2u) {
            const uint32_t quarter = warp & 3u, n = n0 + quarter * 32u + lane;
            const bool live = n < a.out_dim;
            const float ws = KIND == kFp8 && live ? __ldg(a.w_scale + n) : 0.0f;
            const float bias = KIND == kNvf4 && live && a.bias != nullptr ? a.bias[n] : 0.0f;
#pragma unroll 1
            for (uint32_t c = 0; c < n_tok; c += 32u) {
                uint32_t r[32];
                tc5::tmem_ld_32x32(tmem_base + ((quarter * 32u) << 16) + c, r);
                const float xs = KIND == kFp8 ? a.x_scale[t0 + min(c + lane, n_tok - 1u)] : 0.0f;
                tc5::tmem_ld_wait();
                TO* out = y + (size_t)(t0 + c) * a.out_dim + n;
                const uint32_t left = live ? n_tok - c : 0u;
#pragma unroll
                for (uint32_t i = 0; i < 32u; ++i) {
                    const float v = __uint_as_float(r[i]);
                    float o;
                    if constexpr (KIND == kFp8) o = v * (__shfl_sync(0xffffffffu, xs, i) * ws);
                    else o = fmaf(v, a.scale2, bias);
                    store_if(out, to_out(o, out), i < left);
                    out += a.out_dim;
                }
            }
            tc5::fence_before_sync();
        }
        __syncthreads();
        if (warp == 1) {
            tc5::fence_after_sync();
            tc5::tmem_dealloc(tmem_base, C::kTmemCols);
        }
        return;
    }
    if (warp >= 2u) {
        const uint32_t quarter = warp & 3u, ch = quarter * 32u + lane;      // a warp reads its own quarter of the tensor-memory lanes
        const uint32_t dst = cluster_addr(tc5::smem_u32(red), ch / cpr) + (rank * n_tok * cpr + ch % cpr) * 4u;
#pragma unroll 1
        for (uint32_t c = 0; c < n_tok; c += 32u) {
            uint32_t r[32];
            tc5::tmem_ld_32x32(tmem_base + ((quarter * 32u) << 16) + c, r);
            tc5::tmem_ld_wait();
            const uint32_t at = dst + c * cpr * 4u, left = n_tok - c;
#pragma unroll
            for (uint32_t i = 0; i < 32u; ++i)
                if (i < left) st_cluster(at + i * cpr * 4u, __uint_as_float(r[i]));
        }
        tc5::fence_before_sync();
    }
    cluster_sync();

    const uint32_t ch_lo = rank * cpr, groups = ch_lo < BM ? min(cpr, BM - ch_lo) / 4u : 0u;   // of four channels
    for (uint32_t i = threadIdx.x; i < groups * n_tok; i += kThreads) {
        const uint32_t tok = i / groups, g = (i - tok * groups) * 4u, n = n0 + ch_lo + g, t = t0 + tok;
        if (n >= a.out_dim) continue;
        const float* part = red + tok * cpr + g;
        float4 sum = *reinterpret_cast<const float4*>(part);
        for (uint32_t s = 1; s < split; ++s) {
            const float4 p = *reinterpret_cast<const float4*>(part + s * n_tok * cpr);
            sum.x += p.x; sum.y += p.y; sum.z += p.z; sum.w += p.w;
        }
        float v[4] = {sum.x, sum.y, sum.z, sum.w};
        const float xs = KIND == kFp8 ? a.x_scale[t] : 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j) {
            const uint32_t nj = min(n + j, a.out_dim - 1u);
            if constexpr (KIND == kFp8) v[j] = v[j] * (xs * __ldg(a.w_scale + nj));
            else v[j] = fmaf(v[j], a.scale2, a.bias != nullptr ? a.bias[nj] : 0.0f);
        }
        TO* out = y + (size_t)t * a.out_dim + n;
        if (a.vec_store) {          // out_dim % 4 == 0: the four channels are all there
            store4<TO>(out, v);
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j)
                if (n + j < a.out_dim) out[j] = to_out(v[j], out);
        }
    }
    if (warp == 1) {
        tc5::fence_after_sync();
        tc5::tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// The CTAs that share a tile of BN tokens (the split of K) in a call: 0 or a cudaError_t.
template <int KIND, uint32_t BN, typename TO>
int plan_split(const Args& a, uint32_t& split, uint32_t& sms) {
    // How many clusters of s CTAs are resident at once (they stay within a GPC).  The driver counts one CTA per SM for
    // a kernel that allocates tensor memory; two run, so twice its answer (148, 74, 45, 33, 26, 22, 15, 15 on a B200).
    static PdkClusterCaps table;
    const uint32_t* resident = nullptr;
    if (int rc = pdk_cluster_caps(table, (const void*)splitk_gemm_kernel<KIND, BN, TO>, kThreads, Cfg<KIND, BN>::kSmemBytes, &resident)) return rc;
    // The largest split whose clusters are all resident at once: more only add start-ups.  K = 5120, N = 5120, 7 tokens
    // (40 tiles): 11.4 us at S = 1, 7.6 at 4, 7.4 at 6, and 11.9 at 7, where a part of the clusters waits for a
    // second turn.  At least two stages per CTA, so that it streams more than it sets up.
    const uint32_t tiles_t = (a.batch + BN - 1u) / BN, tiles_w = (a.out_dim + BM - 1u) / BM;
    split = a.num_kb / 2u < kMaxSplit ? a.num_kb / 2u : kMaxSplit;
    while (split > 1u && (uint64_t)tiles_t * tiles_w > 2u * resident[split]) --split;
    // It has to save a CTA more slabs (0.3 us each) than the meeting of the partial sums costs, which grows with the tokens of a
    // tile.  us whole / split: fp8 K = 1024, N = 1024: 3.6 / 3.4 at 1 token, 3.7 / 4.4 at 32, 5.3 / 7.1 at 128; nvfp4 K = 1024, N = 5120:
    // 3.1 / 3.8 at 1, 4.7 / 8.4 at 128; K = 2048, N = 5120: 4.7 / 4.5 at 1, 4.8 / 5.3 at 32.  Over 1500 random shapes
    // (K = 1024 ... 17408, N = 512 ... 27648, 1 ... 8192 tokens) this choice is within 1.2 % of the best of all eight splits on average.
    // Several tiles of 64 tokens count as tiles of 128, there are as many more of them (nvfp4 K = 3584, N = 1088, 265 tokens: 7.3 whole, 7.9 split).
    const uint32_t tokens = tiles_t > 1u ? (BN < 128u ? 128u : BN) : a.batch, saved = split > 1u ? a.num_kb - (a.num_kb + split - 1u) / split : 0u;
    if (KIND == kFp8 ? saved * 12u <= 6u * 12u + tokens : saved * 16u <= 4u * 16u + tokens) split = 1u;
    if (split == 0u) split = 1u;
    sms = resident[1];
    return 0;
}

template <int KIND, uint32_t BN, typename TO>
int launch_bn(const void* data, const void* xq, Args& a, uint32_t row_bytes, uint32_t split, cudaStream_t st) {
    using C = Cfg<KIND, BN>;
    CUtensorMap tw, tx;
    if (int rc = pdk_make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, data, row_bytes, a.out_dim, row_bytes, BKB, BM)) return rc;
    if (int rc = pdk_make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, row_bytes, a.batch, row_bytes, BKB, BN)) return rc;
    auto kern = splitk_gemm_kernel<KIND, BN, TO>;
    const uint32_t tiles_t = (a.batch + BN - 1u) / BN, tiles_w = (a.out_dim + BM - 1u) / BM;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdk_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    // one launch, unless a grid axis cannot hold the tiles (numbering them along x instead cost a division per CTA, 0.1 us)
    constexpr uint32_t kAxis = 65535u;
    for (a.tile_w0 = 0u; a.tile_w0 < tiles_w; a.tile_w0 += kAxis)
        for (a.tile_t0 = 0u; a.tile_t0 < tiles_t; a.tile_t0 += kAxis) {
            const uint32_t nt = tiles_t - a.tile_t0, nw = tiles_w - a.tile_w0;
            cfg.gridDim = dim3(split, nt < kAxis ? nt : kAxis, nw < kAxis ? nw : kAxis);
            if (cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, tx, a); e != cudaSuccess) return (int)e;
        }
    return pdk_launch_status();
}

template <int KIND, typename TO>
int launch(const void* data, const void* xq, Args& a, uint32_t row_bytes, cudaStream_t st) {
    a.num_kb = (row_bytes + BKB - 1u) / BKB;
    a.vec_store = (a.out_dim & 3u) == 0u && pdk_aligned(a.y, 4u * sizeof(TO)) ? 1u : 0u;
    a.sf_vec = pdk_aligned(a.x_sf, 16) ? 1u : 0u;
    a.err = pdk_error_word();
    uint32_t split = 1u, sms = 0u;
    if (a.batch <= 32u) {
        if (int rc = plan_split<KIND, 32, TO>(a, split, sms)) return rc;
        return launch_bn<KIND, 32, TO>(data, xq, a, row_bytes, split, st);
    }
    if (int rc = plan_split<KIND, 64, TO>(a, split, sms)) return rc;
    if (a.batch > 64u) {
        // Tiles of 64 or of 128 tokens (figures: us with 128 / with 64).  64 while they are all resident, two CTAs per SM: a tile starts and ends sooner,
        // and there are twice as many to fill the chip (fp8 1024 x 5120, 100 tokens 6.3 / 5.0, 160 tokens 6.9 / 5.1; 5120 x 17408, 128 tokens
        // 23.6 / 20.7; nvfp4 5120 x 5120, 200 tokens 13.1 / 9.6; beyond it fp8 1024 x 25600, 96 tokens 8.5 / 10.8).  128
        //  - where 64 leaves a CTA more slabs of K and the tokens are few (fp8 8192 x 9728: 65 tokens 18.5 / 22.9, 17408 x 5120, 80 tokens 20.8 / 23.0);
        //  - for up to 80 tokens on a split row: 128 moves no more partial sums than there are tokens, and a second tile is
        //    mostly padding (fp8 2048 x 2560, 65 tokens 6.5 / 7.1; nvfp4 10240 x 632, 68 tokens 6.4 / 6.8; even at 80);
        //  - for long rows of many tiles: 64 reads each weight twice as often, and L2 paces that (fp8 14592 x 3528, 323 tokens, 19152 slabs in all:
        //    25.2 / 35.2; 15104 x 2424, 283 tokens, 11210: 20.5 / 23.5; 9728 x 2264, 332 tokens, 8208: even);
        //  - above 512 tokens, where 64 was not measured.
        // Over 260 shapes of 65 ... 512 tokens: 0.90 of the time with 128 alone, 1 % over the better of the two; longer by more than 3 % on five,
        // 8 % at worst (fp8 15872 x 3608, 87 tokens 15.1 / 16.3).  More weight on the slabs mends those and loses as much elsewhere
        // (nvfp4 9216 x 11160, 123 tokens 17.3 / 16.2).
        uint32_t split128 = 1u;
        if (int rc = plan_split<KIND, 128, TO>(a, split128, sms)) return rc;
        const uint64_t tiles = (uint64_t)((a.batch + 63u) / 64u) * ((a.out_dim + BM - 1u) / BM);
        const uint32_t slabs = (a.num_kb + split - 1u) / split, slabs128 = (a.num_kb + split128 - 1u) / split128;
        if (tiles > 2u * sms || a.batch > 512u || (a.batch <= 80u && split128 > 1u) || (slabs > slabs128 && 3u * (slabs - slabs128) + 40u > a.batch) ||
            (a.num_kb > 64u && a.num_kb * tiles > 8000u && a.batch > 128u))
            return launch_bn<KIND, 128, TO>(data, xq, a, row_bytes, split128, st);
    }
    return launch_bn<KIND, 64, TO>(data, xq, a, row_bytes, split, st);
}

}  // namespace

// Whether a pair kernel (256 x 256 tiles, two SMs each) beats this file's 128 x 128 tiles for a prompt.  Per SM the
// pair tile moves fewer shared-memory bytes per flop, but it starts later and its time hardly falls below that of one full
// tile.  So the line falls with K, and lies at many small tiles where K is short.  Measured on a B200 (434 random shapes of 129 ...
// 8192 tokens; the rule is within 1 % of the faster one on average, and 4 % behind it at worst where it used to choose
// the other), us here / pair: fp8 K = 1024, N = 5120: 22.4 / 28.4 at 2500 tokens (800 small tiles); K = 2048, N = 5120: 31.0 / 32.4
// there; K = 5120, N = 5120, 200 tokens: 15.3 / 21.6, N = 17408, 2500 tokens: 225 / 157.  nvfp4, whose pair kernel also has a 128-token tile and
// re-tiles the activation scales first: K = 1024, N = 17408: 18.1 / 19.5 at 700 tokens, 34.5 / 32.5 at 1500; K = 8192, N = 9472: 108 / 83
// at 2500.  Up to 128 tokens, one token tile, the weight stream decides and this kernel keeps the call.
bool pdk_prefer_pair(uint32_t batch, uint32_t out_dim, uint32_t row_bytes, bool nvf4) {
    if (batch <= 128u) return false;
    const uint64_t small = (uint64_t)((batch + 127u) / 128u) * ((out_dim + 127u) / 128u), slabs = (row_bytes + BKB - 1u) / BKB;
    return small > 100u && (small - 100u) * slabs > (nvf4 ? 8000u : 6000u);
}

int pdk_f8row_gemm_splitk(const void* data, const void* w_scale, const void* xq, const void* x_scale, void* y, uint32_t in_dim,
                          uint32_t out_dim, uint32_t batch, bool bf16, cudaStream_t st) {
    Args a{};
    a.w_scale = (const float*)w_scale; a.x_scale = (const float*)x_scale; a.y = y;
    a.in_dim = in_dim; a.out_dim = out_dim; a.batch = batch;
    return bf16 ? launch<kFp8, __nv_bfloat16>(data, xq, a, in_dim, st) : launch<kFp8, float>(data, xq, a, in_dim, st);
}

int pdk_nvf4_gemm_splitk(const void* data, const void* scale_tiled, const void* bias, const void* xq, const void* xs, void* y,
                         float scale2, uint32_t in_dim, uint32_t out_dim, uint32_t batch, bool bf16, cudaStream_t st) {
    Args a{};
    a.w_sf = (const uint8_t*)scale_tiled; a.x_sf = (const uint8_t*)xs; a.bias = (const float*)bias; a.scale2 = scale2; a.y = y;
    a.in_dim = in_dim; a.out_dim = out_dim; a.batch = batch;
    const uint32_t row_bytes = in_dim >> 1;
    return bf16 ? launch<kNvf4, __nv_bfloat16>(data, xq, a, row_bytes, st) : launch<kNvf4, float>(data, xq, a, row_bytes, st);
}
