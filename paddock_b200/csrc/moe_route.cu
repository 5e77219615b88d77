// moe_route.cu - MoE routing around the grouped expert GEMMs: top-k router,
// expert alignment (token permutation into expert-contiguous blocks),
// activation preparation for the expert GEMMs, and the fixed-order
// slot combine.
#include <cuda_fp8.h>

#include "moe_route.cuh"
#include "pdk_common.cuh"

namespace {

// ---------------------------------------------------------------- top-k router (moe_route.cuh)
__global__ void moe_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias, uint32_t n_expert,
                                uint32_t k, uint32_t* __restrict__ out_idx, float* __restrict__ out_w,
                                uint32_t batch) {
    pdk_pdl_wait_then_launch();   // dependent launch: may start while the previous kernel of the stream drains
    const uint32_t token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (token >= batch) return;
    moe_route::topk_warp(logits + (size_t)token * n_expert, bias, n_expert, k, threadIdx.x & 31u,
                         out_idx + (size_t)token * k, out_w + (size_t)token * k);
}

// ---------------------------------------------------------------- expert alignment
// Groups the (token, slot) pairs by expert into blocks of `bm` entries, padding
// each expert's last block.  One CTA; a warp owns experts warp, warp+nwarps, ...
// and walks the pair list in order with ballots, so entries inside an expert
// keep ascending pair order (the layout is a pure function of the routing).
//   sorted_row[b*bm + i]  source token row, or PDK_MOE_PAD
//   sorted_slot[b*bm + i] which of the token's k picks
//   block_expert[b]       expert of block b, PDK_MOE_PAD past the used blocks
__global__ void __launch_bounds__(1024)
moe_align_kernel(const uint32_t* __restrict__ idx, uint32_t* __restrict__ sorted_row,
                 uint32_t* __restrict__ sorted_slot, uint32_t* __restrict__ block_expert, uint32_t rows,
                 uint32_t n_active, uint32_t n_expert, uint32_t bm, uint32_t max_blocks, uint32_t staged) {
    extern __shared__ uint32_t ash[];
    uint32_t* count = ash;               // [n_expert]
    uint32_t* boff = ash + n_expert;     // [n_expert + 1] first block of each expert
    uint32_t* sidx = boff + n_expert + 1u;  // [npairs] when `staged`: every warp rescans the whole list
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nwarp = blockDim.x >> 5;
    const uint32_t npairs = rows * n_active;
    for (uint32_t e = tid; e < n_expert; e += blockDim.x) count[e] = 0;
    __syncthreads();
    for (uint32_t p = tid; p < npairs; p += blockDim.x) {
        const uint32_t e = idx[p];
        if (staged) sidx[p] = e;
        if (e < n_expert) atomicAdd(&count[e], 1u);
    }
    __syncthreads();
    const uint32_t* pick = staged ? sidx : idx;
    if (tid == 0) {
        uint32_t b = 0;
        for (uint32_t e = 0; e < n_expert; ++e) {
            boff[e] = b;
            b += (count[e] + bm - 1u) / bm;
        }
        boff[n_expert] = b;
    }
    __syncthreads();
    const uint32_t used = min(boff[n_expert], max_blocks);
    for (uint32_t b = used + tid; b < max_blocks; b += blockDim.x) block_expert[b] = PDK_MOE_PAD;
    for (uint32_t e = warp; e < n_expert; e += nwarp) {
        const uint32_t b0 = boff[e], nb = boff[e + 1] - b0;
        for (uint32_t b = lane; b < nb; b += 32u)
            if (b0 + b < max_blocks) block_expert[b0 + b] = e;
        uint32_t pos = b0 * bm;
        for (uint32_t base = 0; base < npairs; base += 32u) {
            const uint32_t p = base + lane;
            const bool mine = p < npairs && pick[p] == e;
            const uint32_t m = __ballot_sync(0xffffffffu, mine);
            if (mine) {
                const uint32_t at = pos + __popc(m & ((1u << lane) - 1u));
                if (at < max_blocks * bm) {
                    sorted_row[at] = p / n_active;
                    sorted_slot[at] = p % n_active;
                }
            }
            pos += __popc(m);
        }
        const uint32_t end = (b0 + nb) * bm;
        for (uint32_t at = pos + lane; at < end; at += 32u)
            if (at < max_blocks * bm) {
                sorted_row[at] = PDK_MOE_PAD;
                sorted_slot[at] = 0;
            }
    }
}

// Same layout, linear work, one CTA: every warp owns a run of consecutive pairs.  It counts them per expert, one thread per
// expert turns the warps' counts into first places, and a second walk over the same pairs, held in registers, places them - in
// shared memory, from where the tables go out in whole lines.  The lanes with the same expert come from one vote per bit of the expert's number: __match_any_sync takes as many turns as there
// are different values.  Needs a [warps][n_expert] table in shared memory.
// pair_pos (may be null): position of pair p | its group's place in a scale record << 30, PDK_MOE_PAD for a pair that has none.
// (With a chunk of 1024 pairs at a time, its table cleared and summed up for each: 16.5 us at 4096 pairs of 128 experts, bound
// by barriers and the serial sums; this way 8.5.)
struct AlignArgs {
    const uint32_t* idx;
    uint32_t *sorted_row, *sorted_slot, *block_expert, *pair_pos;
    uint32_t rows, n_active, n_expert, bm, max_blocks, staged;   // staged: positions in shared memory first
};
constexpr uint32_t kAlignHeld = 4u;   // chunks of 32 pairs a warp keeps in registers

__device__ __forceinline__ void align_cta(const AlignArgs& a, uint32_t* ash) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nwarp = blockDim.x >> 5, ne = a.n_expert;
    uint32_t* count = ash;                // [ne] entries per expert
    uint32_t* boff = count + ne;          // [ne + 1] first block of each expert
    uint32_t* table = boff + ne + 1u;     // [nwarp][ne] entries, then the warp's next place among its expert's
    uint32_t* sums = table + nwarp * ne;  // [64] blocks of 32 experts each (up to 2048 experts)
    uint32_t* mine = table + warp * ne;
    const uint32_t npairs = a.rows * a.n_active, cap = a.max_blocks * a.bm;
    const uint32_t chunks = (npairs + 32u * nwarp - 1u) / (32u * nwarp), p0 = warp * chunks * 32u + lane;
    uint32_t held[kAlignHeld];
#pragma unroll
    for (uint32_t c = 0; c < kAlignHeld; ++c)
        held[c] = c < chunks && p0 + c * 32u < npairs ? a.idx[p0 + c * 32u] : 0xFFFFFFFFu;
    for (uint32_t e = lane; e < ne; e += 32u) mine[e] = 0u;
    __syncwarp();
    const uint32_t bits = 32u - __clz(ne);   // ne itself stands for every number that is no expert's
    auto peers_of = [&](uint32_t e) {
        const uint32_t v = min(e, ne);
        uint32_t m = 0xffffffffu;
        for (uint32_t i = 0; i < bits; ++i) {
            const uint32_t b = (v >> i) & 1u, ones = __ballot_sync(0xffffffffu, b);
            m &= b ? ones : ~ones;
        }
        return m;
    };
    uint32_t peers_held[kAlignHeld];
    auto add = [&](uint32_t e, uint32_t peers) {
        if (e < ne && (peers & ((1u << lane) - 1u)) == 0u) mine[e] += __popc(peers);
        __syncwarp();
    };
#pragma unroll
    for (uint32_t c = 0; c < kAlignHeld; ++c)
        if (c < chunks) { peers_held[c] = peers_of(held[c]); add(held[c], peers_held[c]); }
    for (uint32_t c = kAlignHeld; c < chunks; ++c) {
        const uint32_t e = p0 + c * 32u < npairs ? a.idx[p0 + c * 32u] : 0xFFFFFFFFu;
        add(e, peers_of(e));
    }
    __syncthreads();
    for (uint32_t e = tid; e < ne; e += blockDim.x) {   // per expert: places before each warp's
        uint32_t run = 0;
        for (uint32_t w = 0; w < nwarp; w += 8u) {
            uint32_t t[8];
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k) t[k] = w + k < nwarp ? table[(w + k) * ne + e] : 0u;
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k)
                if (w + k < nwarp) { table[(w + k) * ne + e] = run; run += t[k]; }
        }
        count[e] = run;
    }
    __syncthreads();
    // exclusive scan of the block counts: a warp per 32 experts, then the sums of the warps before
    const uint32_t turns = (ne + 31u) >> 5;
    for (uint32_t t = warp; t < turns; t += nwarp) {
        const uint32_t e = t * 32u + lane;
        const uint32_t nb = e < ne ? (count[e] + a.bm - 1u) / a.bm : 0u;
        uint32_t inc = nb;
#pragma unroll
        for (uint32_t d = 1; d < 32u; d <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += up;
        }
        if (e < ne) boff[e] = inc - nb;
        if (lane == 31u) sums[t] = inc;
    }
    uint32_t* place_of = sums + 64u;      // [cap] when staged: the pair at a position
    if (a.staged)
        for (uint32_t at = tid; at < cap; at += blockDim.x) place_of[at] = PDK_MOE_PAD;
    __syncthreads();
    for (uint32_t e = tid; e <= ne; e += blockDim.x) {
        uint32_t before = 0;
        for (uint32_t t = 0; t < (e == ne ? turns : e >> 5); ++t) before += sums[t];
        boff[e] = e == ne ? before : boff[e] + before;
    }
    __syncthreads();
    const uint32_t used = min(boff[ne], a.max_blocks);
    auto put = [&](uint32_t p, uint32_t e, uint32_t peers) {
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        const bool live = e < ne;
        const uint32_t place = live ? mine[e] + rank : 0u;
        __syncwarp();
        if (live && rank == 0u) mine[e] = place + __popc(peers);
        __syncwarp();
        if (p >= npairs) return;
        const uint32_t at = live ? boff[e] * a.bm + place : cap;
        if (at < cap) {
            if (a.staged) place_of[at] = p;
            else { a.sorted_row[at] = p / a.n_active; a.sorted_slot[at] = p % a.n_active; }
        }
        if (a.pair_pos) a.pair_pos[p] = at < cap ? at | ((a.bm == 8u ? place >> 3 : at >> 3) & 3u) << 30 : PDK_MOE_PAD;
    };
#pragma unroll
    for (uint32_t c = 0; c < kAlignHeld; ++c)
        if (c < chunks) put(p0 + c * 32u, held[c], peers_held[c]);
    for (uint32_t c = kAlignHeld; c < chunks; ++c) {
        const uint32_t p = p0 + c * 32u, e = p < npairs ? a.idx[p] : 0xFFFFFFFFu;
        put(p, e, peers_of(e));
    }
    for (uint32_t b = used + tid; b < a.max_blocks; b += blockDim.x) a.block_expert[b] = PDK_MOE_PAD;
    for (uint32_t e = tid; e < ne; e += blockDim.x) {
        for (uint32_t b = boff[e]; b < boff[e + 1u] && b < a.max_blocks; ++b) a.block_expert[b] = e;
        if (!a.staged)   // padding of the expert's last block
            for (uint32_t at = boff[e] * a.bm + count[e]; at < boff[e + 1u] * a.bm && at < cap; ++at) {
                a.sorted_row[at] = PDK_MOE_PAD;
                a.sorted_slot[at] = 0;
            }
    }
    if (!a.staged) return;
    __syncthreads();
    for (uint32_t at = tid; at < used * a.bm; at += blockDim.x) {
        const uint32_t p = place_of[at];
        a.sorted_row[at] = p == PDK_MOE_PAD ? PDK_MOE_PAD : p / a.n_active;
        a.sorted_slot[at] = p == PDK_MOE_PAD ? 0u : p % a.n_active;
    }
}

__global__ void __launch_bounds__(1024) moe_align_rank_kernel(const AlignArgs a) {
    extern __shared__ uint32_t ash[];
    pdk_pdl_wait_then_launch();   // dependent launch: may start while the previous kernel of the stream drains
    align_cta(a, ash);
}

// ---------------------------------------------------------------- activation prep
// f32 rows -> the B operand of the expert GEMMs: f16 with one power-of-two step
// 2^e per row chosen so that amax / 2^e lies in [2^14, 2^15).  bf16 activations
// are carried exactly (8 significant bits fit in f16's 11); general f32 ones are
// rounded to 11 significant bits.
// Layout per row and 32-element block, 64 bytes: for t = 0..3 the eight halves
//   [x(4t), x(4t+2), x(4t+1), x(4t+3), x(16+4t), x(16+4t+2), x(16+4t+1), x(16+4t+3)]
// which is one lane's B registers for the block's two mmas.
__global__ void __launch_bounds__(256)
moe_prep_act_kernel(const float* __restrict__ x, uint8_t* __restrict__ xq, float* __restrict__ xscale, uint32_t dim) {
    __shared__ float wmax[8];
    const uint32_t row = blockIdx.x, tid = threadIdx.x;
    const float* xr = x + (size_t)row * dim;
    float a = 0.0f;
    for (uint32_t i = tid; i < dim; i += 256u) {
        const float v = fabsf(xr[i]);
        a = fmaxf(a, v == v ? v : 0.0f);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, off));
    if ((tid & 31u) == 0u) wmax[tid >> 5] = a;
    __syncthreads();
    float amax = 0.0f;
    for (int w = 0; w < 8; ++w) amax = fmaxf(amax, wmax[w]);
    int e = 0;
    if (amax > 0.0f && amax < 3.0e38f) {
        (void)frexpf(amax, &e);   // amax in [2^(e-1), 2^e)
        e -= 15;                  // amax / 2^e in [2^14, 2^15)
        e = max(e, -100);
    }
    const float inv = ldexpf(1.0f, -e);
    if (tid == 0) xscale[row] = ldexpf(1.0f, e);
    uint8_t* out = xq + (size_t)row * dim * 2u;
    for (uint32_t u = tid; u < (dim >> 3); u += 256u) {  // one thread per (block, t): 8 elements -> 16 bytes
        const uint32_t blk = u >> 2, t = u & 3u;
        const float4 p = *reinterpret_cast<const float4*>(xr + blk * 32u + 4u * t);
        const float4 q = *reinterpret_cast<const float4*>(xr + blk * 32u + 16u + 4u * t);
        const __half2 h0 = __floats2half2_rn(p.x * inv, p.z * inv), h1 = __floats2half2_rn(p.y * inv, p.w * inv);
        const __half2 h2 = __floats2half2_rn(q.x * inv, q.z * inv), h3 = __floats2half2_rn(q.y * inv, q.w * inv);
        uint4 o;
        o.x = *reinterpret_cast<const uint32_t*>(&h0);
        o.y = *reinterpret_cast<const uint32_t*>(&h1);
        o.z = *reinterpret_cast<const uint32_t*>(&h2);
        o.w = *reinterpret_cast<const uint32_t*>(&h3);
        *reinterpret_cast<uint4*>(out + (size_t)blk * 64u + t * 16u) = o;
    }
}

// ---------------------------------------------------------------- slot combine
// A thread per four columns of a row; the slots' loads of a thread are in flight together, four at a time.  Bound by memory where
// rows are many.  Where they are narrow too, a block takes several (NARROW, up to 512 columns and from 1024 rows on), and no call
// has more than 16 blocks per SM: a block per row starts blocks and does little else (70000 rows of 32 columns 68 -> 4.1 us, 5000 of
// 64, 8 slots, 5.7 -> 2.4, 5000 of 516 5.85 -> 4.8; 1024 of 2880, 4 slots, 5.5 either way; several rows a block cost 64 rows of
// 128 columns 1.4 -> 1.56).
template <bool NARROW>
__global__ void __launch_bounds__(256)
moe_slot_combine_kernel(const float4* __restrict__ part, float4* __restrict__ residual, uint32_t embd4, uint32_t n_active,
                        uint32_t rows) {
    pdk_pdl_wait_then_launch();   // dependent launch: may start while the previous kernel of the stream drains
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= embd4) return;
    const uint32_t step = NARROW ? gridDim.y * blockDim.y : gridDim.y;
    for (size_t t = NARROW ? blockIdx.y * blockDim.y + threadIdx.y : blockIdx.y; t < rows; t += step) {
        const float4* p = part + t * n_active * embd4 + r;
        float4 d = residual[t * embd4 + r];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t k = 0; k < n_active; k += 4u) {  // fixed slot order: bit-reproducible
            float4 v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j)
                if (k + j < n_active) v[j] = __ldcs(p + (size_t)(k + j) * embd4);
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j)
                if (k + j < n_active) { acc.x += v[j].x; acc.y += v[j].y; acc.z += v[j].z; acc.w += v[j].w; }
        }
        d.x += acc.x; d.y += acc.y; d.z += acc.z; d.w += acc.w;
        residual[t * embd4 + r] = d;
    }
}

}  // namespace

// slot 29, packs/cuda/src/attn/decode.cuh:1392-1500 (launcher gemm/f32_qkv.cuh:1137-1150)
PDK_EXPORT int pd_moe_topk_batch(const void* logits, const void* bias, uint32_t n_expert, uint32_t k, void* out_idx,
                                 void* out_w, uint32_t batch, void* stream) {
    if (batch == 0) return 0;
    if (n_expert == 0 || n_expert > 512u || k == 0 || k > 16u || k > n_expert) return cudaErrorInvalidValue;
    return pdk_launch_pdl(moe_topk_kernel, dim3((batch + 3u) / 4u), dim3(128), 0, (cudaStream_t)stream,
                          (const float*)logits, (const float*)bias, n_expert, k, (uint32_t*)out_idx, (float*)out_w, batch);
}

// shared memory of align_cta without and with the staged positions
static size_t align_smem(uint32_t n_expert, uint32_t warps) { return ((size_t)(warps + 2u) * n_expert + 65u) * sizeof(uint32_t); }

static int align_impl(const void* idx, void* sorted_row, void* sorted_slot, void* block_expert, void* pair_pos, uint32_t rows,
                      uint32_t n_active, uint32_t n_expert, uint32_t bm, uint32_t max_blocks, void* stream) {
    if (rows == 0 || n_expert == 0) return 0;
    if (bm == 0 || (bm & (bm - 1u)) || n_expert > 4096u) return cudaErrorInvalidValue;
    static const cudaError_t attr_rank =
        cudaFuncSetAttribute(moe_align_rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    // a warp per 32 pairs, up to 32 warps: with few pairs the counts of the idle ones would only be cleared and summed
    const uint64_t pairs = (uint64_t)rows * n_active;
    const uint32_t warps = pairs >= 1024u ? 32u : pairs <= 128u ? 4u : (uint32_t)((pairs + 31u) / 32u);
    const size_t base = align_smem(n_expert, warps), places = (size_t)max_blocks * bm * sizeof(uint32_t);
    const uint32_t in_smem = base + places <= 200u * 1024u ? 1u : 0u;
    if (attr_rank == cudaSuccess && base <= 200u * 1024u && n_expert <= 2048u) {
        const AlignArgs a{(const uint32_t*)idx, (uint32_t*)sorted_row, (uint32_t*)sorted_slot, (uint32_t*)block_expert,
                          (uint32_t*)pair_pos, rows, n_active, n_expert, bm, max_blocks, in_smem};
        return pdk_launch_pdl(moe_align_rank_kernel, dim3(1), dim3(32u * warps), base + (in_smem ? places : 0u), (cudaStream_t)stream, a);
    }
    if (pair_pos) return cudaErrorInvalidValue;
    // many experts: the scan kernel, one warp per expert
    size_t shmem = (size_t)(2u * n_expert + 1u) * sizeof(uint32_t);
    // the pick list is staged in shared memory when it fits (up to 200 KB)
    const size_t list = (size_t)rows * n_active * sizeof(uint32_t);
    const uint32_t staged = shmem + list <= 200u * 1024u ? 1u : 0u;
    if (staged) shmem += list;
    static const cudaError_t attr_rc =
        cudaFuncSetAttribute(moe_align_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (attr_rc != cudaSuccess) return (int)attr_rc;
    moe_align_kernel<<<1, 1024, shmem, (cudaStream_t)stream>>>((const uint32_t*)idx, (uint32_t*)sorted_row,
                                                               (uint32_t*)sorted_slot, (uint32_t*)block_expert, rows,
                                                               n_active, n_expert, bm, max_blocks, staged);
    return pdk_launch_status();
}

// slot 146, packs/cuda/src/gemm/f32_qkv.cuh:1269-1279 (kernel attn/decode.cuh:2316-2396)
PDK_EXPORT int pd_moe_align_bm(const void* idx, void* sorted_row, void* sorted_slot, void* block_expert,
                               uint32_t rows, uint32_t n_active, uint32_t n_expert, uint32_t bm, uint32_t max_blocks,
                               void* stream) {
    return align_impl(idx, sorted_row, sorted_slot, block_expert, nullptr, rows, n_active, n_expert, bm, max_blocks, stream);
}

// No slot: moe_align_bm that also leaves every pair's position for pdk_moe_prep_tokens_f4, u32[rows * n_active]: the position |
// its group's place in a scale record << 30, or PDK_MOE_PAD where the pair has no expert or no room.  bm 8 or 32, up to 1500
// experts, positions below 2^30.
PDK_EXPORT int pdk_moe_align_pos(const void* idx, void* sorted_row, void* sorted_slot, void* block_expert, void* pair_pos,
                                 uint32_t rows, uint32_t n_active, uint32_t n_expert, uint32_t bm, uint32_t max_blocks,
                                 void* stream) {
    if (rows == 0 || n_expert == 0) return 0;
    if ((bm != 8u && bm != 32u) || n_expert > 1500u || !pair_pos || max_blocks >= (1u << 25)) return cudaErrorInvalidValue;
    return align_impl(idx, sorted_row, sorted_slot, block_expert, pair_pos, rows, n_active, n_expert, bm, max_blocks, stream);
}

// slot 34, packs/cuda/src/attn/decode.cuh:2316-2396: blocks of 32 entries
PDK_EXPORT int pd_moe_align(const void* idx, void* sorted_row, void* sorted_slot, void* block_expert, uint32_t rows,
                            uint32_t n_active, uint32_t n_expert, uint32_t max_blocks, void* stream) {
    return pd_moe_align_bm(idx, sorted_row, sorted_slot, block_expert, rows, n_active, n_expert, 32u, max_blocks,
                           stream);
}

// No slot: the activation step in front of the expert GEMMs (the reference's
// chain quantizes to int8 here, packs/cuda/src/attn/decode.cuh:2981-3004).
// x f32[rows][dim] -> xq f16[rows][dim] (fragment order) + xscale f32[rows]; dim % 32 == 0.
PDK_EXPORT int pdk_moe_prep_act(const void* x, void* xq, void* xscale, uint32_t dim, uint32_t rows, void* stream) {
    if (rows == 0 || dim == 0) return 0;
    if ((dim & 31u) != 0u || !pdk_aligned(x, 16) || !pdk_aligned(xq, 16)) return cudaErrorInvalidValue;
    moe_prep_act_kernel<<<rows, 256, 0, (cudaStream_t)stream>>>((const float*)x, (uint8_t*)xq, (float*)xscale, dim);
    return pdk_launch_status();
}

// slot 91, packs/cuda/src/moe/mmq.cuh:447-483
PDK_EXPORT int pd_moe_slot_combine(const void* part, void* residual, uint32_t embd, uint32_t n_active, uint32_t rows,
                                   void* stream) {
    if (rows == 0 || embd == 0) return 0;
    if ((embd & 3u) != 0u || !pdk_aligned(part, 16) || !pdk_aligned(residual, 16)) return cudaErrorInvalidValue;
    const uint32_t embd4 = embd >> 2, nx = (embd4 + 255u) / 256u;
    const bool narrow = embd4 <= 128u && rows >= 1024u;
    const uint32_t cols = narrow ? embd4 : ((embd4 + nx - 1u) / nx + 31u) & ~31u, rows_per_block = narrow ? 256u / cols : 1u;
    const uint64_t blocks = ((uint64_t)rows + rows_per_block - 1u) / rows_per_block;
    const uint32_t cap = (16u * (uint32_t)pdk_sm_count() + nx - 1u) / nx;
    return pdk_launch_pdl(narrow ? moe_slot_combine_kernel<true> : moe_slot_combine_kernel<false>,
                          dim3(nx, (uint32_t)(blocks < cap ? blocks : cap)), dim3(cols, rows_per_block), 0, (cudaStream_t)stream,
                          (const float4*)part, (float4*)residual, embd4, n_active, rows);
}
