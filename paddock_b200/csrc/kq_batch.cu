// kq_batch.cu - Q4_K, Q5_K, Q6_K, Q4_0 and Q8_0 planes times 1..16 tokens per launch on mma.sync f16, weights exact.
//
// The work is a stream of weights; what the kernel is built around is what it costs to get a weight byte in front of
// the tensor core and a scale behind it:
//
//   * weights come as TMA boxes of 16 rows x one super-block (a "unit") into a ring that every warp owns and refills
//     itself; the scale records as 8-byte cp.async copies on the same mbarrier.  Fetched by plain loads, a Q6_K unit is
//     34 requests that touch eight rows each, and the L1 request rate (about 270 cycles a unit) set the time;
//   * a code is its own f16 operand: the bit pattern of q in 0..63 is the subnormal number q 2^-24, which the tensor core
//     multiplies exactly.  A high nibble stays where it is (16 q 2^-24; its block's scale is divided by 16), so two weights
//     cost one AND (an AND-OR with the high bits of Q5_K / Q6_K) and no conversion.  Q8_0's int8 codes are raised by 128 on the way (XOR);
//   * activations: per token and unit a power of two brings the largest element below 2^10, and x = hi + lo in two f16
//     terms (22 bits, exact for bf16 values).  Both terms accumulate into one f32 tile, so a block is folded into the unit's
//     sum with four FFMAs per 16 x 8 tile (an int8 fold takes eight IMADs at half their rate, and an s8 m16n8k16 for
//     Q6_K's 16-weight blocks takes the tensor pipe as long, 8 cycles, as an f16 one).  Up to four tokens the terms are columns of
//     their own: one mma and half the fragment bytes per step;
//   * the min term (Q4_K, Q5_K), the -32 (Q6_K), the -8 (Q4_0) and the -128 (Q8_0) are products of the block scales with the block
//     sums of x: one or two more MMAs per unit.
//
// Split: a cluster of S CTAs shares a run of 16-row tiles, each CTA one part of K - its part of the activations (4 bytes
// per element and token) has to fit beside the ring, and narrow planes fill the chip that way.  A CTA's (tile, unit)
// pairs are one sequence, cut into equal runs for its 16 warps whatever the tile count; a warp leaves one partial tile per
// tile that it touched, and the partials meet once per round (as many tiles as shared memory holds partials of; one,
// mostly), in a fixed order, across the cluster in distributed shared memory: the same sum whatever the timing, no
// scratch, no zeroing of y, one launch.
//
// Measured on a B200 (us; up to 4 tokens: terms as two mmas -> as columns).  Q6_K, K = 17408, N = 5003: 28.2 -> 26.0 at 2 tokens, 27.8 -> 25.6 at 3,
// 28.7 -> 26.5 at 4, 34.1 at 8; K = 5120, N = 25600: 33.2 -> 30.4 at 2, 38 at 8, 76 at 16.  Q4_K, K = 17408, N = 5120: 23.6 -> 20.6 at 2; Q4_0, K = 5120,
// N = 25600: 25.4 -> 21.5.  Q8_0 (a GEMV per token before): 7424 x 520, 8 tokens 108 -> 6.7; 2816 x 6016, 16 tokens 96 -> 16.
// What bounds it from 5 tokens: the shared memory pipe (118 wavefronts per unit, 64 of them the activation fragments: 13 of
// the 25 us of Q4_K, K = 5120, N = 25600 at 2 tokens with two mmas) and issue slots (450 instructions per unit).  Tiles of 32 rows halve the fragments but double the ring's stages, so that
// fewer fit: 24.7 us at 1 token, but 45 at 8 and no plan at all for Q6_K, not kept.
#include "cluster_caps.cuh"
#include "kq_plan.cuh"
#include "tc5.cuh"

namespace {

using namespace kq;
using tc5::cluster_addr;
using tc5::cluster_sync;
using tc5::st_cluster;
static_assert(kMaxSplit == kPdkMaxCluster, "cluster_caps.cuh asks for these sizes");

struct Args {
    const uint8_t* recs;
    const float* x;            // f32 activations, or null:
    const int8_t* xq;          // int8 activations ...
    const float* xq_scale;     // ... with one scale per 32 elements
    const float* bias;         // [out_dim] or null
    float* y;
    uint32_t in_dim, out_dim, batch, stages, ku_max, round_tiles;
    unsigned int* err;
};

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// byte `i` of the scale words as a float (times 1/16 for a block whose codes sit 4 bits up); `bias` is what the byte
// was raised by.  2^23 + byte is exact, and so is the product that takes it off again.
__device__ __forceinline__ float scale_f(uint32_t w, uint32_t i, bool up, float bias) {
    const float f = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | i));
    return up ? fmaf(f, 0.0625f, -(8388608.0f + bias) * 0.0625f) : f - (8388608.0f + bias);
}

// HL: up to four tokens.  The mma's columns are (token, term) pairs: one mma and an 8-byte fragment per step where a column per
// token takes two mmas and 16 bytes, and the two terms' sums are added when a tile is done.
template <int F, uint32_t NT, bool HL>
__global__ void __launch_bounds__(kWarps * 32u, 1)
kq_batch_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const Args a) {
    using T = Fmts<F>;
    constexpr uint32_t NCOLS = NT * 8u, kThreads = kWarps * 32u;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, t = lane & 3u;
    const uint32_t split = gridDim.x, rank = blockIdx.x;   // the cluster spans x
    const uint32_t n_unit = a.in_dim >> 8, n_tiles = (a.out_dim + kRows - 1u) / kRows;
    const uint32_t u_lo = rank * n_unit / split, ku = (rank + 1u) * n_unit / split - u_lo;
    const uint32_t t_lo = (uint32_t)((uint64_t)blockIdx.y * n_tiles / gridDim.y);
    const uint32_t t_hi = (uint32_t)((uint64_t)(blockIdx.y + 1u) * n_tiles / gridDim.y);
    const Layout L = layout<F, NT>(a.stages, a.batch, a.ku_max, a.round_tiles);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.off_bar) + warp * a.stages;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.off_bar + kWarps * a.stages * 8u);
    const tc5::WaitCtx ctx{abort_flag, a.err};
    uint8_t* box0 = smem + warp * a.stages * kBox0;
    uint8_t* box1 = smem + L.off_box1 + warp * a.stages * T::kBox1;
    uint8_t* recs = smem + L.off_rec + warp * a.stages * T::kRecs;
    float* red = reinterpret_cast<float*>(smem + L.off_red);

    pdk_pdl_launch_dependents();
    if (lane == 0u) {
        for (uint32_t s = 0; s < a.stages; ++s) tc5::mbar_init(&bars[s], 33u);   // expected bytes + 32 lanes' record copies
        tc5::mbar_fence_init();
    }
    if (tid == 0u) *abort_flag = 0;
    __syncwarp();

    // ---- the warp's load cursor
    const uint64_t stream_once = tc5::l2_policy_evict_first();
    uint32_t l_tile = 0u, l_u = 0u, rec_off[2];
    const uint8_t* rec_src = a.recs;
    constexpr uint32_t kPieces = T::kRec / 8u, kCopies = (kRows * kPieces + 31u) / 32u;   // eight-byte pieces of a row's record, copies of a lane
    auto seek = [&](uint32_t tile, uint32_t u) {
        l_tile = tile;
        l_u = u;
        const uint32_t row0 = min(tile * kRows, a.out_dim - 1u), last = a.out_dim - 1u - row0;
        rec_src = a.recs + ((size_t)row0 * n_unit + u_lo + u) * T::kRec;
#pragma unroll
        for (uint32_t i = 0; i < kCopies; ++i) {
            const uint32_t c = i * 32u + lane, r = c / kPieces;
            rec_off[i] = min(r, last) * n_unit * T::kRec + (c - kPieces * r) * 8u;
        }
    };
    auto issue = [&](uint32_t s) {
        const uint32_t u = u_lo + l_u;
        tc5::mbar_arrive_expect_tx_elect(&bars[s], kBox0 + T::kBox1);
        tc5::tma_load_2d_hint_elect(box0 + s * kBox0, &tm0, &bars[s], (int32_t)(u * T::kUnit), (int32_t)(l_tile * kRows), stream_once);
        if constexpr (T::kBox1 != 0u)
            tc5::tma_load_2d_hint_elect(box1 + s * T::kBox1, &tm1, &bars[s], (int32_t)(u * T::kUnit + 128u), (int32_t)(l_tile * kRows), stream_once);
        const uint32_t dst = tc5::smem_u32(recs + s * T::kRecs) + lane * 8u;
#pragma unroll
        for (uint32_t i = 0; i < kCopies; ++i)
            if (i == 0u || lane < 16u) cp_async8(dst + i * 256u, rec_src + rec_off[i]);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc5::smem_u32(&bars[s])) : "memory");
        rec_src += T::kRec;
        if (++l_u == ku) seek(l_tile + 1u, 0u);
    };
    uint32_t stage = 0u, phase = 0u;
    bool ok = true;

    for (uint32_t r0 = t_lo; r0 < t_hi; r0 += a.round_tiles) {
        const uint32_t nt = min(a.round_tiles, t_hi - r0), total = nt * ku;
        const uint32_t f_lo = warp * total / kWarps, f_hi = (warp + 1u) * total / kWarps, mine = f_hi - f_lo;
        uint32_t c_tile = f_lo / ku, c_u = f_lo - c_tile * ku;
        seek(r0 + c_tile, c_u);
        const uint32_t pre = min(mine, a.stages);
        // weights depend on nothing the previous kernel in the stream writes: the ring fills before the wait for it
        for (uint32_t i = 0, s = stage; i < pre && ok; ++i) {
            issue(s);
            if (++s == a.stages) s = 0u;
        }
        if (r0 == t_lo) {
            pdk_pdl_wait();
            // ---- the activation image, one warp per (token, unit), eight elements per lane.  Step s (16 elements of k) of a
            // unit is 64 bytes, lane t's 16 = {hi(e0,e2), hi(e1,e3), lo(e0,e2), lo(e1,e3)} of the four elements it feeds
            const uint32_t tasks = a.batch * ku;
            auto load8 = [&](uint32_t task, float (&v)[8]) {
                if (task >= tasks) return;
                const uint32_t tok = task / ku, ul = task - tok * ku;
                const size_t e0 = (size_t)tok * a.in_dim + (u_lo + ul) * 256u + lane * 8u;
                if (a.x != nullptr) {
                    const float4 p = *reinterpret_cast<const float4*>(a.x + e0), q = *reinterpret_cast<const float4*>(a.x + e0 + 4u);
                    v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
                } else {
                    const int2 q = *reinterpret_cast<const int2*>(a.xq + e0);
                    const float s = a.xq_scale[e0 >> 5];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = (float)(int8_t)((i < 4 ? q.x >> (8 * i) : q.y >> (8 * (i - 4))) & 0xff) * s;
                }
            };
            float next[2][8];       // two tasks ahead: a task is one L2 round trip
            load8(warp, next[0]);
            load8(warp + kWarps, next[1]);
            for (uint32_t task = warp; task < tasks; task += kWarps) {
                const uint32_t tok = task / ku, ul = task - tok * ku;
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) { v[i] = next[0][i]; next[0][i] = next[1][i]; }
                load8(task + 2u * kWarps, next[1]);
                float amax = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
                // non-negative floats order as their bit patterns; amax < 2^ex: x 2^(10 - ex) stays below 2^10, a sum of
                // 32 below the f16 range
                const uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
                const int ex = bits == 0u ? 0 : min(128, max((int)(bits >> 23) - 126, -100));
                const float mul = __uint_as_float((uint32_t)(137 - ex) << 23), back = __uint_as_float((uint32_t)(117 + ex) << 23);
                float sum = 0.0f;
                uint8_t* dst = smem + L.off_b + tok * L.pitch + ul * 1024u +
                               (F == kQ6K ? (lane >> 1) * 64u + (lane & 1u) * 32u : (lane >> 2) * 128u + (lane & 3u) * 16u);
#pragma unroll
                for (uint32_t j = 0; j < 2u; ++j) {
                    uint32_t hi[2], lo[2];
#pragma unroll
                    for (uint32_t p = 0; p < 2u; ++p) {
                        const float e = v[4u * j + p] * mul, f = v[4u * j + p + 2u] * mul;
                        const __half2 h = __floats2half2_rn(e, f);
                        hi[p] = h2_bits(h);
                        lo[p] = h2_bits(__floats2half2_rn(e - __low2float(h), f - __high2float(h)));
                        sum += e + f;
                    }
                    *reinterpret_cast<uint4*>(dst + j * (F == kQ6K ? 16u : 64u)) = make_uint4(hi[0], hi[1], lo[0], lo[1]);
                }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                if constexpr (F != kQ6K) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                constexpr uint32_t kPer = 32u / T::kBlocks;      // lanes per block
                if ((lane & (kPer - 1u)) == 0u) {
                    __half* xs = reinterpret_cast<__half*>(smem + L.off_xs) + (ul * a.batch + tok) * 2u * T::kBlocks + lane / kPer;
                    const __half h = __float2half_rn(sum);
                    xs[0] = h;
                    xs[T::kBlocks] = __float2half_rn(sum - __half2float(h));
                }
                if (lane == 0u) reinterpret_cast<float*>(smem + L.off_step)[ul * a.batch + tok] = back;
            }
            __syncthreads();
        }

        // ---- the stream.  mma row g is row 2g (g < 4) or 2g - 7 of its half of the tile: the four rows whose 8-byte reads
        // fall into one pass of the banks are then 0,2,4,6 or 1,3,5,7, which the 128-byte swizzle puts on distinct banks
        const uint32_t row = g < 4u ? 2u * g : 2u * g - 7u;
        uint32_t col[NT], even[NT], odd[NT];       // columns past the batch repeat its last token
#pragma unroll
        for (uint32_t n = 0; n < NT; ++n) {
            col[n] = min(HL ? g >> 1 : g + 8u * n, a.batch - 1u);
            even[n] = min(HL ? t : 2u * t + 8u * n, a.batch - 1u);
            odd[n] = HL ? even[n] : min(2u * t + 1u + 8u * n, a.batch - 1u);
        }
        float acc[NT][4];
#pragma unroll
        for (uint32_t n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.0f;
        const float* ustep = reinterpret_cast<const float*>(smem + L.off_step);
        constexpr uint32_t kSteps = F == kQ6K ? 1u : 2u;
        constexpr float kBias = F == kQ6K ? 128.0f : 0.0f;
        constexpr bool kF16Scales = F == kQ40 || F == kQ80;

        for (uint32_t q = 0; q < mine; ++q) {
            ok = __all_sync(0xffffffffu, ok && tc5::mbar_wait(&bars[stage], phase, ctx, tc5::kErrFullWait, 0x50u + warp));
            if (!ok) break;
            const uint8_t* b0 = box0 + stage * kBox0;
            const uint8_t* b1 = box1 + stage * T::kBox1;
            const uint8_t* rb = recs + stage * T::kRecs + row * T::kRec;
            float U[NT][4];
#pragma unroll
            for (uint32_t n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) U[n][i] = 0.0f;
            const uint8_t* bp[NT];
#pragma unroll
            for (uint32_t n = 0; n < NT; ++n) bp[n] = smem + L.off_b + col[n] * L.pitch + c_u * 1024u + t * 16u + (HL ? (g & 1u) * 8u : 0u);

            uint32_t sw[2][4];     // the scale bytes (Q6: raised by 128; Q4_0, Q8_0: eight f16 scales)
            uint2 high[2];         // Q5: the high-bit bytes 8t .. 8t+7
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                const uint32_t* rp = reinterpret_cast<const uint32_t*>(rb + h * 8u * T::kRec) + (kF16Scales ? 0 : 1);
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i)
                    sw[h][i] = (F == kQ6K) ? rp[i] ^ 0x80808080u : (kF16Scales || i < 2u) ? rp[i] : 0u;
                if constexpr (F == kQ5K) high[h] = *reinterpret_cast<const uint2*>(b1 + (row + h * 8u) * 32u + t * 8u);
            }
            // A pair of blocks shares its bytes: the low nibbles' block and the high nibbles' (Q8_0: blocks p and 4 + p, of the two boxes)
#pragma unroll
            for (uint32_t p = 0; p < T::kBlocks / 2u; ++p) {
                // Q6: p = half * 4 + h * 2 + (run & 1)
                const uint32_t nh = p >> 2, hb = (p >> 1) & 1u, r01 = p & 1u;
                uint32_t x[2][kSteps], z[2][kSteps];
#pragma unroll
                for (uint32_t h = 0; h < 2u; ++h) {
                    const uint32_t r = row + h * 8u;
                    if constexpr (F == kQ6K) {
                        const uint32_t c = 4u * nh + 2u * r01 + hb;
                        x[h][0] = *reinterpret_cast<const uint32_t*>(b0 + r * 128u + ((c ^ (row & 7u)) << 4) + t * 4u);
                        z[h][0] = *reinterpret_cast<const uint32_t*>(b1 + r * 64u + (((2u * nh + hb) ^ ((row >> 1) & 3u)) << 4) + t * 4u);
                    } else {
                        const uint32_t at = r * 128u + (((2u * p + (t >> 1)) ^ (row & 7u)) << 4) + (t & 1u) * 8u;
                        const uint2 v = *reinterpret_cast<const uint2*>(b0 + at);
                        x[h][0] = v.x;
                        x[h][kSteps - 1u] = v.y;
                        const uint2 w = F == kQ80 ? *reinterpret_cast<const uint2*>(b1 + at) : high[h];
                        z[h][0] = w.x;
                        z[h][kSteps - 1u] = w.y;
                    }
                }
#pragma unroll
                for (uint32_t up = 0; up < 2u; ++up) {
                    const uint32_t b = F == kQ6K ? 8u * nh + 2u * (r01 + 2u * up) + hb : F == kQ80 ? 4u * up + p : 2u * p + up;
                    const uint32_t mq = up ? 0x00F000F0u : 0x000F000Fu;
                    float d[NT][4];
#pragma unroll
                    for (uint32_t j = 0; j < kSteps; ++j) {
                        uint32_t A[4];       // {row g, row g + 8} x {bytes 0, 2 | bytes 1, 3}
#pragma unroll
                        for (uint32_t h = 0; h < 2u; ++h) {
                            const uint32_t xv = x[h][j], zv = z[h][j];
                            if constexpr (F == kQ6K) {
                                const uint32_t mh = up ? 0x03000300u : 0x00300030u, sh = r01 ? 2u : 4u;
                                A[h] = (xv & mq) | ((zv << sh) & mh);
                                A[2u + h] = ((xv >> 8) & mq) | ((zv >> (8u - sh)) & mh);
                            } else if constexpr (F == kQ80) {
                                // int8 raised by 128: 0..255, subnormal too
                                const uint32_t wv = (up ? zv : xv) ^ 0x80808080u;
                                A[h] = wv & 0x00FF00FFu;
                                A[2u + h] = (wv >> 8) & 0x00FF00FFu;
                            } else {
                                A[h] = xv & mq;
                                A[2u + h] = (xv >> 8) & mq;
                                if constexpr (F == kQ5K) {
                                    // bit b of a byte goes to bit 4 of its code (up: 8, the code being 4 bits up)
                                    const uint32_t mh = up ? 0x01000100u : 0x00100010u, to = up ? 8u : 4u;
                                    A[h] |= (to >= b ? zv << (to - b) : zv >> (b - to)) & mh;
                                    A[2u + h] |= (zv >> (8u + b - to)) & mh;
                                }
                            }
                        }
                        if constexpr (HL) {
                            const uint2 v = *reinterpret_cast<const uint2*>(bp[0] + (b * kSteps + j) * 64u);
                            if (j == 0u) mma_f16_z(d[0], A, v.x, v.y);
                            else mma_f16(d[0], A, v.x, v.y);
                            continue;
                        }
                        uint4 v[NT];
#pragma unroll
                        for (uint32_t n = 0; n < NT; ++n) v[n] = *reinterpret_cast<const uint4*>(bp[n] + (b * kSteps + j) * 64u);
#pragma unroll
                        for (uint32_t n = 0; n < NT; ++n)
                            if (j == 0u) mma_f16_z(d[n], A, v[n].x, v[n].y);
                            else mma_f16(d[n], A, v[n].x, v[n].y);
#pragma unroll
                        for (uint32_t n = 0; n < NT; ++n) mma_f16(d[n], A, v[n].z, v[n].w);
                    }
                    float s[2];
#pragma unroll
                    for (uint32_t h = 0; h < 2u; ++h) {
                        if constexpr (F == kQ80) {
                            const __half2 v = *reinterpret_cast<const __half2*>(&sw[h][b >> 1]);
                            s[h] = (b & 1u) ? __high2float(v) : __low2float(v);
                        } else if constexpr (F == kQ40) {
                            const __half2 v = *reinterpret_cast<const __half2*>(&sw[h][p]);
                            s[h] = up ? __high2float(v) * 0.0625f : __low2float(v);
                        } else {
                            s[h] = scale_f(sw[h][b >> 2], b & 3u, up != 0u, kBias);
                        }
                    }
#pragma unroll
                    for (uint32_t n = 0; n < NT; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) U[n][i] = fmaf(s[i >> 1], d[n][i], U[n][i]);
                }
            }
            // ---- scales x block sums
            const uint32_t sel = (t & 1u) ? 0x4342u : 0x4140u;     // bytes 2 (t & 1), + 1 into the halves
            const bool odd_w = (t & 2u) != 0u;
            uint32_t A[4], dd[2];
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                const uint32_t* rp = reinterpret_cast<const uint32_t*>(rb + h * 8u * T::kRec);
                dd[h] = rp[0];
                if constexpr (F == kQ6K) {
                    // int8 scales as f16: 1024 + (sc + 128) by bit pattern, less 1152
                    const __half2 off = __floats2half2_rn(1152.0f, 1152.0f);
                    const uint32_t e = __byte_perm(odd_w ? sw[h][1] : sw[h][0], 0x64646464u, sel);
                    const uint32_t f = __byte_perm(odd_w ? sw[h][3] : sw[h][2], 0x64646464u, sel);
                    A[h] = h2_bits(__hsub2(*reinterpret_cast<const __half2*>(&e), off));
                    A[2u + h] = h2_bits(__hsub2(*reinterpret_cast<const __half2*>(&f), off));
                } else if constexpr (kF16Scales) {
                    A[h] = A[2u + h] = rp[t];
                } else {
                    A[h] = A[2u + h] = __byte_perm(rp[3u + (t >> 1)], 0u, sel);
                }
            }
            const __half2 dh[2] = {*reinterpret_cast<const __half2*>(&dd[0]), *reinterpret_cast<const __half2*>(&dd[1])};
#pragma unroll
            for (uint32_t n = 0; n < NT; ++n) {
                const uint32_t* xs = reinterpret_cast<const uint32_t*>(smem + L.off_xs + (c_u * a.batch + col[n]) * T::kBlocks * 4u);
                float M[4];
                const bool takes = !HL || (g & 1u) == 0u;     // the first term's column has both terms' sums
                auto xsum = [&](uint32_t i) { return takes ? xs[i] : 0u; };
                mma_f16_z(M, A, xsum(t), xsum(4u + t));      // Q4 / Q5: A twice along k, the high terms, then the low ones
                if constexpr (F == kQ6K) mma_f16(M, A, xsum(8u + t), xsum(12u + t));
                const float* st = ustep + c_u * a.batch;
                const float se = st[even[n]], so = st[odd[n]];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float dg = __low2float(dh[i >> 1]) * 16777216.0f;
                    float v;
                    if constexpr (kF16Scales) v = fmaf(U[n][i], 16777216.0f, (F == kQ80 ? -128.0f : -8.0f) * M[i]);
                    else if constexpr (F == kQ6K) v = dg * fmaf(-32.0f / 16777216.0f, M[i], U[n][i]);
                    else v = dg * U[n][i] - __high2float(dh[i >> 1]) * (M[i] * 16777216.0f);
                    acc[n][i] = fmaf((i & 1) ? so : se, v, acc[n][i]);
                }
            }
            __syncwarp();
            if (q + a.stages < mine) issue(stage);
            if (++stage == a.stages) { stage = 0u; phase ^= 1u; }

            if (++c_u == ku || q + 1u == mine) {
                // the (tile, warp) pairs that meet increase by one or two from each partial to the next: slot = tile + warp
                float* dst = red + (size_t)(c_tile + warp) * kRows * NCOLS;
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) {
                    if constexpr (HL) {
                        dst[row * NCOLS + t] = acc[n][0] + acc[n][1];
                        dst[(row + 8u) * NCOLS + t] = acc[n][2] + acc[n][3];
                    } else {
                        float* to = dst + row * NCOLS + n * 8u + 2u * t;
                        *reinterpret_cast<float2*>(to) = make_float2(acc[n][0], acc[n][1]);
                        *reinterpret_cast<float2*>(to + 8u * NCOLS) = make_float2(acc[n][2], acc[n][3]);
                    }
                    acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
                }
                c_u = 0u;
                ++c_tile;
            }
        }
        if (!ok)      // copies already issued still land in this CTA's shared memory
            for (int i = 0; i < 64; ++i) __nanosleep(1000);

        // ---- the partials meet.  Row r of the round belongs to rank r / rpo
        __syncthreads();
        if (split > 1u) cluster_sync();        // every CTA of the cluster is done with its ring
        const uint32_t rows = nt * kRows, rpo = (rows + split - 1u) / split;
        const uint32_t part = tc5::smem_u32(smem);
        // Only calls on Q8_0 planes have a bias.  Where the other formats' instances for 5 and more tokens asked for it too it cost them 0.1 to
        // 0.2 us, and 10 % where a cluster stores many rows (Q4_K 7424 x 5707, 11 tokens 25.0 us, 22.6 without).  Up to four tokens the
        // question stays: without it the compiler's main loops are 1 to 2 % slower on large planes (Q6_K 17408 x 5003, 3 tokens 25.5 -> 25.8,
        // Q4_K 17408 x 5120 19.9 -> 20.3), and small ones gain as much (Q5_K 1280 x 2778, 2 tokens 4.48 -> 4.38).
        auto with_bias = [&](float v, uint32_t n) {
            if constexpr (F == kQ80 || HL) return a.bias ? v + a.bias[n] : v;
            return v;
        };
        for (uint32_t i = tid; i < rows * a.batch; i += kThreads) {
            const uint32_t tok = i / rows, r = i - tok * rows, tl = r / kRows;
            const uint32_t w_lo = (tl * ku * kWarps + kWarps - 1u) / total, w_hi = ((tl * ku + ku - 1u) * kWarps + kWarps - 1u) / total;
            const float* p = red + (size_t)r * NCOLS + tok;
            float v = p[w_lo * kRows * NCOLS];
            for (uint32_t w = w_lo + 1u; w <= w_hi; ++w)
                if (w * total / kWarps != (w + 1u) * total / kWarps) v += p[w * kRows * NCOLS];    // a warp without a unit left nothing
            if (split > 1u) {
                const uint32_t owner = r / rpo;
                st_cluster(cluster_addr(part, owner) + ((rank * a.batch + tok) * rpo + (r - owner * rpo)) * 4u, v);
            } else if (r0 * kRows + r < a.out_dim) {
                a.y[(size_t)tok * a.out_dim + r0 * kRows + r] = with_bias(v, r0 * kRows + r);
            }
        }
        if (split > 1u) {
            // the next round's TMA boxes land where these stores went
            asm volatile("fence.proxy.async;" ::: "memory");
            __syncwarp();
            cluster_sync();
            const float* got = reinterpret_cast<const float*>(smem);
            const uint32_t own = min(rows - min(rows, rank * rpo), rpo);
            for (uint32_t i = tid; i < own * a.batch; i += kThreads) {
                const uint32_t tok = i / own, r = i - tok * own, n = r0 * kRows + rank * rpo + r;
                float v = 0.0f;
                for (uint32_t s = 0; s < split; ++s) v += got[(s * a.batch + tok) * rpo + r];
                if (n < a.out_dim) a.y[(size_t)tok * a.out_dim + n] = with_bias(v, n);
            }
        }
        if (r0 + a.round_tiles < t_hi) {
            asm volatile("fence.proxy.async;" ::: "memory");   // generic accesses above, TMA boxes next
            __syncthreads();
        }
    }
}

// Clusters of s CTAs that are resident at once: one CTA per SM.
template <int F, uint32_t NT, bool HL>
int cluster_caps(const uint32_t** cap) {
    static PdkClusterCaps table;
    return pdk_cluster_caps(table, (const void*)kq_batch_kernel<F, NT, HL>, kWarps * 32u, kSmemMax, cap);
}

template <int F, uint32_t NT, bool HL>
int launch(const void* data, const void* recs, const float* bias, const float* x, const int8_t* xq, const float* xq_scale, float* y,
           uint32_t in_dim, uint32_t out_dim, uint32_t batch, cudaStream_t st) {
    constexpr uint32_t kThreads = kWarps * 32u;
    auto kern = kq_batch_kernel<F, NT, HL>;
    const uint32_t* cap = nullptr;
    if (int rc = cluster_caps<F, NT, HL>(&cap)) return rc;
    Plan p;
    if (!make_plan<F, NT>(p, cap, in_dim, out_dim, batch)) return -1;
    using T = Fmts<F>;
    const uint64_t pitch = (uint64_t)(in_dim >> 8) * T::kUnit;
    CUtensorMap t0, t1;
    if (int rc = pdk_make_tmap_2d(&t0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, data, pitch, out_dim, pitch, 128u, kRows)) return rc;
    t1 = t0;
    if constexpr (F == kQ5K) {
        if (int rc = pdk_make_tmap_2d_dense(&t1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, data, pitch, out_dim, pitch, 32u, kRows)) return rc;
    } else if constexpr (F == kQ6K) {
        if (int rc = pdk_make_tmap_2d_sw64(&t1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, data, pitch, out_dim, pitch, 64u, kRows)) return rc;
    }
    const Args a{(const uint8_t*)recs, x, xq, xq_scale, bias, y, in_dim, out_dim, batch, p.stages, p.ku, p.round_tiles, pdk_error_word()};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.split, p.clusters);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdk_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, t0, t1, a);
    return e == cudaSuccess ? pdk_launch_status() : (int)e;
}

template <int F>
int launch_f(const void* data, const void* recs, const float* x, const int8_t* xq, const float* xs, float* y, uint32_t in_dim,
             uint32_t out_dim, uint32_t batch, cudaStream_t st, const float* bias = nullptr) {
    if (batch <= 4u) return launch<F, 1, true>(data, recs, bias, x, xq, xs, y, in_dim, out_dim, batch, st);
    return batch <= 8u ? launch<F, 1, false>(data, recs, bias, x, xq, xs, y, in_dim, out_dim, batch, st)
                       : launch<F, 2, false>(data, recs, bias, x, xq, xs, y, in_dim, out_dim, batch, st);
}

}  // namespace

// y f32 [batch][out_dim] for 1 <= batch <= 16 tokens through a repacked plane of `dtype` (ggml type id).  Activations are f32
// x [batch][in_dim], or (x == nullptr) int8 xq with one f32 scale per 32 elements.  Returns 0 / a cudaError_t, or -1
// when the shape is outside the plan (K not a multiple of 256, or so long that the activations of one eighth of it do not fit).
int pdk_kq_batch(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xq_scale, float* y,
                 uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype, cudaStream_t st) {
    if (batch == 0u || batch > 16u || in_dim == 0u || (in_dim & 255u) != 0u || out_dim > 0x40000000u) return -1;
    switch (dtype) {
        case 12u: return launch_f<kQ4K>(data, scales, x, xq, xq_scale, y, in_dim, out_dim, batch, st);
        case 2u: return launch_f<kQ40>(data, scales, x, xq, xq_scale, y, in_dim, out_dim, batch, st);
        case 13u: return launch_f<kQ5K>(data, scales, x, xq, xq_scale, y, in_dim, out_dim, batch, st);
        case 14u: return launch_f<kQ6K>(data, scales, x, xq, xq_scale, y, in_dim, out_dim, batch, st);
        default: return -1;
    }
}

// The estimate of the plan for 9 .. 16 tokens of a Q4_K or Q4_0 plane (kq_plan.cuh: super-blocks of a warp); 0 = none.  Without a device, a B200's.
float pdk_kq_batch_cost(uint32_t in_dim, uint32_t out_dim, uint32_t batch) {
    static const uint32_t b200[kMaxSplit + 1u] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    const uint32_t* cap = nullptr;
    if (cluster_caps<kQ4K, 2, false>(&cap) != 0) {
        (void)cudaGetLastError();
        cap = b200;
    }
    Plan p;
    if (batch <= 8u || batch > 16u || out_dim > 0x40000000u) return 0.0f;
    return make_plan<kQ4K, 2>(p, cap, in_dim, out_dim, batch) ? p.cost : 0.0f;
}

// The same for repacked Q8_0 planes (data int8 [out_dim][in_dim], scale f16 [out_dim][in_dim / 32], bias [out_dim] or null).
int pdk_kq_batch_q8(const void* data, const void* scale, const float* bias, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                    uint32_t batch, cudaStream_t st) {
    if (batch == 0u || batch > 16u || in_dim == 0u || (in_dim & 255u) != 0u || out_dim > 0x40000000u || !pdk_aligned(scale, 8)) return -1;
    return launch_f<kQ80>(data, scale, x, nullptr, nullptr, y, in_dim, out_dim, batch, st, bias);
}
