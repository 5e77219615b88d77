// kquant.cu - Q4_K: dequant, repack and the decode GEMV / small-batch GEMM over
// the repacked planes.
//
// Repacked layout (the byte budget the engine allocates: 128 B + 24 B per
// 256-weight super-block; every super-block is self-contained because the
// repack call is only told a super-block count):
//   data   : the 128 nibble bytes verbatim: group G (32 bytes) byte l holds
//            element G*64 + l (low nibble) and element G*64 + 32 + l (high nibble);
//   scales : 24-byte record {f16 d, f16 dmin, u8 sc[8], u8 m[8], 4 pad bytes}
//            with the 6-bit (scale, min) pairs unpacked to bytes.
// Dequant value of element l of sub-block j: (d*sc_j)*q - (dmin*m_j).
//
// One token runs the integer tensor-core GEMVs (gemv_ring.cu, gemv_i8.cu), 2..64 tokens the kernel that batch_route picks; the
// plain kernel below serves what is outside all their plans.
#include <cmath>
#include <cstdlib>

#include "pdk_common.cuh"
#include "q4k_runs.cuh"

// kquant_more.cu: Q5_K, Q6_K, Q4_0
bool pdk_kq_more_has(uint32_t dtype);
int pdk_kq_more_dequant(const void* src, void* dst, uint64_t n_super, uint32_t dtype, cudaStream_t st);
int pdk_kq_more_repack(const void* src, void* dst_data, void* dst_scales, uint64_t n_super, uint32_t dtype,
                       cudaStream_t st);
int pdk_kq_more_gemm(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                     uint32_t batch, uint32_t dtype, cudaStream_t st);
int pdk_q4k_gemv_i8_q8act(const void* data, const void* scales, const int8_t* xq, const float* xq_scale, float* y,
                          uint32_t in_dim, uint32_t out_dim, cudaStream_t st);
int pdk_q4k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                    uint32_t out_dim, cudaStream_t st);
int pdk_q4_0_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                     uint32_t out_dim, cudaStream_t st);
int pdk_q5k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                    uint32_t out_dim, cudaStream_t st);
int pdk_iq4xs_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                      cudaStream_t st);  // gemv_i8.cu
int pdk_q6k_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim,
                    uint32_t out_dim, cudaStream_t st);  // gemv_ring.cu
// kq_batch.cu: 1..16 tokens of every format here, f32 or int8 activations; -1 = shape outside its plan
int pdk_kq_batch(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xq_scale, float* y,
                 uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype, cudaStream_t st);
float pdk_kq_batch_cost(uint32_t in_dim, uint32_t out_dim, uint32_t batch);   // of its plan for 9..16 tokens; 0 = none
// q4k_batch_i8.cu: 1..8 tokens, same operands and return convention
int pdk_q4k_batch_i8(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xq_scale,
                     float* y, uint32_t in_dim, uint32_t out_dim, uint32_t batch, cudaStream_t st);
int pdk_q5k_batch_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                     uint32_t batch, cudaStream_t st);
// q4k_tc5.cu: 1..32 tokens on tcgen05 (f16 weights); same operands and return convention
int pdk_q4k_tc5(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xq_scale, float* y,
                uint32_t in_dim, uint32_t out_dim, uint32_t batch, cudaStream_t st);
int pdk_q4_0_tc5(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                 uint32_t batch, cudaStream_t st);

namespace {

// ggml get_scale_min_k4: unpack 6-bit pair j of the 12 packed scale bytes.
__device__ __forceinline__ void scale_min_k4(const uint8_t* s, uint32_t j, uint32_t* sc, uint32_t* m) {
    if (j < 4u) {
        *sc = s[j] & 63u;
        *m = s[j + 4u] & 63u;
    } else {
        *sc = (s[j + 4u] & 0xFu) | ((uint32_t)(s[j - 4u] >> 6) << 4);
        *m = (uint32_t)(s[j + 4u] >> 4) | ((uint32_t)(s[j] >> 6) << 4);
    }
}

// One warp per super-block; lane l writes element l of each of the 8
// sub-blocks, so every store instruction covers one 128-byte line.
__global__ void q4k_dequant_kernel(const uint8_t* __restrict__ src, float* __restrict__ dst, uint64_t n_super) {
    const uint64_t b = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= n_super) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint8_t* s = src + b * 144u;
    const float d = __half2float(*reinterpret_cast<const __half*>(s));
    const float dmin = __half2float(*reinterpret_cast<const __half*>(s + 2));
    float* y = dst + b * 256u;
#pragma unroll
    for (uint32_t j = 0; j < 8u; ++j) {
        uint32_t sc, m;
        scale_min_k4(s + 4, j, &sc, &m);
        const float dj = __fmul_rn(d, (float)sc), mj = __fmul_rn(dmin, (float)m);
        const uint32_t q = s[16u + (j >> 1) * 32u + lane];
        const uint32_t v = (j & 1u) ? (q >> 4) : (q & 0xFu);
        y[j * 32u + lane] = __fsub_rn(__fmul_rn(dj, (float)v), mj);
    }
}

// Repack of 16-byte aligned planes.  A raw super-block is nine 16-byte vectors - header, then the nibble payload as the plane
// stores it.  The payload goes through as it is, eight lanes per super-block, so that a warp's store is four whole
// 128-byte lines; one thread per super-block unpacks the header into the record.  Every load of a thread is in flight before
// its first store.  HBM bound; 5120 x 25600: 60.5 us with the word-per-lane kernel below (a warp per super-block, one 4-byte load in
// flight per thread), 24.8 us now (151.6 MB, 0.94 of the HBM copy rate; 26.6 with nine
// consecutive lanes per super-block, whose stores begin and end inside lines).  Plain loads: with ld.global.nc.L1::no_allocate here the
// repack takes as long, but the decode GEMV reads a plane of the same bytes slower ever after (18.10 against 17.92 us; Q8_0, the same
// in elementwise.cu, 16.67 against 15.95), until something rewrites it - measured, the mechanism is not known.
constexpr uint32_t kRepackDepth = 4, kRepackThreads = 256, kRepackSupers = kRepackThreads * kRepackDepth / 8u;
__global__ void __launch_bounds__(kRepackThreads)
q4k_repack16_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst_data, uint2* __restrict__ dst_scales, uint64_t n_super) {
    const uint64_t s0 = (uint64_t)blockIdx.x * kRepackSupers;
    uint4 v[kRepackDepth], head;
#pragma unroll
    for (uint32_t i = 0; i < kRepackDepth; ++i) {
        const uint32_t at = i * kRepackThreads + threadIdx.x;
        if (s0 + (at >> 3) < n_super) v[i] = src[(s0 + (at >> 3)) * 9u + 1u + (at & 7u)];
    }
    const uint64_t b = s0 + threadIdx.x;
    const bool mine = threadIdx.x < kRepackSupers && b < n_super;
    if (mine) head = src[b * 9u];
#pragma unroll
    for (uint32_t i = 0; i < kRepackDepth; ++i) {
        const uint32_t at = i * kRepackThreads + threadIdx.x;
        if (s0 + (at >> 3) < n_super) dst_data[s0 * 8u + at] = v[i];
    }
    if (!mine) return;
    // scale bytes 0..3 | 4..7 | 8..11 = y | z | w: pairs 0..3 are the low six bits of the first two words,
    // pairs 4..7 the nibbles of the third under the top two bits of those words
    const uint32_t sc_lo = head.y & 0x3f3f3f3fu, m_lo = head.z & 0x3f3f3f3fu;
    const uint32_t sc_hi = (head.w & 0x0f0f0f0fu) | ((head.y >> 2) & 0x30303030u);
    const uint32_t m_hi = ((head.w >> 4) & 0x0f0f0f0fu) | ((head.z >> 2) & 0x30303030u);
    uint2* rec = dst_scales + b * 3u;
    rec[0] = make_uint2(head.x, sc_lo);
    rec[1] = make_uint2(sc_hi, m_lo);
    rec[2] = make_uint2(m_hi, 0u);
}

// Any alignment the slot takes: one warp per super-block, lane l moves one 4-byte word of the nibble payload
// (the source payload at 144*b + 16 is 4-byte aligned when the plane is);
// lanes 0..7 unpack one (sc, m) pair each into the record.
__global__ void q4k_repack_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst_data,
                                  uint8_t* __restrict__ dst_scales, uint64_t n_super) {
    const uint64_t b = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= n_super) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint8_t* s = src + b * 144u;
    reinterpret_cast<uint32_t*>(dst_data + b * 128u)[lane] = reinterpret_cast<const uint32_t*>(s + 16)[lane];
    uint8_t* rec = dst_scales + b * 24u;
    if (lane < 8u) {
        uint32_t sc, m;
        scale_min_k4(s + 4, lane, &sc, &m);
        rec[4u + lane] = (uint8_t)sc;
        rec[12u + lane] = (uint8_t)m;
    } else if (lane < 12u) {
        rec[lane - 8u] = s[lane - 8u];  // f16 d, f16 dmin
    } else if (lane < 16u) {
        rec[8u + lane] = 0;             // pad bytes 20..23
    }
}

// ===========================================================================
// Plain-load f32 kernel, one token: the route for shapes outside the tensor-core kernels' plans.  A warp owns
// one output row at a time; lane l reads word l of each super-block (a coalesced 128-byte line).
// ===========================================================================
constexpr uint32_t kWarps = 8;

constexpr uint32_t UNROLL = 10;

__global__ void __launch_bounds__(kWarps * 32)
q4k_gemv_kernel(const uint8_t* __restrict__ data, const uint8_t* __restrict__ scales,
                const float* __restrict__ x, float* __restrict__ y, uint32_t in_dim, uint32_t out_dim) {
    extern __shared__ __align__(16) float xsf[];  // [in_dim]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid * 4u; i < in_dim; i += blockDim.x * 4u)
        *reinterpret_cast<float4*>(xsf + i) = *reinterpret_cast<const float4*>(x + i);
    __syncthreads();

    const uint32_t n_super = in_dim >> 8;
    // word `lane` of the payload = ggml group G, word w of that group
    const uint32_t G = lane >> 3, w = lane & 7u;
    const uint32_t koff = G * 64u + w * 4u;  // first low-nibble element inside the super-block
    for (uint32_t row = blockIdx.x * kWarps + warp; row < out_dim; row += gridDim.x * kWarps) {
        const uint8_t* drow = data + (size_t)row * n_super * 128u;
        const uint8_t* srow = scales + (size_t)row * n_super * 24u;
        float acc = 0.0f;
        for (uint32_t sb0 = 0; sb0 < n_super; sb0 += UNROLL) {
            uint32_t q[UNROLL];
            uint32_t dd[UNROLL];
            uint32_t scm[UNROLL];
#pragma unroll
            for (uint32_t u = 0; u < UNROLL; ++u) {
                const uint32_t sb = sb0 + u;
                if (sb < n_super) {
                    q[u] = pdk_ldg_stream4(drow + sb * 128u + lane * 4u);
                    const uint8_t* rec = srow + sb * 24u;
                    dd[u] = *reinterpret_cast<const uint32_t*>(rec);
                    const uint32_t s2 = *reinterpret_cast<const uint16_t*>(rec + 4u + 2u * G);
                    const uint32_t m2 = *reinterpret_cast<const uint16_t*>(rec + 12u + 2u * G);
                    scm[u] = s2 | (m2 << 16);
                } else {
                    q[u] = 0u; dd[u] = 0u; scm[u] = 0u;
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < UNROLL; ++u) {
                const uint32_t sb = sb0 + u;
                if (sb >= n_super) break;
                const __half2 dh = *reinterpret_cast<const __half2*>(&dd[u]);
                const float d = __low2float(dh), dmin = __high2float(dh);
                const float d_lo = d * (float)(scm[u] & 0xffu), d_hi = d * (float)((scm[u] >> 8) & 0xffu);
                const float m_lo = dmin * (float)((scm[u] >> 16) & 0xffu), m_hi = dmin * (float)(scm[u] >> 24);
                const uint32_t k = sb * 256u + koff;
                const float4 xl = *reinterpret_cast<const float4*>(xsf + k);
                const float4 xh = *reinterpret_cast<const float4*>(xsf + k + 32u);
                float sl = (float)(q[u] & 0xFu) * xl.x;
                sl = fmaf((float)((q[u] >> 8) & 0xFu), xl.y, sl);
                sl = fmaf((float)((q[u] >> 16) & 0xFu), xl.z, sl);
                sl = fmaf((float)((q[u] >> 24) & 0xFu), xl.w, sl);
                float sh = (float)((q[u] >> 4) & 0xFu) * xh.x;
                sh = fmaf((float)((q[u] >> 12) & 0xFu), xh.y, sh);
                sh = fmaf((float)((q[u] >> 20) & 0xFu), xh.z, sh);
                sh = fmaf((float)(q[u] >> 28), xh.w, sh);
                const float xsl = (xl.x + xl.y) + (xl.z + xl.w);
                const float xsh = (xh.x + xh.y) + (xh.z + xh.w);
                acc += (d_lo * sl - m_lo * xsl) + (d_hi * sh - m_hi * xsh);
            }
        }
        const float v = pdk_warp_sum(acc);
        if (lane == 0) y[row] = v;
    }
}

int launch_plain(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim, cudaStream_t st) {
    const size_t smem = (size_t)in_dim * sizeof(float);
    auto kern = q4k_gemv_kernel;
    if (smem > 48u * 1024u) {
        if (smem > 200u * 1024u) return cudaErrorNotSupported;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)(kWarps * 32u), smem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    uint32_t grid = (uint32_t)pdk_sm_count() * (uint32_t)per_sm;
    const uint32_t need = (out_dim + kWarps - 1u) / kWarps;
    if (grid > need) grid = need;
    kern<<<grid, kWarps * 32u, smem, st>>>((const uint8_t*)data, (const uint8_t*)scales, x, y, in_dim, out_dim);
    return pdk_launch_status();
}

// PDK_Q4K_PLAIN=1 forces the plain-load kernel (A/B switch, read once).
bool force_plain() {
    static const bool v = [] {
        const char* e = getenv("PDK_Q4K_PLAIN");
        return e && e[0] == '1';
    }();
    return v;
}

enum Route : int { kRouteKq = 1, kRouteI8 = 2, kRouteTc5 = 3 };

// From how many tokens on the tcgen05 kernel takes a Q4_K call: 9, where kq_beats_tc5 agrees.  PDK_Q4K_TC5_MIN (read once) sets it by hand, and
// then no estimate has a say (Q4_0: from 9 tokens); 0 = never.
struct Tc5Min {
    uint32_t tokens;
    bool by_hand;
};
const Tc5Min& tc5_min() {
    static const Tc5Min v = [] {
        const char* e = getenv("PDK_Q4K_TC5_MIN");
        return e ? Tc5Min{(uint32_t)atoi(e), true} : Tc5Min{9u, false};
    }();
    return v;
}

// Where kq_batch.cu (clusters over K, any width) beats the integer kernel of q4k_batch_i8.cu (Q4_K, Q5_K up to 8 tokens), whose
// time hardly falls below that of one round of 64-row CTAs while kq_batch splits K until the chip is full and grows with tokens
// and plane.  Measured over 480 random shapes of both formats (K = 1024 ... 17408, N = 512 ... 27648; the rule is 1.1 % off the
// faster one on average), us kq_batch / integer:
//   K > 9216: the integer kernel's activation image leaves no L1: K = 11008, N = 2304, 2 tokens 10.2 / 41.5, N = 6208, 8 tokens 22.3 / 42.4;
//   below, N (tokens + 8) against 680 sqrt(K): K = 8192, N = 3000, 8 tokens 11.8 / 14.3; K = 4096, N = 4096: 7.0 / 8.1 at 3, 9.6 / 8.1 at 8;
//   K = 5120, N = 25600: 26.2 / 21.2 at 2, 32.1 / 22.2 at 8;
//   narrow planes at short K, where both take a few us: kq_batch is one launch and keeps 22 activation bits where the
//   integer kernel keeps 15.  K = 1024, N = 4096, 4 tokens: 4.6 / 5.5 launched one by one, 4.3 / 3.6 in a replayed graph.
bool kq_beats_i8(uint32_t in_dim, uint32_t out_dim, uint32_t batch) {
    if (in_dim > 9216u || (float)out_dim * (float)(batch + 8u) <= 680.0f * sqrtf((float)in_dim)) return true;
    const uint64_t limit = batch <= 2u ? 30000000u : batch <= 4u ? 20000000u : 10000000u;
    return (uint64_t)out_dim * (in_dim + 2048u) <= limit;
}

// 9 and more tokens of Q4_K or Q4_0, the first 32 of them: both kernels' times in us, fitted to 434 timings (K = 1024 ... 16384, N = 512 ... 27648,
// 9 ... 32 tokens; the choice is 0.3 % off the faster one on average).  tcgen05 takes up to 32 tokens for one price, the run of its busiest CTA
// (q4k_runs.cuh).  kq_batch pays for weights x tokens, 16 tokens a pass, but fills the chip whatever N is and has exact weights; where
// K is so long that the activations leave room for the partial sums of a tile or two, its plan takes many rounds and is the price instead.
// Measured (us, kq_batch / tcgen05): Q4_K 9728 x 1100, 9 tokens 10.9 / 19.3, 16 tokens 12.5 / 19.6; 9728 x 3000, 9 tokens 17.3 / 19.4; 12800 x 5000, 12 tokens
// 30.3 / 24.2; 5120 x 2560, 16 tokens 12.4 / 12.2; 9728 x 520, 32 tokens 20.1 / 19.6; Q4_0 14848 x 2112, 16 tokens 55.1 / 26.9 (nine rounds).
bool kq_beats_tc5(uint32_t in_dim, uint32_t out_dim, uint32_t batch) {
    const uint32_t left = batch < 32u ? batch : 32u, passes = (left + 15u) / 16u, take = (left + passes - 1u) / passes;
    const float tc5 = q4k_runs::launch_us(in_dim, out_dim, left, (uint32_t)pdk_sm_count());
    const float kq = 5.0f + (float)in_dim / 3000.0f + 0.1f * ((float)take - 9.0f) +
                     (float)out_dim * (float)in_dim * (2.25e-7f + 1.0e-8f * (float)take);
    if ((float)passes * kq >= tc5) return false;
    const float cost = pdk_kq_batch_cost(in_dim, out_dim, take);
    return cost != 0.0f && (float)passes * 1.2f * cost < tc5;
}

// The kernel that a pass over `batch` tokens asks first.  Q4_0 up to 8 tokens: kq_batch against the tcgen05 kernel (which costs the same
// at 4 and at 16 tokens) is 0.4 % off the faster one over 180 random shapes, up to 5 times faster, at most 18 % slower (K = 5120,
// N = 25600: 26.4 / 29.2 us at 4 tokens; N = 9472: 16.2 / 15.2 at 8).  Q5_K from 9 tokens on: two passes of the integer kernel would
// be faster on wide planes (K = 5120, N = 25600, 16 tokens: 51.6 against 64.5 us), but kq_batch keeps 22 activation bits.
Route batch_route(uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype) {
    const Tc5Min& min = tc5_min();
    const uint32_t from = dtype == PDK_KQ_Q4K ? min.tokens : dtype == PDK_KQ_Q4_0 && min.tokens != 0u ? 9u : 0u;
    if (from != 0u && batch >= from) return !min.by_hand && kq_beats_tc5(in_dim, out_dim, batch) ? kRouteKq : kRouteTc5;
    if ((dtype == PDK_KQ_Q4K || dtype == PDK_KQ_Q5K) && batch <= 8u && !kq_beats_i8(in_dim, out_dim, batch)) return kRouteI8;
    return kRouteKq;
}

// Up to 16 tokens of `batch` through kq_batch.cu, in passes of one width (17 tokens are 9 + 8: the weights are read once per
// pass whatever its width), or fewer where K is so long that their activations do not fit.  The tokens done, or -(cudaError_t) - 1.
int kq_pass(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xs, float* y, uint32_t in_dim,
            uint32_t out_dim, uint32_t batch, uint32_t dtype, cudaStream_t st) {
    const uint32_t passes = (batch + 15u) / 16u;
    for (uint32_t take = (batch + passes - 1u) / passes; take != 0u; take = take > 8u ? 8u : take / 2u) {
        const int rc = pdk_kq_batch(data, scales, x, xq, xs, y, in_dim, out_dim, take, dtype, st);
        if (rc == 0) return (int)take;
        if (rc != -1) return -rc - 1;
    }
    return 0;
}

// 2 <= tokens of a Q4_K, Q4_0, Q5_K or Q6_K plane on the tensor paths: up to 32 tokens per launch on tcgen05, up to 8 on the
// integer kernel, and whatever is not theirs or outside their plans up to 16 on kq_batch.cu.  Activations f32 (x) or, for Q4_K, int8 with
// per-32 scales (xq, xs).  Returns the number of tokens done (all of them unless a shape is outside every plan), or
// -(cudaError_t) - 1 on a launch error.
int small_batch(const void* data, const void* scales, const float* x, const int8_t* xq, const float* xs, float* y,
                uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype, cudaStream_t st) {
    uint32_t b = 0;
    while (b < batch) {
        const uint32_t left = batch - b;
        const float* xb = x ? x + (size_t)b * in_dim : nullptr;
        const int8_t* qb = xq ? xq + (size_t)b * in_dim : nullptr;
        const float* sb = xs ? xs + (size_t)b * (in_dim >> 5) : nullptr;
        float* yb = y + (size_t)b * out_dim;
        uint32_t take = left < 32u ? left : 32u;
        int rc = -1;
        switch (batch_route(in_dim, out_dim, left, dtype)) {
            case kRouteTc5:
                rc = dtype == PDK_KQ_Q4K ? pdk_q4k_tc5(data, scales, xb, qb, sb, yb, in_dim, out_dim, take, st)
                                         : pdk_q4_0_tc5(data, scales, xb, yb, in_dim, out_dim, take, st);
                break;
            case kRouteI8:
                rc = dtype == PDK_KQ_Q4K ? pdk_q4k_batch_i8(data, scales, xb, qb, sb, yb, in_dim, out_dim, take, st)
                                         : pdk_q5k_batch_i8(data, scales, xb, yb, in_dim, out_dim, take, st);
                break;
            default: break;
        }
        if (rc == -1) {
            const int done = kq_pass(data, scales, xb, qb, sb, yb, in_dim, out_dim, left, dtype, st);
            if (done < 0) return done;
            if (done == 0) break;
            take = (uint32_t)done;
            rc = 0;
        }
        if (rc != 0) return -rc - 1;
        b += take;
    }
    return (int)b;
}

int gemm_any(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
             uint32_t batch, cudaStream_t st) {
    uint32_t done = 0;
    if (!force_plain()) {
        if (batch == 1u) {
            const int rc = pdk_q4k_gemv_i8(data, scales, x, y, in_dim, out_dim, st);
            if (rc != -1) return rc;
        }
        const int n = small_batch(data, scales, x, nullptr, nullptr, y, in_dim, out_dim, batch, PDK_KQ_Q4K, st);
        if (n < 0) return -n - 1;
        done = (uint32_t)n;
    }
    for (; done < batch; ++done)      // outside every plan
        if (int rc = launch_plain(data, scales, x + (size_t)done * in_dim, y + (size_t)done * out_dim, in_dim, out_dim, st)) return rc;
    return 0;
}

// Q4_0 / Q5_K / Q6_K decode GEMV on the integer tensor path; -1 = shape outside the kernels' plan
int more_gemv_i8(const void* data, const void* scales, const float* x, float* y, uint32_t in_dim, uint32_t out_dim,
                 uint32_t dtype, cudaStream_t st) {
    if (dtype == PDK_KQ_Q4_0) return pdk_q4_0_gemv_i8(data, scales, x, y, in_dim, out_dim, st);
    if (dtype == PDK_KQ_Q5K) return pdk_q5k_gemv_i8(data, scales, x, y, in_dim, out_dim, st);
    if (dtype == PDK_KQ_Q6K) return pdk_q6k_gemv_i8(data, scales, x, y, in_dim, out_dim, st);
    if (dtype == PDK_KQ_IQ4XS) return pdk_iq4xs_gemv_i8(data, scales, x, y, in_dim, out_dim, st);
    return -1;
}

int check_gemv(const void* data, const void* scales, const void* x, const void* y, uint32_t in_dim, uint32_t dtype) {
    if (dtype != PDK_KQ_Q4K && !pdk_kq_more_has(dtype))
        return cudaErrorInvalidValue;
    if (in_dim == 0u || (in_dim & 255u) != 0u) return cudaErrorInvalidValue;
    if (!pdk_aligned(data, 16) || !pdk_aligned(scales, 8) || !pdk_aligned(x, 16) || !pdk_aligned(y, 4))
        return cudaErrorInvalidValue;
    return 0;
}

}  // namespace

PDK_EXPORT int pd_kquant_dequant(const void* src, void* dst, uint64_t n_super, uint32_t dtype, void* stream) {
    if (n_super == 0) return 0;
    if (pdk_kq_more_has(dtype)) return pdk_kq_more_dequant(src, dst, n_super, dtype, (cudaStream_t)stream);
    if (dtype != PDK_KQ_Q4K) return cudaErrorInvalidValue;
    if (!pdk_aligned(src, 2) || !pdk_aligned(dst, 4)) return cudaErrorInvalidValue;
    const uint64_t blocks = (n_super + 7u) / 8u;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    q4k_dequant_kernel<<<(uint32_t)blocks, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)src, (float*)dst, n_super);
    return pdk_launch_status();
}

PDK_EXPORT int pd_kquant_repack(const void* src, void* dst_data, void* dst_scales, uint64_t n_super, uint32_t dtype,
                                void* stream) {
    if (n_super == 0) return 0;
    if (pdk_kq_more_has(dtype))
        return pdk_kq_more_repack(src, dst_data, dst_scales, n_super, dtype, (cudaStream_t)stream);
    if (dtype != PDK_KQ_Q4K) return cudaErrorInvalidValue;
    if (!pdk_aligned(src, 4) || !pdk_aligned(dst_data, 4)) return cudaErrorInvalidValue;
    const uint64_t blocks = (n_super + 7u) / 8u;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    if (pdk_aligned(src, 16) && pdk_aligned(dst_data, 16) && pdk_aligned(dst_scales, 8)) {
        const uint64_t ctas = (n_super + kRepackSupers - 1u) / kRepackSupers;
        q4k_repack16_kernel<<<(uint32_t)ctas, kRepackThreads, 0, (cudaStream_t)stream>>>((const uint4*)src, (uint4*)dst_data,
                                                                                      (uint2*)dst_scales, n_super);
        return pdk_launch_status();
    }
    q4k_repack_kernel<<<(uint32_t)blocks, 256, 0, (cudaStream_t)stream>>>(
        (const uint8_t*)src, (uint8_t*)dst_data, (uint8_t*)dst_scales, n_super);
    return pdk_launch_status();
}

PDK_EXPORT int pd_kquant_gemv(const void* data, const void* scales, const void* x, void* y, uint32_t in_dim,
                              uint32_t out_dim, uint32_t dtype, void* stream) {
    if (out_dim == 0) return 0;
    if (int rc = check_gemv(data, scales, x, y, in_dim, dtype)) return rc;
    if (dtype != PDK_KQ_Q4K && !force_plain() && pdk_aligned(data, 16)) {
        const int rc = more_gemv_i8(data, scales, (const float*)x, (float*)y, in_dim, out_dim, dtype, (cudaStream_t)stream);
        if (rc != -1) return rc;
    }
    if (dtype != PDK_KQ_Q4K)
        return pdk_kq_more_gemm(data, scales, (const float*)x, (float*)y, in_dim, out_dim, 1u, dtype, (cudaStream_t)stream);
    return gemm_any(data, scales, (const float*)x, (float*)y, in_dim, out_dim, 1u, (cudaStream_t)stream);
}

PDK_EXPORT int pdk_kquant_gemm_route(uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype) {
    const bool known = dtype == PDK_KQ_Q4K || dtype == PDK_KQ_Q4_0 || dtype == PDK_KQ_Q5K || dtype == PDK_KQ_Q6K;
    return known && batch >= 2u && batch <= 64u ? (int)batch_route(in_dim, out_dim, batch, dtype) : 0;
}

PDK_EXPORT int pdk_kquant_gemm_f32(const void* data, const void* scales, const void* x, void* y, uint32_t in_dim,
                                   uint32_t out_dim, uint32_t batch, uint32_t dtype, void* stream) {
    if (out_dim == 0 || batch == 0) return 0;
    if (batch > 64u) return cudaErrorInvalidValue;
    if (int rc = check_gemv(data, scales, x, y, in_dim, dtype)) return rc;
    if ((dtype == PDK_KQ_Q4_0 || dtype == PDK_KQ_Q5K || dtype == PDK_KQ_Q6K) && batch >= 2u && !force_plain()) {
        const int done = small_batch(data, scales, (const float*)x, nullptr, nullptr, (float*)y, in_dim, out_dim, batch, dtype, (cudaStream_t)stream);
        if (done < 0) return -done - 1;
        if ((uint32_t)done == batch) return 0;
        x = (const float*)x + (size_t)done * in_dim;   // outside every plan: the routes below take what is left
        y = (float*)y + (size_t)done * out_dim;
        batch -= (uint32_t)done;
    }
    if (dtype != PDK_KQ_Q4K && !force_plain() && pdk_aligned(data, 16)) {
        // one token, and IQ4_XS, which has no batch kernel: one decode GEMV per token (17-29 us each at K=5120
        // N=25600, the later ones partly from L2) beats the plain f32 kernel's 165 us per four tokens
        int rc = 0;
        for (uint32_t b = 0; b < batch && rc == 0; ++b)
            rc = more_gemv_i8(data, scales, (const float*)x + (size_t)b * in_dim, (float*)y + (size_t)b * out_dim, in_dim,
                              out_dim, dtype, (cudaStream_t)stream);
        if (rc != -1) return rc;  // -1 comes from the first call (the plan depends on the shape alone): nothing is done yet
    }
    if (dtype != PDK_KQ_Q4K)
        return pdk_kq_more_gemm(data, scales, (const float*)x, (float*)y, in_dim, out_dim, batch, dtype,
                                (cudaStream_t)stream);
    return gemm_any(data, scales, (const float*)x, (float*)y, in_dim, out_dim, batch, (cudaStream_t)stream);
}

// ---------------------------------------------------------------- int8 activation operands (W4A8 slots)
namespace {

// One warp per 32-element block: scale = amax / 127, q = RN(x / scale) clamped to +-127;
// optionally the two per-16 sums of q as f32 (packs/cuda/src/attn/decode.cuh:2981-3004, 3041-3068).
__global__ void quantize_q8_kernel(const float* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale,
                                   float* __restrict__ sums, uint32_t n_blocks) {
    const uint32_t b = blockIdx.x * 8u + (threadIdx.x >> 5), d = threadIdx.x & 31u;
    if (b >= n_blocks) return;
    const float v = x[(size_t)b * 32u + d];
    float a = fabsf(v);
#pragma unroll
    for (uint32_t s = 16; s > 0; s >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, s));
    const float scl = a * (1.0f / 127.0f);
    if (d == 0) scale[b] = scl;
    const float inv = scl > 0.0f ? 1.0f / scl : 0.0f;
    int qi = __float2int_rn(v * inv);
    qi = qi < -127 ? -127 : (qi > 127 ? 127 : qi);
    q[(size_t)b * 32u + d] = (int8_t)qi;
    if (sums != nullptr) {
        int s16 = qi;
#pragma unroll
        for (uint32_t s = 8; s > 0; s >>= 1) s16 += __shfl_xor_sync(0xffffffffu, s16, s);
        if ((d & 15u) == 0u) sums[(size_t)b * 2u + (d >> 4)] = (float)s16;
    }
}

// x[i] = q[i] * scale[i / 32]: the f32 activations the batch kernels take
__global__ void q8_act_widen_kernel(const int8_t* __restrict__ q, const float* __restrict__ scale, float* __restrict__ x,
                                    uint64_t n4) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const uint32_t w = reinterpret_cast<const uint32_t*>(q)[i];
    const float s = scale[i >> 3];
    reinterpret_cast<float4*>(x)[i] = make_float4((float)(int8_t)(w & 0xff) * s, (float)(int8_t)((w >> 8) & 0xff) * s,
                                                  (float)(int8_t)((w >> 16) & 0xff) * s, (float)(int8_t)(w >> 24) * s);
}

int w4a8_gemm(const void* data, const void* scales, const void* xq, const void* xs, void* part, void* y,
              uint32_t in_dim, uint32_t out_dim, uint32_t batch, uint32_t dtype, cudaStream_t st) {
    if (out_dim == 0 || batch == 0) return 0;
    if (batch > 64u) return cudaErrorInvalidValue;
    if (int rc = check_gemv(data, scales, xq, y, in_dim, dtype)) return rc;
    if (dtype != PDK_KQ_Q4K) return cudaErrorNotSupported;
    if (batch == 1u) {
        const int rc = pdk_q4k_gemv_i8_q8act(data, scales, (const int8_t*)xq, (const float*)xs, (float*)y, in_dim, out_dim, st);
        if (rc >= 0) return rc;
    }
    if (!force_plain() && pdk_aligned(xq, 8)) {
        const int done = small_batch(data, scales, nullptr, (const int8_t*)xq, (const float*)xs, (float*)y, in_dim,
                                     out_dim, batch, PDK_KQ_Q4K, st);
        if (done < 0) return -done - 1;
        if ((uint32_t)done == batch) return 0;
        // outside every plan: the widening route takes what is left
        xq = (const int8_t*)xq + (size_t)done * in_dim;
        xs = (const float*)xs + (size_t)done * (in_dim >> 5);
        y = (float*)y + (size_t)done * out_dim;
        batch -= (uint32_t)done;
    }
    // the batch kernels take f32 activations: widen q * scale into the caller's partial
    // buffer (>= 8 * out_dim * batch floats by the slot's contract)
    if (part == nullptr || !pdk_aligned(part, 16) || !pdk_aligned(xq, 4) || (uint64_t)in_dim > 8ull * out_dim)
        return cudaErrorInvalidValue;
    const uint64_t n4 = (uint64_t)batch * in_dim / 4u;
    q8_act_widen_kernel<<<(uint32_t)((n4 + 255u) / 256u), 256, 0, st>>>((const int8_t*)xq, (const float*)xs, (float*)part, n4);
    return gemm_any(data, scales, (const float*)part, (float*)y, in_dim, out_dim, batch, st);
}

}  // namespace

// slot 18, packs/cuda/src/gemm/f32_qkv.cuh:283-292
PDK_EXPORT int pd_quantize_q8(const void* x, void* q, void* scale, uint32_t n, void* stream) {
    const uint32_t n_blocks = n >> 5;
    if (n_blocks == 0) return 0;
    quantize_q8_kernel<<<(n_blocks + 7u) / 8u, 256, 0, (cudaStream_t)stream>>>((const float*)x, (int8_t*)q, (float*)scale,
                                                                               nullptr, n_blocks);
    return pdk_launch_status();
}

// slot 218, packs/cuda/src/gemm/f32_qkv.cuh:304-311: also the per-16 sums of q (f32 [n/16])
PDK_EXPORT int pd_quantize_q8_sums(const void* x, void* q, void* scale, void* sums, uint32_t n, void* stream) {
    const uint32_t n_blocks = n >> 5;
    if (n_blocks == 0) return 0;
    if (sums == nullptr) return cudaErrorInvalidValue;
    quantize_q8_kernel<<<(n_blocks + 7u) / 8u, 256, 0, (cudaStream_t)stream>>>((const float*)x, (int8_t*)q, (float*)scale,
                                                                               (float*)sums, n_blocks);
    return pdk_launch_status();
}

// slot 217, packs/cuda/src/quant/kquant_w4a8.cuh:1266-1330: decode GEMV on int8 activations.
// xsums (the min term's per-16 sums) is accepted and not needed: the kernel rebuilds its
// own sums from q * scale.  Shapes outside the GEMV kernel's plan answer "not supported"
// (there is no scratch argument to widen the activations into).
PDK_EXPORT int pd_kquant_gemv_w4a8(const void* data, const void* scales, const void* xq, const void* xs,
                                   const void* xsums, void* y, uint32_t in_dim, uint32_t out_dim, uint32_t dtype,
                                   void* stream) {
    (void)xsums;
    if (out_dim == 0) return 0;
    if (int rc = check_gemv(data, scales, xq, y, in_dim, dtype)) return rc;
    if (dtype != PDK_KQ_Q4K) return cudaErrorNotSupported;
    const int rc = pdk_q4k_gemv_i8_q8act(data, scales, (const int8_t*)xq, (const float*)xs, (float*)y, in_dim, out_dim,
                                         (cudaStream_t)stream);
    return rc >= 0 ? rc : (int)cudaErrorNotSupported;
}

// slot 212, packs/cuda/src/quant/kquant_w4a8.cuh:2364-2430: batch <= 64, y f32 [batch][out_dim];
// `part` (>= 8 * out_dim * batch floats) is used as scratch for the widened activations.
PDK_EXPORT int pd_kquant_gemm_mma_ks(const void* data, const void* scales, const void* xq, const void* xs,
                                     const void* xsums, void* part, void* y, uint32_t in_dim, uint32_t out_dim,
                                     uint32_t batch, uint32_t dtype, void* stream) {
    (void)xsums;
    return w4a8_gemm(data, scales, xq, xs, part, y, in_dim, out_dim, batch, dtype, (cudaStream_t)stream);
}

// slot 837, packs/cuda/src/quant/kquant_w4a8_sb.cuh:300-353: same contract as slot 212
PDK_EXPORT int pd_kquant_gemm_w4a8_sb(const void* data, const void* scales, const void* xq, const void* xs,
                                      const void* xsums, void* part, void* y, uint32_t in_dim, uint32_t out_dim,
                                      uint32_t batch, uint32_t dtype, void* stream) {
    (void)xsums;
    return w4a8_gemm(data, scales, xq, xs, part, y, in_dim, out_dim, batch, dtype, (cudaStream_t)stream);
}
