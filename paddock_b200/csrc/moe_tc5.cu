// moe_tc5.cu - MXFP4 expert GEMMs on the block-scaled tcgen05 path.
//
// An MXFP4 plane needs no weight transformation to run on kind::mxf4nvf4:
//   * the repacked data plane is already 16 packed e2m1 bytes per 32 weights.  The
//     tensor core reads byte j of a block as the element pair (2j, 2j+1) where ggml
//     means (j, j+16); a dot product does not care as long as the activations are
//     packed in the same order, and the whole block shares one scale;
//   * the E8M0 block scale 2^(s-127) becomes two equal UE4M3 per-16 scales
//     2^(s - emax + 8) plus one per-plane factor scale2 = 2^(emax - 135), emax being
//     the largest scale byte of the plane.  Powers of two from 2^-9 to 2^8 are exact in
//     UE4M3, so every block within 17 binades of the plane's largest is exact; smaller
//     ones flush to zero (below 2^-17 of the largest weight block).
// Activations keep more than 4 bits by being expanded into four NVFP4 terms,
//   x * 2^-e = t0 + t1/16 + t2/256 + t3/4096,  t_k = nvfp4(16^k * residual_k),
// which sit side by side in the token dimension of one MMA (32 columns per group of 8
// tokens, moe_grouped.cuh); the epilogue adds the four.  What is
// left of a 16-element group after four terms is below 1e-3 of the group's largest
// element.  No weight passes through a register: at decode widths the kernel is a
// pure stream of 4.25 bits per weight.
//
// Launch order of one MoE block (host side in planes.py):
//   pd_moe_topk_batch, pdk_moe_align_pos (decode widths: pdk_moe_route_few for both)
//   pdk_moe_prep_tokens_f4 (each token's term rows to its pairs' positions)
//   pdk_*_moe_gate_up_tc5 (gate, up and the unit)  or  pdk_*_moe_gemm_tc5_ahead (gate and up, raw)
//   pdk_moe_prep_pairs_f4 (the unit where it is still to do, term rows)
//   pdk_*_moe_gemm_tc5_ahead (down, scattered to (token, slot) rows and multiplied by the routing weight)
//   pd_moe_slot_combine
#include <cuda_fp8.h>

#include "moe_grouped.cuh"
#include "moe_route.cuh"

namespace {

using namespace nvf4tc5;

// ---------------------------------------------------------------- weight scale planes

__global__ void mxfp4_emax_kernel(const uint8_t* __restrict__ scale, uint64_t n, uint32_t* __restrict__ meta) {
    uint32_t m = 0u;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, (uint32_t)scale[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31u) == 0u && m) atomicMax(meta, m);
}

// E8M0 byte relative to the plane's largest -> UE4M3 byte of 2^(s - emax + 8)
__device__ __forceinline__ uint32_t e8m0_to_ue4m3(uint32_t s, uint32_t emax) {
    const int k = (int)s - (int)emax + 8;  // <= 8
    if (k >= -6) return (uint32_t)(k + 7) << 3;
    if (k >= -9) return 1u << (k + 9);     // subnormals 2^-9, 2^-8, 2^-7
    return 0u;
}

// scale u8 [expert][rows][nblk]  ->  tiled [expert][row tile][slab][2048]: for row tile rt
// (128 rows) and slab kb (256 elements = 8 blocks) four 512-byte cells, one per MMA step j:
//   byte l*16 + c*4 + b of cell j = ue4m3 of block kb*8 + j*2 + b/2 of row rt*128 + c*32 + l
// (rows past `rows` and blocks past nblk read as 0).  One thread per 4-byte word.
__global__ void mxfp4_tile_scales_kernel(const uint8_t* __restrict__ scale, uint32_t* __restrict__ tiled,
                                         uint32_t rows, uint32_t nblk, uint32_t row_tiles, uint32_t num_kb,
                                         uint32_t* __restrict__ meta) {
    const uint32_t emax = meta[0];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        reinterpret_cast<float*>(meta)[1] = emax >= 9u ? __uint_as_float((emax - 8u) << 23) : 0.0f;  // 2^(emax - 135)
    const uint32_t expert = blockIdx.y;
    const uint32_t words = row_tiles * num_kb * 512u;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x) {
        const uint32_t c = w & 3u, l = (w >> 2) & 31u, j = (w >> 7) & 3u, rec = w >> 9;
        const uint32_t kb = rec % num_kb, rt = rec / num_kb;
        const uint32_t row = rt * 128u + c * 32u + l;
        uint32_t out = 0u;
        if (row < rows) {
            const uint8_t* srow = scale + ((size_t)expert * rows + row) * nblk;
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                const uint32_t blk = kb * 8u + j * 2u + h;
                if (blk < nblk) out |= (e8m0_to_ue4m3(srow[blk], emax) * 0x0101u) << (16u * h);
            }
        }
        tiled[(size_t)expert * words + w] = out;
    }
}

// NVFP4 expert planes carry UE4M3 per-16 scales already: scale u8 [expert][rows][in_dim/16]
// -> the same records, byte l*16 + c*4 + b of cell j = scale[row rt*128 + c*32 + l][kb*16 + j*4 + b].
__global__ void nvf4_moe_tile_scales_kernel(const uint8_t* __restrict__ scale, uint32_t* __restrict__ tiled,
                                            uint32_t rows, uint32_t sf_row, uint32_t row_tiles, uint32_t num_kb) {
    const uint32_t expert = blockIdx.y;
    const uint32_t words = row_tiles * num_kb * 512u;
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x) {
        const uint32_t c = w & 3u, l = (w >> 2) & 31u, j = (w >> 7) & 3u, rec = w >> 9;
        const uint32_t kb = rec % num_kb, rt = rec / num_kb;
        const uint32_t row = rt * 128u + c * 32u + l, off = kb * 16u + j * 4u;
        uint32_t out = 0u;
        if (row < rows && off < sf_row)  // sf_row % 4 == 0
            out = *reinterpret_cast<const uint32_t*>(scale + ((size_t)expert * rows + row) * sf_row + off);
        tiled[(size_t)expert * words + w] = out;
    }
}

// ---------------------------------------------------------------- activations: four NVFP4 terms

// Two f32 -> one byte of two e2m1 codes (RN-even, saturating; low nibble = lo), and the byte's two values back as f32.
__device__ __forceinline__ uint32_t e2m1x2_rn(float2 v) {
    uint16_t byte;
    asm("{\n\t.reg .b8 q;\n\tcvt.rn.satfinite.e2m1x2.f32 q, %1, %2;\n\tmov.b16 %0, {q, 0};\n\t}" : "=h"(byte) : "f"(v.y), "f"(v.x));
    return byte;
}
__device__ __forceinline__ float2 e2m1x2_value(uint32_t byte) {
    uint32_t h2;
    asm("{\n\t.reg .b8 q, z;\n\tmov.b16 {q, z}, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, q;\n\t}" : "=r"(h2) : "h"((uint16_t)byte));
    return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}
// two f32 operations per instruction
__device__ __forceinline__ float2 mul2(float2 v, float s) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmul.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(v.x), "f"(v.y), "f"(s));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 v, float s, float2 w) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, e;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %6};\n\t"
        "fma.rn.f32x2 e, a, b, c;\n\tmov.b64 {%0, %1}, e;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(v.x), "f"(v.y), "f"(s), "f"(w.x), "f"(w.y));
    return d;
}
__device__ __forceinline__ float rcp_approx(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// One 16-element scale group, r[8] = its pairs in code order (byte i of a term's 8 bytes = pair i), values below 512: the four
// terms' codes, handed to put(term, codes), and the four scale bytes as one word.  The residual stays unscaled; the power 16^k of term k sits
// in its scale's factor (exact), and the last term leaves none.  The kernels around it are bound by issue: this is half the
// instructions of the form that scaled 16 residuals up per term, divided by the scale and worked on single floats.  One copy of a
// term's code: what a launch runs once per thread it fetches into the instruction cache first.  The reciprocal is the approximate
// instruction, but of a value with three bits of mantissa: for every scale byte and term it is the rounded quotient's bits.
template <class Put>
__device__ __forceinline__ uint32_t quantize_group(float2 (&r)[8], Put&& put) {
    float up = 1.0f / 6.0f, down = 1.329227995784916e36f;   // 2^120
    uint32_t word = 0u;
#pragma unroll 1
    for (uint32_t term = 0; term < 4u; ++term) {
        float m = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) m = fmaxf(m, fmaxf(fabsf(r[k].x), fabsf(r[k].y)));
        uint32_t s = (uint32_t)__nv_cvt_float_to_fp8(m * up, __NV_SATFINITE, __NV_E4M3);
        if (s == 0u) s = 1u;
        // an e4m3 byte's exponent and mantissa are an f32's, 120 binades lower
        const float sc = __uint_as_float(s << 20) * down;
        const float inv = rcp_approx(sc);
        uint32_t w[2] = {0u, 0u};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t byte = e2m1x2_rn(mul2(r[k], inv));
            w[k >> 2] |= byte << (8 * (k & 3));
            if (term < 3u) r[k] = fma2(e2m1x2_value(byte), -sc, r[k]);
        }
        put(term, make_uint2(w[0], w[1]));
        word |= (m > 0.0f ? s : 0u) << (8u * term);
        up *= 16.0f;
        down *= 0.0625f;
    }
    return word;
}

struct PrepArgs {
    const float* x;              // mode 0: [src rows][dim]; mode 1: gate [positions][dim]
    const float* up;             // mode 1: up [positions][dim]
    const uint32_t* sorted_row;  // [positions]; PDK_MOE_PAD = padding (zeros are written)
    const uint32_t* block_expert;  // [blocks]; PDK_MOE_PAD = unused block (its sorted_row entries are not defined; its rows are left as they are)
    uint8_t* xq;                 // [groups of 8 positions][32][dim/2]
    uint8_t* xs;                 // tiled: [records][slab][4 cells][512], the weight scale records' layout
    float* xstep;                // [positions] power of two the row was divided by
    uint32_t dim, bm, mode;  // mode 0 gather, 1 gated (x = gate, up), 2 relu(x)^2 of x [positions][dim],
                             // 3 one row: position 0 = x, the rest padding; the kernel writes the tables itself
    uint32_t* tables;        // mode 3: sorted_row[bm], block_expert[1] (written here), then f32 scale2 = table_scale2
    float table_scale2;
    uint32_t natural;        // 0: ggml MXFP4 element order (byte j = elements j, j+16); 1: byte j = elements 2j, 2j+1
    float alpha, limit, up_add;
};

// Where block b's positions keep their scale bytes.  A record holds 128 term rows = four groups of 8 tokens: a 32-token block
// is a record, and 8-token blocks share one by fours, counted from the first block of their expert (`same(b)`: whether
// block b belongs to it), at the first block of the four.  Every warp finds the run's start for itself.
template <class Same>
__device__ __forceinline__ void record_place(uint32_t pos, uint32_t bm, Same same, uint32_t& rec, uint32_t& col) {
    const uint32_t b = pos / bm;
    rec = b;
    col = (pos >> 3) & 3u;
    if (bm != 8u) return;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t first = b;
    for (;;) {
        const uint32_t below = lane + 1u;
        const uint32_t other = __ballot_sync(0xffffffffu, first < below || !same(first - below));
        const uint32_t n = other ? (uint32_t)__ffs(other) - 1u : 32u;
        first -= n;
        if (n < 32u) break;
    }
    col = (b - first) & 3u;
    rec = b - col;
}

// Four lanes' scale bytes of the four terms, transposed: lane j of the four gets term j's, groups in byte order.
__device__ __forceinline__ uint32_t scale_word(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t a = __shfl_xor_sync(0xffffffffu, v, 1);
    v = lane & 1u ? __byte_perm(v, a, 0x3715) : __byte_perm(v, a, 0x6240);   // even lane: terms 0 and 2 of both, odd: 1 and 3
    const uint32_t b = __shfl_xor_sync(0xffffffffu, v, 2);
    return lane & 2u ? __byte_perm(v, b, 0x3276) : __byte_perm(v, b, 0x5410);
}

// One CTA per block position; groups of eight without a token return before this.  Position (block b, token i) writes four term rows of its group of 8 tokens,
// row term * 8 + i % 8 of the group's 32.  A 16-element scale group of the tensor core's element order is the
// two 8-runs (h*8 .. h*8+7) and (16 + h*8 .. 16 + h*8+7) of a 32-element block.
__device__ __forceinline__ void prep_position(const PrepArgs& a, uint32_t pos, uint32_t src, uint32_t rec, uint32_t col) {
    const uint32_t tid = threadIdx.x;
    const uint32_t groups = a.dim >> 4, kh = a.dim >> 1;
    __shared__ float s_red[8];
    const bool pad = src == PDK_MOE_PAD;
    const float* row = (a.mode == 0u || a.mode == 3u) ? a.x + (size_t)(pad ? 0u : src) * a.dim : a.x + (size_t)pos * a.dim;
    const float* urow = a.up + (size_t)pos * a.dim;

    auto load8 = [&](uint32_t off, float (&v)[8]) {
        const float4 p = *reinterpret_cast<const float4*>(row + off);
        const float4 q = *reinterpret_cast<const float4*>(row + off + 4u);
        v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
        if (a.mode == 1u) {
            const float4 r = *reinterpret_cast<const float4*>(urow + off);
            const float4 t = *reinterpret_cast<const float4*>(urow + off + 4u);
            const float u[8] = {r.x, r.y, r.z, r.w, t.x, t.y, t.z, t.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                // gated unit: (xg * sigmoid(alpha * xg)) * (yu + up_add); OpenAI variant (reference/ops.rs:27-36)
                // = alpha 1.702, limit 7, up_add 1; plain SwiGLU = alpha 1, limit inf, up_add 0
                const float xg = fminf(v[k], a.limit);
                const float yu = fminf(fmaxf(u[k], -a.limit), a.limit);
                v[k] = (xg / (1.0f + __expf(-a.alpha * xg))) * (yu + a.up_add);
            }
        } else if (a.mode == 2u) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float r = fmaxf(v[k], 0.0f);
                v[k] = r * r;
            }
        }
    };
    // first element of scale group g's two 8-runs
    auto run_base = [&](uint32_t g, uint32_t& lo_at, uint32_t& hi_at) {
        if (a.natural) { lo_at = g * 16u; hi_at = g * 16u + 8u; }
        else { lo_at = (g >> 1) * 32u + (g & 1u) * 8u; hi_at = lo_at + 16u; }
    };

    // ---- the row's largest magnitude -> the power of two that brings it into [256, 512).
    // When the CTA has a thread per group (dim <= 4096) the row is read once and kept in
    // registers across the reduction.
    const uint32_t num_kb = (a.dim + 255u) >> 8;
    const bool single = num_kb * 16u <= blockDim.x;
    float lo0[8], hi0[8];
    float amax = 0.0f;
    if (!pad)
        for (uint32_t g = tid; g < groups; g += blockDim.x) {
            uint32_t lo_at, hi_at;
            run_base(g, lo_at, hi_at);
            load8(lo_at, lo0);
            load8(hi_at, hi0);
#pragma unroll
            for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fmaxf(fabsf(lo0[k]), fabsf(hi0[k])));
        }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    if ((tid & 31u) == 0u) s_red[tid >> 5] = amax;
    __syncthreads();
    amax = 0.0f;
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) amax = fmaxf(amax, s_red[w]);
    // amax = m * 2^ex with m in [1, 2): divide by 2^(ex - 8)
    const int ex = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 127;
    const bool live = !pad && amax > 0.0f && ex > -110 && ex < 120;
    const float inv_step = live ? __uint_as_float((uint32_t)(127 - (ex - 8)) << 23) : 0.0f;
    if (tid == 0) a.xstep[pos] = live ? __uint_as_float((uint32_t)(127 + (ex - 8)) << 23) : 0.0f;

    // ---- four terms per 16-element group
    const uint32_t r0 = pos & 7u;
    uint8_t* xq_rows = a.xq + ((size_t)(pos >> 3) * 32u + r0) * kh;
    uint8_t* xs_row = a.xs + (size_t)rec * num_kb * 2048u + r0 * 16u + col * 4u;
    for (uint32_t base = 0; base < num_kb * 16u; base += blockDim.x) {   // whole warps: scale_word shuffles
        const uint32_t g = base + tid;
        // scale byte of group g and term row r: record slab g/16, cell (g/4)%4, byte r*16 + col*4 + g%4
        // (four threads write their groups' bytes of a term as one word)
        uint8_t* xs_g = xs_row + (size_t)(g >> 4) * 2048u + ((g >> 2) & 3u) * 512u;
        uint32_t sb = 0u;
        auto put = [&](uint32_t term, uint2 codes) {
            *reinterpret_cast<uint2*>(xq_rows + (size_t)(term * 8u) * kh + (size_t)g * 8u) = codes;
        };
        // padding and all-zero rows: zero term rows and scale bytes, none of the term arithmetic; the record's cells
        // past K must read as zero too
        if (live && g < groups) {
            if (!single) {
                uint32_t lo_at, hi_at;
                run_base(g, lo_at, hi_at);
                load8(lo_at, lo0);
                load8(hi_at, hi0);
            }
            float2 r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                // ggml order: byte k = (lo run k, hi run k); natural: byte k = lo run (2k, 2k+1), byte 4+k = hi run (2k, 2k+1)
                r[k] = mul2(!a.natural ? make_float2(lo0[k], hi0[k])
                            : k < 4    ? make_float2(lo0[2 * (k & 3)], lo0[2 * (k & 3) + 1])
                                       : make_float2(hi0[2 * (k & 3)], hi0[2 * (k & 3) + 1]), inv_step);
            sb = quantize_group(r, put);
        } else if (g < groups) {
#pragma unroll 1
            for (uint32_t term = 0; term < 4u; ++term) put(term, make_uint2(0u, 0u));
        }
        const uint32_t word = scale_word(sb);
        if (g < num_kb * 16u) *reinterpret_cast<uint32_t*>(xs_g + (g & 3u) * 128u) = word;
    }
}

__global__ void __launch_bounds__(256) moe_prep_f4_kernel(const PrepArgs a) {
    pdk_pdl_wait_then_launch();   // dependent launch: may start while the previous kernel of the stream drains
    const uint32_t pos = blockIdx.x, b = pos / a.bm;
    uint32_t src, rec, col;
    if (a.mode == 3u) {
        src = pos == 0u ? 0u : PDK_MOE_PAD;
        rec = col = 0u;
        if (threadIdx.x == 0) {
            a.tables[pos] = src;
            if (pos == 0u) {
                a.tables[a.bm] = 0u;  // block 0 belongs to expert 0
                reinterpret_cast<float*>(a.tables)[a.bm + 1u] = a.table_scale2;
            }
        }
    } else {
        // Blocks of 8: the table words are requested together, one after the other they were a good part of a short call (60 tokens, 4 of
        // 128 experts, 2880: 6.3 us, this way 5.5).  Blocks of 32 have many empty groups, for which one word is enough (1024 tokens: together 25.9
        // us, this way 24.6).
        const bool small = a.bm == 8u;
        const uint32_t lane = threadIdx.x & 31u, e = a.block_expert[b];
        const uint32_t before = small && lane < b ? a.block_expert[b - 1u - lane] : PDK_MOE_PAD;
        uint32_t group = small ? a.sorted_row[pos & ~7u] : 0u;
        if (small) src = a.sorted_row[pos];
        if (e == PDK_MOE_PAD) return;   // an unused block: the GEMMs skip it, nothing reads its rows
        if (!small) {
            src = a.sorted_row[pos];
            if (src == PDK_MOE_PAD) group = a.sorted_row[pos & ~7u];
        }
        if (src == PDK_MOE_PAD && group == PDK_MOE_PAD) return;   // nor a group without a token
        record_place(pos, a.bm, [&](uint32_t q) { return (q == b - 1u - lane ? before : a.block_expert[q]) == e; }, rec, col);
    }
    prep_position(a, pos, src, rec, col);
}

// The preparations by pair: one CTA per row that has a token, none for padding.
//   kTokens  a token's row is quantized once and written to the positions of all its k pairs, where a CTA per position read and
//            quantized it k times (1024 tokens of 2880, 4 of 128 experts: 26.2 -> 12.4 us);
//   the others: the row at pair p's own position, as it is, gate and up through the gated unit, or relu^2.  A CTA per position
//            meets as many empty ones as live ones where experts hold ragged blocks (the same call: 31 -> 28 us; 60 tokens, 240 rows at 1264 positions: 7.7 -> 4).
// Positions without a pair are left as they are: their columns of the GEMM are never read.
enum PrepKind : uint32_t { kTokens = 0u, kRows = 1u, kGatedRows = 2u, kSquaredRows = 3u };
struct TokenArgs {
    const float *x, *up;        // kTokens: [rows][dim]; else [positions][dim] (x = gate with kGatedRows)
    const uint32_t* pair_pos;   // [rows][k]
    uint8_t *xq, *xs;
    float* xstep;
    uint32_t dim, k, bm, natural;
    float alpha, limit, up_add;
};

template <uint32_t KIND>
__global__ void __launch_bounds__(256) moe_prep_pairs_kernel(const TokenArgs a) {
    __shared__ float s_red[8];
    __shared__ uint32_t s_pos[16];
    pdk_pdl_wait_then_launch();
    const uint32_t tid = threadIdx.x, groups = a.dim >> 4, kh = a.dim >> 1, num_kb = (a.dim + 255u) >> 8;
    size_t row = blockIdx.x;
    const uint32_t k = KIND == kTokens ? a.k : 1u;
    if (KIND == kTokens) {
        if (tid < k) s_pos[tid] = a.pair_pos[row * k + tid];
    } else {
        const uint32_t at = a.pair_pos[row];
        if (at == PDK_MOE_PAD) return;
        if (tid == 0u) s_pos[0] = at;
        row = at & 0x3FFFFFFFu;
    }
    const float* x = a.x + row * a.dim;
    const float* up = a.up + row * a.dim;
    auto load4 = [&](uint32_t at) {
        float4 v = *reinterpret_cast<const float4*>(x + at);
        if (KIND == kGatedRows) {
            const float4 u = *reinterpret_cast<const float4*>(up + at);
            // gated unit: (xg * sigmoid(alpha * xg)) * (yu + up_add); OpenAI variant (reference/ops.rs:27-36) = alpha 1.702, limit 7,
            // up_add 1; plain SwiGLU = alpha 1, limit inf, up_add 0
            auto unit = [&](float g, float w) {
                const float xg = fminf(g, a.limit), yu = fminf(fmaxf(w, -a.limit), a.limit);
                return (xg / (1.0f + __expf(-a.alpha * xg))) * (yu + a.up_add);
            };
            v = make_float4(unit(v.x, u.x), unit(v.y, u.y), unit(v.z, u.z), unit(v.w, u.w));
        }
        if (KIND == kSquaredRows) {
            auto sq = [](float g) { const float r = fmaxf(g, 0.0f); return r * r; };
            v = make_float4(sq(v.x), sq(v.y), sq(v.z), sq(v.w));
        }
        return v;
    };
    auto load = [&](uint32_t g, float2 (&r)[8]) {   // in code order, as prep_position
        const uint32_t lo_at = a.natural ? g * 16u : (g >> 1) * 32u + (g & 1u) * 8u, hi_at = lo_at + (a.natural ? 8u : 16u);
        const float4 p = load4(lo_at), q = load4(lo_at + 4u), u = load4(hi_at), v = load4(hi_at + 4u);
        if (a.natural) {
            r[0] = make_float2(p.x, p.y); r[1] = make_float2(p.z, p.w); r[2] = make_float2(q.x, q.y); r[3] = make_float2(q.z, q.w);
            r[4] = make_float2(u.x, u.y); r[5] = make_float2(u.z, u.w); r[6] = make_float2(v.x, v.y); r[7] = make_float2(v.z, v.w);
        } else {
            r[0] = make_float2(p.x, u.x); r[1] = make_float2(p.y, u.y); r[2] = make_float2(p.z, u.z); r[3] = make_float2(p.w, u.w);
            r[4] = make_float2(q.x, v.x); r[5] = make_float2(q.y, v.y); r[6] = make_float2(q.z, v.z); r[7] = make_float2(q.w, v.w);
        }
    };
    float2 r[8] = {};
    float amax = 0.0f;
    for (uint32_t g = tid; g < groups; g += blockDim.x) {
        load(g, r);
#pragma unroll
        for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fmaxf(fabsf(r[k].x), fabsf(r[k].y)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    if ((tid & 31u) == 0u) s_red[tid >> 5] = amax;
    __syncthreads();
    amax = 0.0f;
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) amax = fmaxf(amax, s_red[w]);
    const int ex = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 127;
    const bool live = amax > 0.0f && ex > -110 && ex < 120;
    const float inv_step = live ? __uint_as_float((uint32_t)(127 - (ex - 8)) << 23) : 0.0f;
    const float step = live ? __uint_as_float((uint32_t)(127 + (ex - 8)) << 23) : 0.0f;
    const bool single = num_kb * 16u <= blockDim.x;
    for (uint32_t base = 0; base < num_kb * 16u; base += blockDim.x) {   // whole warps: scale_word shuffles
        const uint32_t g = base + tid;
        uint32_t sb = 0u;
        auto put = [&](uint32_t term, uint2 codes) {
            for (uint32_t s = 0; s < k; ++s) {
                const uint32_t at = s_pos[s];
                if (at == PDK_MOE_PAD) continue;
                const uint32_t pos = at & 0x3FFFFFFFu;
                *reinterpret_cast<uint2*>(a.xq + ((size_t)(pos >> 3) * 32u + (pos & 7u) + term * 8u) * kh + (size_t)g * 8u) = codes;
            }
        };
        if (live && g < groups) {
            if (!single) load(g, r);
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = mul2(r[k], inv_step);
            sb = quantize_group(r, put);
        } else if (g < groups) {
#pragma unroll 1
            for (uint32_t term = 0; term < 4u; ++term) put(term, make_uint2(0u, 0u));
        }
        const uint32_t word = scale_word(sb);
        if (g >= num_kb * 16u) continue;
        for (uint32_t s = 0; s < k; ++s) {
            const uint32_t at = s_pos[s];
            if (at == PDK_MOE_PAD) continue;
            const uint32_t pos = at & 0x3FFFFFFFu, col = at >> 30, r0 = pos & 7u, b = pos / a.bm, rec = a.bm == 8u ? b - col : b;
            *reinterpret_cast<uint32_t*>(a.xs + ((size_t)rec * num_kb + (g >> 4)) * 2048u + ((g >> 2) & 3u) * 512u + r0 * 16u +
                                         col * 4u + (g & 3u) * 128u) = word;
            if (g == 0u) a.xstep[pos] = step;
        }
    }
}

// Decode widths (rows * k <= 32 pairs): routing, alignment and the first activation preparation in
// one launch.  Every CTA (one per block position, as above) routes the few tokens itself - a warp
// per token for the top-k, one warp for the alignment of at most 32 pairs: rank inside an expert
// from __match_any_sync, first block of an expert from the block counts of the lower experts - and
// then prepares its own position; CTA 0 also leaves the routing tables in global memory for the
// GEMMs and the combine.  The layout is moe_align's: blocks in ascending expert order, a block's
// entries in ascending pair order, unused blocks marked PDK_MOE_PAD.
struct RouteArgs {
    const float* logits;     // [rows][n_expert]
    const float* bias;       // [n_expert] or null
    uint32_t* idx;           // out [rows][k]
    float* w;                // out [rows][k]
    uint32_t* sorted_row;    // out [max_blocks * bm]
    uint32_t* sorted_slot;   // out [max_blocks * bm]
    uint32_t* block_expert;  // out [max_blocks]
    uint32_t rows, k, n_expert, max_blocks;
};
constexpr uint32_t kRouteMaxPos = 32u * 32u;

// The tables of the few tokens, in shared memory (256 threads).
struct RouteTables {
    uint32_t idx[32], row[kRouteMaxPos], slot[kRouteMaxPos], bexp[32], pos[32];   // pos: pair -> position
    float w[32];
};
__device__ __forceinline__ void route_few(const RouteArgs& r, uint32_t bm, RouteTables& s) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t npairs = r.rows * r.k, n_pos = r.max_blocks * bm;
    if (warp < r.rows) moe_route::topk_warp(r.logits + (size_t)warp * r.n_expert, r.bias, r.n_expert, r.k, lane, s.idx + warp * r.k, s.w + warp * r.k);
    for (uint32_t p = tid; p < n_pos; p += blockDim.x) { s.row[p] = PDK_MOE_PAD; s.slot[p] = 0u; }
    if (tid < 32u) { s.bexp[tid] = PDK_MOE_PAD; s.pos[tid] = PDK_MOE_PAD; }
    __syncthreads();
    if (warp == 0u) {
        const bool valid = lane < npairs;
        const uint32_t e = valid ? s.idx[lane] : 0x80000000u + lane;     // idle lanes: distinct keys that match nobody
        const uint32_t grp = __match_any_sync(0xffffffffu, e);
        const uint32_t rank = __popc(grp & ((1u << lane) - 1u)), cnt = __popc(grp);
        const uint32_t nblk = (valid && rank == 0u) ? (cnt + bm - 1u) / bm : 0u;   // counted once, by the group's first lane
        uint32_t first = 0u;
        for (uint32_t q = 0; q < 32u; ++q) {
            const uint32_t eq = __shfl_sync(0xffffffffu, e, q), nq = __shfl_sync(0xffffffffu, nblk, q);
            if (eq < e) first += nq;
        }
        if (valid) {
            const uint32_t blk = first + rank / bm, at = blk * bm + rank % bm;
            if (blk < r.max_blocks) {
                s.row[at] = lane / r.k;
                s.slot[at] = lane % r.k;
                s.pos[lane] = at | ((bm == 8u ? rank >> 3 : at >> 3) & 3u) << 30;
                if (rank % bm == 0u) s.bexp[blk] = e;
            }
        }
    }
    __syncthreads();
}
__device__ __forceinline__ void route_store(const RouteArgs& r, uint32_t bm, const RouteTables& s) {
    const uint32_t tid = threadIdx.x, npairs = r.rows * r.k;
    if (tid < npairs) { r.idx[tid] = s.idx[tid]; r.w[tid] = s.w[tid]; }
    for (uint32_t p = tid; p < r.max_blocks * bm; p += blockDim.x) { r.sorted_row[p] = s.row[p]; r.sorted_slot[p] = s.slot[p]; }
    if (tid < r.max_blocks) r.block_expert[tid] = s.bexp[tid];
}

__global__ void __launch_bounds__(256) moe_route_few_kernel(const RouteArgs r, uint32_t* __restrict__ pair_pos, uint32_t bm) {
    __shared__ RouteTables s;
    pdk_pdl_wait_then_launch();
    route_few(r, bm, s);
    route_store(r, bm, s);
    if (threadIdx.x < r.rows * r.k) pair_pos[threadIdx.x] = s.pos[threadIdx.x];
}

__global__ void __launch_bounds__(256) moe_route_prep_f4_kernel(const PrepArgs a, const RouteArgs r) {
    __shared__ RouteTables s;
    pdk_pdl_wait_then_launch();
    route_few(r, a.bm, s);
    if (blockIdx.x == 0u) route_store(r, a.bm, s);
    const uint32_t pos = blockIdx.x, b = pos / a.bm, e = s.bexp[b], src = s.row[pos];
    if (e == PDK_MOE_PAD) return;   // an unused block
    if (src == PDK_MOE_PAD && s.row[pos & ~7u] == PDK_MOE_PAD) return;
    uint32_t rec, col;
    record_place(pos, a.bm, [&](uint32_t q) { return s.bexp[q] == e; }, rec, col);
    prep_position(a, pos, src, rec, col);
}

}  // namespace

// No counterpart in the reference (its B200 MoE kernels run mma.sync on int8 activations):
// E8M0 scale plane [n_expert][rows][in_dim/32] -> tiled UE4M3 scale records
// [n_expert][ceil(rows/128)][ceil(in_dim/256)][2048] for pdk_mxfp4_moe_gemm_tc5, plus
// meta = {u32 largest scale byte, f32 scale2 = 2^(largest - 135)} (8 bytes, device memory).
// Load-time call; three launches on `stream`.
PDK_EXPORT int pdk_mxfp4_tc5_tile_scales(const void* scale, void* tiled, void* meta, uint32_t rows, uint32_t in_dim,
                                         uint32_t n_expert, void* stream) {
    if (rows == 0 || n_expert == 0) return 0;
    if (in_dim == 0 || (in_dim & 63u) != 0u || !pdk_aligned(tiled, 16) || !pdk_aligned(meta, 8))
        return cudaErrorInvalidValue;
    auto st = (cudaStream_t)stream;
    const uint32_t nblk = in_dim >> 5, row_tiles = (rows + 127u) / 128u, num_kb = (in_dim + 255u) >> 8;
    cudaError_t e = cudaMemsetAsync(meta, 0, 8, st);
    if (e != cudaSuccess) return (int)e;
    const uint64_t n = (uint64_t)n_expert * rows * nblk;
    const uint64_t want = (n + 1023u) / 1024u;
    mxfp4_emax_kernel<<<(uint32_t)(want < 1184u ? want : 1184u), 256, 0, st>>>((const uint8_t*)scale, n, (uint32_t*)meta);
    const uint32_t words = row_tiles * num_kb * 512u;
    mxfp4_tile_scales_kernel<<<dim3((words + 255u) / 256u < 64u ? (words + 255u) / 256u : 64u, n_expert), 256, 0, st>>>(
        (const uint8_t*)scale, (uint32_t*)tiled, rows, nblk, row_tiles, num_kb, (uint32_t*)meta);
    return pdk_launch_status();
}

// No counterpart in the reference: block positions -> four NVFP4 term rows each.
//   mode 0: position p takes row sorted_row[p] of x f32 [rows][dim]            (`up` unused)
//   mode 1: position p takes swiglu(x[p], up[p]) of the raw gate / up outputs f32 [positions][dim]
// Writes xq u8 [max_blocks*4*bm][dim/2] (term t of position p in row p/8*32 + t*8 + p%8), xs u8 [max_blocks][ceil(dim/256)][2048]
// (scale records in the weight scale records' layout, one for the 128 term rows of four groups of eight: with bm 8 four blocks of
// a run share the first one's; bytes of term rows that are not there are left alone), xstep f32 [max_blocks*bm].
// dim % 32 == 0, bm 8 or 32.
static uint32_t prep_threads(uint32_t dim) {
    const uint32_t per_row = ((dim + 255u) >> 8) * 16u;  // scale groups incl. the zero tail of the last record
    return per_row <= 256u ? (per_row + 31u) & ~31u : 256u;
}
static int prep_impl(const void* x, const void* up, const void* sorted_row, const void* block_expert, void* xq, void* xs,
                     void* xstep, uint32_t dim, uint32_t bm, uint32_t max_blocks, uint32_t mode, uint32_t natural,
                     float alpha, float limit, float up_add, void* stream) {
    if (max_blocks == 0) return 0;
    if (dim == 0 || (dim & 31u) != 0u || (bm != 8u && bm != 32u)) return cudaErrorInvalidValue;
    if (!pdk_aligned(x, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(xs, 4) || (mode == 1u && !pdk_aligned(up, 16)))
        return cudaErrorInvalidValue;
    PrepArgs a{};
    a.x = (const float*)x; a.up = (const float*)up; a.sorted_row = (const uint32_t*)sorted_row;
    a.block_expert = (const uint32_t*)block_expert;
    a.xq = (uint8_t*)xq; a.xs = (uint8_t*)xs; a.xstep = (float*)xstep;
    a.dim = dim; a.bm = bm; a.mode = mode; a.natural = natural; a.alpha = alpha; a.limit = limit; a.up_add = up_add;
    return pdk_launch_pdl(moe_prep_f4_kernel, dim3(max_blocks * bm), dim3(prep_threads(dim)), 0, (cudaStream_t)stream, a);
}

PDK_EXPORT int pdk_moe_prep_act_f4(const void* x, const void* up, const void* sorted_row, const void* block_expert,
                                   void* xq, void* xs, void* xstep, uint32_t dim, uint32_t bm, uint32_t max_blocks,
                                   uint32_t mode, float alpha, float limit, void* stream) {
    if (mode > 1u) return cudaErrorInvalidValue;
    return prep_impl(x, up, sorted_row, block_expert, xq, xs, xstep, dim, bm, max_blocks, mode, 0u, alpha, limit, 1.0f,
                     stream);
}

// The rows of x f32 [rows][dim] to the positions of their pairs (pair_pos u32 [rows][k], pdk_moe_align_pos):
// the same term rows, scale records and steps there as pdk_moe_prep_act_f4 (natural 0) or ..._f4n (1) in mode 0; positions of padding
// are left alone.
PDK_EXPORT int pdk_moe_prep_tokens_f4(const void* x, const void* pair_pos, void* xq, void* xs, void* xstep, uint32_t dim, uint32_t k,
                                      uint32_t rows, uint32_t bm, uint32_t natural, void* stream) {
    if (rows == 0 || k == 0) return 0;
    if (dim == 0 || (dim & 31u) != 0u || (bm != 8u && bm != 32u) || natural > 1u || k > 16u || !pair_pos) return cudaErrorInvalidValue;
    if (!pdk_aligned(x, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(xs, 16)) return cudaErrorInvalidValue;
    TokenArgs a{};
    a.x = (const float*)x; a.pair_pos = (const uint32_t*)pair_pos; a.xq = (uint8_t*)xq; a.xs = (uint8_t*)xs; a.xstep = (float*)xstep;
    a.dim = dim; a.k = k; a.bm = bm; a.natural = natural;
    return pdk_launch_pdl(moe_prep_pairs_kernel<kTokens>, dim3(rows), dim3(prep_threads(dim)), 0, (cudaStream_t)stream, a);
}

// Position rows to term rows for the pairs' positions only: x f32 [positions][dim] as it is (mode 0, the rows of
// pdk_*_moe_gate_up_tc5), gate = x and up through the gated unit (mode 1) or relu(x)^2 (mode 2).  pair_pos u32 [pairs] as above;
// natural, alpha, limit and up_add as in pdk_moe_prep_act_f4 / ..._f4n, and the same rows, records and steps at these positions.
PDK_EXPORT int pdk_moe_prep_pairs_f4(const void* x, const void* up, const void* pair_pos, void* xq, void* xs, void* xstep, uint32_t dim,
                                     uint32_t bm, uint32_t pairs, uint32_t mode, uint32_t natural, float alpha, float limit, float up_add,
                                     void* stream) {
    if (pairs == 0) return 0;
    if (dim == 0 || (dim & 31u) != 0u || (bm != 8u && bm != 32u) || natural > 1u || mode > 2u || !pair_pos) return cudaErrorInvalidValue;
    if (!pdk_aligned(x, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(xs, 16) || (mode == 1u && (!up || !pdk_aligned(up, 16))))
        return cudaErrorInvalidValue;
    TokenArgs a{};
    a.x = (const float*)x; a.up = (const float*)up; a.pair_pos = (const uint32_t*)pair_pos;
    a.xq = (uint8_t*)xq; a.xs = (uint8_t*)xs; a.xstep = (float*)xstep;
    a.dim = dim; a.bm = bm; a.natural = natural; a.alpha = alpha; a.limit = limit; a.up_add = up_add;
    auto kern = mode == 0u ? moe_prep_pairs_kernel<kRows> : mode == 1u ? moe_prep_pairs_kernel<kGatedRows> : moe_prep_pairs_kernel<kSquaredRows>;
    return pdk_launch_pdl(kern, dim3(pairs), dim3(prep_threads(dim)), 0, (cudaStream_t)stream, a);
}

// No counterpart in the reference.  moe_topk_batch + moe_align_bm + pdk_moe_prep_act_f4 (mode 0) in one
// launch for decode widths: rows * k <= 32 pairs, rows <= 8, n_expert <= 512, max_blocks <= 32.  Writes
// the same idx / w / sorted_row / sorted_slot / block_expert the three calls would, and the term rows.
static int route_prep_impl(const void* logits, const void* router_bias, const void* x, void* idx, void* w, void* sorted_row,
                           void* sorted_slot, void* block_expert, void* xq, void* xs, void* xstep, uint32_t n_expert, uint32_t k,
                           uint32_t rows, uint32_t dim, uint32_t bm, uint32_t max_blocks, uint32_t natural, void* stream) {
    if (rows == 0 || max_blocks == 0) return 0;
    if (rows > 8u || k == 0 || k > 16u || rows * k > 32u || n_expert == 0 || n_expert > 512u || k > n_expert ||
        max_blocks > 32u || (bm != 8u && bm != 32u) || max_blocks * bm > kRouteMaxPos || dim == 0 || (dim & 31u) != 0u)
        return cudaErrorInvalidValue;
    if (!pdk_aligned(x, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(xs, 16) || !pdk_aligned(logits, 4)) return cudaErrorInvalidValue;
    PrepArgs a{};
    a.x = (const float*)x;
    a.xq = (uint8_t*)xq; a.xs = (uint8_t*)xs; a.xstep = (float*)xstep;
    a.dim = dim; a.bm = bm; a.mode = 0u; a.natural = natural; a.alpha = 1.0f; a.limit = 0.0f; a.up_add = 0.0f;
    RouteArgs r{};
    r.logits = (const float*)logits; r.bias = (const float*)router_bias;
    r.idx = (uint32_t*)idx; r.w = (float*)w;
    r.sorted_row = (uint32_t*)sorted_row; r.sorted_slot = (uint32_t*)sorted_slot; r.block_expert = (uint32_t*)block_expert;
    r.rows = rows; r.k = k; r.n_expert = n_expert; r.max_blocks = max_blocks;
    return pdk_launch_pdl(moe_route_prep_f4_kernel, dim3(max_blocks * bm), dim3(256), 0, (cudaStream_t)stream, a, r);
}

// moe_topk_batch + pdk_moe_align_pos in one small launch, with pdk_moe_route_prep_f4's limits.  Unlike that call it leaves the
// preparation to pdk_moe_prep_tokens_f4, under which the expert GEMM behind it requests its weights already.
PDK_EXPORT int pdk_moe_route_few(const void* logits, const void* router_bias, void* idx, void* w, void* sorted_row, void* sorted_slot,
                                 void* block_expert, void* pair_pos, uint32_t n_expert, uint32_t k, uint32_t rows, uint32_t bm,
                                 uint32_t max_blocks, void* stream) {
    if (rows == 0 || max_blocks == 0) return 0;
    if (rows > 8u || k == 0 || k > 16u || rows * k > 32u || n_expert == 0 || n_expert > 512u || k > n_expert ||
        max_blocks > 32u || (bm != 8u && bm != 32u) || max_blocks * bm > kRouteMaxPos || !pair_pos)
        return cudaErrorInvalidValue;
    RouteArgs r{};
    r.logits = (const float*)logits; r.bias = (const float*)router_bias;
    r.idx = (uint32_t*)idx; r.w = (float*)w;
    r.sorted_row = (uint32_t*)sorted_row; r.sorted_slot = (uint32_t*)sorted_slot; r.block_expert = (uint32_t*)block_expert;
    r.rows = rows; r.k = k; r.n_expert = n_expert; r.max_blocks = max_blocks;
    return pdk_launch_pdl(moe_route_few_kernel, dim3(1), dim3(256), 0, (cudaStream_t)stream, r, (uint32_t*)pair_pos, bm);
}

PDK_EXPORT int pdk_moe_route_prep_f4(const void* logits, const void* router_bias, const void* x, void* idx, void* w,
                                     void* sorted_row, void* sorted_slot, void* block_expert, void* xq, void* xs, void* xstep,
                                     uint32_t n_expert, uint32_t k, uint32_t rows, uint32_t dim, uint32_t bm,
                                     uint32_t max_blocks, void* stream) {
    return route_prep_impl(logits, router_bias, x, idx, w, sorted_row, sorted_slot, block_expert, xq, xs, xstep, n_expert, k, rows,
                           dim, bm, max_blocks, 0u, stream);
}

// The same for NVFP4 expert planes (natural element order).
PDK_EXPORT int pdk_moe_route_prep_f4n(const void* logits, const void* router_bias, const void* x, void* idx, void* w,
                                      void* sorted_row, void* sorted_slot, void* block_expert, void* xq, void* xs, void* xstep,
                                      uint32_t n_expert, uint32_t k, uint32_t rows, uint32_t dim, uint32_t bm,
                                      uint32_t max_blocks, void* stream) {
    return route_prep_impl(logits, router_bias, x, idx, w, sorted_row, sorted_slot, block_expert, xq, xs, xstep, n_expert, k, rows,
                           dim, bm, max_blocks, 1u, stream);
}

// The same for NVFP4 expert planes: term rows packed in the natural element order (byte j = elements
// 2j, 2j+1, as ModelOpt checkpoints store their weights).  mode 0 gather; mode 1 gated unit
// (min(g, limit) * sigmoid(alpha * that)) * (clamp(u, +-limit) + up_add) - plain SwiGLU is alpha 1,
// limit inf, up_add 0; mode 2 relu(x)^2 of x f32 [positions][dim] (the non-gated experts).
PDK_EXPORT int pdk_moe_prep_act_f4n(const void* x, const void* up, const void* sorted_row, const void* block_expert,
                                    void* xq, void* xs, void* xstep, uint32_t dim, uint32_t bm, uint32_t max_blocks,
                                    uint32_t mode, float alpha, float limit, float up_add, void* stream) {
    if (mode > 2u) return cudaErrorInvalidValue;
    return prep_impl(x, up, sorted_row, block_expert, xq, xs, xstep, dim, bm, max_blocks, mode, 1u, alpha, limit, up_add,
                     stream);
}

// No counterpart in the reference (slots 88 / 89 are its mma.sync kernels on int8 activations):
// grouped expert GEMM over blocks aligned with block size bm.  Plane p (w*_data repacked MXFP4
// data [n_expert][out_dim][in_dim/2], w*_sf / w*_meta from pdk_mxfp4_tc5_tile_scales, bias
// [n_expert][out_dim] or NULL) times the term rows of pdk_moe_prep_act_f4.
//   scatter 0: out_p f32 [max_blocks*bm][out_dim] in block order, raw (bias added); one or two planes
//              (w1_data NULL = one)
//   scatter 1: out0 = part f32 [rows*n_active][out_dim], row (sorted_row, sorted_slot), times topk_w
// in_dim % 64 == 0, max_blocks <= 1024.
namespace {
struct PlaneArgs { const void *data, *sf, *bias; const float* scale2; };
struct RowArgs { const void *xq, *xs, *xstep, *block_expert, *sorted_row, *sorted_slot, *topk_w; };
struct UnitArgs { float alpha, limit, up_add; };
constexpr uint32_t kAhead = 0x10000u;   // beside a kind: moe_gemm::Args::ahead
}  // namespace

static int gemm_impl(const PlaneArgs& w0, const PlaneArgs& w1, void* out0, void* out1, const RowArgs& r, uint32_t in_dim,
                     uint32_t out_dim, uint32_t n_expert, uint32_t bm, uint32_t max_blocks, uint32_t n_active, uint32_t kind,
                     uint32_t scale2_per_expert, const UnitArgs& unit, void* stream) {
    if (max_blocks == 0 || out_dim == 0 || n_expert == 0) return 0;
    if (in_dim == 0 || (in_dim & 63u) != 0u || (bm != 8u && bm != 32u) || max_blocks > moe_gemm::kMaxBlocks)
        return cudaErrorInvalidValue;
    if (!pdk_aligned(w0.data, 16) || !pdk_aligned(w0.sf, 16) || !pdk_aligned(r.xq, 16) || !pdk_aligned(r.xs, 16) ||
        !pdk_aligned(w0.scale2, 4) || (w1.data && (!pdk_aligned(w1.data, 16) || !pdk_aligned(w1.sf, 16))))
        return cudaErrorInvalidValue;
    const uint32_t ahead = kind & kAhead ? 1u : 0u;
    kind &= ~kAhead;
    if (kind == moe_gemm::kScatter && (w1.data || !r.sorted_slot || !r.topk_w)) return cudaErrorInvalidValue;
    if (kind == moe_gemm::kGated && !w1.data) return cudaErrorInvalidValue;
    const PlaneArgs& wb = w1.data ? w1 : w0;
    const uint32_t kbytes = in_dim >> 1;
    CUtensorMap tw0, tw1, tx;
    const uint64_t wrows = (uint64_t)n_expert * out_dim;
    if (int rc = pdk_make_tmap_2d(&tw0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w0.data, kbytes, wrows, kbytes, BKB, BM)) return rc;
    if (int rc = pdk_make_tmap_2d(&tw1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wb.data, kbytes, wrows, kbytes, BKB, BM)) return rc;
    if (int rc = pdk_make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, r.xq, kbytes, (uint64_t)max_blocks * 4u * bm, kbytes,
                                  BKB, 32u))
        return rc;
    moe_gemm::Args a{};
    a.w_sf[0] = (const uint8_t*)w0.sf; a.w_sf[1] = (const uint8_t*)wb.sf;
    a.scale2[0] = w0.scale2; a.scale2[1] = wb.scale2;
    a.scale2_per_expert = scale2_per_expert;
    a.bias[0] = (const float*)w0.bias; a.bias[1] = (const float*)w1.bias;
    a.out[0] = (float*)out0; a.out[1] = (float*)out1;
    a.x_sf = (const uint8_t*)r.xs; a.xstep = (const float*)r.xstep;
    a.block_expert = (const uint32_t*)r.block_expert; a.sorted_row = (const uint32_t*)r.sorted_row;
    a.sorted_slot = (const uint32_t*)r.sorted_slot; a.topk_w = (const float*)r.topk_w;
    a.in_dim = in_dim; a.out_dim = out_dim; a.max_blocks = max_blocks; a.n_planes = w1.data ? 2u : 1u;
    a.n_active = n_active; a.scatter = kind == moe_gemm::kScatter; a.ahead = ahead; a.block_shift = bm == 32u ? 2u : 0u;
    a.alpha = unit.alpha; a.limit = unit.limit; a.up_add = unit.up_add; a.err_word = pdk_error_word();
    auto st = (cudaStream_t)stream;
    // The gated unit needs gate and up in one CTA.  One plane, blocks of 32: where an expert has a block or a little more on average,
    // half of the experts spill a few tokens into the next one, and tiles of up to six groups save that pass over the weights
    // (1024 tokens, 4 of 128 experts, 2880 x 2880: down 150 -> 130 us).  From 48 tokens an expert on, runs are long and the tensor core is what
    // they wait for: tiles of four groups in stages of two slabs (down of 1000 tokens an expert, 2048 x 2048: 54.2 -> 42.8 us, of 256,
    // 2880 x 768: 126 -> 104; but of 44, 1664 x 2176: 78 -> 85).  Blocks of 8: six groups instead of four 0.97 to 1.08 times
    // the time over 40 shapes, 1.00 on average.
    using namespace moe_gemm;
    if (kind == kGated) return launch<6, 2, kGated, 12>(tw0, tw1, tx, a, st);
    if (bm == 8u) return launch<4, 1, kPlain, 8>(tw0, tw1, tx, a, st);
    // max_blocks has room for a partly filled block of every expert
    const uint64_t tokens = max_blocks > n_expert ? (uint64_t)(max_blocks - n_expert) * bm : 0u;
    return tokens > 48ull * n_expert ? launch<4, 1, kPlain, 8, false, true>(tw0, tw1, tx, a, st)
                                     : launch<6, 1, kPlain, 8>(tw0, tw1, tx, a, st);
}

PDK_EXPORT int pdk_mxfp4_moe_gemm_tc5(const void* w0_data, const void* w0_sf, const void* w0_meta, const void* w0_bias,
                                      void* out0, const void* w1_data, const void* w1_sf, const void* w1_meta,
                                      const void* w1_bias, void* out1, const void* xq, const void* xs,
                                      const void* xstep, const void* block_expert, const void* sorted_row,
                                      const void* sorted_slot, const void* topk_w, uint32_t in_dim, uint32_t out_dim,
                                      uint32_t n_expert, uint32_t bm, uint32_t max_blocks, uint32_t n_active,
                                      uint32_t scatter, void* stream) {
    if (!pdk_aligned(w0_meta, 8) || w0_meta == nullptr || (w1_data && w1_meta == nullptr)) return cudaErrorInvalidValue;
    return gemm_impl({w0_data, w0_sf, w0_bias, (const float*)w0_meta + 1},
                     {w1_data, w1_sf, w1_bias, w1_meta ? (const float*)w1_meta + 1 : nullptr}, out0, out1,
                     {xq, xs, xstep, block_expert, sorted_row, sorted_slot, topk_w}, in_dim, out_dim, n_expert, bm, max_blocks,
                     n_active, scatter ? moe_gemm::kScatter : moe_gemm::kPlain, 0u, {}, stream);
}

// The same where block_expert, sorted_row and sorted_slot were written before the launch in front of this one in the stream began (as
// they are behind pdk_moe_prep_*: the preparations release the next launch only when everything before them is complete): the
// tiles are laid out and the first weights requested while that launch runs.
PDK_EXPORT int pdk_mxfp4_moe_gemm_tc5_ahead(const void* w0_data, const void* w0_sf, const void* w0_meta, const void* w0_bias,
                                      void* out0, const void* w1_data, const void* w1_sf, const void* w1_meta,
                                      const void* w1_bias, void* out1, const void* xq, const void* xs,
                                      const void* xstep, const void* block_expert, const void* sorted_row,
                                      const void* sorted_slot, const void* topk_w, uint32_t in_dim, uint32_t out_dim,
                                      uint32_t n_expert, uint32_t bm, uint32_t max_blocks, uint32_t n_active,
                                      uint32_t scatter, void* stream) {
    if (!pdk_aligned(w0_meta, 8) || w0_meta == nullptr || (w1_data && w1_meta == nullptr)) return cudaErrorInvalidValue;
    return gemm_impl({w0_data, w0_sf, w0_bias, (const float*)w0_meta + 1},
                     {w1_data, w1_sf, w1_bias, w1_meta ? (const float*)w1_meta + 1 : nullptr}, out0, out1,
                     {xq, xs, xstep, block_expert, sorted_row, sorted_slot, topk_w}, in_dim, out_dim, n_expert, bm, max_blocks,
                     n_active, (scatter ? moe_gemm::kScatter : moe_gemm::kPlain) | kAhead, 0u, {}, stream);
}

// Gate, up and the gated unit (pdk_moe_prep_act_f4n has its formula) in one launch: h f32 [max_blocks*bm][out_dim] in block
// order, rows of padding left alone.  The tables are older than the launch in front
// (pdk_mxfp4_moe_gemm_tc5_ahead).  The raw gate and up rows are never written: at 1024 tokens, 4 experts each, 2880 wide
// they were 94 MB out and 94 MB back in.
PDK_EXPORT int pdk_mxfp4_moe_gate_up_tc5(const void* gate_data, const void* gate_sf, const void* gate_meta, const void* gate_bias,
                                         const void* up_data, const void* up_sf, const void* up_meta, const void* up_bias, void* h,
                                         const void* xq, const void* xs, const void* xstep, const void* block_expert,
                                         const void* sorted_row, uint32_t in_dim, uint32_t out_dim, uint32_t n_expert, uint32_t bm,
                                         uint32_t max_blocks, float alpha, float limit, float up_add, void* stream) {
    if (!pdk_aligned(gate_meta, 8) || !gate_meta || !up_meta || !up_data) return cudaErrorInvalidValue;
    return gemm_impl({gate_data, gate_sf, gate_bias, (const float*)gate_meta + 1}, {up_data, up_sf, up_bias, (const float*)up_meta + 1},
                     h, nullptr, {xq, xs, xstep, block_expert, sorted_row, nullptr, nullptr}, in_dim, out_dim, n_expert, bm, max_blocks,
                     1u, moe_gemm::kGated | kAhead, 0u, {alpha, limit, up_add}, stream);
}

// ---- NVFP4 expert planes (crates/paddock-engine/src/gpu/types.rs:176-226: data [expert*rows][in/2],
// scale e4m3 [expert*rows][in/16], scale2 f32 [expert]) on the same grouped GEMM.  No counterpart slot
// is served: the reference's NVFP4 MoE kernels take its Tiled64 / CutBlk plane orders.

// scale -> tiled records [n_expert][ceil(rows/128)][ceil(in_dim/256)][2048].  in_dim % 64 == 0.
PDK_EXPORT int pdk_nvf4_moe_tile_scales(const void* scale, void* tiled, uint32_t rows, uint32_t in_dim,
                                        uint32_t n_expert, void* stream) {
    if (rows == 0 || n_expert == 0) return 0;
    if (in_dim == 0 || (in_dim & 63u) != 0u || !pdk_aligned(tiled, 16) || !pdk_aligned(scale, 4))
        return cudaErrorInvalidValue;
    const uint32_t row_tiles = (rows + 127u) / 128u, num_kb = (in_dim + 255u) >> 8;
    const uint32_t words = row_tiles * num_kb * 512u;
    nvf4_moe_tile_scales_kernel<<<dim3((words + 255u) / 256u < 64u ? (words + 255u) / 256u : 64u, n_expert), 256, 0,
                                  (cudaStream_t)stream>>>((const uint8_t*)scale, (uint32_t*)tiled, rows, in_dim >> 4,
                                                          row_tiles, num_kb);
    return pdk_launch_status();
}

// pdk_mxfp4_moe_gemm_tc5 with NVFP4 planes: w*_sf from pdk_nvf4_moe_tile_scales, w*_scale2 f32 [n_expert],
// term rows from pdk_moe_prep_act_f4n.
PDK_EXPORT int pdk_nvf4_moe_gemm_tc5(const void* w0_data, const void* w0_sf, const void* w0_scale2, const void* w0_bias,
                                     void* out0, const void* w1_data, const void* w1_sf, const void* w1_scale2,
                                     const void* w1_bias, void* out1, const void* xq, const void* xs, const void* xstep,
                                     const void* block_expert, const void* sorted_row, const void* sorted_slot,
                                     const void* topk_w, uint32_t in_dim, uint32_t out_dim, uint32_t n_expert,
                                     uint32_t bm, uint32_t max_blocks, uint32_t n_active, uint32_t scatter,
                                     void* stream) {
    if (w0_scale2 == nullptr || (w1_data && w1_scale2 == nullptr)) return cudaErrorInvalidValue;
    return gemm_impl({w0_data, w0_sf, w0_bias, (const float*)w0_scale2}, {w1_data, w1_sf, w1_bias, (const float*)w1_scale2}, out0,
                     out1, {xq, xs, xstep, block_expert, sorted_row, sorted_slot, topk_w}, in_dim, out_dim, n_expert, bm, max_blocks,
                     n_active, scatter ? moe_gemm::kScatter : moe_gemm::kPlain, 1u, {}, stream);
}

PDK_EXPORT int pdk_nvf4_moe_gemm_tc5_ahead(const void* w0_data, const void* w0_sf, const void* w0_scale2, const void* w0_bias,
                                     void* out0, const void* w1_data, const void* w1_sf, const void* w1_scale2,
                                     const void* w1_bias, void* out1, const void* xq, const void* xs, const void* xstep,
                                     const void* block_expert, const void* sorted_row, const void* sorted_slot,
                                     const void* topk_w, uint32_t in_dim, uint32_t out_dim, uint32_t n_expert,
                                     uint32_t bm, uint32_t max_blocks, uint32_t n_active, uint32_t scatter,
                                     void* stream) {
    if (w0_scale2 == nullptr || (w1_data && w1_scale2 == nullptr)) return cudaErrorInvalidValue;
    return gemm_impl({w0_data, w0_sf, w0_bias, (const float*)w0_scale2}, {w1_data, w1_sf, w1_bias, (const float*)w1_scale2}, out0,
                     out1, {xq, xs, xstep, block_expert, sorted_row, sorted_slot, topk_w}, in_dim, out_dim, n_expert, bm, max_blocks,
                     n_active, (scatter ? moe_gemm::kScatter : moe_gemm::kPlain) | kAhead, 1u, {}, stream);
}

PDK_EXPORT int pdk_nvf4_moe_gate_up_tc5(const void* gate_data, const void* gate_sf, const void* gate_scale2, const void* gate_bias,
                                        const void* up_data, const void* up_sf, const void* up_scale2, const void* up_bias, void* h,
                                        const void* xq, const void* xs, const void* xstep, const void* block_expert,
                                        const void* sorted_row, uint32_t in_dim, uint32_t out_dim, uint32_t n_expert, uint32_t bm,
                                        uint32_t max_blocks, float alpha, float limit, float up_add, void* stream) {
    if (!gate_scale2 || !up_scale2 || !up_data) return cudaErrorInvalidValue;
    return gemm_impl({gate_data, gate_sf, gate_bias, (const float*)gate_scale2}, {up_data, up_sf, up_bias, (const float*)up_scale2}, h,
                     nullptr, {xq, xs, xstep, block_expert, sorted_row, nullptr, nullptr}, in_dim, out_dim, n_expert, bm, max_blocks, 1u,
                     moe_gemm::kGated | kAhead, 1u, {alpha, limit, up_add}, stream);
}

// ---------------------------------------------------------------- W4A16 decode GEMV on the same kernels
// pd_nvf4_gemv (slot 394) hands over the checkpoint's NVFP4 plane (row-major scales) and one f32
// activation vector.  On the tensor-core route the vector becomes four NVFP4 term rows (one
// "block" of one token) in a library-resident scratch slice and the grouped GEMM runs with one
// expert, gathering the weight scales from the row-major plane.  Two launches; the plane is
// streamed once at 4.5 bits per weight.  One scratch slice per stream for the first two streams
// that come here (the pack allocates nothing); other callers get -1 and take the plain kernel.
namespace {
constexpr uint32_t kGemvMaxK = 16384;
constexpr size_t kGemvXs = 128, kGemvXq = kGemvXs + (size_t)(kGemvMaxK / 256u) * 2048u;
constexpr size_t kGemvSlice = ((kGemvXq + 32u * (kGemvMaxK / 2u)) + 1023u) & ~(size_t)1023u;
constexpr int kGemvLanes = 2;
__device__ __align__(1024) uint8_t g_gemv_scratch[kGemvLanes][kGemvSlice];

PDK_SLICE_TABLE(gemv_slice_table, g_gemv_scratch, kGemvSlice, kGemvLanes);
uint8_t* gemv_slice(cudaStream_t st) { return gemv_slice_table.slice(st); }
}  // namespace

// 0 / cudaError_t, or -1 when the route does not apply (in_dim not a multiple of 64 or above 16384,
// no scratch slice for this stream) and the caller should use its own kernel.
int pdk_nvf4_gemv_tc5(const void* data, const void* scale, const void* bias, const void* x, void* y, float scale2,
                      uint32_t in_dim, uint32_t out_dim, cudaStream_t st) {
    if ((in_dim & 63u) != 0u || in_dim > kGemvMaxK || !pdk_aligned(data, 16) || !pdk_aligned(scale, 4) ||
        !pdk_aligned(x, 16))
        return -1;
    uint8_t* sl = gemv_slice(st);
    if (sl == nullptr) return -1;
    uint32_t* tables = reinterpret_cast<uint32_t*>(sl);          // sorted_row[8], block_expert[1], f32 scale2
    float* xstep = reinterpret_cast<float*>(sl + 64);
    uint8_t* xs = sl + kGemvXs;
    uint8_t* xq = sl + kGemvXq;
    PrepArgs pa{};
    pa.x = (const float*)x; pa.xq = xq; pa.xs = xs; pa.xstep = xstep;
    pa.dim = in_dim; pa.bm = 8u; pa.mode = 3u; pa.natural = 1u; pa.tables = tables; pa.table_scale2 = scale2;
    if (int rc = pdk_launch_pdl(moe_prep_f4_kernel, dim3(8), dim3(prep_threads(in_dim)), 0, st, pa))
        return rc;
    const uint32_t kbytes = in_dim >> 1;
    CUtensorMap tw, tx;
    if (int rc = pdk_make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, data, kbytes, out_dim, kbytes, BKB, BM)) return rc;
    if (int rc = pdk_make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, kbytes, 32u, kbytes, BKB, 32u)) return rc;
    moe_gemm::Args a{};
    a.w_sf[0] = a.w_sf[1] = (const uint8_t*)scale;
    a.scale2[0] = a.scale2[1] = reinterpret_cast<const float*>(tables) + 9;
    a.bias[0] = (const float*)bias;
    a.out[0] = (float*)y;
    a.x_sf = xs; a.xstep = xstep;
    a.block_expert = tables + 8; a.sorted_row = tables;
    a.in_dim = in_dim; a.out_dim = out_dim; a.max_blocks = 1u; a.n_planes = 1u; a.n_active = 1u;
    a.err_word = pdk_error_word();
    return moe_gemm::launch<4, 1, moe_gemm::kPlain, 4, true>(tw, tw, tx, a, st);
}
