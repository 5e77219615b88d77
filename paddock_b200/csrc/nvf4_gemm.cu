// nvf4_gemm.cu - NVFP4 x NVFP4 GEMM on tcgen05 with hardware block scaling: entry points and the choice
// of kernel.
//
//   y[t][n] = scale2 * sum over 16-element blocks b of
//             e4m3(ws[n][b]) * e4m3(xs[t][b]) * sum_{k in b} e2m1(W[n][k]) * e2m1(X[t][k])   (+ bias[n])
//
// tcgen05.mma kind::mxf4nvf4 reads packed e2m1 operands straight from shared memory (K = 64 per
// instruction) and applies both operands' per-16 UE4M3 scales from tensor memory, so no weight ever
// passes through a register.  Prompts with enough 256 x 256 tiles run on pairs of SMs (nvf4_gemm2.cu),
// everything else - decode widths, narrow planes - on the K-split kernel (splitk_gemm.cu).
#include <cstdlib>

#include "nvf4_tc5.cuh"

// nvf4_gemm2.cu: prefill widths on pairs of SMs
int pdk_nvf4_gemm_pair_f32(const void*, const void*, const void*, const void*, const void*, void*, float, uint32_t, uint32_t,
                           uint32_t, cudaStream_t);
int pdk_nvf4_gemm_pair_bf16(const void*, const void*, const void*, const void*, const void*, void*, float, uint32_t, uint32_t,
                            uint32_t, cudaStream_t);

// nvf4_elem.cu; plane: the records are a weight plane's
int pdk_nvf4_tile_scales(const void* scale, void* tiled, uint32_t in_dim, uint32_t out_dim, bool plane, cudaStream_t st);
// splitk_gemm.cu
bool pdk_prefer_pair(uint32_t batch, uint32_t out_dim, uint32_t row_bytes, bool nvf4);
int pdk_nvf4_gemm_splitk(const void* data, const void* scale_tiled, const void* bias, const void* xq, const void* xs, void* y,
                         float scale2, uint32_t in_dim, uint32_t out_dim, uint32_t batch, bool bf16, cudaStream_t st);

namespace {

using namespace nvf4tc5;

// PDK_NVF4_PAIR=0 keeps every call on the K-split kernel (A/B switch, read once).
bool pair_enabled() {
    static const bool v = [] {
        const char* e = getenv("PDK_NVF4_PAIR");
        return !(e && e[0] == '0');
    }();
    return v;
}

// Scratch for the pair kernel's re-tiled activation scales: a 4-byte gather per token row and 64
// K-elements costs the L2 as many requests again as the operand boxes, one 2 KB bulk copy per slab does
// not.  The buffer lives in the library (the pack allocates nothing at run time); one slice per stream,
// for the first kXsfLanes streams that make such calls - further streams, and calls too large for a
// slice, take the K-split kernel's whole tiles, which bring the scales through registers: 8192 tokens, K = 17408, N = 4096
// (9.4 MB of records) 300 us, 4096 tokens, K = N = 5120 66 us where the pair kernel takes 59.
constexpr size_t kXsfSliceBytes = 8u << 20;  // batch * in_dim / 16 bytes, padded to 128 tokens
constexpr int kXsfLanes = 2;
__device__ __align__(1024) uint8_t g_xsf_scratch[kXsfLanes][kXsfSliceBytes];

PDK_SLICE_TABLE(xsf_slice_table, g_xsf_scratch, kXsfSliceBytes, kXsfLanes);
uint8_t* xsf_slice(cudaStream_t st, size_t need) {
    if (need > kXsfSliceBytes) return nullptr;
    return xsf_slice_table.slice(st);
}

template <typename TO>
int launch(const void* data, const void* scale_tiled, const void* bias, const void* xq, const void* xs, void* y,
           float scale2, uint32_t in_dim, uint32_t out_dim, uint32_t batch, cudaStream_t st) {
    if (out_dim == 0 || batch == 0) return 0;
    if (in_dim == 0 || (in_dim & 255u) != 0u) return cudaErrorInvalidValue;
    if (!pdk_aligned(data, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(scale_tiled, 16) || !pdk_aligned(xs, 4) ||
        !pdk_aligned(y, sizeof(TO)))
        return cudaErrorInvalidValue;
    if (pair_enabled() && pdk_prefer_pair(batch, out_dim, in_dim >> 1, true)) {
        const size_t need = (size_t)((batch + 127u) / 128u) * (in_dim >> 8) * kSfBytes;
        if (uint8_t* xt = xsf_slice(st, need)) {
            if (int rc = pdk_nvf4_tile_scales(xs, xt, in_dim, batch, false, st)) return rc;
            if constexpr (sizeof(TO) == 4) return pdk_nvf4_gemm_pair_f32(data, scale_tiled, bias, xq, xt, y, scale2, in_dim, out_dim, batch, st);
            else return pdk_nvf4_gemm_pair_bf16(data, scale_tiled, bias, xq, xt, y, scale2, in_dim, out_dim, batch, st);
        }
    }
    return pdk_nvf4_gemm_splitk(data, scale_tiled, bias, xq, xs, y, scale2, in_dim, out_dim, batch, sizeof(TO) == 2u, st);
}

}  // namespace

// slot 852, packs/cuda/src/gemm/dense_nvf4_tc5.cuh:1216-1263.  `part` / `part_floats`
// (the reference's K-split partial planes) are accepted and unused: the K split here
// meets in distributed shared memory.
PDK_EXPORT int pd_nvf4_gemm_tc5w(const void* data, const void* scale_tiled, const void* bias, const void* xq,
                                 const void* xs, void* y, float scale2, uint32_t in_dim, uint32_t out_dim,
                                 uint32_t batch, void* part, uint64_t part_floats, void* stream) {
    (void)part;
    (void)part_floats;
    return launch<float>(data, scale_tiled, bias, xq, xs, y, scale2, in_dim, out_dim, batch, (cudaStream_t)stream);
}

// No slot: slot 852 with bf16 output.
PDK_EXPORT int pdk_nvf4_gemm_bf16(const void* data, const void* scale_tiled, const void* bias, const void* xq,
                                  const void* xs, void* y, float scale2, uint32_t in_dim, uint32_t out_dim,
                                  uint32_t batch, void* stream) {
    return launch<__nv_bfloat16>(data, scale_tiled, bias, xq, xs, y, scale2, in_dim, out_dim, batch,
                                 (cudaStream_t)stream);
}
