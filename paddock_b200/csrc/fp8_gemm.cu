// fp8_gemm.cu - row-scaled e4m3 GEMM: entry points and the choice of kernel.
//
//   y[t][n] = ( sum_k e4m3(Xq[t][k]) * e4m3(W[n][k]) ) * xs[t] * ws[n]
//
// Prompts with enough 256 x 256 tiles run on pairs of SMs (fp8_gemm2.cu), everything else - decode
// widths, narrow planes - on the K-split kernel (splitk_gemm.cu).  Scales touch only the epilogue: the
// accumulation is the exact product sum.
#include <cstdlib>

#include "tc5.cuh"

// fp8_gemm2.cu: the same GEMM on pairs of SMs
int pdk_f8row_gemm_pair_f32(const void*, const void*, const void*, const void*, void*, uint32_t, uint32_t, uint32_t, cudaStream_t);
int pdk_f8row_gemm_pair_bf16(const void*, const void*, const void*, const void*, void*, uint32_t, uint32_t, uint32_t, cudaStream_t);
// splitk_gemm.cu
bool pdk_prefer_pair(uint32_t batch, uint32_t out_dim, uint32_t row_bytes, bool nvf4);
int pdk_f8row_gemm_splitk(const void* data, const void* w_scale, const void* xq, const void* x_scale, void* y, uint32_t in_dim,
                          uint32_t out_dim, uint32_t batch, bool bf16, cudaStream_t st);

namespace {

// PDK_F8_PAIR=0 keeps every call on the K-split kernel (A/B switch, read once).
bool pair_enabled() {
    static const bool v = [] {
        const char* e = getenv("PDK_F8_PAIR");
        return !(e && e[0] == '0');
    }();
    return v;
}

template <typename TO>
int launch(const void* data, const void* w_scale, const void* xq, const void* x_scale, void* y, uint32_t in_dim,
           uint32_t out_dim, uint32_t batch, cudaStream_t st) {
    if (out_dim == 0 || batch == 0) return 0;
    if (in_dim == 0 || (in_dim & 15u) != 0u) return cudaErrorInvalidValue;
    if (!pdk_aligned(data, 16) || !pdk_aligned(xq, 16) || !pdk_aligned(w_scale, 4) || !pdk_aligned(x_scale, 4) ||
        !pdk_aligned(y, sizeof(TO)))
        return cudaErrorInvalidValue;
    if (pair_enabled() && pdk_prefer_pair(batch, out_dim, in_dim, false)) {
        if constexpr (sizeof(TO) == 4) return pdk_f8row_gemm_pair_f32(data, w_scale, xq, x_scale, y, in_dim, out_dim, batch, st);
        else return pdk_f8row_gemm_pair_bf16(data, w_scale, xq, x_scale, y, in_dim, out_dim, batch, st);
    }
    return pdk_f8row_gemm_splitk(data, w_scale, xq, x_scale, y, in_dim, out_dim, batch, sizeof(TO) == 2u, st);
}

}  // namespace

// slot 184, packs/cuda/src/gemm/dense_f8_decode.cuh:4638-4722: f32 output
PDK_EXPORT int pd_f8row_gemm(const void* data, const void* w_rowscale, const void* xq, const void* x_rowscale,
                             void* y, uint32_t in_dim, uint32_t out_dim, uint32_t batch, void* stream) {
    return launch<float>(data, w_rowscale, xq, x_rowscale, y, in_dim, out_dim, batch, (cudaStream_t)stream);
}

// slot 855, packs/cuda/src/gemm/dense_nvf4_tc5.cuh:1480-1515: same contract
PDK_EXPORT int pd_f8row_gemm_tc5x(const void* data, const void* w_rowscale, const void* xq, const void* x_rowscale,
                                  void* y, uint32_t in_dim, uint32_t out_dim, uint32_t batch, void* stream) {
    return launch<float>(data, w_rowscale, xq, x_rowscale, y, in_dim, out_dim, batch, (cudaStream_t)stream);
}

// No slot: the same GEMM with bf16 output (halves the store traffic of a prefill)
PDK_EXPORT int pdk_f8row_gemm_bf16(const void* data, const void* w_rowscale, const void* xq, const void* x_rowscale,
                                   void* y, uint32_t in_dim, uint32_t out_dim, uint32_t batch, void* stream) {
    return launch<__nv_bfloat16>(data, w_rowscale, xq, x_rowscale, y, in_dim, out_dim, batch, (cudaStream_t)stream);
}
