#include <stdlib.h>

#include "gemv_inst.cuh"
namespace b200 {
int launch_gemv_nk_f32(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_t<float, false>(a, fmt, swiglu, st); }
int launch_gemv_nk_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_nk_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_mma_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_mma_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_q_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_q_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_rs_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_rs_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_nk(const GemvArgs &a, int dtype, int fmt, bool swiglu, cudaStream_t st) {
    if (swiglu && (a.N != 2 * a.inter)) {
        set_error("gemv: SwiGLU epilogue needs N == 2*inter");
        return B200_ERR_INVALID_ARG;
    }
    const bool b16 = dtype == B200_BF16 || dtype == B200_F16;
    // 16-bit activations, 2..16 tokens, no prologue: the weights stream past activations in registers (gemv_rs.cuh; one token of quantised weights keeps the
    // kernel with the prologue below, one dense token the SIMT kernel: a single row leaves the matrix instructions seven eighths empty)
    if (b16 && a.M >= 2 && a.M <= 16) {
        const int rc = dtype == B200_BF16 ? launch_gemv_rs_bf16(a, fmt, swiglu, st) : launch_gemv_rs_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    // shapes whose ring does not fit beside it: activations in shared memory (gemv_mma.cuh)
    if (b16 && a.M >= 2 && a.M <= 16) {
        const int rc = dtype == B200_BF16 ? launch_gemv_mma_bf16(a, fmt, swiglu, st) : launch_gemv_mma_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    // weight-only quantised, 16-bit activations, one token (more where the kernels above refuse): dequant into mma fragments with the SIMT GEMV's fused
    // prologue (gemv_q.cuh)
    if (b16 && fmt != WF_DENSE && a.M <= 8) {
        const int rc = dtype == B200_BF16 ? launch_gemv_q_bf16(a, fmt, swiglu, st) : launch_gemv_q_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    if (a.M > 4) return B200_ERR_UNSUPPORTED;
    switch (dtype) {
        case B200_F32: return launch_gemv_nk_f32(a, fmt, swiglu, st);
        case B200_F16: return launch_gemv_nk_f16(a, fmt, swiglu, st);
        case B200_BF16: return launch_gemv_nk_bf16(a, fmt, swiglu, st);
    }
    set_error("gemv: unknown dtype %d", dtype);
    return B200_ERR_INVALID_ARG;
}
}
