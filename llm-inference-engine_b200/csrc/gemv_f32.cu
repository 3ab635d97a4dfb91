#include <stdlib.h>

#include "gemv_inst.cuh"
#include "gemv_sr.cuh"
namespace b200 {
int launch_gemv_nk_f32(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_t<float, false>(a, fmt, swiglu, st); }
int launch_gemv_nk_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_nk_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_mma_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_mma_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_qd_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_qd_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_rs_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_rs_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st);
int launch_gemv_nk(const GemvArgs &a, int dtype, int fmt, bool swiglu, cudaStream_t st) {
    if (swiglu && (a.N != 2 * a.inter)) {
        set_error("gemv: SwiGLU epilogue needs N == 2*inter");
        return B200_ERR_INVALID_ARG;
    }
    const bool b16 = dtype == B200_BF16 || dtype == B200_F16;
    // up to 8 tokens of INT4 weights, up to 16 of dense rows of at most 3072 k: straight from global memory into registers (gemv_qd.cuh, with both sides' times)
    if (a.finish && fmt != WF_DENSE) return B200_ERR_UNSUPPORTED;
    if (b16 && fmt != WF_FP8) {
        const int rc = dtype == B200_BF16 ? launch_gemv_qd_bf16(a, fmt, swiglu, st) : launch_gemv_qd_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    if (a.norm && fmt == WF_INT4) return B200_ERR_UNSUPPORTED;  // (no other kernel keeps the norm kernel's bits)
    if (a.finish) return B200_ERR_UNSUPPORTED;  // (in gemv_rs.cuh the ending cost every other caller 0.6 to 1.1 %)
    // 16-bit activations, no prologue: 2..16 tokens, and one token of FP8 weights, past which the weights stream with the activations in registers
    // (gemv_rs.cuh).  One dense token keeps the SIMT kernel and its fused norm: its weights alone fill the memory pipe, and the norm launch would come on
    // top.  One FP8 token, 4 layers, norm kernel + gemv_rs against the kernel with the fused norm that was here (ctx 1024): 7B size 238 us against 245, 70B-shaped
    // shard 204 against 230, 2048-wide 130 against 142.
    if (b16 && (a.M >= 2 || fmt != WF_DENSE) && a.M <= 16) {
        const int rc = dtype == B200_BF16 ? launch_gemv_rs_bf16(a, fmt, swiglu, st) : launch_gemv_rs_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    // what its ring leaves out (rows of more than 4096 k with so many outputs that their sums fill the SM): activations in shared memory (gemv_mma.cuh)
    if (b16 && (a.M >= 2 || fmt != WF_DENSE) && a.M <= 16) {
        const int rc = dtype == B200_BF16 ? launch_gemv_mma_bf16(a, fmt, swiglu, st) : launch_gemv_mma_f16(a, fmt, swiglu, st);
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    if (a.M > 4) return B200_ERR_UNSUPPORTED;
    // one token of short rows (fp32: up to four), norm in front or not: whole rows per warp (gemv_sr.cuh, with both sides' times)
    {
        const int rc = dtype == B200_F32 ? launch_gemv_sr_t<float>(a, fmt, swiglu, st) : dtype == B200_BF16 ? launch_gemv_sr_t<__nv_bfloat16>(a, fmt, swiglu, st) : dtype == B200_F16 ? launch_gemv_sr_t<__half>(a, fmt, swiglu, st) : B200_ERR_UNSUPPORTED;
        if (rc != B200_ERR_UNSUPPORTED) return rc;
    }
    switch (dtype) {
        case B200_F32: return launch_gemv_nk_f32(a, fmt, swiglu, st);
        case B200_F16: return launch_gemv_nk_f16(a, fmt, swiglu, st);
        case B200_BF16: return launch_gemv_nk_bf16(a, fmt, swiglu, st);
    }
    set_error("gemv: unknown dtype %d", dtype);
    return B200_ERR_INVALID_ARG;
}
}
