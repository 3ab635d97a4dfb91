#include "gemv_qd.cuh"
namespace b200 {
int launch_gemv_qd_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_qd_t<__nv_bfloat16>(a, fmt, swiglu, st); }
int launch_gemv_rs_bf16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_rs_t<__nv_bfloat16>(a, fmt, swiglu, st); }
}
