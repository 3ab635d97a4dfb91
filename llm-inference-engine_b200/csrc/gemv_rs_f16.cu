#include "gemv_qd.cuh"
namespace b200 {
int launch_gemv_qd_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_qd_t<__half>(a, fmt, swiglu, st); }
int launch_gemv_rs_f16(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) { return launch_gemv_rs_t<__half>(a, fmt, swiglu, st); }
}
