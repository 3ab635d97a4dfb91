// gemv_sr.cuh -- the decode-shaped linear of short dense rows for one token (fp32: up to four) with its norm in front: y[M,N] = norm(x)[M,K] * W^T, W packed [N,K].
// Reference: launchLinearGemm (src/kernels/linear.cu:10-87) behind launchFusedAddBiasResidualAndRMSNorm / launchRMSNorm (src/layers/self_decoder.cpp:24-122).
//
// What bounds it: the launch itself.  A model of 1024 or 2048 channels has 4 to 20 MB per linear, 1 to 3 us of HBM time; gemv.cuh splits a row over eight warps
// (4 numbers of 1024 for a lane), hands every pair of rows through two barriers to a reducer warp and starts with a ring's worth of barriers and bulk copies.
// Here a warp owns whole rows, two at a time (SwiGLU: a gate row and its up row), and streams them into registers; nothing is shared between warps but the
// activations, and the first 8 KB of every warp are on their way before griddepcontrol.wait.  Units are dealt over the SMs first, then over an SM's warps.
// A lane adds 4 (16-bit: 8) chains of products, the warp adds the lanes: fp32 multiply-adds in a fixed order (deterministic).  Neither that order nor the norm's
// depends on the number of tokens: a token's result has the same bits whatever is beside it.
// fp32 sums: relative to 64 bits 8.7e-8 / 8.9e-8 / 9.0e-8 at 1024 / 1408 / 1536 k (8192 rows of normal numbers; gemv.cuh 9.4e-8 / 9.1e-8 / 9.2e-8; all of a lane's
// products of one chain in a row 9.1e-8 / 9.5e-8 / 9.6e-8, and 2 to 4 tokens 1 to 4 % less time).
// Measured (four layers, context 129, us per step, gemv.cuh -> here): fp32, 1024 wide, feed-forward 1408, 1 / 2 / 3 / 4 tokens 96 / 141 / 175 / 194 -> 81 / 96 / 122 / 130;
// bf16, 2048 wide, 1 token 133 -> 102.  With gemv.cuh's prologue, one token's norm after another, 2 and 4 fp32 tokens gained little: 184 -> 178 and 238 -> 239, another context.
#pragma once
#include "gemv.cuh"

namespace b200 {

constexpr int kSrWarps = 8, kSrSlot = 4, kSrRing = 2;  // 16-byte pieces of a row per lane and slot, slots in flight per warp

template <typename T, bool kSwiGLU, int MB>
__global__ void __launch_bounds__(kSrWarps * 32, 2)
gemv_sr_kernel(const GemvArgs a) {
    constexpr int V = Elem<T>::kVec, C = V / 4;
    extern __shared__ __align__(16) float xs[];  // [MB][K]; 16-bit: the halves of a warp's 256 numbers apart, so that 16-byte reads of neighbours touch
    __shared__ float red[MB][kSrWarps];
    GemvArgs b = a;
    b.tp.world = 0;  // (never set here: the exchange's registers are not wanted)
    const int K = a.K, N = a.N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pieces = K / (32 * V), units = kSwiGLU ? a.inter : (N + 1) / 2, step = gridDim.x * kSrWarps;
    const int slots = (pieces + kSrSlot - 1) / kSrSlot;
    auto row = [&](int u, int r) { return kSwiGLU ? u + r * a.inter : min(2 * u + r, N - 1); };

    struct Slot {
        uint4 w[kSrSlot][2];
    };
    Slot ring[kSrRing];
    int lu = warp * gridDim.x + blockIdx.x, lp = 0;  // the slot to load next
    auto load = [&](Slot &s) {
        if (lu >= units) return;
#pragma unroll
        for (int j = 0; j < kSrSlot; ++j) {
            const int p = min(lp * kSrSlot + j, pieces - 1);  // (past the row: its last piece, not used)
#pragma unroll
            for (int r = 0; r < 2; ++r) s.w[j][r] = ld_stream_v4(reinterpret_cast<const T *>(a.w) + (size_t)row(lu, r) * K + (p * 32 + lane) * V);
        }
        if (++lp == slots) lp = 0, lu += step;
    };
#pragma unroll
    for (int i = 0; i < kSrRing; ++i) load(ring[i]);
    // the norm's weights do not depend on the kernel in front either
    T *const gs = reinterpret_cast<T *>(xs + (size_t)MB * K);
    const bool norm = a.norm && a.gamma;
    if (norm)
        for (int i = threadIdx.x; i < K / V; i += kSrWarps * 32) st_v4(gs + (size_t)i * V, ld_v4(reinterpret_cast<const T *>(a.gamma) + (size_t)i * V));
    pdl_wait();
    pdl_launch_dependents();
    {   // Activations, one token per 8 / MB warps: x (+ residual) -> T; residual_out <- that (CTA 0); (+ bias) -> T; norm, rounded where the un-fused kernels round
        constexpr int TT = kSrWarps * 32 / MB;  // threads of a token
        const int m = threadIdx.x / TT, t = threadIdx.x - m * TT;
        float ss[MB] = {};  // squares, summed as by 8 warps whatever MB is: a token's norm has the same bits beside any others
        auto place = [&](int i, int c) { return reinterpret_cast<float4 *>(xs + (size_t)m * K + (i >> 5) * 32 * V + c * 128 + (i & 31) * 4); };
        if (m < a.M) {
#pragma unroll (4 / MB)
            for (int i0 = t; i0 < K / V; i0 += MB * TT) {
#pragma unroll
                for (int w = 0; w < MB; ++w) {
                    const int i = i0 + w * TT;
                    if (i >= K / V) break;
                    float f[V];
                    gemv_prenorm_vec<T>(b, 0u, m, i, f, true);
#pragma unroll
                    for (int j = 0; j < V; ++j) ss[w] = fmaf(f[j], f[j], ss[w]);
#pragma unroll
                    for (int c = 0; c < C; ++c) *place(i, c) = make_float4(f[4 * c], f[4 * c + 1], f[4 * c + 2], f[4 * c + 3]);
                }
            }
        }
        if (norm) {  // (every thread scales what it has written)
#pragma unroll
            for (int w = 0; w < MB; ++w) {
                ss[w] = warp_sum(ss[w]);
                if (lane == 0) red[m][w * (kSrWarps / MB) + warp % (kSrWarps / MB)] = ss[w];
            }
            __syncthreads();
            float total = 0.0f;
#pragma unroll
            for (int w = 0; w < kSrWarps; ++w) total += red[m][w];
            const float rs = rsqrtf(total / (float)K + a.eps);
            if (m < a.M) {
#pragma unroll 4
                for (int i = t; i < K / V; i += TT) {
                    float f[V], g[V];
                    unpack16<T>(ld_v4(gs + (size_t)i * V), g);
#pragma unroll
                    for (int c = 0; c < C; ++c) load_vec<4>(reinterpret_cast<const float *>(place(i, c)), f + 4 * c);
#pragma unroll
                    for (int j = 0; j < V; ++j) f[j] = (f[j] * g[j]) * rs;
                    round_vec<T>(f);
#pragma unroll
                    for (int c = 0; c < C; ++c) *place(i, c) = make_float4(f[4 * c], f[4 * c + 1], f[4 * c + 2], f[4 * c + 3]);
                }
            }
        }
    }
    __syncthreads();

    int u = warp * gridDim.x + blockIdx.x, at = 0;
    float acc[MB][2][V] = {};
    // fp32: a slot's products are summed before they join the row's, chains of 4 and of K / 512 terms instead of one of K / 128
    constexpr bool kSplit = sizeof(T) == 4;
    while (u < units) {
#pragma unroll
        for (int i = 0; i < kSrRing; ++i) {
            if (u >= units) break;
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                if (MB > 1 && m >= a.M) break;
                float part[2][V] = {};
                float(&to)[2][V] = kSplit ? part : acc[m];
#pragma unroll
                for (int j = 0; j < kSrSlot; ++j) {
                    if (at * kSrSlot + j >= pieces) break;
                    float w[2][V], x[V];
                    unpack16<T>(ring[i].w[j][0], w[0]), unpack16<T>(ring[i].w[j][1], w[1]);
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        load_vec<4>(xs + (size_t)m * K + (at * kSrSlot + j) * 32 * V + c * 128 + lane * 4, x + 4 * c);
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int v = 0; v < V; ++v) to[r][v] = fmaf(w[r][v], x[v], to[r][v]);
                }
                if constexpr (kSplit) {
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int v = 0; v < V; ++v) acc[m][r][v] += part[r][v];
                }
            }
            load(ring[i]);
            if (++at < slots) continue;
            at = 0;
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                if (MB > 1 && m >= a.M) break;
                float s[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
#pragma unroll
                    for (int o = V / 2; o > 0; o >>= 1)
#pragma unroll
                        for (int v = 0; v < o; ++v) acc[m][r][v] += acc[m][r][v + o];
                    s[r] = warp_sum(acc[m][r][0]);
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[m][r][v] = 0.0f;
                }
                if constexpr (kSwiGLU) {
                    const float g = round_to<T>(s[0]), up = round_to<T>(s[1]);  // (the un-fused reference stores gate / up in T before SiLU reads them)
                    if (lane == 0) {
                        const float v = (g / (1.0f + expf(-g))) * up;
                        if (a.y_f32) reinterpret_cast<float *>(a.y)[(size_t)m * a.inter + u] = v;
                        else reinterpret_cast<T *>(a.y)[(size_t)m * a.inter + u] = Elem<T>::from_f(v);
                    }
                } else if (lane < 2 && 2 * u + lane < N) {
                    const float v = lane ? s[1] : s[0];
                    if (a.y_f32) reinterpret_cast<float *>(a.y)[(size_t)m * N + 2 * u + lane] = v;
                    else reinterpret_cast<T *>(a.y)[(size_t)m * N + 2 * u + lane] = Elem<T>::from_f(v);
                }
            }
            u += step;
        }
    }
}

// The rows' length says whether a launch is mostly its start -- it alone, so that a token's bits do not depend on those beside it: one fp32 token of 2048 / 2688 k has
// 16 to 44 MB per linear, for which gemv.cuh holds 192 KB per SM in flight (four layers 188 us there, 194 here), so 2 to 4 of them run there too (four layers,
// context 129, 2 / 4 tokens 208 / 286 us there, 177 / 238 here).
// B200_ERR_UNSUPPORTED (no error text): other formats, long rows, rows that are no whole number of a warp's pieces, tensor-parallel ends
template <typename T>
static int launch_gemv_sr_t(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) {
    if (fmt != WF_DENSE || a.M < 1 || a.M > (sizeof(T) == 4 ? 4 : 1) || a.K > (sizeof(T) == 4 ? 1536 : 3072) || a.K % (32 * Elem<T>::kVec) != 0 || !all_aligned16({a.w, a.x})) return B200_ERR_UNSUPPORTED;
    if (a.tp.world > 1 || a.push.n > 0 || (a.norm && !all_aligned16({a.res_in, a.res_out, a.bias, a.gamma}))) return B200_ERR_UNSUPPORTED;
    const int units = swiglu ? a.inter : (a.N + 1) / 2, sms = sm_count();
    const dim3 grid(units <= sms ? std::max(1, units) : units <= sms * kSrWarps ? sms : 2 * sms);
    const size_t smem = (size_t)(a.M <= 2 ? a.M : 4) * a.K * sizeof(float) + (size_t)a.K * sizeof(T);
    auto go = [&](auto kern) -> int {
        if (!allow_smem(reinterpret_cast<const void *>(kern), 64 * 1024, 100 * 1024)) return cuda_status("gemv_sr cudaFuncSetAttribute");
        launch_pdl(kern, grid, dim3(kSrWarps * 32), smem, st, true, a);
        return cuda_status("gemv_sr launch");
    };
    if constexpr (sizeof(T) == 4) {
        if (a.M == 2) return swiglu ? go(gemv_sr_kernel<T, true, 2>) : go(gemv_sr_kernel<T, false, 2>);
        if (a.M > 2) return swiglu ? go(gemv_sr_kernel<T, true, 4>) : go(gemv_sr_kernel<T, false, 4>);
    }
    return swiglu ? go(gemv_sr_kernel<T, true, 1>) : go(gemv_sr_kernel<T, false, 1>);
}

}  // namespace b200
