// gemv_qd.cuh -- the decode-shaped linear for INT4 weights of 1..8 tokens and dense weights of short rows of 1..16, streamed from global memory STRAIGHT INTO
// REGISTERS: y[M,N] = x[M,K] * W^T, W packed [N,K], in groups of 128 k (W4A16) or dense 16-bit.
// Reference: launchLinearGemm (src/kernels/linear.cu:10-87) at the decode shapes of src/layers/self_attention.cpp:79-86,131-138, src/layers/ffn.cpp:105-139.
//
// What bounds it: latency and instructions, not the 0.6 to 7 us that a 7B layer's INT4 linears take to read.  In gemv_rs.cuh a unit of 16 rows passes a barrier,
// 16 warps with two quantisation groups each, a second barrier and one reducer warp, and the parameters of a unit are waited for where they are loaded.  Here
//   * a warp owns a slice of k of 16 weight rows and walks it in pairs of groups (dense: in groups) through a ring of registers: a pair's place is loaded again as
//     soon as it has been multiplied, up to 64 KB (dense: 128) in flight per SM without a barrier between a load and its use, and two groups' chains of products
//     keep the tensor pipe from waiting for its own results.  (K = 4096, N = 12288, where this takes 8.2 us: two buffers of four groups 10.6, one group at a time
//     in three CTAs per SM 9.2);
//   * 16 warps per SM, as one CTA where a row is long (a slice is then at least two pairs and the activations are staged once per SM), else as two CTAs, so that a
//     unit's sum does not stop all of them: K = 4096, N = 12288 8.3 us with two against 9.1 with one, K = 2048, N = 5376 3.1 against 4.6, K = 8192, N = 10240
//     14.5 against 13.3, K = 12288, N = 1536 7.3 against 5.7;
//   * the first weights and parameters are requested before griddepcontrol.wait; one __syncthreads per unit: the warps leave their tiles in one of two buffers,
//     the first threads add them in a fixed order (deterministic).
// Fragments, dequantisation and arithmetic are those of gemv_rs.cuh's quantised units: exact integers in f16, fp32 sums, the group's scale once per 128 k.
// Dense weights: a launch's start rather than its instructions; its CTAs wait for no barrier and no ring.  Their sums are shorter chains in the tensor cores than
// gemv_rs.cuh's (fp32 outputs of K = 4096: 1.08e-7 from 64 bits against 1.42e-7).
// (Codes multiplied as they are, as subnormal f16, with the zero points' part taken off afterwards, need five instructions instead of nine for eight weights and
// were no faster; the tensor cores align a product by its operands' exponents, so the codes' leading zeros cost bits of the sum.)
// Measured, us per launch in a chain, 1 / 4 / 8 tokens (gemv_rs -> here): K = 4096: N = 12288 11.3 / 11.9 / 12.5 -> 8.2 / 9.1 / 10.4, N = 4096
// 5.1 / 5.5 / 6.0 -> 4.2 / 5.1 / 6.1, N = 22016 16.9 / 17.5 / 18.0 -> 13.4 / 14.3 / 15.5; K = 11008, N = 4096 12.0 / 12.7 / 14.1 -> 9.4 / 10.5 / gemv_rs.
// Dense, 1 (gemv.cuh) / 8 / 16 tokens (gemv_rs.cuh -> here): K = 2048: N = 6176 7.4 / 7.6 / 9.0 -> 5.0 / 5.8 / 6.5, N = 2048 3.8 / 3.7 / 4.4 -> 2.5 / 2.9 / 3.4;
// K = 1024, N = 1536 3.2 / 2.8 / 3.3 -> 1.8 / 1.9 / 2.3.
#pragma once
#include "gemv_rs.cuh"

namespace b200 {

template <typename T> __device__ __forceinline__ void mma_any(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) mma_bf16(c, a0, a1, a2, a3, b0, b1);
    else mma_f16f16(c, a0, a1, a2, a3, b0, b1);
}

constexpr int kQdRows = 16;
constexpr int kQdRing = 2;              // slots of weights in flight per warp, see below
constexpr int kQdTileRow = 20;          // fp32 values of a token in a warp's tile: [8 NT tokens][16 rows + 4]
// dynamic shared memory of an SM's one CTA of 16 warps or two of 8, at most: what is in flight (64 KB, dense 128) needs L1 beside it
__host__ __device__ constexpr size_t qd_smem(int fmt, int warps) { return (size_t)(fmt == WF_INT4 ? 160 : 108) * 1024 * warps / 16; }
// groups of 128 k per slot: INT4 two of them (2 KB of 16 rows), dense weights one (4 KB)
__host__ __device__ constexpr int qd_groups(int fmt) { return fmt == WF_INT4 ? 2 : 1; }

template <typename T, int FMT, bool kSwiGLU, int NT, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
gemv_qd_kernel(const GemvArgs a) {
    static_assert(FMT == WF_DENSE || (FMT == WF_INT4 && NT == 1), "dense, or INT4 of up to 8 tokens");
    constexpr bool kDense = FMT == WF_DENSE;
    constexpr int R = kQdRows, P = qd_groups(FMT), LD = kDense ? 4 : 1, GB = kDense ? 256 : 64;  // 16-byte loads and bytes of a row per group
    constexpr int TILE = 8 * NT * kQdTileRow;
    extern __shared__ __align__(128) unsigned char smem[];
    const int K = a.K, N = a.N, groups = K / 128;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int units = kSwiGLU ? (a.inter + R / 2 - 1) / (R / 2) : (N + R - 1) / R;
    const int g0 = groups * warp / NW, ng = groups * (warp + 1) / NW - g0;  // this warp's groups of every row
    const int slots = (ng + P - 1) / P;
    // (rows past the last: a live row's weights, whose sums nobody stores)
    auto live_row = [&](int u, int r) -> int { return kSwiGLU ? ((r & 1) ? a.inter : 0) + min((R / 2) * u + (r >> 1), a.inter - 1) : min(R * u + r, N - 1); };

    struct Slot {
        uint4 w[P][LD][2];        // this lane's 32 weights of rows g and g + 8 in each group (dense: 8 of each 32 k)
        unsigned short s, z;      // INT4: scale bits and zero point of row lane % 16 in group lane / 16
    };
    Slot ring[kQdRing];
    const unsigned char *wa, *wb;   // the slot to load next: rows g and g + 8 of unit lu at slot lp
    size_t par = 0;
    int lu = blockIdx.x, lp = 0;
    auto open_unit = [&]() {
        const size_t at = (size_t)g0 * GB + 16 * t, row_bytes = (size_t)groups * GB;
        wa = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g) * row_bytes + at;
        wb = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g + 8) * row_bytes + at;
        if (!kDense) par = (size_t)live_row(lu, lane & 15) * groups + g0;
    };
    auto load = [&](Slot &p) {
        if (lu >= units) return;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int q = min(P * lp + j, ng - 1);  // (a missing second group: the first once more, which no activation meets)
#pragma unroll
            for (int i = 0; i < LD; ++i) p.w[j][i][0] = ld_stream_v4(wa + GB * q + 64 * i), p.w[j][i][1] = ld_stream_v4(wb + GB * q + 64 * i);
        }
        if constexpr (!kDense) {
            const size_t at = par + min(P * lp + (lane >> 4), ng - 1);
            // (as they come: a shift or an or here would wait for them)
            asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(p.s) : "l"(reinterpret_cast<const unsigned short *>(a.scales) + at));
            asm volatile("ld.global.nc.u8 %0, [%1];" : "=h"(p.z) : "l"(reinterpret_cast<const uint8_t *>(a.zeros) + at));
        }
        if (++lp == slots) {
            lp = 0, lu += gridDim.x;
            if (lu < units) open_unit();
        }
    };

    // ---- the first slots are on their way before the activations are there
    if (ng > 0) {
        open_unit();
#pragma unroll
        for (int i = 0; i < kQdRing; ++i) load(ring[i]);
    }
    pdl_wait();
    pdl_launch_dependents();

    // activations, [token][group][i][t] 16-byte pieces in the order in which a lane's loads meet them: the 8 k at 32 i + 8 t (dense), or (INT4, in f16) at
    // 32 t + 8 i.  One block of zeros for the slots past M
    const int xstride = 2 * K + 64;  // bytes: the rows of tokens g and g + 1 fall on different banks
    for (int idx = threadIdx.x; idx < a.M * (K / 8); idx += NW * 32) {
        const int m = idx / (K / 8), p8 = idx - m * (K / 8);
        const uint4 f = rs_fragment<T, FMT>(ld_v4(reinterpret_cast<const T *>(a.x) + (size_t)8 * idx));
        *reinterpret_cast<uint4 *>(smem + (size_t)m * xstride + (kDense ? p8 : (p8 & ~15) + (p8 & 3) * 4 + ((p8 >> 2) & 3)) * 16) = f;
    }
    unsigned char *const zeros = smem + (size_t)a.M * xstride;
    if (threadIdx.x < 16) *reinterpret_cast<uint4 *>(zeros + 16 * threadIdx.x) = make_uint4(0u, 0u, 0u, 0u);
    float *const red = reinterpret_cast<float *>(zeros + 256);  // [2][warp][tile]
    __syncthreads();
    const unsigned char *x0[NT];
    int xstep[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int m = g + 8 * i;
        x0[i] = m < a.M ? smem + (size_t)m * xstride + (size_t)g0 * 256 + 16 * t : zeros + 16 * t, xstep[i] = m < a.M ? 256 : 0;
    }

    float acc[NT][4] = {};  // [row g (+8)][token 2t (+1)] of each eight tokens
    int u = blockIdx.x, h = 0;
    auto finish = [&]() {  // the unit's last group is in: the warps' tiles become 16 rows of every token
        float *tile = red + (size_t)((h & 1) * NW + warp) * TILE;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                tile[(8 * i + 2 * t + (e & 1)) * kQdTileRow + g + 8 * (e >> 1)] = acc[i][e];
                acc[i][e] = 0.0f;
            }
        __syncthreads();
        if (warp * 2 < a.M) {  // (whole warps: two tokens each)
            const int r = lane & 15, m = warp * 2 + (lane >> 4);
            float v = 0.0f;
#pragma unroll
            for (int w2 = 0; w2 < NW; ++w2) v += red[(size_t)((h & 1) * NW + w2) * TILE + m * kQdTileRow + r];
            const bool ok = m < a.M && (kSwiGLU ? (R / 2) * u + (r >> 1) < a.inter : R * u + r < N);
            if constexpr (kSwiGLU) {
                // the un-fused reference stores gate / up in T before SiLU reads them
                const float rounded = round_to<T>(v), up = __shfl_down_sync(0xffffffffu, rounded, 1);
                if (ok && (r & 1) == 0) {
                    const float sv = (rounded / (1.0f + expf(-rounded))) * up;
                    const size_t o = (size_t)m * a.inter + (R / 2) * u + (r >> 1);
                    if (a.y_f32) reinterpret_cast<float *>(a.y)[o] = sv;
                    else reinterpret_cast<T *>(a.y)[o] = Elem<T>::from_f(sv);
                }
            } else if (ok) {
                const size_t o = (size_t)m * N + R * u + r;
                if (a.y_f32) reinterpret_cast<float *>(a.y)[o] = v;
                else reinterpret_cast<T *>(a.y)[o] = Elem<T>::from_f(v);
            }
        }
        ++h;
    };
    auto multiply = [&](const Slot &p, int at) {
        if constexpr (kDense) {
            float c[2][NT][4] = {};  // two chains
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 &e = p.w[0][i][0], &f = p.w[0][i][1];
                uint4 x[NT];
#pragma unroll
                for (int n = 0; n < NT; ++n) x[n] = *reinterpret_cast<const uint4 *>(x0[n] + (size_t)at * xstep[n] + 64 * i);
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_any<T>(c[0][n], e.x, f.x, e.y, f.y, x[n].x, x[n].y);
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_any<T>(c[1][n], e.z, f.z, e.w, f.w, x[n].z, x[n].w);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int y = 0; y < 4; ++y) acc[n][y] += c[0][n][y] + c[1][n][y];
        } else {
            // two groups, two chains of products each: one group's chains alone leave the tensor pipe waiting for its own results
            const bool both = at + 1 < ng;
            const unsigned char *const xp[2] = {x0[0] + (size_t)at * xstep[0], both ? x0[0] + (size_t)(at + 1) * xstep[0] : zeros + 16 * t};
            uint32_t sz;
            asm volatile("mov.b32 %0, {%1, %2};" : "=r"(sz) : "h"(p.s), "h"(p.z));
            uint32_t pa[P], pb[P], zpa[P], nza[P], zpb[P], nzb[P];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                pa[j] = __shfl_sync(0xffffffffu, sz, 16 * j + g), pb[j] = __shfl_sync(0xffffffffu, sz, 16 * j + g + 8);
                mma_int4_consts(pa[j] >> 16, zpa[j], nza[j]);
                mma_int4_consts(pb[j] >> 16, zpb[j], nzb[j]);
            }
            float c0[P][4] = {}, c1[P][4] = {};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint4 xv[P];
                uint32_t e[P][4], f[P][4];
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const uint4 &ra = p.w[j][0][0], &rb = p.w[j][0][1];
                    xv[j] = *reinterpret_cast<const uint4 *>(xp[j] + 64 * i);
                    mma_deq_int4(i == 0 ? ra.x : i == 1 ? ra.y : i == 2 ? ra.z : ra.w, zpa[j], nza[j], e[j]);
                    mma_deq_int4(i == 0 ? rb.x : i == 1 ? rb.y : i == 2 ? rb.z : rb.w, zpb[j], nzb[j], f[j]);
                }
#pragma unroll
                for (int j = 0; j < P; ++j) mma_f16f16(c0[j], e[j][0], f[j][0], e[j][1], f[j][1], xv[j].x, xv[j].y);
#pragma unroll
                for (int j = 0; j < P; ++j) mma_f16f16(c1[j], e[j][2], f[j][2], e[j][3], f[j][3], xv[j].z, xv[j].w);
            }
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const unsigned short la = (unsigned short)pa[j], lb = (unsigned short)pb[j];
                const float sa = Elem<T>::to_f(*reinterpret_cast<const T *>(&la)), sb = Elem<T>::to_f(*reinterpret_cast<const T *>(&lb));
                if (j == 0 || both) {
#pragma unroll
                    for (int y = 0; y < 4; ++y) acc[0][y] = fmaf(y < 2 ? sa : sb, c0[j][y] + c1[j][y], acc[0][y]);
                }
            }
        }
    };
    if (ng == 0) {  // (fewer groups than warps: a warp without any has only its barriers)
        for (; u < units; u += gridDim.x) finish();
        return;
    }
    for (int at = 0;;) {
#pragma unroll
        for (int i = 0; i < kQdRing; ++i) {
            if (u >= units) return;
            multiply(ring[i], at);
            load(ring[i]);
            if ((at += P) >= ng) {
                finish();
                u += gridDim.x, at = 0;
            }
        }
    }
}

// host side ----------------------------------------------------------------------------------------------------------
inline size_t gemv_qd_smem(int M, int K, int warps) { return (size_t)M * (2 * (size_t)K + 64) + 256 + (size_t)2 * warps * (M > 8 ? 16 : 8) * kQdTileRow * sizeof(float); }
template <typename T, int FMT, bool SW, int NT, int NW>
static int launch_gemv_qd_inst(const GemvArgs &a, int units, cudaStream_t st) {
    auto kern = gemv_qd_kernel<T, FMT, SW, NT, NW>;
    const size_t smem = gemv_qd_smem(a.M, a.K, NW);
    if (smem > qd_smem(FMT, NW)) return B200_ERR_UNSUPPORTED;
    if (!allow_smem(reinterpret_cast<const void *>(kern), qd_smem(FMT, NW), qd_smem(FMT, 16) + 2048)) return cuda_status("gemv_qd cudaFuncSetAttribute");
    launch_pdl(kern, dim3(std::max(1, std::min(units, 16 / NW * sm_count()))), dim3(NW * 32), smem, st, true, a);
    return cuda_status("gemv_qd launch");
}

// B200_ERR_UNSUPPORTED (no error text): what gemv_rs refuses, FP8, more than 8 tokens of INT4, long dense rows, activations that two CTAs of an SM cannot both
// hold, and the partial of a tensor-parallel linear.  Every choice depends on the tokens, the row's length and the output's type alone: a row's result has the
// same bits whatever rows are beside it.
template <typename T>
static int launch_gemv_qd_t(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) {
    if (fmt == WF_FP8 || (fmt == WF_INT4 && (a.group != 128 || a.M > 8)) || a.M < 1 || a.M > 16 || a.K % 128 != 0 || !aligned16(a.w) || !aligned16(a.x)) return B200_ERR_UNSUPPORTED;
    if (a.tp.world > 1 || a.norm || a.push.n > 0 || (swiglu && a.inter % 8 != 0)) return B200_ERR_UNSUPPORTED;
    const int units = swiglu ? (a.inter + kQdRows / 2 - 1) / (kQdRows / 2) : (a.N + kQdRows - 1) / kQdRows;
#define B200_QD_GO(FMTC, SW, NT) (wide ? launch_gemv_qd_inst<T, FMTC, SW, NT, 16>(a, units, st) : launch_gemv_qd_inst<T, FMTC, SW, NT, 8>(a, units, st))
    if (fmt == WF_INT4) {
        const bool wide = a.K >= 8192;
        return swiglu ? B200_QD_GO(WF_INT4, true, 1) : B200_QD_GO(WF_INT4, false, 1);
    }
    // Dense rows of at most 3072 k: there the start is most of a launch.  Longer ones fill gemv_rs.cuh's 200 KB ring before their wait, behind an attention or a
    // norm kernel, where this holds 128 KB (four layers, 2 / 8 tokens: 7B size 386 / 377 us there, 403 / 411 here; 2048 wide 155 / 169 there, 149 / 150 here; a
    // 70B-shaped shard, whose down projection has 3584 k, 286 / 296 there, 330 / 344 with it here and 273 / 287 without).  A vocabulary's fp32 logits of more than
    // 8 tokens stay there as well (50257 x 2048, 16 tokens: 58.1 us a head there, 59.0 here).
    if (a.K > 3072 || (a.M > 8 && a.y_f32)) return B200_ERR_UNSUPPORTED;
    const bool wide = a.M > 8 ? a.K >= 2048 : a.K > 2048;
    if (a.M <= 8) return swiglu ? B200_QD_GO(WF_DENSE, true, 1) : B200_QD_GO(WF_DENSE, false, 1);
    return swiglu ? B200_QD_GO(WF_DENSE, true, 2) : B200_QD_GO(WF_DENSE, false, 2);
#undef B200_QD_GO
}

}  // namespace b200
