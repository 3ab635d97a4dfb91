// gemv_qd.cuh -- the decode-shaped linear for 1..8 tokens and INT4 weights, streamed from global memory STRAIGHT INTO REGISTERS:
// y[M,N] = x[M,K] * W^T, W packed [N,K] in groups of 128 k (W4A16), 16-bit activations.
// Reference: launchLinearGemm (src/kernels/linear.cu:10-87) at the decode shapes of src/layers/self_attention.cpp:79-86,131-138, src/layers/ffn.cpp:105-139.
//
// What bounds it: latency and instructions, not the 0.6 to 7 us that a 7B layer's linears take to read.  In gemv_rs.cuh a unit of 16 rows passes a barrier, 16
// warps with two quantisation groups each, a second barrier and one reducer warp, and the parameters of a unit are waited for where they are loaded.  Here
//   * a warp owns a slice of k of 16 weight rows and walks it in pairs of groups through a ring of registers: a pair's place is loaded again as soon as it has
//     been multiplied, up to 64 KB in flight per SM without a barrier between a load and its use, and two groups' chains of products keep the tensor pipe from
//     waiting for its own results.  (K = 4096, N = 12288, where this takes 8.2 us: two buffers of four groups 10.6, one group at a time in three CTAs per SM 9.2);
//   * 16 warps per SM, as one CTA where a row is long or the units are few (a slice is then at least a pair and the activations are staged once per SM), else as
//     two CTAs, so that a unit's sum does not stop all of them: K = 4096, N = 12288 8.3 us with two against 9.1 with one, K = 2048, N = 5376 3.1 against 4.6,
//     K = 8192, N = 10240 14.5 against 13.3, K = 12288, N = 1536 7.3 against 5.7;
//   * the first weights and parameters are requested before griddepcontrol.wait; one __syncthreads per unit: the warps leave their tiles in one of two buffers,
//     the first threads add them in a fixed order (deterministic).
// Fragments, dequantisation and arithmetic are those of gemv_rs.cuh's quantised units: exact integers in f16, fp32 sums, the group's scale once per 128 k.
// (Codes multiplied as they are, as subnormal f16, with the zero points' part taken off afterwards, need five instructions instead of nine for eight weights and
// were no faster; the tensor cores align a product by its operands' exponents, so the codes' leading zeros cost bits of the sum.)
// Measured, us per launch in a chain, 1 / 4 / 8 tokens (gemv_rs -> here): K = 4096: N = 12288 11.3 / 11.9 / 12.5 -> 8.2 / 9.1 / 10.4, N = 4096
// 5.1 / 5.5 / 6.0 -> 3.9 / 4.3 / 4.8, N = 22016 16.9 / 17.5 / 18.0 -> 13.4 / 14.3 / 15.5; K = 11008, N = 4096 12.0 / 12.7 / 14.1 -> 9.4 / 10.5 / gemv_rs.
#pragma once
#include "gemv_rs.cuh"

namespace b200 {

constexpr int kQdRows = 16;
constexpr int kQdTile = 8 * 20;         // fp32 values of one warp's tile: [8 tokens][16 rows + 4]
constexpr int kQdRing = 2;              // pairs of quantisation groups in flight per warp, four 16-byte loads of a lane each
constexpr size_t kQdSmem = 160 * 1024;  // dynamic shared memory of an SM's one CTA of 16 warps or two of 8, at most: the 64 KB in flight need L1 beside it

template <typename T, bool kSwiGLU, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
gemv_qd_kernel(const GemvArgs a) {
    constexpr int R = kQdRows, P = 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const int K = a.K, N = a.N, groups = K / 128;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int units = kSwiGLU ? (a.inter + R / 2 - 1) / (R / 2) : (N + R - 1) / R;
    const int g0 = groups * warp / NW, ng = groups * (warp + 1) / NW - g0;  // this warp's groups of every row
    const int pairs = (ng + P - 1) / P;
    // (rows past the last: a live row's weights, whose sums nobody stores)
    auto live_row = [&](int u, int r) -> int { return kSwiGLU ? ((r & 1) ? a.inter : 0) + min((R / 2) * u + (r >> 1), a.inter - 1) : min(R * u + r, N - 1); };

    struct Pair {
        uint4 w[P][2];           // this lane's 32 weights of rows g and g + 8 in either group
        unsigned short s, z;     // scale bits and zero point of row lane % 16 in group lane / 16
    };
    Pair ring[kQdRing];
    const unsigned char *wa, *wb;   // the pair to load next: rows g and g + 8 of unit lu at pair lp
    size_t par;
    int lu = blockIdx.x, lp = 0;
    auto open_unit = [&]() {
        const size_t at = (size_t)g0 * 64 + 16 * t, row_bytes = (size_t)K / 2;
        wa = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g) * row_bytes + at;
        wb = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g + 8) * row_bytes + at;
        par = (size_t)live_row(lu, lane & 15) * groups + g0;
    };
    auto load = [&](Pair &p) {
        if (lu >= units) return;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int q = min(P * lp + j, ng - 1);  // (a missing second group: the first once more, which no activation meets)
            p.w[j][0] = ld_stream_v4(wa + 64 * q), p.w[j][1] = ld_stream_v4(wb + 64 * q);
        }
        const size_t at = par + min(P * lp + (lane >> 4), ng - 1);
        // (as they come: a shift or an or here would wait for them)
        asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(p.s) : "l"(reinterpret_cast<const unsigned short *>(a.scales) + at));
        asm volatile("ld.global.nc.u8 %0, [%1];" : "=h"(p.z) : "l"(reinterpret_cast<const uint8_t *>(a.zeros) + at));
        if (++lp == pairs) {
            lp = 0, lu += gridDim.x;
            if (lu < units) open_unit();
        }
    };

    // ---- the first pairs are on their way before the activations are there
    if (ng > 0) {
        open_unit();
#pragma unroll
        for (int i = 0; i < kQdRing; ++i) load(ring[i]);
    }
    pdl_wait();
    pdl_launch_dependents();

    // activations in f16, [token][group][i][t] 16-byte pieces: a lane's piece i of a group is the 8 k at 32 t + 8 i.  One block of zeros for the slots past M
    const int xstride = 2 * K + 64;  // bytes: the rows of tokens g and g + 1 fall on different banks
    for (int idx = threadIdx.x; idx < a.M * (K / 8); idx += NW * 32) {
        const int m = idx / (K / 8), p8 = idx - m * (K / 8);
        const uint4 f = rs_fragment<T, WF_INT4>(ld_v4(reinterpret_cast<const T *>(a.x) + (size_t)8 * idx));
        *reinterpret_cast<uint4 *>(smem + (size_t)m * xstride + ((p8 & ~15) + (p8 & 3) * 4 + ((p8 >> 2) & 3)) * 16) = f;
    }
    unsigned char *const zeros = smem + (size_t)a.M * xstride;
    if (threadIdx.x < 16) *reinterpret_cast<uint4 *>(zeros + 16 * threadIdx.x) = make_uint4(0u, 0u, 0u, 0u);
    float *const red = reinterpret_cast<float *>(zeros + 256);  // [2][warp][tile]
    __syncthreads();
    const unsigned char *const x0 = g < a.M ? smem + (size_t)g * xstride + (size_t)g0 * 256 + 16 * t : zeros + 16 * t;
    const int xstep = g < a.M ? 256 : 0;

    float acc[4] = {};  // [row g (+8)][token 2t (+1)]
    int u = blockIdx.x, h = 0;
    auto finish = [&]() {  // the unit's last group is in: eight warps' tiles become 16 rows of every token
        float *tile = red + (size_t)((h & 1) * NW + warp) * kQdTile;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            tile[(2 * t + (e & 1)) * 20 + g + 8 * (e >> 1)] = acc[e];
            acc[e] = 0.0f;
        }
        __syncthreads();
        if (warp * 2 < a.M) {  // (whole warps: two tokens each)
            const int r = lane & 15, m = warp * 2 + (lane >> 4);
            float v = 0.0f;
#pragma unroll
            for (int w2 = 0; w2 < NW; ++w2) v += red[(size_t)((h & 1) * NW + w2) * kQdTile + m * 20 + r];
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
    // two groups, two chains of products each: one group's chains alone leave the tensor pipe waiting for its own results
    auto multiply = [&](const Pair &p, int at) {
        const bool both = at + 1 < ng;
        const unsigned char *const xp[P] = {x0 + (size_t)at * xstep, both ? x0 + (size_t)(at + 1) * xstep : zeros + 16 * t};
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
                xv[j] = *reinterpret_cast<const uint4 *>(xp[j] + 64 * i);
                mma_deq_int4(i == 0 ? p.w[j][0].x : i == 1 ? p.w[j][0].y : i == 2 ? p.w[j][0].z : p.w[j][0].w, zpa[j], nza[j], e[j]);
                mma_deq_int4(i == 0 ? p.w[j][1].x : i == 1 ? p.w[j][1].y : i == 2 ? p.w[j][1].z : p.w[j][1].w, zpb[j], nzb[j], f[j]);
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
                for (int y = 0; y < 4; ++y) acc[y] = fmaf(y < 2 ? sa : sb, c0[j][y] + c1[j][y], acc[y]);
            }
        }
    };
    if (ng == 0) {  // (K < 1024: a warp without groups has only its barriers)
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
inline size_t gemv_qd_smem(int M, int K, int warps) {
    return (size_t)M * (2 * (size_t)K + 64) + 256 + (size_t)2 * warps * kQdTile * sizeof(float);
}
template <typename T, bool SW, int NW>
static int launch_gemv_qd_inst(const GemvArgs &a, int units, cudaStream_t st) {
    auto kern = gemv_qd_kernel<T, SW, NW>;
    const size_t smem = gemv_qd_smem(a.M, a.K, NW);
    if (smem > kQdSmem * NW / 16) return B200_ERR_UNSUPPORTED;
    if (!allow_smem(reinterpret_cast<const void *>(kern), kQdSmem)) return cuda_status("gemv_qd cudaFuncSetAttribute");
    launch_pdl(kern, dim3(std::max(1, std::min(units, 16 / NW * sm_count()))), dim3(NW * 32), smem, st, true, a);
    return cuda_status("gemv_qd launch");
}

// B200_ERR_UNSUPPORTED (no error text): what gemv_rs refuses, and other formats, more than 8 tokens, activations that two CTAs of an SM cannot both hold, and
// the partial of a tensor-parallel linear.
template <typename T>
static int launch_gemv_qd_t(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) {
    if (fmt != WF_INT4 || a.group != 128 || a.M < 1 || a.M > 8 || a.K % 128 != 0 || !aligned16(a.w) || !aligned16(a.x)) return B200_ERR_UNSUPPORTED;
    if (a.tp.world > 1 || a.norm || a.push.n > 0 || (swiglu && a.inter % 8 != 0)) return B200_ERR_UNSUPPORTED;
    const int units = swiglu ? (a.inter + kQdRows / 2 - 1) / (kQdRows / 2) : (a.N + kQdRows - 1) / kQdRows;
    if (a.K >= 8192 || (a.K >= 4096 && units <= 2 * sm_count())) return swiglu ? launch_gemv_qd_inst<T, true, 16>(a, units, st) : launch_gemv_qd_inst<T, false, 16>(a, units, st);
    return swiglu ? launch_gemv_qd_inst<T, true, 8>(a, units, st) : launch_gemv_qd_inst<T, false, 8>(a, units, st);
}

}  // namespace b200
