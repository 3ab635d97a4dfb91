// gemv_qd.cuh -- the decode-shaped linear for INT4 weights of 1..8 tokens and dense weights of short rows of 1..16, streamed from global memory STRAIGHT INTO
// REGISTERS: y[M,N] = x[M,K] * W^T, W packed [N,K], in groups of 128 k (W4A16) or dense 16-bit.
// Reference: launchLinearGemm (src/kernels/linear.cu:10-87) at the decode shapes of src/layers/self_attention.cpp:79-86,131-138, src/layers/ffn.cpp:105-139.
//
// What bounds it: latency and instructions, not the 0.6 to 7 us that a 7B layer's INT4 linears take to read.  In gemv_rs.cuh a unit of 16 rows passes a barrier,
// 16 warps with two quantisation groups each, a second barrier and one reducer warp, and the parameters of a unit are waited for where they are loaded.  Here
//   * a warp owns one or two slices of k of 16 weight rows and walks them in slots of two groups (dense: of one) through a ring of registers: a slot's place is
//     loaded again as soon as it has been multiplied, up to 64 KB (dense: 128) in flight per SM without a barrier between a load and its use, and two groups' chains
//     of products keep the tensor pipe from waiting for its own results.  (K = 4096, N = 12288, where this takes 8.5 us: two buffers of four groups 10.6, one
//     group at a time in three CTAs per SM 9.2);
//   * 16 warps per SM, as two CTAs where both hold the activations, so that a unit's sum does not stop all of them (K = 4096, N = 12288 8.5 us with two against 9.4
//     with one, K = 2048, N = 5376 2.8 against 4.9), else as one: longer rows (K > 4096, dense > 2048) and more tokens;
//   * the first weights and parameters are requested before griddepcontrol.wait; one __syncthreads per unit (and part, below): the warps leave their tiles in one of
//     two buffers, the first threads add them in a fixed order (deterministic).
// A token's result does not depend on how many are beside it, though the form does:
//   * INT4: everything is summed in the order of gemv_rs.cuh, which takes the tokens that no form holds (K = 11008 from 7 on).  Fragments, dequantisation and
//     arithmetic are its own: exact integers in f16, fp32 sums, the group's scale once per 128 k; then parts of at most 32 groups, of every part 16 slices, of every
//     slice a tile.  So a part of a long row costs a barrier: K = 11008, N = 4096 10.3 us where one sum over each warp's whole slice took 9.3, K = 8192, N = 10240 14.9
//     for 13.8; all parts' tiles at once behind one barrier 10.6 and 14.4.
//   * dense: the sums of eight warps in order, or of sixteen two by two, which are the same where a warp of eight has at most two groups (K <= 2048).
// Dense weights: a launch's start rather than its instructions; its CTAs wait for no barrier and no ring.  Their sums are shorter chains in the tensor cores than
// gemv_rs.cuh's (fp32 outputs of K = 4096: 1.08e-7 from 64 bits against 1.42e-7).
// (Codes multiplied as they are, as subnormal f16, with the zero points' part taken off afterwards, need five instructions instead of nine for eight weights and
// were no faster; the tensor cores align a product by its operands' exponents, so the codes' leading zeros cost bits of the sum.)
// Measured, us per launch in a chain, 1 / 4 / 8 tokens (gemv_rs -> here): K = 4096: N = 12288 11.2 / 11.8 / 12.3 -> 8.5 / 9.3 / 10.5, N = 4096
// 5.1 / 5.5 / 6.0 -> 4.0 / 4.9 / 5.2, N = 22016 16.7 / 17.4 / 17.7 -> 13.3 / 14.2 / 16.5; K = 11008, N = 4096 12.0 / 12.6 / 14.0 -> 10.3 / 11.4 / gemv_rs;
// K = 8192, N = 10240 17.6 / 18.2 / 19.6 -> 14.9 / 16.0 / 17.6; K = 5120, N = 5120 9.6 / 9.8 / 10.2 -> 8.9 / 9.6 / 10.4 (its 20 groups a part are one or two to a slot).
// Dense, 1 (gemv.cuh) / 8 / 16 tokens (gemv_rs.cuh -> here): K = 2048: N = 6176 7.3 / 7.6 / 9.0 -> 5.3 / 6.0 / 6.6, N = 2048 3.8 / 3.6 / 4.3 -> 2.6 / 3.0 / 3.5;
// K = 1024, N = 1536 3.1 / 2.8 / 3.2 -> 1.8 / 1.9 / 2.4; K = 1536, N = 3072 4.4 / 4.1 / 5.0 -> 2.6 / 3.0 / 3.9; K = 3072, N = 3072 5.7 / 5.9 / 7.1 -> 4.2 / 4.8 / 5.9.
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
// groups of 128 k per slot: INT4 two of them (2 KB of 16 rows), dense weights one (4 KB)
__host__ __device__ constexpr int qd_groups(int fmt) { return fmt == WF_INT4 ? 2 : 1; }
// What a warp's slot is.  INT4 (a slice has at most two groups, where rows have at most 2048 k one): its two slices; one of its two slices; its only slice of a part.
// Dense: a group of its slice, with at most 108 KB of shared memory per SM, or 148
enum { QD_TWO_SLICES, QD_SLICE, QD_PART, QD_DENSE, QD_DENSE_LARGE };
// Dynamic shared memory of an SM's one CTA of 16 warps or two of 8, at most: what is in flight (64 KB, dense 128) needs L1 beside it.  With 148 KB dense loads no
// longer have all of theirs: K = 2048, N = 6176 of 1 / 8 / 16 tokens 5.8 / 6.5 / 6.7 us for 5.3 / 6.0 / 6.6; for K = 3072 and 16 tokens, which 108 KB do not hold, 5.9 (gemv_rs 7.1)
__host__ __device__ constexpr size_t qd_smem(int mode, int warps) { return (size_t)(mode == QD_DENSE ? 108 : mode == QD_DENSE_LARGE ? 148 : 160) * 1024 * warps / 16; }

// NORM: one INT4 token with the residual add and RMSNorm in front (GemvArgs), in the norm kernel's order and roundings: the same bits as with a launch in
// between.  Four 7B layers, one token: 203.0 us with norm kernels, 199.2 here (202.4 with the gains asked for behind the sum).
template <typename T, int FMT, bool kSwiGLU, int NT, int NW, int MODE, bool NORM = false>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
gemv_qd_kernel(const GemvArgs a) {
    static_assert(FMT == WF_DENSE || (FMT == WF_INT4 && NT == 1 && (MODE == QD_PART) == (NW == 16)), "dense, or INT4 of up to 8 tokens");
    constexpr bool kDense = FMT == WF_DENSE;
    constexpr int R = kQdRows, P = qd_groups(FMT), LD = kDense ? 4 : 1, GB = kDense ? 256 : 64;  // 16-byte loads and bytes of a row per group
    constexpr int TILE = 8 * NT * kQdTileRow, TILES = kDense ? NW : 16;
    extern __shared__ __align__(128) unsigned char smem[];
    const int K = a.K, N = a.N, groups = K / 128;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int units = kSwiGLU ? (a.inter + R / 2 - 1) / (R / 2) : (N + R - 1) / R;
    // (rows past the last: a live row's weights, whose sums nobody stores)
    auto live_row = [&](int u, int r) -> int { return kSwiGLU ? ((r & 1) ? a.inter : 0) + min((R / 2) * u + (r >> 1), a.inter - 1) : min(R * u + r, N - 1); };

    struct Slot {
        uint4 w[P][LD][2];        // this lane's 32 weights of rows g and g + 8 in each group (dense: 8 of each 32 k)
        unsigned short s, z;      // INT4: scale bits and zero point of row lane % 16 in group lane / 16
    };
    Slot ring[kQdRing];
    // This warp's slots in every unit, as groups [first, first + count).  Dense: the groups of its slice one by one.  INT4: its two slices are [0] and [1], in one
    // slot or in two; or [0] is its slice of a row's first part, `step` groups further that of the next, and [1] its slice of the last part
    struct Span {
        int first, count;
    } span[2];
    int slots = 1, step = 0;
    if constexpr (kDense) {
        span[0].first = groups * warp / NW, slots = groups * (warp + 1) / NW - span[0].first;
        step = 1;
    } else if constexpr (MODE == QD_PART) {
        slots = (groups + 31) / 32, step = (groups + slots - 1) / slots, slots = (groups + step - 1) / step;  // (the parts of gemv_rs.cuh)
        const int last = groups - (slots - 1) * step;
        span[0].first = step * warp / 16, span[0].count = step * (warp + 1) / 16 - span[0].first;
        span[1].first = last * warp / 16, span[1].count = last * (warp + 1) / 16 - span[1].first;
        span[1].first += (slots - 1) * step;
    } else {
        const int mid = groups * (2 * warp + 1) / 16;
        span[0].first = groups * warp / 8, span[0].count = mid - span[0].first;
        span[1].first = mid, span[1].count = groups * (warp + 1) / 8 - mid;
        slots = MODE == QD_SLICE ? 2 : 1;
    }
    // the groups of slot s
    auto first_of = [&](int s) { return kDense ? span[0].first + s : MODE == QD_SLICE ? span[s].first : MODE == QD_PART && s + 1 == slots ? span[1].first : span[0].first + s * step; };
    auto count_of = [&](int s) { return kDense ? 1 : MODE == QD_SLICE ? span[s].count : MODE == QD_TWO_SLICES ? span[0].count + span[1].count : s + 1 == slots ? span[1].count : span[0].count; };
    const unsigned char *wa, *wb;   // the slot to load next: rows g and g + 8 of unit lu at slot lp
    size_t par = 0;
    int lu = blockIdx.x, lp = 0;
    auto open_unit = [&]() {
        const size_t row_bytes = (size_t)groups * GB;
        wa = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g) * row_bytes + 16 * t;
        wb = reinterpret_cast<const unsigned char *>(a.w) + (size_t)live_row(lu, g + 8) * row_bytes + 16 * t;
        if (!kDense) par = (size_t)live_row(lu, lane & 15) * groups;
    };
    auto load = [&](Slot &p, int s) {
        if (lu >= units) return;
        const int at = min(first_of(s), groups - 1), more = count_of(s) > 1;  // (a missing group: a live one, which no activation meets)
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int q = (at + j * more) * GB;
#pragma unroll
            for (int i = 0; i < LD; ++i) p.w[j][i][0] = ld_stream_v4(wa + q + 64 * i), p.w[j][i][1] = ld_stream_v4(wb + q + 64 * i);
        }
        if constexpr (!kDense) {
            const size_t where = par + at + (lane >> 4) * more;
            // (as they come: a shift or an or here would wait for them)
            asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(p.s) : "l"(reinterpret_cast<const unsigned short *>(a.scales) + where));
            asm volatile("ld.global.nc.u8 %0, [%1];" : "=h"(p.z) : "l"(reinterpret_cast<const uint8_t *>(a.zeros) + where));
        }
        if (MODE == QD_SLICE ? s == 1 : ++lp == slots) {
            lp = 0, lu += gridDim.x;
            if (lu < units) open_unit();
        }
    };
    // ---- the first slots are on their way before the activations are there
    if (slots > 0) {
        if (lu < units) open_unit();
#pragma unroll
        for (int i = 0; i < kQdRing; ++i) load(ring[i], MODE == QD_SLICE ? i : lp);
    }
    // (the gains do not depend on the kernel in front either: those of a thread's first rows of eight)
    constexpr int GN = NORM ? 512 / (NW * 32) : 1;
    uint4 gain[GN];
    if constexpr (NORM) {
#pragma unroll
        for (int v = 0; v < GN; ++v) {
            const int i = threadIdx.x + v * NW * 32;
            if (a.gamma && i < K / 8) gain[v] = ld_v4(reinterpret_cast<const T *>(a.gamma) + (size_t)8 * i);
        }
    }
    pdl_wait();
    pdl_launch_dependents();

    // activations, [token][group][i][t] 16-byte pieces in the order in which a lane's loads meet them: the 8 k at 32 i + 8 t (dense), or (INT4, in f16) at
    // 32 t + 8 i.  One block of zeros for the slots past M
    const int xstride = 2 * K + 64;  // bytes: the rows of tokens g and g + 1 fall on different banks
    if constexpr (NORM) {
        __shared__ float sums[16];
        constexpr int vt = 512;  // threads of the norm kernel: one of ours does the work of one or two of them
        auto place = [&](int i) { return smem + ((i & ~15) + (i & 3) * 4 + ((i >> 2) & 3)) * 16; };
#pragma unroll
        for (int v = threadIdx.x; v < vt; v += NW * 32) {
            float ss = 0.0f;
            for (int i = v; i < K / 8; i += vt) {
                float f[8];
                unpack16<T>(ld_v4(reinterpret_cast<const T *>(a.x) + (size_t)8 * i), f);
                if (a.res_in) {
                    float r[8];
                    unpack16<T>(ld_v4(reinterpret_cast<const T *>(a.res_in) + (size_t)8 * i), r);
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = round_to<T>(f[e] + r[e]);
                }
                if (a.res_out && blockIdx.x == 0) st_v4(reinterpret_cast<T *>(a.res_out) + (size_t)8 * i, pack16<T>(f));
                if (a.bias) {
                    float b[8];
                    unpack16<T>(ld_v4(reinterpret_cast<const T *>(a.bias) + (size_t)8 * i), b);
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = round_to<T>(f[e] + b[e]);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
                *reinterpret_cast<uint4 *>(place(i)) = pack16<T>(f);  // (exact: f is of T)
            }
            ss = warp_sum(ss);
            if (lane == 0) sums[v >> 5] = ss;
        }
        __syncthreads();
        const float scale = rsqrtf(warp_sum(lane < (vt >> 5) ? sums[lane & 15] : 0.0f) / (float)K + a.eps);
#pragma unroll
        for (int w = 0; w < GN; ++w)
            for (int v = threadIdx.x + w * NW * 32, i = v; i < K / 8; i += vt) {
                float f[8], g[8];
                unpack16<T>(*reinterpret_cast<const uint4 *>(place(i)), f);
                if (a.gamma) {
                    unpack16<T>(i == v ? gain[w] : ld_v4(reinterpret_cast<const T *>(a.gamma) + (size_t)8 * i), g);
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = (f[e] * g[e]) * scale;
                }
                *reinterpret_cast<uint4 *>(place(i)) = rs_fragment<T, FMT>(pack16<T>(f));
            }
    } else
    for (int idx = threadIdx.x; idx < a.M * (K / 8); idx += NW * 32) {
        const int m = idx / (K / 8), p8 = idx - m * (K / 8);
        const uint4 f = rs_fragment<T, FMT>(ld_v4(reinterpret_cast<const T *>(a.x) + (size_t)8 * idx));
        *reinterpret_cast<uint4 *>(smem + (size_t)m * xstride + (kDense ? p8 : (p8 & ~15) + (p8 & 3) * 4 + ((p8 >> 2) & 3)) * 16) = f;
    }
    unsigned char *const zeros = smem + (size_t)a.M * xstride;
    if (threadIdx.x < 16) *reinterpret_cast<uint4 *>(zeros + 16 * threadIdx.x) = make_uint4(0u, 0u, 0u, 0u);
    float *const red = reinterpret_cast<float *>(zeros + 256);  // [2][slice][tile]
    __syncthreads();
    const unsigned char *x0[NT];
    int xstep[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        const int m = g + 8 * i;
        x0[i] = m < a.M ? smem + (size_t)m * xstride + 16 * t : zeros + 16 * t, xstep[i] = m < a.M ? 256 : 0;
    }

    float acc[NT][4] = {};  // dense: [row g (+8)][token 2t (+1)] of each eight tokens
    float sum = 0.0f;       // a reducing thread's: the parts before this one
    int u = blockIdx.x, at = 0, h = 0;  // the slot to multiply next
    auto hand_over = [&](int slice, const float (&c)[NT][4]) {
        float *tile = red + (size_t)((h & 1) * TILES + slice) * TILE;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) tile[(8 * i + 2 * t + (e & 1)) * kQdTileRow + g + 8 * (e >> 1)] = c[i][e];
    };
    auto finish = [&](bool last) {  // the slices' tiles of a part are in: they become 16 rows of every token
        __syncthreads();
        if (warp * 2 < a.M) {  // (whole warps: two tokens each)
            const int r = lane & 15, m = warp * 2 + (lane >> 4);
            const float *mine = red + (size_t)(h & 1) * TILES * TILE + m * kQdTileRow + r;
            float v = 0.0f;
            if constexpr (kDense && NW == 16) {  // (a warp of the other form has the groups of two of these)
#pragma unroll
                for (int w2 = 0; w2 < TILES; w2 += 2) v += mine[(size_t)w2 * TILE] + mine[(size_t)(w2 + 1) * TILE];
            } else {
#pragma unroll
                for (int w2 = 0; w2 < TILES; ++w2) v += mine[(size_t)w2 * TILE];
            }
            if constexpr (MODE == QD_PART) {
                v += sum, sum = last ? 0.0f : v;
                if (!last) {
                    ++h;
                    return;
                }
            }
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
                if (kDense && a.finish) v = bias_act<T>(v, a.out_bias, R * u + r, a.out_act);
                if (a.y_f32) reinterpret_cast<float *>(a.y)[o] = v;
                else reinterpret_cast<T *>(a.y)[o] = Elem<T>::from_f(v);
            }
        }
        ++h;
    };
    // slot s of the unit at hand; INT4: hands over its slice or slices
    auto multiply = [&](const Slot &p, int s) {
        const int at = first_of(s);
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
            const int n = count_of(s);
            const unsigned char *const xp[2] = {n > 0 ? x0[0] + (size_t)at * xstep[0] : zeros + 16 * t, n > 1 ? x0[0] + (size_t)(at + 1) * xstep[0] : zeros + 16 * t};
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
            float d[2][1][4] = {};  // (QD_TWO_SLICES: of either slice)
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const unsigned short la = (unsigned short)pa[j], lb = (unsigned short)pb[j];
                const float sa = Elem<T>::to_f(*reinterpret_cast<const T *>(&la)), sb = Elem<T>::to_f(*reinterpret_cast<const T *>(&lb));
                float(&to)[4] = d[MODE == QD_TWO_SLICES ? j : 0][0];
                if (n > j) {
#pragma unroll
                    for (int y = 0; y < 4; ++y) to[y] = fmaf(y < 2 ? sa : sb, c0[j][y] + c1[j][y], to[y]);
                }
            }
            if constexpr (MODE == QD_TWO_SLICES) {
                // (a warp with one group: it is the first slice's or the second's)
                if (span[0].count == 0) hand_over(2 * warp, d[1]), hand_over(2 * warp + 1, d[0]);
                else hand_over(2 * warp, d[0]), hand_over(2 * warp + 1, d[1]);
            } else {
                hand_over(MODE == QD_SLICE ? 2 * warp + s : warp, d[0]);
            }
        }
    };
    if constexpr (kDense) {
        if (slots == 0) {  // (fewer groups than warps: a warp without any has only its barriers)
            for (; u < units; u += gridDim.x) hand_over(warp, acc), finish(true);
            return;
        }
    }
    for (;;) {
#pragma unroll
        for (int i = 0; i < kQdRing; ++i) {
            if (u >= units) return;
            multiply(ring[i], MODE == QD_SLICE ? i : at);
            load(ring[i], MODE == QD_SLICE ? i : lp);
            const bool last = MODE == QD_SLICE ? i == 1 : at + 1 == slots;
            if constexpr (kDense) {
                if (last) {
                    hand_over(warp, acc);
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int y = 0; y < 4; ++y) acc[n][y] = 0.0f;
                }
            }
            if (MODE == QD_PART || last) finish(last);
            ++at;
            if (last) u += gridDim.x, at = 0;
        }
    }
}

// host side ----------------------------------------------------------------------------------------------------------
inline size_t gemv_qd_smem(int M, int K, int fmt, int warps) {
    return (size_t)M * (2 * (size_t)K + 64) + 256 + (size_t)2 * (fmt == WF_INT4 ? 16 : warps) * (M > 8 ? 16 : 8) * kQdTileRow * sizeof(float);
}
template <typename T, int FMT, bool SW, int NT, int NW, int MODE, bool NORM = false>
static int launch_gemv_qd_inst(const GemvArgs &a, int units, cudaStream_t st) {
    auto kern = gemv_qd_kernel<T, FMT, SW, NT, NW, MODE, NORM>;
    const size_t smem = gemv_qd_smem(a.M, a.K, FMT, NW);
    if (smem > qd_smem(MODE, NW)) return B200_ERR_UNSUPPORTED;
    if (!allow_smem(reinterpret_cast<const void *>(kern), qd_smem(MODE, NW), qd_smem(MODE, 16) + 2048)) return cuda_status("gemv_qd cudaFuncSetAttribute");
    launch_pdl(kern, dim3(std::max(1, std::min(units, 16 / NW * sm_count()))), dim3(NW * 32), smem, st, true, a);
    return cuda_status("gemv_qd launch");
}

// B200_ERR_UNSUPPORTED (no error text): what gemv_rs refuses, FP8, more than 8 tokens of INT4, long dense rows, INT4 activations that an SM does not hold beside what
// is in flight, and the partial of a tensor-parallel linear.
template <typename T>
static int launch_gemv_qd_t(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) {
    if (fmt == WF_FP8 || (fmt == WF_INT4 && (a.group != 128 || a.M > 8)) || a.M < 1 || a.M > 16 || a.K % 128 != 0 || !aligned16(a.w) || !aligned16(a.x)) return B200_ERR_UNSUPPORTED;
    if (a.norm && (fmt != WF_INT4 || a.M != 1 || a.K > 16384 || !all_aligned16({a.res_in, a.res_out, a.bias, a.gamma}))) return B200_ERR_UNSUPPORTED;
    if (a.tp.world > 1 || a.push.n > 0 || (swiglu && a.inter % 8 != 0)) return B200_ERR_UNSUPPORTED;
    const int units = swiglu ? (a.inter + kQdRows / 2 - 1) / (kQdRows / 2) : (a.N + kQdRows - 1) / kQdRows;
    auto fits = [&](int mode, int warps) { return gemv_qd_smem(a.M, a.K, fmt, warps) <= qd_smem(mode, warps); };
    if (fmt == WF_INT4) {
        const int mode = a.K > 4096 || !fits(QD_SLICE, 8) ? QD_PART : a.K > 2048 ? QD_SLICE : QD_TWO_SLICES;
#define B200_QD_GO(SW, NORM) (mode == QD_PART ? launch_gemv_qd_inst<T, WF_INT4, SW, 1, 16, QD_PART, NORM>(a, units, st) \
                        : mode == QD_SLICE ? launch_gemv_qd_inst<T, WF_INT4, SW, 1, 8, QD_SLICE, NORM>(a, units, st) : launch_gemv_qd_inst<T, WF_INT4, SW, 1, 8, QD_TWO_SLICES, NORM>(a, units, st))
        if (a.norm) return swiglu ? B200_QD_GO(true, true) : B200_QD_GO(false, true);
        return swiglu ? B200_QD_GO(true, false) : B200_QD_GO(false, false);
#undef B200_QD_GO
    }
    // Dense rows of at most 3072 k: there the start is most of a launch.  Longer ones fill gemv_rs.cuh's 200 KB ring before their wait, behind an attention or a
    // norm kernel, where this holds 128 KB (four layers, 2 / 8 tokens: 7B size 386 / 377 us there, 403 / 411 here; 2048 wide 155 / 169 there, 149 / 150 here; a
    // 70B-shaped shard, whose down projection has 3584 k, 286 / 296 there, 330 / 344 with it here and 273 / 287 without).  A vocabulary's fp32 logits of 16 rows, norm and
    // top-k included: 1024 x 32000 41.7 us there, 30.3 here; 2048 x 32000 41.9 and 41.7; 2048 x 50257 58.2 and 59.6.
    if (a.K > 3072) return B200_ERR_UNSUPPORTED;
    const bool wide = a.K > 2048 || !fits(QD_DENSE, 8);
#define B200_QD_GO(SW) (a.M <= 8 ? (wide ? launch_gemv_qd_inst<T, WF_DENSE, SW, 1, 16, QD_DENSE>(a, units, st) : launch_gemv_qd_inst<T, WF_DENSE, SW, 1, 8, QD_DENSE>(a, units, st)) \
                        : !wide ? launch_gemv_qd_inst<T, WF_DENSE, SW, 2, 8, QD_DENSE>(a, units, st) : fits(QD_DENSE, 16) ? launch_gemv_qd_inst<T, WF_DENSE, SW, 2, 16, QD_DENSE>(a, units, st) \
                        : launch_gemv_qd_inst<T, WF_DENSE, SW, 2, 16, QD_DENSE_LARGE>(a, units, st))
    return swiglu ? B200_QD_GO(true) : B200_QD_GO(false);
#undef B200_QD_GO
}

}  // namespace b200
