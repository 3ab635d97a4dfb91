// chunk_recurrence.cu -- the token-parallel form of two recurrences over a matrix state (gla.cu, recurrent.cu) for long portions:
//     gated linear attention   S_t = diag(g_t) S_(t-1) + k_t v_t^T                                          o_t = S_t^T q_t
//     gated delta rule         S~ = diag(g_t) S_(t-1);  u_t = beta_t (v_t - S~^T k_t);  S_t = S~ + k_t u_t^T     o_t = S_t^T q_t
// The serial form takes one dependent step per token.  Here a portion is cut into chunks of kC tokens; with p_t the product of the chunk's
// decays up to token t, e_s the product after token s, and S_0 the state the chunk starts from,
//     u   = Tb (V - Kp S_0)         Kp = rows k_t * p_t,  Tb = (I + diag(beta) A)^-1 diag(beta),  A[t,s] = sum_i k_t k_s prod_(s<r<=t) g_r, s < t
//     o   = Qp S_0 + P u            Qp = rows q_t * p_t,  P[t,s] = sum_i q_t k_s prod_(s<r<=t) g_r, s <= t
//     S_C = diag(p_C) S_0 + Ke^T u  Ke = rows k_s * e_s
// (linear attention: u = V), so the serial part is one step of small matrix products per chunk.  Every decay factor is a product of decays
// formed forward in time, never a quotient: it is at most 1, and one that underflows stands for a contribution that is gone.
//   chunk_factors_kernel  one CTA per (chunk, head), all chunks at once: Qp, Kp, Ke, P, p_C, Tb as plain rows
//   chunk_scan_kernel     one CTA per (16 columns of S, head, sequence) walks the chunks, S^T in shared memory and in registers
// All products are fp32 multiply-adds; a chunk's decay products are formed in 64 bits and rounded once.  mma.sync on operands split in two TF32 halves was
// here first (182 us for the first case below, 203 for the second): 22 of 24 bits and sums that are cut off put read-outs up to 2.1 and states up to 5 times
// as far from 64 bits as the serial kernels'; now 0.46 to 1.05 times (fp32 vectors, dim 64 and 128, 64 to 4096 tokens, decays near 1, around 0.7 and 0.15).
// tcgen05 has no fp32 form.
// Measured (B200, 8 heads, dim 128, vdim 256; factors + scan against the serial kernel): linear attention of 4096 tokens 37 + 326 against 690 us, delta rule of
// 1500, 511 and 900 tokens 40 + 289 against 401.
#include "hybrid_ops.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kC = 32;      // tokens per chunk
constexpr int kCols = 16;   // columns of S per CTA of the scan (the M of its matrix instructions)

// one (chunk, head) block, rows as they are: Qp [kC x DK], (delta rule: Kp [kC x DK]), Ke [kC x DK], P [kC x kC], p_C [DK], (Tb [kC x kC])
template <int DK, bool DELTA> struct Block {
    static constexpr int kQp = 0, kKp = kC * DK, kKe = (DELTA ? 2 : 1) * kC * DK, kP = kKe + kC * DK, kG = kP + kC * kC, kTb = kG + DK;
    static constexpr int kFloats = kTb + (DELTA ? kC * kC : 0);
};
__host__ __device__ constexpr int block_floats(int dk, bool delta) { return (delta ? 3 : 2) * kC * dk + (delta ? 2 : 1) * kC * kC + dk; }

// where a head's vectors of a token are: q, k, v rows of one array of type TQ (element offsets), the decays in an fp32 array
struct ChunkSource {
    const void *rows;
    int ld, q_off, k_off, v_off;
    const float *decay;
    int decay_ld, decay_off, decay_dim;  // decay_dim: numbers per head (dim: one per key channel; 1: one for all of them)
    const float *beta;  // one number per head and token (delta rule), or NULL
    int beta_ld;
    float q_scale;
};

struct ChunkMap {
    const int *seq_start, *seq_pos0, *seq_slot;
    int heads, group;      // heads per key head
    int vdim;
    int min_tokens;        // shorter portions are another kernel's
    int first, count;      // chunks [first, first + count) of every portion run now
    int packed;            // 1: block index from the packed row (all chunks of the batch fit); 0: `count` blocks per sequence
};
__device__ __forceinline__ int block_base(const ChunkMap &m, int s) { return m.packed ? m.seq_start[s] / kC + s : s * m.count; }

// CH (2 or 4) consecutive shared floats in one access: a lane's channels, CH floats from its neighbour's
template <int CH> __device__ __forceinline__ void load_channels(const float *p, float *f) {
    if constexpr (CH == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
    } else {
        const float2 v = *reinterpret_cast<const float2 *>(p);
        f[0] = v.x, f[1] = v.y;
    }
}

template <typename TQ, int DK, bool DELTA>
__global__ void __launch_bounds__(256, 4)
chunk_factors_kernel(const ChunkSource src, const ChunkMap map, float *__restrict__ blocks) {
    constexpr int P = DK + 4;  // row pitch: rows read by neighbouring lanes start four banks apart
    constexpr int CH = DK / 32;
    extern __shared__ __align__(16) float sm[];
    float *ks = sm, *qs = ks + kC * P, *gs = qs + kC * P;  // [kC][P] each
    float *As = gs + kC * P, *Ps = As + kC * 36;           // [kC][36]
    double *half_prod = reinterpret_cast<double *>(Ps + kC * 36);  // [2][DK]
    float *bs = reinterpret_cast<float *>(half_prod + 2 * DK);     // [kC]
    const int s = blockIdx.z, h = blockIdx.y, hk = h / map.group;
    const int len = map.seq_start[s + 1] - map.seq_start[s];
    const int c = map.first + blockIdx.x;
    if (len < map.min_tokens || c * kC >= len) return;
    const int t0 = map.seq_start[s] + c * kC, nt = min(kC, len - c * kC);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // tokens past the portion's end: no key, no query, no decay.  Eight channels per thread and step, their loads in flight together
#pragma unroll
    for (int it = 0; it < kC * DK / 8 / 256; ++it) {
        const int idx = tid + it * 256, t = idx / (DK / 8), i = (idx - t * (DK / 8)) * 8;
        const bool live = t < nt;
        const size_t tok = (size_t)(t0 + min(t, nt - 1));
        const TQ *row = static_cast<const TQ *>(src.rows) + tok * src.ld + hk * DK + i;
        const float *dec = src.decay + tok * src.decay_ld + src.decay_off + (src.decay_dim == 1 ? h : h * DK + i);
        float k[8], q[8], g[8];
        load8<TQ>(row + src.k_off, k);
        load8<TQ>(row + src.q_off, q);
        if (src.decay_dim == 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) g[e] = dec[0];
        } else {
            load8<float>(dec, g);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            k[e] = live ? k[e] : 0.0f;
            q[e] = live ? q[e] * src.q_scale : 0.0f;
            g[e] = live ? g[e] : 1.0f;
        }
#pragma unroll
        for (int e = 0; e < 8; e += 4) {
            *reinterpret_cast<float4 *>(ks + t * P + i + e) = make_float4(k[e], k[e + 1], k[e + 2], k[e + 3]);
            *reinterpret_cast<float4 *>(qs + t * P + i + e) = make_float4(q[e], q[e + 1], q[e + 2], q[e + 3]);
            *reinterpret_cast<float4 *>(gs + t * P + i + e) = make_float4(g[e], g[e + 1], g[e + 2], g[e + 3]);
        }
    }
    for (int idx = tid; idx < 2 * kC * 36; idx += 256) As[idx] = 0.0f;
    if (DELTA && tid < kC) bs[tid] = tid < nt ? src.beta[(size_t)(t0 + tid) * src.beta_ld + h] : 0.0f;
    __syncthreads();

    // the two 16 x 16 blocks on the diagonal: a source token's key is carried forward, decayed step by step (a lane owns CH channels).  A warp carries FOUR
    // sources, so a target's rows are read from shared memory once for the four, and their four (eight) sums fold into one another on the way through the
    // warp: six (nine) shuffles instead of five for each.  (One source at a time: shared memory 0.68 busy, 45 us for 4096 tokens x 8 heads.)
    {
        const int b = warp >> 2, s0 = 16 * b + 4 * (warp & 3);
        float e[4][CH];
#pragma unroll
        for (int x = 0; x < 4; ++x) load_channels<CH>(ks + (s0 + x) * P + lane * CH, e[x]);
        for (int t = s0; t < 16 * b + 16; ++t) {
            float gt[CH], kt[CH], qt[CH], pv[4] = {}, av[4] = {};
            load_channels<CH>(gs + t * P + lane * CH, gt);
            load_channels<CH>(qs + t * P + lane * CH, qt);
            if (DELTA) load_channels<CH>(ks + t * P + lane * CH, kt);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int c2 = 0; c2 < CH; ++c2) {
                    if (t > s0 + x) e[x][c2] *= gt[c2];
                    if (DELTA) av[x] = fmaf(e[x][c2], kt[c2], av[x]);
                    pv[x] = fmaf(e[x][c2], qt[c2], pv[x]);
                }
            // (targets before a source: computed along, not stored)
            // (folded in 64 bits: seven levels of rounding in 32 were what set a read-out's error with strong decays)
            auto other = [](double v, int x) { return __shfl_xor_sync(0xffffffffu, v, x); };
            if (DELTA) {  // the lower half of the warp ends with p, the upper with a; source 2 (lane bit 8) + (lane bit 4)
                const bool up = lane & 16, up8 = lane & 8, up4 = lane & 4;
                double w[4], y[2];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = (double)(up ? av[x] : pv[x]) + (double)__shfl_xor_sync(0xffffffffu, up ? pv[x] : av[x], 16);
#pragma unroll
                for (int x = 0; x < 2; ++x) y[x] = (up8 ? w[2 + x] : w[x]) + other(up8 ? w[x] : w[2 + x], 8);
                double z = (up4 ? y[1] : y[0]) + other(up4 ? y[0] : y[1], 4);
                z += other(z, 2);
                z += other(z, 1);
                const int sr = s0 + 2 * (up8 ? 1 : 0) + (up4 ? 1 : 0);
                if ((lane & 3) == 0) {
                    if (!up && t >= sr) Ps[t * 36 + sr] = (float)z;
                    if (up && t > sr) As[t * 36 + sr] = (float)z;
                }
            } else {  // source 2 (lane bit 16) + (lane bit 8)
                const bool up = lane & 16, up8 = lane & 8;
                double y[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) y[x] = (double)(up ? pv[2 + x] : pv[x]) + (double)__shfl_xor_sync(0xffffffffu, up ? pv[x] : pv[2 + x], 16);
                double z = (up8 ? y[1] : y[0]) + other(up8 ? y[0] : y[1], 8);
                z += other(z, 4);
                z += other(z, 2);
                z += other(z, 1);
                const int sr = s0 + 2 * (up ? 1 : 0) + (up8 ? 1 : 0);
                if ((lane & 7) == 0 && t >= sr) Ps[t * 36 + sr] = (float)z;
            }
        }
    }
    __syncthreads();

    using B = Block<DK, DELTA>;
    static_assert(B::kFloats == block_floats(DK, DELTA), "the scratch is sized by block_floats");
    float *blk = blocks + ((size_t)(block_base(map, s) + blockIdx.x) * map.heads + h) * B::kFloats;
    // a thread owns a channel of one half of the chunk: products from the half's start and to its end.  In 64 bits, rounded once: products rounded decay by
    // decay leave a state whose decays are near 1 1.2 times as far from 64 bits as the serial kernels do
    const int half = tid / DK, i = tid - half * DK;
    if (half < 2) {
        double g = 1.0;
#pragma unroll 8
        for (int t = 0; t < 16; ++t) g *= (double)gs[(16 * half + t) * P + i];
        half_prod[half * DK + i] = g;
    }
    __syncthreads();
    if (half < 2) {
        const double before = half ? half_prod[i] : 1.0, after = half ? 1.0 : half_prod[DK + i];
        if (half == 0) blk[B::kG + i] = (float)(half_prod[i] * half_prod[DK + i]);
        double g = 1.0;
#pragma unroll 4
        for (int t = 15; t >= 0; --t) {  // g: after token t, to the end of the half
            const int row = 16 * half + t;
            blk[B::kKe + row * DK + i] = (float)((double)ks[row * P + i] * (g * after));
            g *= (double)gs[row * P + i];
        }
        g = 1.0;
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
            const int row = 16 * half + t;
            const float k = ks[row * P + i], q = qs[row * P + i];
            g *= (double)gs[row * P + i];
            const double p = before * g;
            if (DELTA) blk[B::kKp + row * DK + i] = (float)((double)k * p);
            blk[B::kQp + row * DK + i] = (float)((double)q * p);
            // the operands of the block below the diagonal replace the raw rows: targets from its start here, sources carried to the first half's end below
            if (half) ks[row * P + i] = k * (float)g, qs[row * P + i] = q * (float)g;
        }
        if (half == 0) {
            g = 1.0;
#pragma unroll 4
            for (int t = 15; t >= 0; --t) {
                ks[t * P + i] *= (float)g;
                g *= (double)gs[t * P + i];
            }
        }
    }
    __syncthreads();
    {  // the 16 x 16 block below the diagonal: one (target, source) pair per thread
        const int t = 16 + (tid >> 4), sr = tid & 15;
        float a[8] = {}, p[8] = {};
#pragma unroll 4
        for (int x = 0; x < DK; x += 4) {
            const int c = x & 4;  // (eight chains)
            const float4 f = *reinterpret_cast<const float4 *>(ks + sr * P + x), q = *reinterpret_cast<const float4 *>(qs + t * P + x);
            p[c] = fmaf(f.x, q.x, p[c]), p[c + 1] = fmaf(f.y, q.y, p[c + 1]), p[c + 2] = fmaf(f.z, q.z, p[c + 2]), p[c + 3] = fmaf(f.w, q.w, p[c + 3]);
            if (DELTA) {
                const float4 k = *reinterpret_cast<const float4 *>(ks + t * P + x);
                a[c] = fmaf(f.x, k.x, a[c]), a[c + 1] = fmaf(f.y, k.y, a[c + 1]), a[c + 2] = fmaf(f.z, k.z, a[c + 2]), a[c + 3] = fmaf(f.w, k.w, a[c + 3]);
            }
        }
        Ps[t * 36 + sr] = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
        if (DELTA) As[t * 36 + sr] = ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
    }
    __syncthreads();
    if (DELTA && warp == 0) {
        // Tb by forward substitution, a column per lane: x_t = beta_t ([t == lane] - sum_(r<t) A[t,r] x_r)
        float x[kC];
#pragma unroll
        for (int t = 0; t < kC; ++t) {
            float d[4] = {t == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int r = 0; r < t; ++r) d[r & 3] = fmaf(-As[t * 36 + r], x[r], d[r & 3]);
            x[t] = bs[t] * ((d[0] + d[1]) + (d[2] + d[3]));
            blk[B::kTb + t * kC + lane] = x[t];
        }
    } else {
        const int first = DELTA ? 32 : 0;
        for (int idx = tid - first; idx < kC * kC; idx += 256 - first) blk[B::kP + idx] = Ps[(idx >> 5) * 36 + (idx & 31)];
    }
}

// ---- the scan
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {  // two multiply-adds in one instruction, each rounded as fmaf rounds
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(*reinterpret_cast<unsigned long long *>(&d))
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)), "l"(*reinterpret_cast<const unsigned long long *>(&c)));
    return d;
}
__device__ __forceinline__ void cp16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// What bounds it: shared memory.  Per chunk the products are (2 or 3) x 32 x DK x 16 multiply-adds of operands that are used once, so they are shared out by how
// little each reads again:
//   read   [Kp; Qp] S   a warp takes 8 columns and a quarter of the rows; 16 lanes share a row, a lane holds its DK / 16 rows of S for the 8 columns in
//                       registers and reads each row of the factors once; eight shuffles fold the lanes' sums into one column per lane pair
//   solve  Tb R, P u    a thread takes a token and two columns, over the tokens up to its own
//   update S            a warp takes 16 rows of S, a lane 2 rows x 4 columns in registers for the whole portion: S <- p_C S, then one multiply-add per token in
//                       the tokens' order (the decayed, smaller ones first), and S^T goes to shared memory for the next read
// One stage of the block: its first part (Qp, Kp, V) is free behind the read and the second (the rest) behind the update, so either arrives while the other
// is used, and two CTAs share an SM.
template <typename TQ, int DK, bool DELTA> struct Scan {
    using B = Block<DK, DELTA>;
    static constexpr int kSP = DK + 4;                             // floats per column of S^T
    static constexpr int kUP = 20;                                 // floats per token of R, u, Qp S
    static constexpr int kVP = sizeof(TQ) == 2 ? 24 : 20;          // elements per staged value row
    static constexpr int kV = B::kFloats, kS = kV + kC * kVP * (int)sizeof(TQ) / 4, kR = kS + kCols * kSP, kQ = kR + kC * kUP, kU = kQ + kC * kUP;
    static constexpr int kFloats = kU + kC * kUP;                  // of shared memory
};

template <typename TQ, int DK, bool DELTA>
__global__ void __launch_bounds__(DK * 2, 2)
chunk_scan_kernel(const ChunkSource src, const ChunkMap map, const float *__restrict__ blocks, float *__restrict__ state, float *__restrict__ o) {
    using Sh = Scan<TQ, DK, DELTA>;
    using B = Block<DK, DELTA>;
    constexpr int NT = DK * 2, NW = NT / 32, KJ = DK / 64;    // threads, warps, 16-byte pieces of a row per lane
    constexpr int ROWS = DELTA ? 2 * kC : kC, PER = ROWS / (NW / 2);  // rows of [Kp; Qp], of a warp
    extern __shared__ __align__(16) float sm[];
    TQ *vs = reinterpret_cast<TQ *>(sm + Sh::kV);
    float *St = sm + Sh::kS, *R = sm + Sh::kR, *Qs = sm + Sh::kQ, *U = sm + Sh::kU;
    const int s = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kCols;
    const int start = map.seq_start[s], len = map.seq_start[s + 1] - start;
    if (len < map.min_tokens || map.first * kC >= len) return;
    const int n_chunks = min(map.count, (len + kC - 1) / kC - map.first);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const float *blk = blocks + ((size_t)block_base(map, s) * map.heads + h) * B::kFloats;
    auto load = [&](int c, int from, int to) {
        const float *b = blk + (size_t)c * map.heads * B::kFloats;
        for (int i = from / 4 + tid; i < to / 4; i += NT) cp16(sm + 4 * i, b + 4 * i);
    };
    auto load_first = [&](int c) {
        load(c, 0, B::kKe);
        constexpr int per = kCols * (int)sizeof(TQ) / 16;      // 16-byte pieces per value row
        for (int i = tid; i < kC * per; i += NT) {
            const int t = min((map.first + c) * kC + i / per, len - 1), e = i % per * (16 / (int)sizeof(TQ));  // past the end: a live row, which no key meets
            cp16(vs + (i / per) * Sh::kVP + e, static_cast<const TQ *>(src.rows) + (size_t)(start + t) * src.ld + src.v_off + h * map.vdim + j0 + e);
        }
        cp_commit();
    };
    load_first(0);
    // this lane's part of S: rows r0, r0 + 1, columns c0 .. c0 + 3
    const int r0 = 16 * w + 2 * (lane & 7), c0 = 4 * (lane >> 3);
    float S[2][4], S0[2][4];
    float *slot = state + ((size_t)map.seq_slot[s] * map.heads + h) * DK * map.vdim + j0;
    const bool fresh = map.first == 0 && map.seq_pos0[s] == 0;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[x][e] = fresh ? 0.0f : slot[(size_t)(r0 + x) * map.vdim + c0 + e];
    auto publish = [&]() {
#pragma unroll
        for (int e = 0; e < 4; ++e) *reinterpret_cast<float2 *>(St + (c0 + e) * Sh::kSP + r0) = make_float2(S[0][e], S[1][e]);
    };
    publish();
    const int t = tid / 8 % kC, cp = 2 * (tid & 7);            // a thread's token and columns of the solve (64-row states: of half the tokens)
    constexpr int TS = NT / 8;                                 // tokens per pass of the solve

    // The products multiply a token's vectors with those of the whole chunk, by zero where one must not see the other: an infinity or a NaN could reach what
    // came before it (0 x inf), and P and Tb gather sums that the serial kernels form token by token.  A chunk whose state or read-outs are not all finite
    // is run again from its first state, token by token, from the tokens' own vectors.
    bool bad = false;
    auto again = [&](int c) {
        const int hk = h / map.group;
        auto total = [&](float (&p)[4], float *buf) {          // sums over the rows of S for this lane's columns; buf [NW][kCols]
#pragma unroll
            for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int x = 1; x < 8; x <<= 1) p[e] += __shfl_xor_sync(0xffffffffu, p[e], x);
                if ((lane & 7) == 0) buf[w * kCols + c0 + e] = p[e];
            }
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                p[e] = 0.0f;
                for (int x = 0; x < NW; ++x) p[e] += buf[x * kCols + c0 + e];
            }
        };
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[x][e] = S0[x][e];
        for (int tt = (map.first + c) * kC, end = min(len, tt + kC); tt < end; ++tt) {
            const size_t tok = (size_t)(start + tt);
            const TQ *row = static_cast<const TQ *>(src.rows) + tok * src.ld;
            const float *dec = src.decay + tok * src.decay_ld + src.decay_off + (src.decay_dim == 1 ? h : h * DK);
            float k[2], q[2], p[4] = {}, u[4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                k[x] = Elem<TQ>::to_f(row[src.k_off + hk * DK + r0 + x]), q[x] = Elem<TQ>::to_f(row[src.q_off + hk * DK + r0 + x]) * src.q_scale;
                const float d = src.decay_dim == 1 ? dec[0] : dec[r0 + x];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S[x][e] *= d;
                    p[e] = fmaf(S[x][e], k[x], p[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) u[e] = Elem<TQ>::to_f(row[src.v_off + h * map.vdim + j0 + c0 + e]);
            if (DELTA) {
                total(p, Qs);
                const float beta = src.beta[tok * src.beta_ld + h];
#pragma unroll
                for (int e = 0; e < 4; ++e) u[e] = beta * (u[e] - p[e]);
            }
            float y[4] = {};
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    S[x][e] = fmaf(k[x], u[e], S[x][e]);
                    y[e] = fmaf(S[x][e], q[x], y[e]);
                }
            total(y, R);
            if (w == 0 && (lane & 7) == 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) o[(tok * map.heads + h) * map.vdim + j0 + c0 + e] = y[e];
            }
            if (!DELTA) __syncthreads();  // (the delta rule's first sum stands between two uses of the second's places)
        }
        publish();
        __syncthreads();
    };
    static_assert(NW * kCols <= kC * Sh::kUP, "the sums of `again` fit where the chunk's were");

    for (int c = 0; c < n_chunks; ++c) {
        cp_wait_all();
        if (__syncthreads_or(bad)) again(c - 1);               // (also: S^T and the first part are there, the second part is free)
        bad = false;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) S0[x][e] = S[x][e];
        load(c, B::kKe, B::kFloats);
        cp_commit();
        {   // read: rows `half` + 2 i of this warp's, 8 columns
            const int half = lane >> 4, l16 = lane & 15, cg = 8 * (w & 1);
            float4 Sr[8][KJ];
#pragma unroll
            for (int e = 0; e < 8; ++e)
#pragma unroll
                for (int j = 0; j < KJ; ++j) Sr[e][j] = *reinterpret_cast<const float4 *>(St + (cg + e) * Sh::kSP + 64 * j + 4 * l16);
            const int col = cg + (lane >> 1 & 4) + (lane >> 1 & 2) + (lane >> 1 & 1);  // the column whose sum this lane ends with
#pragma unroll 4
            for (int i = 0; i < PER / 2; ++i) {
                const int row = (w >> 1) * PER + 2 * i + half;  // (delta rule: rows kC .. are Kp's)
                float2 a2[8] = {};
#pragma unroll
                for (int j = 0; j < KJ; ++j) {
                    const float4 f = *reinterpret_cast<const float4 *>(sm + B::kQp + row * DK + 64 * j + 4 * l16);
#pragma unroll
                    for (int e = 0; e < 8; ++e) a2[e] = fma2(make_float2(f.z, f.w), make_float2(Sr[e][j].z, Sr[e][j].w), fma2(make_float2(f.x, f.y), make_float2(Sr[e][j].x, Sr[e][j].y), a2[e]));
                }
                float a[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) a[e] = a2[e].x + a2[e].y;
                const bool b8 = lane & 8, b4 = lane & 4, b2 = lane & 2;
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e] = (b8 ? a[e + 4] : a[e]) + __shfl_xor_sync(0xffffffffu, b8 ? a[e] : a[e + 4], 8);
#pragma unroll
                for (int e = 0; e < 2; ++e) a[e] = (b4 ? a[e + 2] : a[e]) + __shfl_xor_sync(0xffffffffu, b4 ? a[e] : a[e + 2], 4);
                a[0] = (b2 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, b2 ? a[0] : a[1], 2);
                a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
                if ((lane & 1) == 0) {
                    if (DELTA && row >= kC) R[(row - kC) * Sh::kUP + col] = Elem<TQ>::to_f(vs[(row - kC) * Sh::kVP + col]) - a[0];
                    else Qs[row * Sh::kUP + col] = a[0];
                }
            }
            if (!DELTA)
                for (int i = tid; i < kC * kCols; i += NT) U[i / kCols * Sh::kUP + i % kCols] = Elem<TQ>::to_f(vs[i / kCols * Sh::kVP + i % kCols]);
        }
        cp_wait_all();
        __syncthreads();                                       // R, Qp S (and u) are there, so is the second part; the first part is free
        if (c + 1 < n_chunks) load_first(c + 1);
        // sums over the tokens up to t of a row of Tb or P with two columns of R or u; `base` joins in front of the last group (see the update)
        auto solve = [&](const float *rows, const float *x, int tt, float2 base) -> float2 {
            float2 y = make_float2(0.0f, 0.0f);
            auto group = [&](int s4) {
                const float4 f = *reinterpret_cast<const float4 *>(rows + tt * kC + s4);
                const float ff[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) y = fma2(make_float2(ff[e], ff[e]), *reinterpret_cast<const float2 *>(x + (s4 + e) * Sh::kUP + cp), y);
            };
            const int last = tt & ~3;
#pragma unroll 2
            for (int s4 = 0; s4 < last; s4 += 4) group(s4);
            y.x += base.x, y.y += base.y;
            group(last);
            return y;
        };
        if (DELTA) {
#pragma unroll
            for (int tt = t; tt < kC; tt += TS) *reinterpret_cast<float2 *>(U + tt * Sh::kUP + cp) = solve(sm + B::kTb, R, tt, make_float2(0.0f, 0.0f));
            __syncthreads();
        }
        {   // update
            // all but the last four of the chunk's tokens are added up apart from the state: with decays near 1 their sum is smaller than it and so are its
            // roundings, with strong ones the last tokens are nearly all of it and round once
            const int live = min(kC, len - (map.first + c) * kC), apart = max(live - 4, 0);
            float2 d[2][2] = {};
            auto add = [&](int x, float2 (&to)[2][2]) {
                const float2 k = *reinterpret_cast<const float2 *>(sm + B::kKe + x * DK + r0);
                const float4 u = *reinterpret_cast<const float4 *>(U + x * Sh::kUP + c0);
                const float2 k0 = make_float2(k.x, k.x), k1 = make_float2(k.y, k.y), lo = make_float2(u.x, u.y), hi = make_float2(u.z, u.w);
                to[0][0] = fma2(k0, lo, to[0][0]), to[0][1] = fma2(k0, hi, to[0][1]);
                to[1][0] = fma2(k1, lo, to[1][0]), to[1][1] = fma2(k1, hi, to[1][1]);
            };
#pragma unroll 4
            for (int x = 0; x < apart; ++x) add(x, d);
            const float2 p = *reinterpret_cast<const float2 *>(sm + B::kG + r0);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) d[x][e] = fma2(make_float2(x ? p.y : p.x, x ? p.y : p.x), make_float2(S[x][2 * e], S[x][2 * e + 1]), d[x][e]);
#pragma unroll 4
            for (int x = apart; x < live; ++x) add(x, d);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) S[x][2 * e] = d[x][e].x, S[x][2 * e + 1] = d[x][e].y;
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int e = 0; e < 4; ++e) bad |= !(fabsf(S[x][e]) < INFINITY);
            publish();
        }
#pragma unroll
        for (int tt = t; tt < kC; tt += TS) {                  // read-outs
            const float2 y = solve(sm + B::kP, U, tt, *reinterpret_cast<const float2 *>(Qs + tt * Sh::kUP + cp));
            const int at = (map.first + c) * kC + tt;
            if (at < len) {
                *reinterpret_cast<float2 *>(o + ((size_t)(start + at) * map.heads + h) * map.vdim + j0 + cp) = y;
                bad |= !(fabsf(y.x) < INFINITY) || !(fabsf(y.y) < INFINITY);
            }
        }
    }
    if (__syncthreads_or(bad)) again(n_chunks - 1);
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) slot[(size_t)(r0 + x) * map.vdim + c0 + e] = S[x][e];
}

template <typename TQ, int DK, bool DELTA>
int launch_chunks_t(const ChunkSource &src, ChunkMap map, float *scratch, size_t scratch_floats, float *state, float *o, int n_seqs, int tokens, int longest,
                    cudaStream_t st) {
    const size_t per_block = (size_t)map.heads * block_floats(DK, DELTA);
    const size_t fit = scratch_floats / per_block;  // (chunk, all heads) blocks the scratch holds
    const int chunks = (longest + kC - 1) / kC;
    map.packed = fit >= (size_t)(tokens / kC + n_seqs + 1);
    map.count = map.packed ? chunks : (int)std::min<size_t>(fit / n_seqs, chunks);
    if (map.count == 0) return B200_ERR_UNSUPPORTED;
    const size_t smem_f = (size_t)(3 * kC * (DK + 4) + 2 * kC * 36 + 4 * DK + kC) * sizeof(float);
    const size_t scan_smem = Scan<TQ, DK, DELTA>::kFloats * sizeof(float);
    auto fk = chunk_factors_kernel<TQ, DK, DELTA>;
    auto sk = chunk_scan_kernel<TQ, DK, DELTA>;
    cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_f);
    cudaFuncSetAttribute(sk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scan_smem);
    for (map.first = 0; map.first < chunks; map.first += map.count) {
        const int n = std::min(map.count, chunks - map.first);
        launch_plain(fk, dim3(n, map.heads, n_seqs), dim3(256), smem_f, st, src, map, scratch);
        launch_plain(sk, dim3(map.vdim / kCols, map.heads, n_seqs), dim3(DK * 2), scan_smem, st, src, map, scratch, state, o);
    }
    return cuda_status("chunk recurrence launch");
}

}  // namespace

size_t chunk_scratch_floats(int heads, int dim, bool delta, int max_tokens, int max_seqs) {
    if (dim != 64 && dim != 128) return 0;
    const size_t per_block = (size_t)heads * block_floats(dim, delta);
    // all chunks of a call at once, or 64 MB of them (never less than one chunk per sequence)
    const size_t all = (size_t)max_tokens / kC + max_seqs + 1, some = std::max<size_t>((64u << 20) / (per_block * sizeof(float)), max_seqs);
    return std::min(all, some) * per_block;
}

int launch_chunk_gla(int dtype, const void *proj, int ld, const float *decay, float *state, float *o, const int *seq_start, const int *seq_pos0,
                     const int *seq_slot, int n_seqs, int heads, int dim, int vdim, float *scratch, size_t scratch_floats, int tokens, int longest,
                     cudaStream_t st) {
    const int es = dtype == B200_F32 ? 4 : 2;
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || ld * es % 16 != 0 || 2 * heads * dim * es % 16 != 0 || !all_aligned16({proj, decay, o, scratch}) || !scratch) return B200_ERR_UNSUPPORTED;
    const ChunkSource src = {proj, ld, 0, heads * dim, 2 * heads * dim, decay, heads * dim, 0, dim, nullptr, 0, 1.0f / sqrtf((float)dim)};
    const ChunkMap map = {seq_start, seq_pos0, seq_slot, heads, 1, vdim, kChunkMinTokens, 0, 0, 0};
    B200_DISPATCH_DTYPE(dtype, {
        return dim == 64 ? launch_chunks_t<T, 64, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st)
                         : launch_chunks_t<T, 128, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st);
    });
    return B200_ERR_UNSUPPORTED;
}

int launch_chunk_delta(const float *rec, float *state, float *o, const int *seq_start, const int *seq_pos0, const int *seq_slot, int n_seqs, int heads,
                       int kv_heads, int dim, int vdim, float *scratch, size_t scratch_floats, int tokens, int longest, cudaStream_t st) {
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || !all_aligned16({rec, o, scratch}) || !scratch) return B200_ERR_UNSUPPORTED;
    const DeltaRow lay = delta_row(heads, kv_heads, dim, vdim);  // (every segment of the row starts on a 16-byte boundary)
    const ChunkSource src = {rec, lay.ld, lay.q, lay.k, lay.v, rec, lay.ld, lay.decay, dim, rec + lay.beta, lay.ld, 1.0f};
    const ChunkMap map = {seq_start, seq_pos0, seq_slot, heads, heads / kv_heads, vdim, kChunkMinTokens, 0, 0, 0};
    return dim == 64 ? launch_chunks_t<float, 64, true>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st)
                     : launch_chunks_t<float, 128, true>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st);
}

int launch_chunk_decay(const float *rec, float *state, float *o, const int *seq_start, const int *seq_pos0, const int *seq_slot, int n_seqs, int heads,
                       int kv_heads, int dim, int vdim, float *scratch, size_t scratch_floats, int tokens, int longest, cudaStream_t st) {
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || !all_aligned16({rec, o, scratch}) || !scratch) return B200_ERR_UNSUPPORTED;
    const DecayRow lay = decay_row(heads, kv_heads, dim, vdim);
    const ChunkSource src = {rec, lay.ld, lay.q, lay.k, lay.v, rec, lay.ld, lay.decay, 1, nullptr, 0, 1.0f};
    const ChunkMap map = {seq_start, seq_pos0, seq_slot, heads, heads / kv_heads, vdim, kChunkMinTokens, 0, 0, 0};
    return dim == 64 ? launch_chunks_t<float, 64, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st)
                     : launch_chunks_t<float, 128, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st);
}

}  // namespace b200

using namespace b200;

extern "C" {

size_t b200_chunk_recurrence_scratch_bytes(int kind, int heads, int dim, int max_tokens, int max_seqs) {
    if (heads < 1 || max_tokens < 0 || max_seqs < 1) return 0;
    return chunk_scratch_floats(heads, dim, kind == B200_MIXER_DELTA, max_tokens, max_seqs) * sizeof(float);
}

int b200_chunk_recurrence(int kind, const void *rows, int ld, const float *decay, float *state, float *o, const int *seq_start, const int *seq_pos0,
                          const int *seq_slot, int n_seqs, int heads, int kv_heads, int dim, int vdim, void *scratch, size_t scratch_bytes, int tokens,
                          int longest, int dtype, b200_stream_t stream) {
    B200_REQUIRE(rows && state && o && seq_start && seq_pos0 && seq_slot && scratch, "chunk_recurrence: null pointer");
    B200_REQUIRE(n_seqs >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0 && tokens >= 0 && longest >= 0, "chunk_recurrence: bad shape");
    if (n_seqs == 0 || longest < kChunkMinTokens) return B200_OK;
    float *sc = static_cast<float *>(scratch);
    const size_t floats = scratch_bytes / sizeof(float);
    const float *rec = static_cast<const float *>(rows);
    if (kind == B200_MIXER_GLA) {
        B200_REQUIRE(decay && kv_heads == heads && ld >= 2 * heads * dim + heads * vdim, "chunk_recurrence: bad gated linear attention");
        return launch_chunk_gla(dtype, rows, ld, decay, state, o, seq_start, seq_pos0, seq_slot, n_seqs, heads, dim, vdim, sc, floats, tokens, longest, as_stream(stream));
    }
    B200_REQUIRE(dtype == B200_F32 && (kind == B200_MIXER_DELTA || kind == B200_MIXER_LINEAR), "chunk_recurrence: kind %d, dtype %d", kind, dtype);
    if (kind == B200_MIXER_DELTA)
        return launch_chunk_delta(rec, state, o, seq_start, seq_pos0, seq_slot, n_seqs, heads, kv_heads, dim, vdim, sc, floats, tokens, longest, as_stream(stream));
    return launch_chunk_decay(rec, state, o, seq_start, seq_pos0, seq_slot, n_seqs, heads, kv_heads, dim, vdim, sc, floats, tokens, longest, as_stream(stream));
}

}  // extern "C"
