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
// Measured (B200, 8 heads, dim 128, vdim 256; factors + scan against the serial kernel): linear attention of 4096 tokens 39 + 218 against 690 us, delta rule of
// 1500, 511 and 900 tokens 42 + 212 against 401.
#include "hybrid_ops.cuh"

#include <algorithm>
#include <type_traits>

namespace b200 {

namespace {

constexpr int kC = 32;      // tokens per chunk
constexpr int kCols = 16;   // columns of S per CTA of the scan

// one (chunk, head) block, rows as the scan has them in shared memory: Qp, (delta rule: Kp,) Ke [kC][kP], P [kC][kTP], p_C [DK], (Tb [kC][kTP])
constexpr int kTP = 40;  // floats per row of P and Tb and per column of V^T
template <int DK, bool DELTA> struct Block {
    static constexpr int kP = DK + 8;  // floats per row of the factors and per column of S^T: rows start 8 banks apart
    static constexpr int kQp = 0, kKp = kC * kP, kKe = (DELTA ? 2 : 1) * kC * kP, kPm = kKe + kC * kP, kG = kPm + kC * kTP, kTb = kG + DK;
    static constexpr int kFloats = kTb + (DELTA ? kC * kTP : 0);
};
__host__ __device__ constexpr int block_floats(int dk, bool delta) { return (delta ? 3 : 2) * kC * (dk + 8) + (delta ? 2 : 1) * kC * kTP + dk; }

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
            blk[B::kKe + row * B::kP + i] = (float)((double)ks[row * P + i] * (g * after));
            g *= (double)gs[row * P + i];
        }
        g = 1.0;
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
            const int row = 16 * half + t;
            const float k = ks[row * P + i], q = qs[row * P + i];
            g *= (double)gs[row * P + i];
            const double p = before * g;
            if (DELTA) blk[B::kKp + row * B::kP + i] = (float)((double)k * p);
            blk[B::kQp + row * B::kP + i] = (float)((double)q * p);
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
            blk[B::kTb + t * kTP + lane] = x[t];
        }
    } else {
        const int first = DELTA ? 32 : 0;
        for (int idx = tid - first; idx < kC * kC; idx += 256 - first) blk[B::kPm + (idx >> 5) * kTP + (idx & 31)] = Ps[(idx >> 5) * 36 + (idx & 31)];
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

// What bounds it: fp32 multiply-adds and shared memory, about evenly: per chunk (2 or 3) x 32 x DK x 16 multiply-adds and as many again for the update, of
// operands that are used once.  Products are thread tiles, so that an operand read serves four multiply-adds:
//   read   [Kp; Qp] S   4 rows x 4 columns per thread over a quarter of k (linear attention: an eighth, and P V joins as 32 more k), four lanes' sums folded
//                       into four outputs of each
//   solve  Tb R, P u    a token and two columns per thread, over the tokens up to its own
//   update S            4 rows x 2 columns per thread, held in registers for the whole portion: S <- p_C S, then one multiply-add per token in the tokens'
//                       order (the decayed, smaller ones first), and S^T goes to shared memory for the next read
// A warp's 16-byte reads have at most eight addresses in each half, on different banks (pitches of 8 or 4 modulo 32 floats).  Linear attention's read and
// update touch different copies of S^T, so a chunk has two barriers; its factors have two stages.  The delta rule has three barriers and one stage, whose first
// part (Qp, Kp) is free behind the read and the second (the rest) behind the update, so either arrives while the other is used.  Two CTAs share an SM.
// Measured (the sizes above): 218 and 212 us; a row of the factors at a time, folded by eight shuffles, 16-byte reads that shared no addresses between
// neighbouring lanes, values waited for within their chunk and factors copied row by row: 326 and 289 us.  Linear attention with read and update in different
// warps of one CTA: 209 us, but 238 against 220 (with the factors) for four portions of 1024.
template <int DK, bool DELTA> struct Scan {
    using B = Block<DK, DELTA>;
    static constexpr int kP = B::kP, kStage = B::kFloats;
    static constexpr int kStages = DELTA ? 1 : 2;
    static constexpr int KW = DELTA ? 1 : DK / 64;      // warps that share the k of a row group (linear attention)
    static constexpr int kS = kStages * kStage, kV = kS + kStages * kCols * kP, kR = kV + kStages * kCols * kTP;
    static constexpr int kUP = 36;                      // floats per column of R^T, (Qp S)^T, u^T: 4 banks apart, for eight columns at a time
    static constexpr int kPart = 20;                    // floats per token of the partial outputs
    static constexpr int kFloats = kR + (DELTA ? 3 * kCols * kUP : KW * kC * kPart);
};

template <typename TQ, int DK, bool DELTA>
__global__ void __launch_bounds__(DK * 2, 2)
chunk_scan_kernel(const ChunkSource src, const ChunkMap map, const float *__restrict__ blocks, float *__restrict__ state, float *__restrict__ o) {
    using Sh = Scan<DK, DELTA>;
    using B = Block<DK, DELTA>;
    constexpr int NT = DK * 2, NW = NT / 32, P = Sh::kP, TP = kTP, UP = Sh::kUP, RW = DK / 32;  // threads, warps, pitches, warps that share the rows of S
    extern __shared__ __align__(16) float sm[];
    float *const St = sm + Sh::kS, *const VT = sm + Sh::kV, *const RT = sm + Sh::kR, *const QT = RT + kCols * UP, *const UT = QT + kCols * UP;
    const int s = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kCols;
    const int start = map.seq_start[s], len = map.seq_start[s + 1] - start;
    if (len < map.min_tokens || map.first * kC >= len) return;
    const int n_chunks = min(map.count, (len + kC - 1) / kC - map.first);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const float *blk = blocks + ((size_t)block_base(map, s) * map.heads + h) * B::kFloats;
    // floats [from, to) of chunk c's block into its stage
    auto load = [&](int c, auto from, auto to) {
        constexpr int at = decltype(from)::value, n = (decltype(to)::value - at) / 4;
        const float *b = blk + (size_t)c * map.heads * B::kFloats + at + 4 * tid;
        float *st = sm + (c % Sh::kStages) * Sh::kStage + at + 4 * tid;
#pragma unroll
        for (int i = 0; i < (n + NT - 1) / NT; ++i)
            if ((i + 1) * NT <= n || tid + i * NT < n) cp16(st + 4 * i * NT, b + 4 * i * NT);
    };
    constexpr std::integral_constant<int, 0> first{};          // (delta rule: the parts of a block, see below)
    constexpr std::integral_constant<int, B::kKe> second{};
    constexpr std::integral_constant<int, B::kFloats> end{};
    // values: a thread's two columns of one or two tokens, on their way in registers for two chunks (32 bytes of every row: one chunk ahead, linear attention
    // waited for them, 60 of 320 us), then columns of V^T
    constexpr int VN = kC * 8 / NT;
    using Pair = typename std::conditional<sizeof(TQ) == 2, uint32_t, float2>::type;
    Pair vreg[2][VN];  // of this chunk's successor and the one behind it, as they come: a conversion at the load would wait for it
    auto load_values = [&](int c, Pair (&to)[VN]) {
#pragma unroll
        for (int x = 0; x < VN; ++x) {
            const int t = min((map.first + c) * kC + (tid >> 3) + x * (NT / 8), len - 1);  // past the end: a live row, which no key meets
            const TQ *v = static_cast<const TQ *>(src.rows) + (size_t)(start + t) * src.ld + src.v_off + h * map.vdim + j0 + 2 * (tid & 7);
            to[x] = *reinterpret_cast<const Pair *>(v);  // (aligned: rows and segments start on 16-byte boundaries)
        }
    };
    auto put_values = [&](int c, const Pair (&from)[VN]) {
        float *to = VT + (c % Sh::kStages) * kCols * TP;
#pragma unroll
        for (int x = 0; x < VN; ++x) {
            const int t = (tid >> 3) + x * (NT / 8), e = 2 * (tid & 7);
            const TQ *v = reinterpret_cast<const TQ *>(&from[x]);
            to[e * TP + t] = Elem<TQ>::to_f(v[0]), to[(e + 1) * TP + t] = Elem<TQ>::to_f(v[1]);
        }
    };
    if constexpr (DELTA) load(0, first, second);
    else load(0, first, end);
    cp_commit();
    load_values(0, vreg[1]);
    load_values(1, vreg[0]);
    put_values(0, vreg[1]);
    // this lane's part of S: rows r0 .. r0 + 3, columns cp and cp + 8
    const int r0 = 4 * ((lane >> 1 & 1) + 2 * (lane >> 3) + 8 * (w % RW)), cp = (lane & 1) + 2 * (lane >> 2 & 1) + 4 * (w / RW);
    float S[4][2], S0[4][2];
    float *slot = state + ((size_t)map.seq_slot[s] * map.heads + h) * DK * map.vdim + j0 + cp;
    const bool fresh = map.first == 0 && map.seq_pos0[s] == 0;
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) S[x][e] = fresh ? 0.0f : slot[(size_t)(r0 + x) * map.vdim + 8 * e];
    auto publish = [&](int c) {  // for chunk c to read
        float *to = St + (c % Sh::kStages) * kCols * P;
#pragma unroll
        for (int e = 0; e < 2; ++e) *reinterpret_cast<float4 *>(to + (cp + 8 * e) * P + r0) = make_float4(S[0][e], S[1][e], S[2][e], S[3][e]);
    };
    publish(0);

    // The products multiply a token's vectors with those of the whole chunk, by zero where one must not see the other: an infinity or a NaN could reach what
    // came before it (0 x inf), and P and Tb gather sums that the serial kernels form token by token.  A chunk whose state or read-outs are not all finite
    // is run again from its first state, token by token, from the tokens' own vectors.
    bool bad = false;
    auto again = [&](int c) {
        const int hk = h / map.group;
        auto total = [&](float (&p)[2], float *buf) {          // sums over the rows of S for this lane's columns; buf [RW][kCols]
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int x = 2; x < 32; x <<= x == 2 ? 2 : 1) p[e] += __shfl_xor_sync(0xffffffffu, p[e], x);  // (the lane bits of r0: 1, 3, 4)
                if ((lane & 26) == 0) buf[w % RW * kCols + cp + 8 * e] = p[e];
            }
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                p[e] = 0.0f;
                for (int x = 0; x < RW; ++x) p[e] += buf[x * kCols + cp + 8 * e];
            }
        };
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) S[x][e] = S0[x][e];
        for (int tt = (map.first + c) * kC, end = min(len, tt + kC); tt < end; ++tt) {
            const size_t tok = (size_t)(start + tt);
            const TQ *row = static_cast<const TQ *>(src.rows) + tok * src.ld;
            const float *dec = src.decay + tok * src.decay_ld + src.decay_off + (src.decay_dim == 1 ? h : h * DK);
            float k[4], q[4], p[2] = {}, u[2];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                k[x] = Elem<TQ>::to_f(row[src.k_off + hk * DK + r0 + x]), q[x] = Elem<TQ>::to_f(row[src.q_off + hk * DK + r0 + x]) * src.q_scale;
                const float d = src.decay_dim == 1 ? dec[0] : dec[r0 + x];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    S[x][e] *= d;
                    p[e] = fmaf(S[x][e], k[x], p[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) u[e] = Elem<TQ>::to_f(row[src.v_off + h * map.vdim + j0 + cp + 8 * e]);
            if (DELTA) {
                total(p, RT + RW * kCols);
                const float beta = src.beta[tok * src.beta_ld + h];
#pragma unroll
                for (int e = 0; e < 2; ++e) u[e] = beta * (u[e] - p[e]);
            }
            float y[2] = {};
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    S[x][e] = fmaf(k[x], u[e], S[x][e]);
                    y[e] = fmaf(S[x][e], q[x], y[e]);
                }
            total(y, RT);
            if (w % RW == 0 && (lane & 26) == 0) {
#pragma unroll
                for (int e = 0; e < 2; ++e) o[(tok * map.heads + h) * map.vdim + j0 + cp + 8 * e] = y[e];
            }
            if (!DELTA) __syncthreads();  // (the delta rule's first sum stands between two uses of the second's places)
        }
        publish(c + 1);
        __syncthreads();
    };
    static_assert(2 * RW * kCols <= Sh::kFloats - Sh::kR, "the sums of `again` fit where the chunk's were");

    // sums of 4 rows x 4 columns over this lane's k: a[i] rows of the first operand, b[j] columns of the second, `step` floats from one access to the next
    auto tile = [&](float2 (&acc)[4][4], const float *const (&a)[4], const float *const (&b)[4], int n, int step) {
#pragma unroll 4
        for (int x = 0; x < n; ++x) {
            float4 f[4], g[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = *reinterpret_cast<const float4 *>(a[i] + x * step), g[i] = *reinterpret_cast<const float4 *>(b[i] + x * step);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    acc[i][j] = fma2(make_float2(f[i].z, f[i].w), make_float2(g[j].z, g[j].w), fma2(make_float2(f[i].x, f[i].y), make_float2(g[j].x, g[j].y), acc[i][j]));
        }
    };
    // four lanes (bits 3 and 4) fold their 16 sums: a lane ends with row ks of the tile
    auto fold4 = [&](const float2 (&acc)[4][4], float (&y)[4]) {
        const bool hi = lane & 16, lo = lane & 8;
        float m[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float u = acc[i][j].x + acc[i][j].y, v = acc[2 + i][j].x + acc[2 + i][j].y;
                m[i][j] = (hi ? v : u) + __shfl_xor_sync(0xffffffffu, hi ? u : v, 16);
            }
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = (lo ? m[1][j] : m[0][j]) + __shfl_xor_sync(0xffffffffu, lo ? m[0][j] : m[1][j], 8);
    };
    // A 16-byte access of a warp takes two cycles where lanes share addresses with the lane beside them (bit 0) or the one after it (bit 1), four where they do not
    // (measured): rows are shared across bit 0, columns across bit 1, and the four lanes of a sum lie eight apart.
    const int ks = lane >> 3, cg = (lane & 1) + 2 * (lane >> 2 & 1), rg = lane >> 1 & 1;
    auto row_of = [&](int g, int i) { return 8 * g + rg + 2 * i; };
    auto col_of = [&](int j) { return cg + 4 * j; };
    // the delta rule's sums over the sources of a token, row t of `rows` with columns st_c and st_c + 8 of x: a thread's own, over the tokens up to its own.  The
    // last four hold the largest terms: they come last, behind `base`, one rounding a term (folded with the others, states came out 1.2 to 1.4 times as far from
    // 64 bits as the serial kernels').  As 4 x 4 tiles over eight lanes this took 2400 instructions of a chunk's 9400 in selects and shuffles.
    const int st_t = (lane & 1) + 2 * (lane >> 4) + 4 * w, st_c = lane >> 1 & 7;
    auto solve = [&](const float *rows, const float *x, int t, float2 y) -> float2 {
        float2 a = make_float2(0.0f, 0.0f), b = a;
        const int last = t & ~3;
#pragma unroll 2
        for (int s4 = 0; s4 < last; s4 += 4) {
            const float4 f = *reinterpret_cast<const float4 *>(rows + t * TP + s4);
            const float4 u = *reinterpret_cast<const float4 *>(x + st_c * UP + s4), v = *reinterpret_cast<const float4 *>(x + (st_c + 8) * UP + s4);
            a = fma2(make_float2(f.z, f.w), make_float2(u.z, u.w), fma2(make_float2(f.x, f.y), make_float2(u.x, u.y), a));
            b = fma2(make_float2(f.z, f.w), make_float2(v.z, v.w), fma2(make_float2(f.x, f.y), make_float2(v.x, v.y), b));
        }
        y.x += a.x + a.y, y.y += b.x + b.y;
        const float4 f = *reinterpret_cast<const float4 *>(rows + t * TP + last);
        const float4 u = *reinterpret_cast<const float4 *>(x + st_c * UP + last), v = *reinterpret_cast<const float4 *>(x + (st_c + 8) * UP + last);
        y = fma2(make_float2(f.x, f.x), make_float2(u.x, v.x), y), y = fma2(make_float2(f.y, f.y), make_float2(u.y, v.y), y);
        return fma2(make_float2(f.w, f.w), make_float2(u.w, v.w), fma2(make_float2(f.z, f.z), make_float2(u.z, v.z), y));
    };

    for (int c = 0; c < n_chunks; ++c) {
        const float *const stage = sm + (c % Sh::kStages) * Sh::kStage, *const Sc = St + (c % Sh::kStages) * kCols * P, *const Vc = VT + (c % Sh::kStages) * kCols * TP;
        cp_wait_all();
        if (__syncthreads_or(bad)) again(c - 1);               // (also: S^T, V^T and the (first part of the) stage are there; what they replace is free)
        bad = false;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) S0[x][e] = S[x][e];
        if constexpr (DELTA) load(c, second, end);
        else if (c + 1 < n_chunks) load(c + 1, first, end);
        cp_commit();
        load_values(c + 2, vreg[1]);
        // ---- read
        if constexpr (DELTA) {
            for (int g = w; g < 2 * kC / 8; g += NW) {         // rows 0 .. kC - 1 are Qp's, then Kp's
                float2 acc[4][4] = {};
                const float *a[4], *b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = stage + row_of(g, i) * P + 4 * ks, b[i] = Sc + col_of(i) * P + 4 * ks;
                tile(acc, a, b, DK / 16, 16);
                float y[4];
                fold4(acc, y);
                const int row = row_of(g, ks);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (row >= kC) RT[col_of(j) * UP + row - kC] = Vc[col_of(j) * TP + row - kC] - y[j];
                    else QT[col_of(j) * UP + row] = y[j];
                }
            }
            cp_wait_all();
            __syncthreads();                                   // R, Qp S are there, so is the second part; Qp, Kp, S^T and V^T are free
            if (c + 1 < n_chunks) load(c + 1, first, second);
            cp_commit();
#pragma unroll
            for (int t = st_t; t < kC; t += 4 * NW) {
                const float2 u = solve(stage + B::kTb, RT, t, make_float2(0.0f, 0.0f));
                UT[st_c * UP + t] = u.x, UT[(st_c + 8) * UP + t] = u.y;
            }
            __syncthreads();
        } else {
            constexpr int KW = Sh::KW;
            const int g = w / KW, kw = w % KW;                 // row group, share of k
            float2 acc[4][4] = {};
            const float *a[4], *b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = stage + row_of(g, i) * P + kw * (DK / KW) + 4 * ks, b[i] = Sc + col_of(i) * P + kw * (DK / KW) + 4 * ks;
            tile(acc, a, b, DK / KW / 16, 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = stage + B::kPm + row_of(g, i) * TP + kw * (kC / KW) + 4 * ks, b[i] = Vc + col_of(i) * TP + kw * (kC / KW) + 4 * ks;
            tile(acc, a, b, kC / KW / 16, 16);
            float y[4];
            fold4(acc, y);
#pragma unroll
            for (int j = 0; j < 4; ++j) RT[(kw * kC + row_of(g, ks)) * Sh::kPart + col_of(j)] = y[j];
        }
        {   // ---- update
            // all but the chunk's last (up to four) tokens are added up apart from the state: with decays near 1 their sum is smaller than it and so are its
            // roundings, with strong ones the last tokens are nearly all of it and round once
            const int last = (min(kC, len - (map.first + c) * kC) - 1) & ~3;  // (tokens past the end: keys of zero)
            constexpr int VP = DELTA ? UP : TP;
            const float *const Ke = stage + B::kKe + r0, *const U = DELTA ? UT : Vc;
            float2 d[2][2] = {};
            auto add = [&](int x) {
                const float4 u0 = *reinterpret_cast<const float4 *>(U + cp * VP + x), u1 = *reinterpret_cast<const float4 *>(U + (cp + 8) * VP + x);
                const float a0[4] = {u0.x, u0.y, u0.z, u0.w}, a1[4] = {u1.x, u1.y, u1.z, u1.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 k = *reinterpret_cast<const float4 *>(Ke + (x + i) * P);
                    const float2 lo = make_float2(k.x, k.y), hi = make_float2(k.z, k.w), v0 = make_float2(a0[i], a0[i]), v1 = make_float2(a1[i], a1[i]);
                    d[0][0] = fma2(lo, v0, d[0][0]), d[0][1] = fma2(hi, v0, d[0][1]);
                    d[1][0] = fma2(lo, v1, d[1][0]), d[1][1] = fma2(hi, v1, d[1][1]);
                }
            };
#pragma unroll 2
            for (int x = 0; x < last; x += 4) add(x);
            const float4 p = *reinterpret_cast<const float4 *>(stage + B::kG + r0);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                d[e][0] = fma2(make_float2(p.x, p.y), make_float2(S[0][e], S[1][e]), d[e][0]);
                d[e][1] = fma2(make_float2(p.z, p.w), make_float2(S[2][e], S[3][e]), d[e][1]);
            }
            add(last);
#pragma unroll
            for (int e = 0; e < 2; ++e) S[0][e] = d[e][0].x, S[1][e] = d[e][0].y, S[2][e] = d[e][1].x, S[3][e] = d[e][1].y;
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) bad |= !(fabsf(S[x][e]) < INFINITY);
            publish(c + 1);
            if (c + 1 < n_chunks) put_values(c + 1, vreg[0]);
#pragma unroll
            for (int x = 0; x < VN; ++x) vreg[0][x] = vreg[1][x];
        }
        // ---- read-outs
        auto finite = [&](float2 y) { return fabsf(y.x) < INFINITY && fabsf(y.y) < INFINITY; };
        auto out = [&](int t) { return o + ((size_t)(start + (map.first + c) * kC + t) * map.heads + h) * map.vdim + j0; };
        const int live = min(kC, len - (map.first + c) * kC);
        if constexpr (DELTA) {
#pragma unroll
            for (int t = st_t; t < kC; t += 4 * NW) {
                const float2 y = solve(stage + B::kPm, UT, t, make_float2(QT[st_c * UP + t], QT[(st_c + 8) * UP + t]));
                if (t < live) {
                    out(t)[st_c] = y.x, out(t)[st_c + 8] = y.y;
                    bad |= !finite(y);
                }
            }
        } else {
            __syncthreads();                                   // the partial sums are there
#pragma unroll
            for (int x = 0; x < VN; ++x) {
                const int t = (tid >> 3) + x * (NT / 8), e = 2 * (tid & 7);
                float2 y = *reinterpret_cast<const float2 *>(RT + t * Sh::kPart + e);
#pragma unroll
                for (int kw = 1; kw < Sh::KW; ++kw) {
                    const float2 z = *reinterpret_cast<const float2 *>(RT + (kw * kC + t) * Sh::kPart + e);
                    y.x += z.x, y.y += z.y;
                }
                if (t < live) {
                    *reinterpret_cast<float2 *>(out(t) + e) = y;
                    bad |= !finite(y);
                }
            }
        }
    }
    if (__syncthreads_or(bad)) again(n_chunks - 1);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) slot[(size_t)(r0 + x) * map.vdim + 8 * e] = S[x][e];
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
    const size_t scan_smem = Scan<DK, DELTA>::kFloats * sizeof(float);
    auto fk = chunk_factors_kernel<TQ, DK, DELTA>;
    auto sk = chunk_scan_kernel<TQ, DK, DELTA>;
    allow_smem(fk);
    allow_smem(sk);
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
