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
//   chunk_factors_kernel  one CTA per (chunk, head), all chunks at once: Kp, Qp, Ke, P, Tb, p_C, stored in the order in which the lanes of
//                         the second kernel's matrix instructions hold them
//   chunk_scan_kernel     one CTA per (16 columns of S, head, sequence): S^T stays in the accumulators of its warps (16 rows of S each) and
//                         is the A operand of the next chunk's products as it stands -- with the key rows taken in the order the
//                         accumulators hold them nothing is shuffled or stored between chunks
// The products run on mma.sync m16n8k8 with every fp32 operand split in two TF32 halves and the three products that matter (the
// low x low one is below fp32's last bit): fp32 accuracy, measured against 64 bits beside the serial kernels.  tcgen05 has no place here: a
// chunk step is a chain of 16 x 64 x 128-sized products whose results are the next one's operands, bound by latency.
// Measured (B200, 8 heads, dim 128, vdim 256): see the dispatch rule at the end of this file.
#include "hybrid_ops.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kC = 32;      // tokens per chunk
constexpr int kCols = 16;   // columns of S per CTA of the scan (the M of its matrix instructions)

// floats of one (chunk, head) block: Qp, Ke [kC x DK], P [kC x kC], p_C [DK]; the delta rule's go on with Kp [kC x DK], Tb [kC x kC]
__host__ __device__ constexpr int block_floats(int dk, bool delta) { return 2 * kC * dk + kC * kC + dk + (delta ? kC * dk + kC * kC : 0); }

// element (t, s) of P or Tb in fragment order: column tile t / 8, two k-steps of 8 per 16-byte piece; the k order inside a step is the
// accumulators' (lane pairs 2j, 2j + 1)
__device__ __forceinline__ int frag_ts(int t, int s) {
    return ((((t >> 3) * 2 + (s >> 4)) * 32 + (t & 7) * 4 + ((s & 7) >> 1)) << 2) + ((s >> 3) & 1) * 2 + (s & 1);
}

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
__global__ void __launch_bounds__(256)
chunk_factors_kernel(const ChunkSource src, const ChunkMap map, float *__restrict__ blocks) {
    constexpr int P = DK + 4;  // row pitch: rows read by neighbouring lanes start four banks apart
    constexpr int CH = DK / 32;
    extern __shared__ __align__(16) float sm[];
    float *ks = sm, *qs = ks + kC * P, *gs = qs + kC * P;  // [kC][P] each
    float *As = gs + kC * P, *Ps = As + kC * 36;           // [kC][36]
    float *half_prod = Ps + kC * 36;                       // [2][DK]
    float *bs = half_prod + 2 * DK;                        // [kC]
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
            if (DELTA) {  // the lower half of the warp ends with p, the upper with a; source 2 (lane bit 8) + (lane bit 4)
                const bool up = lane & 16, up8 = lane & 8, up4 = lane & 4;
                float w[4], y[2];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = (up ? av[x] : pv[x]) + __shfl_xor_sync(0xffffffffu, up ? pv[x] : av[x], 16);
#pragma unroll
                for (int x = 0; x < 2; ++x) y[x] = (up8 ? w[2 + x] : w[x]) + __shfl_xor_sync(0xffffffffu, up8 ? w[x] : w[2 + x], 8);
                float z = (up4 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, up4 ? y[0] : y[1], 4);
                z += __shfl_xor_sync(0xffffffffu, z, 2);
                z += __shfl_xor_sync(0xffffffffu, z, 1);
                const int sr = s0 + 2 * (up8 ? 1 : 0) + (up4 ? 1 : 0);
                if ((lane & 3) == 0) {
                    if (!up && t >= sr) Ps[t * 36 + sr] = z;
                    if (up && t > sr) As[t * 36 + sr] = z;
                }
            } else {  // source 2 (lane bit 16) + (lane bit 8)
                const bool up = lane & 16, up8 = lane & 8;
                float y[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) y[x] = (up ? pv[2 + x] : pv[x]) + __shfl_xor_sync(0xffffffffu, up ? pv[x] : pv[2 + x], 16);
                float z = (up8 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, up8 ? y[0] : y[1], 8);
                z += __shfl_xor_sync(0xffffffffu, z, 4);
                z += __shfl_xor_sync(0xffffffffu, z, 2);
                z += __shfl_xor_sync(0xffffffffu, z, 1);
                const int sr = s0 + 2 * (up ? 1 : 0) + (up8 ? 1 : 0);
                if ((lane & 7) == 0 && t >= sr) Ps[t * 36 + sr] = z;
            }
        }
    }
    __syncthreads();

    float *qp = blocks + ((size_t)(block_base(map, s) + blockIdx.x) * map.heads + h) * block_floats(DK, DELTA);
    float *ke = qp + kC * DK, *pf = ke + kC * DK, *gc = pf + kC * kC, *kp = gc + DK, *tf = kp + kC * DK;
    // a thread owns a channel of one half of the chunk: products from the half's start and to its end
    const int half = tid / DK, i = tid - half * DK;
    if (half < 2) {
        float g = 1.0f;
#pragma unroll
        for (int t = 0; t < 16; ++t) g *= gs[(16 * half + t) * P + i];
        half_prod[half * DK + i] = g;
    }
    __syncthreads();
    if (half < 2) {
        const float before = half ? half_prod[i] : 1.0f, after = half ? 1.0f : half_prod[DK + i];
        if (half == 0) gc[i] = half_prod[i] * half_prod[DK + i];
        float g = 1.0f, kk[16], suffix[16];
#pragma unroll
        for (int t = 15; t >= 0; --t) {  // suffix[t]: the decays after token t, to the end of the half
            suffix[t] = g;
            g *= gs[(16 * half + t) * P + i];
        }
        g = 1.0f;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int row = 16 * half + t;
            const float k = ks[row * P + i], q = qs[row * P + i];
            g *= gs[row * P + i];
            const int at = ((((row >> 3) * (DK / 16) + (i >> 4)) * 32 + (row & 7) * 4 + ((i & 7) >> 1)) << 2) + ((i >> 3) & 1) * 2 + (i & 1);
            if (DELTA) kp[at] = k * (before * g);
            qp[at] = q * (before * g);
            kk[t] = k * (suffix[t] * after);
            // the operands of the block below the diagonal replace the raw rows: sources carried to the half's end, targets from its start
            ks[row * P + i] = half ? k * g : k * suffix[t];
            if (half) qs[row * P + i] = q * g;
        }
        // Ke: column tile i / 8, a 16-byte piece per four tokens
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4 *>(ke + ((((i >> 3) * 2 + half) * 32 + (i & 7) * 4 + j) << 2)) = make_float4(kk[2 * j], kk[2 * j + 1], kk[8 + 2 * j], kk[9 + 2 * j]);
    }
    __syncthreads();
    {  // the 16 x 16 block below the diagonal: one (target, source) pair per thread
        const int t = 16 + (tid >> 4), sr = tid & 15;
        float a[4] = {}, p[4] = {};
#pragma unroll 4
        for (int x = 0; x < DK; x += 4) {
            const float4 f = *reinterpret_cast<const float4 *>(ks + sr * P + x), q = *reinterpret_cast<const float4 *>(qs + t * P + x);
            p[0] = fmaf(f.x, q.x, p[0]), p[1] = fmaf(f.y, q.y, p[1]), p[2] = fmaf(f.z, q.z, p[2]), p[3] = fmaf(f.w, q.w, p[3]);
            if (DELTA) {
                const float4 k = *reinterpret_cast<const float4 *>(ks + t * P + x);
                a[0] = fmaf(f.x, k.x, a[0]), a[1] = fmaf(f.y, k.y, a[1]), a[2] = fmaf(f.z, k.z, a[2]), a[3] = fmaf(f.w, k.w, a[3]);
            }
        }
        Ps[t * 36 + sr] = (p[0] + p[1]) + (p[2] + p[3]);
        if (DELTA) As[t * 36 + sr] = (a[0] + a[1]) + (a[2] + a[3]);
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
            tf[frag_ts(t, lane)] = x[t];
        }
    } else {
        const int first = DELTA ? 32 : 0;
        for (int idx = tid - first; idx < kC * kC; idx += 256 - first) pf[frag_ts(idx >> 5, idx & 31)] = Ps[(idx >> 5) * 36 + (idx & 31)];
    }
}

// ---- the scan
struct Split { uint32_t hi, lo; };
__device__ __forceinline__ Split split_tf32(float v) {
    Split r;  // hi: v rounded to TF32's 11 significant bits; lo: what is left (exact), of which the instruction reads 11 bits again
    r.hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
    r.lo = __float_as_uint(v - __uint_as_float(r.hi));
    return r;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// A operand of one k-step in both halves; EXACT: its values have at most 11 significant bits and no low half
struct FragA { uint32_t hi[4], lo[4]; };
__device__ __forceinline__ FragA split_a(float a0, float a1, float a2, float a3) {
    FragA f;
    const float v[4] = {a0, a1, a2, a3};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const Split sp = split_tf32(v[e]);
        f.hi[e] = sp.hi, f.lo[e] = sp.lo;
    }
    return f;
}
template <bool EXACT_A>
__device__ __forceinline__ void mma_split(float (&d)[4], const FragA &a, float b0, float b1) {
    const Split x = split_tf32(b0), y = split_tf32(b1);
    mma_tf32(d, a.hi, x.lo, y.lo);  // the small products first
    if (!EXACT_A) mma_tf32(d, a.lo, x.hi, y.hi);
    mma_tf32(d, a.hi, x.hi, y.hi);
}
__device__ __forceinline__ void cp16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// A CTA has DK / 16 warps; warp w holds rows 16 w .. 16 w + 15 of S for the CTA's kCols columns, transposed, as two accumulator tiles.
template <typename TQ, int DK, bool DELTA>
__global__ void __launch_bounds__(DK * 2)
chunk_scan_kernel(const ChunkSource src, const ChunkMap map, const float *__restrict__ blocks, float *__restrict__ state, float *__restrict__ o, int stages) {
    constexpr int NW = DK / 16, NT = NW * 32;
    constexpr int NY = DELTA ? 8 : 4;                         // 8-row tiles of [Kp; Qp] (linear attention: Qp alone)
    constexpr int VP = sizeof(TQ) == 2 ? 24 : 20;             // elements per staged value row (16-byte pieces, rows off the same bank)
    constexpr int RED = 72;                                   // floats per column of a warp's partial products
    constexpr int RP = 40;
    constexpr int BF = block_floats(DK, DELTA);
    extern __shared__ __align__(16) float sm[];
    constexpr int stage_floats = BF + kC * VP * (int)sizeof(TQ) / 4;
    float *red = sm + (size_t)stages * stage_floats;          // [NW][kCols][RED]
    float *Rt = red + NW * kCols * RED, *Qs = Rt + kCols * RP; // [kCols][RP]: V - Kp S_0 and Qp S_0, transposed
    const int s = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * kCols;
    const int start = map.seq_start[s], len = map.seq_start[s + 1] - start;
    if (len < map.min_tokens || map.first * kC >= len) return;
    const int n_chunks = min(map.count, (len + kC - 1) / kC - map.first);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const float *blk = blocks + ((size_t)block_base(map, s) * map.heads + h) * BF;
    auto load = [&](int c, int buf) {
        float *dst = sm + (size_t)buf * stage_floats;
        const float *b = blk + (size_t)c * map.heads * BF;
        for (int i = tid; i < BF / 4; i += NT) cp16(dst + 4 * i, b + 4 * i);
        TQ *vs = reinterpret_cast<TQ *>(dst + BF);
        constexpr int per = kCols * (int)sizeof(TQ) / 16;      // 16-byte pieces per value row
        const int t0 = (map.first + c) * kC;
        for (int i = tid; i < kC * per; i += NT) {
            const int t = min(t0 + i / per, len - 1), e = i % per * (16 / (int)sizeof(TQ));  // past the end: a live row, which no key meets
            cp16(vs + (i / per) * VP + e, static_cast<const TQ *>(src.rows) + (size_t)(start + t) * src.ld + src.v_off + h * map.vdim + j0 + e);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, 0);
    // S^T tiles: accumulator n, element (column g (+8), row 16 w + 8 n + 2 t4 (+1))
    float S[2][4];
    float *slot = state + ((size_t)map.seq_slot[s] * map.heads + h) * DK * map.vdim + j0;
    const bool fresh = map.first == 0 && map.seq_pos0[s] == 0;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = 16 * w + 8 * n + 2 * t4 + (e & 1), col = g + 8 * (e >> 1);
            S[n][e] = fresh ? 0.0f : slot[(size_t)r * map.vdim + col];
        }
    for (int c = 0; c < n_chunks; ++c) {
        const int buf = stages == 2 ? c & 1 : 0;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (stages == 2 && c + 1 < n_chunks) load(c + 1, buf ^ 1);
        const float *qp = sm + (size_t)buf * stage_floats, *ke = qp + kC * DK, *pf = ke + kC * DK, *gc = pf + kC * kC, *kp = gc + DK, *tf = kp + kC * DK;
        const TQ *vs = reinterpret_cast<const TQ *>(qp + BF);
        // this warp's share of ([Kp; Qp] S_0)^T: k = its 16 rows of S
        {
            float y[NY][4];
            const FragA a0 = split_a(S[0][0], S[0][2], S[0][1], S[0][3]), a1 = split_a(S[1][0], S[1][2], S[1][1], S[1][3]);
#pragma unroll
            for (int n = 0; n < NY; ++n) {
                const float4 b = *reinterpret_cast<const float4 *>((DELTA && n < 4 ? kp : qp) + ((((n & 3) * NW + w) * 32 + lane) << 2));
#pragma unroll
                for (int e = 0; e < 4; ++e) y[n][e] = 0.0f;
                mma_split<false>(y[n], a0, b.x, b.y);
                mma_split<false>(y[n], a1, b.z, b.w);
            }
            float *r = red + w * kCols * RED;
#pragma unroll
            for (int n = 0; n < NY; ++n) {
                *reinterpret_cast<float2 *>(r + g * RED + 8 * n + 2 * t4) = make_float2(y[n][0], y[n][1]);
                *reinterpret_cast<float2 *>(r + (g + 8) * RED + 8 * n + 2 * t4) = make_float2(y[n][2], y[n][3]);
            }
        }
        __syncthreads();
        // the warps' shares are added up, in order: token tq + 16 e of a column
        for (int idx = tid; idx < kCols * 16; idx += NT) {
            const int col = idx >> 4, tq = idx & 15;
#pragma unroll
            for (int e = 0; e < NY / 2; ++e) {
                float v = 0.0f;
#pragma unroll
                for (int x = 0; x < NW; ++x) v += red[(x * kCols + col) * RED + tq + 16 * e];
                if (DELTA && e < 2) Rt[col * RP + tq + 16 * e] = Elem<TQ>::to_f(vs[(tq + 16 * e) * VP + col]) - v;
                else Qs[col * RP + tq + 16 * (e & 1)] = v;
            }
        }
        __syncthreads();
        // u^T [column, token]: A operand k-step j = tokens 8 j .. 8 j + 7 (every warp forms all of it: cheaper than handing it round)
        FragA u[4];
        if (DELTA) {
            FragA r[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 lo = *reinterpret_cast<const float2 *>(Rt + g * RP + 8 * j + 2 * t4), hi = *reinterpret_cast<const float2 *>(Rt + (g + 8) * RP + 8 * j + 2 * t4);
                r[j] = split_a(lo.x, hi.x, lo.y, hi.y);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float d[4] = {};
#pragma unroll
                for (int jp = 0; jp <= n / 2; ++jp) {
                    const float4 b = *reinterpret_cast<const float4 *>(tf + (((n * 2 + jp) * 32 + lane) << 2));
                    mma_split<false>(d, r[2 * jp], b.x, b.y);
                    if (2 * jp + 1 <= n) mma_split<false>(d, r[2 * jp + 1], b.z, b.w);
                }
                u[n] = split_a(d[0], d[2], d[1], d[3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = 8 * j + 2 * t4;
                u[j] = split_a(Elem<TQ>::to_f(vs[t * VP + g]), Elem<TQ>::to_f(vs[t * VP + g + 8]), Elem<TQ>::to_f(vs[(t + 1) * VP + g]), Elem<TQ>::to_f(vs[(t + 1) * VP + g + 8]));
            }
        }
        constexpr bool EXACT_U = !DELTA && sizeof(TQ) == 2;  // 16-bit values fit one TF32 half
        // S^T <- S^T diag(p_C) + u^T Ke
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float2 gg = *reinterpret_cast<const float2 *>(gc + 16 * w + 8 * n + 2 * t4);
            S[n][0] *= gg.x, S[n][1] *= gg.y, S[n][2] *= gg.x, S[n][3] *= gg.y;
            float d[4] = {};
#pragma unroll
            for (int jp = 0; jp < 2; ++jp) {
                const float4 b = *reinterpret_cast<const float4 *>(ke + ((((2 * w + n) * 2 + jp) * 32 + lane) << 2));
                mma_split<EXACT_U>(d, u[2 * jp], b.x, b.y);
                mma_split<EXACT_U>(d, u[2 * jp + 1], b.z, b.w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) S[n][e] += d[e];
        }
        // o^T = (Qp S_0)^T + u^T P^T: token tiles over the warps
        for (int n = w; n < 4; n += NW) {
            float d[4] = {};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j <= n) {
                    const float2 b = *reinterpret_cast<const float2 *>(pf + (((n * 2 + (j >> 1)) * 32 + lane) << 2) + 2 * (j & 1));
                    mma_split<EXACT_U>(d, u[j], b.x, b.y);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 8 * n + 2 * t4 + (e & 1), col = g + 8 * (e >> 1), tt = (map.first + c) * kC + t;
                if (tt < len) o[((size_t)(start + tt) * map.heads + h) * map.vdim + j0 + col] = d[e] + Qs[col * RP + t];
            }
        }
        if (stages == 1) {
            __syncthreads();
            if (c + 1 < n_chunks) load(c + 1, 0);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) slot[(size_t)(16 * w + 8 * n + 2 * t4 + (e & 1)) * map.vdim + g + 8 * (e >> 1)] = S[n][e];
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
    const size_t smem_f = (size_t)(3 * kC * (DK + 4) + 2 * kC * 36 + 2 * DK + kC) * sizeof(float);
    constexpr int VP = sizeof(TQ) == 2 ? 24 : 20;
    const size_t stage = block_floats(DK, DELTA) * sizeof(float) + kC * VP * sizeof(TQ), rest = (size_t)(DK / 16 * kCols * 72 + 2 * kCols * 40) * sizeof(float);
    // one CTA per SM at most: two stages hide the block's arrival; more CTAs than SMs: one stage, two CTAs per SM hide each other's.  (Rings of four to
    // six stages filled by bulk copies, one CTA per SM: 196 us against 188 for linear attention, 238 against 198 for the delta rule -- a chunk's time is
    // its chain of products, not its block's arrival.)
    const int ctas = map.vdim / kCols * map.heads * n_seqs, stages = ctas <= sm_count() ? 2 : 1;
    auto fk = chunk_factors_kernel<TQ, DK, DELTA>;
    auto sk = chunk_scan_kernel<TQ, DK, DELTA>;
    cudaFuncSetAttribute(fk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_f);
    cudaFuncSetAttribute(sk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * stage + rest));
    for (map.first = 0; map.first < chunks; map.first += map.count) {
        const int n = std::min(map.count, chunks - map.first);
        launch_pdl(fk, dim3(n, map.heads, n_seqs), dim3(256), smem_f, st, false, src, map, scratch);
        launch_pdl(sk, dim3(map.vdim / kCols, map.heads, n_seqs), dim3(DK * 2), stages * stage + rest, st, false, src, map, scratch, state, o, stages);
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
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || ld * es % 16 != 0 || 2 * heads * dim * es % 16 != 0 || !aligned16(proj) || !scratch) return B200_ERR_UNSUPPORTED;
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
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || !aligned16(rec) || !scratch) return B200_ERR_UNSUPPORTED;
    const DeltaRow lay = delta_row(heads, kv_heads, dim, vdim);  // (every segment of the row starts on a 16-byte boundary)
    const ChunkSource src = {rec, lay.ld, lay.q, lay.k, lay.v, rec, lay.ld, lay.decay, dim, rec + lay.beta, lay.ld, 1.0f};
    const ChunkMap map = {seq_start, seq_pos0, seq_slot, heads, heads / kv_heads, vdim, kChunkMinTokens, 0, 0, 0};
    return dim == 64 ? launch_chunks_t<float, 64, true>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st)
                     : launch_chunks_t<float, 128, true>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st);
}

int launch_chunk_decay(const float *rec, float *state, float *o, const int *seq_start, const int *seq_pos0, const int *seq_slot, int n_seqs, int heads,
                       int kv_heads, int dim, int vdim, float *scratch, size_t scratch_floats, int tokens, int longest, cudaStream_t st) {
    if ((dim != 64 && dim != 128) || vdim % kCols != 0 || !aligned16(rec) || !scratch) return B200_ERR_UNSUPPORTED;
    const DecayRow lay = decay_row(heads, kv_heads, dim, vdim);
    const ChunkSource src = {rec, lay.ld, lay.q, lay.k, lay.v, rec, lay.ld, lay.decay, 1, nullptr, 0, 1.0f};
    const ChunkMap map = {seq_start, seq_pos0, seq_slot, heads, heads / kv_heads, vdim, kChunkMinTokens, 0, 0, 0};
    return dim == 64 ? launch_chunks_t<float, 64, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st)
                     : launch_chunks_t<float, 128, false>(src, map, scratch, scratch_floats, state, o, n_seqs, tokens, longest, st);
}

}  // namespace b200
