// attention_token.cu -- attention of decoded tokens over the paged key / value pool: one CTA per (token, key head, run of its keys), all query heads of the key
// head at once.  Covers the masks and scores of attention_chunked.cu and attention_scored.cu for 16-bit engines; those files keep a per-token kernel for the rest.
// Scores, weights and sums are fp32, two multiply-adds an instruction; the products of a key row and of a value row serve all query heads of their key head.
//
// A token's keys are cut into blocks by its own context alone (128 keys up to 4096, see block_keys), every block's weights and sums are formed in the same way, and
// the blocks are added up first to last: a token's bits are the same whatever is beside it.  How many CTAs share the blocks out follows the batch: few tokens take a
// CTA per block, whose sums go through scratch to the last CTA of the token to arrive (a counter that returns to zero by itself; nobody waits); with many tokens a
// CTA goes through all blocks of its own.
//
// What bounds it: round trips and instructions.  A CTA per (token, QUERY head) read, unpacked and addressed every key and value row once per query head and looked a
// row's page up in global memory before it could ask for the row: 36 thousand instructions for 513 keys of one head, half of the issue slots, and eight round trips
// one behind the other.  Here the pages of a run lie in shared memory, a block's value rows are on their way while its weights are formed, and the next block's key
// rows while its sums are folded.
// Measured (B200, us per launch in a decode step; bf16, dim 128, 16 query heads of 4 key heads): 16 tokens of 513 keys 17 with a CTA per query head, 16.2 here, 16 of 900
// 19.2, 32 of 1001 31.9, one of 200 / 900 10.3 / 11.7; with keys shared out by what else is in the batch, which gave a token other bits in other company, 14.9,
// 17.7, 30.0, 9.5 / 11.4.  Blocks of keys as CTAs of their own at every batch size: 25.6 for 16 of 900, 46 for 32 of 1001.  Key rows asked for at their use in place
// of behind the block before: 11.2 for one of 900, 34.3 for 32 of 1001.
#include "hybrid_ops.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kPageT = B200_KV_PAGE_SIZE;
constexpr int kThreads = 256, kWarpsT = kThreads / 32, kSlots = kThreads / 4;  // four lanes share a key row
constexpr int kBlock = 2 * kSlots, kBlocks = 32, kMostKeys = 1024;             // keys of a block; blocks of a token until they would hold more than kMostKeys
constexpr int kMostBlocks = kWarpsT * 64 / 4;                                  // (three numbers of a block and head lie where the warps' parts were)

struct TokenAttnArgs {
    TokenAttn in;
    int blocks;     // head blocks of G query heads per key head
    int block_max;  // keys of a block, at most
    int run;        // blocks that a CTA goes through, at most
    int item_blocks;  // blocks that the scratch holds of every token and head block
};

__host__ __device__ inline int first_key(int pos, int window, int chunk) {
    int first = window > 0 && pos >= window ? pos - window + 1 : 0;
    if (chunk > 0 && pos - pos % chunk > first) first = pos - pos % chunk;
    return first;
}
// Keys of a block: of the token's own number of keys and of nothing else.  128 are what the lanes take in one round.
__host__ __device__ inline int block_keys(int nkeys) {
    if (nkeys <= kBlocks * kBlock) return kBlock;
    int blocks = nkeys > kBlocks * kMostKeys ? (nkeys + kMostKeys - 1) / kMostKeys : kBlocks;
    if (blocks > kMostBlocks) blocks = kMostBlocks;
    return ((nkeys + blocks - 1) / blocks + 7) & ~7;
}

// The sums of one more block onto those of the blocks before it, whose largest score is m0, of weights formed below the block's own largest score m1.
struct Fold {
    float of_old, of_new, top;
    __device__ __forceinline__ Fold(float m0, float m1) {
        top = fmaxf(m0, m1);
        const float t = top == -INFINITY ? 0.0f : top;  // (no weight so far: all of them stay zero)
        of_old = expf(m0 - t), of_new = expf(m1 - t);
    }
};
__device__ __forceinline__ float fold(float old, float of_old, float now, float of_new) { return fmaf(now, of_new, __fmul_rn(old, of_old)); }

__device__ __forceinline__ float2 fma2t(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(*reinterpret_cast<unsigned long long *>(&d))
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)), "l"(*reinterpret_cast<const unsigned long long *>(&c)));
    return d;
}
template <typename T> __device__ __forceinline__ void unpack_pairs(const uint4 &raw, float2 (&f)[4]) {
    float v[8];
    unpack16<T>(raw, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = make_float2(v[2 * i], v[2 * i + 1]);
}

template <typename T, int G>
__global__ void __launch_bounds__(kThreads, 2)
token_attn_kernel(const TokenAttnArgs args) {
    constexpr int ROWS = G == 8 ? 4 : 8;              // value rows of a thread on their way
    constexpr int NE = G >= 2 ? G * 128 / kThreads : 1;  // elements of the result that a thread adds up, of 128 columns
    const TokenAttn &a = args.in;
    extern __shared__ __align__(16) float sm[];
    const int4 token = a.tokens[blockIdx.x];  // {sequence, row, 1, position}: one access where row, position and sequence by turns were two behind one another
    const int t = token.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = a.heads / a.kv_heads, g = blockIdx.y / args.blocks, h0 = g * group + (blockIdx.y - g * args.blocks) * G, live = min(G, (g + 1) * group - h0);
    const int dim = a.dim, vdim = a.vdim;
    const int pos = token.w;
    const int first = first_key(pos, a.window, a.chunk);
    const int nkeys = pos - first + 1, per = block_keys(nkeys), nblocks = (nkeys + per - 1) / per, ctas = (nblocks + args.run - 1) / args.run;
    const int b0 = blockIdx.z * args.run, b1 = min(b0 + args.run, nblocks);
    if (b0 >= b1) return;  // (fewer blocks than another token has)
    const int run0 = b0 * per, run1 = min(b1 * per, nkeys);  // this CTA's keys, counted from the first

    float *const qs = sm, *const sc = qs + G * dim, *const part = sc + (size_t)args.block_max * G, *const red = part + kWarpsT * G * vdim;  // sums of weights and the maxima of every other block [3][warps][G]
    float *const whole = red + 3 * kWarpsT * G;                               // [G]: the factors of the result
    int *const pages = reinterpret_cast<int *>(whole + G);
    __shared__ int last_one;
    const int page0 = (first + run0) / kPageT;
    for (int i = tid; i <= (first + run1 - 1) / kPageT - page0; i += kThreads) pages[i] = a.block_table[(size_t)token.x * a.mpps + page0 + i];
    if (tid < dim) {  // (dim <= the CTA's threads)
        const T *q = static_cast<const T *>(a.q) + ((size_t)t * a.heads + h0) * dim + tid;
#pragma unroll
        for (int h = 0; h < G; ++h) qs[h * dim + tid] = Elem<T>::to_f(q[min(h, live - 1) * dim]);
    }
    __syncthreads();
    auto row = [&](const void *pool, int j, int d) {  // key j: its row in a pool of rows of d
        const int p = first + j;
        return static_cast<const T *>(pool) + (((size_t)pages[p / kPageT - page0] * a.kv_heads + g) * kPageT + p % kPageT) * d;
    };

    // The four lanes' parts of the 2 G products of a lane group's two keys fold into one another: a lane ends with HQ heads of one key, whole (lane bit 1: which key,
    // bit 0: which heads).
    constexpr int HQ = G >= 2 ? G / 2 : 1;
    const int hq = G >= 2 ? (lane & 1) * HQ : 0;
    const int sub = lane & 3, pieces = dim / 8;
    uint4 keys[2][4];
    auto request_keys = [&](int j0, int end) {  // rows j0 + slot and j0 + kSlots + slot (past the end: the last)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const T *kr = row(a.k_pool, min(j0 + (tid >> 2) + u * kSlots, end - 1), dim);
#pragma unroll
            for (int i = 0; i < 4; ++i) keys[u][i] = ld_v4(kr + min(4 * i + sub, pieces - 1) * 8);
        }
    };
    const int vshift = 31 - __clz(vdim), tpr = vdim / 8, groups = kThreads >> (vshift - 3), kg = tid >> (vshift - 3), c0 = (tid & (tpr - 1)) * 8;
    uint4 raw[ROWS];
    auto request = [&](int j, int end) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) raw[i] = ld_v4(row(a.v_pool, min(j + i * groups, end - 1), vdim) + c0);
    };
    auto folded = [&](int i) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) v += part[(size_t)w * G * vdim + i];
        return v;
    };
    auto maxima = [&](int b) { return red + (1 + (b & 1)) * kWarpsT * G; };  // (a warp may form the next block's while another still folds this one's)
    auto largest = [&](int b, int h) {
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) m = fmaxf(m, maxima(b)[w * G + h]);
        return m;
    };
    auto total = [&](int h) {
        float l = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) l += red[w * G + h];
        return l;
    };
    const int item = blockIdx.x * gridDim.y + blockIdx.y, stride = G * (vdim + 2);
    float *const all = a.part + (size_t)item * args.item_blocks * stride;  // a block: [G] maxima, [G] sums of weights, [G][vdim]
    float out[NE], out_m[NE], out_l[NE];  // of the elements tid, tid + kThreads, ... of [G][vdim]: their sums, the largest score and the weights of their heads
#pragma unroll
    for (int e = 0; e < NE; ++e) out[e] = 0.0f, out_m[e] = -INFINITY, out_l[e] = 0.0f;

    request_keys(run0, min(run0 + per, run1));
    for (int b = b0; b < b1; ++b) {
        const int k0 = b * per, n = min(per, nkeys - k0), end = k0 + n;
        // ---- scores: two keys per lane group and round
        float mx[HQ];
#pragma unroll
        for (int h = 0; h < HQ; ++h) mx[h] = -INFINITY;
        for (int j0 = 0; j0 + warp * 8 < n; j0 += kBlock) {  // (the same for all lanes of a warp: the shuffles take every one)
            if (j0 > 0) request_keys(k0 + j0, end);
            float2 acc[2][G] = {};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (4 * i >= pieces) break;  // (dim is a multiple of 32: the four lanes have a piece each, or none)
                float2 f[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u) unpack_pairs<T>(keys[u][i], f[u]);
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float4 *qp = reinterpret_cast<const float4 *>(qs + h * dim + (4 * i + sub) * 8);
                    const float4 q0 = qp[0], q1 = qp[1];
                    const float2 q[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y), make_float2(q1.z, q1.w)};
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[u][h] = fma2t(q[e], f[u][e], acc[u][h]);
                }
            }
            float w[G], y[HQ];
            const bool up2 = lane & 2, up1 = lane & 1;
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const float p = acc[0][h].x + acc[0][h].y, q = acc[1][h].x + acc[1][h].y;
                w[h] = (up2 ? q : p) + __shfl_xor_sync(0xffffffffu, up2 ? p : q, 2);
            }
            if constexpr (G >= 2) {
#pragma unroll
                for (int h = 0; h < HQ; ++h) y[h] = (up1 ? w[HQ + h] : w[h]) + __shfl_xor_sync(0xffffffffu, up1 ? w[h] : w[HQ + h], 1);
            } else {
                y[0] = w[0] + __shfl_xor_sync(0xffffffffu, w[0], 1);
            }
            const int j = j0 + (tid >> 2) + (up2 ? kSlots : 0);
            if (j < n) {
                const float dist = (float)(nkeys - 1 - k0 - j);
#pragma unroll
                for (int h = 0; h < HQ; ++h) {
                    const int hh = h0 + min(hq + h, live - 1);
                    float v = y[h];
                    v *= a.scale;
                    if (a.softcap > 0.0f) v = a.softcap * tanhf(v / a.softcap);
                    if (a.dist_r1) v -= __ldg(a.dist_r1 + hh) * log1pf(__ldg(a.dist_r2 + hh) * dist);
                    if (a.slope) v = fmaf(-__ldg(a.slope + hh), dist, v);
                    if (a.sigmoid) v = 1.0f / (1.0f + expf(-(v + (a.head_bias ? __ldg(a.head_bias + hh) : 0.0f))));
                    sc[j * G + hq + h] = v;
                    mx[h] = fmaxf(mx[h], v);
                }
            }
        }
        // a thread's first value rows are on their way while the weights are formed
        request(k0 + kg, end);
        if (!a.sigmoid) {
#pragma unroll
            for (int h = 0; h < HQ; ++h) {
#pragma unroll
                for (int x = G >= 2 ? 2 : 1; x < 32; x <<= 1) mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], x));
                if (lane < (G >= 2 ? 2 : 1)) maxima(b)[warp * G + hq + h] = mx[h];
            }
            __syncthreads();
            const float m = largest(b, tid % G), top = m == -INFINITY ? 0.0f : m;  // (a block whose scores are all minus infinity has weights of zero, another may not)
            float sum = 0.0f;  // of head tid % G
            for (int i = tid; i < n * G; i += kThreads) {
                const float e = expf(sc[i] - top);
                sc[i] = e;
                sum += e;
            }
#pragma unroll
            for (int x = G; x < 32; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            if (lane < G) red[warp * G + lane] = sum;
        }
        __syncthreads();

        // ---- weighted sum of the values
        float2 o[G][4] = {};
        for (int j = kg; j < n; j += ROWS * groups) {
            if (j != kg) request(k0 + j, end);
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                if (j + i * groups >= n) break;
                float2 f[4];
                unpack_pairs<T>(raw[i], f);
                float w[G];
                const float *at = sc + (size_t)(j + i * groups) * G;
                if constexpr (G >= 4) {
#pragma unroll
                    for (int h = 0; h < G; h += 4) load_n<float, 4>(at + h, w + h);
                } else {
#pragma unroll
                    for (int h = 0; h < G; ++h) w[h] = at[h];
                }
#pragma unroll
                for (int h = 0; h < G; ++h) {
                    const float2 ww = make_float2(w[h], w[h]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[h][e] = fma2t(ww, f[e], o[h][e]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < G; ++h) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                for (int x = tpr; x < 32; x <<= 1) o[h][e].x += __shfl_xor_sync(0xffffffffu, o[h][e].x, x), o[h][e].y += __shfl_xor_sync(0xffffffffu, o[h][e].y, x);
            if (lane < tpr) {
                float4 *to = reinterpret_cast<float4 *>(part + (size_t)(warp * G + h) * vdim + c0);
                to[0] = make_float4(o[h][0].x, o[h][0].y, o[h][1].x, o[h][1].y), to[1] = make_float4(o[h][2].x, o[h][2].y, o[h][3].x, o[h][3].y);
            }
        }
        if (b + 1 < b1) request_keys(end, min(end + per, run1));
        __syncthreads();
        // ---- the block's sums onto those before it, or to the scratch
        if (ctas == 1) {
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const int i = tid + e * kThreads;
                if (i >= G * vdim) break;
                const float p = folded(i);
                if (a.sigmoid) {
                    out[e] += p;
                } else {
                    const Fold f(out_m[e], largest(b, i >> vshift));
                    out[e] = fold(out[e], f.of_old, p, f.of_new), out_l[e] = fold(out_l[e], f.of_old, total(i >> vshift), f.of_new), out_m[e] = f.top;
                }
            }
        } else {
            float *const mine = all + (size_t)b * stride;
            if (!a.sigmoid && tid < G) __stcg(mine + tid, largest(b, tid)), __stcg(mine + G + tid, total(tid));
            for (int i = tid; i < G * vdim; i += kThreads) __stcg(mine + 2 * G + i, folded(i));
        }
    }

    const float *sink = a.sigmoid ? nullptr : a.sink;
    auto factor = [&](int h, float m, float l) {  // of a head's sums in its result; the sink: a logit with no key and no value, counted once, it may be the largest
        const float s = sink ? sink[h0 + min(h, live - 1)] : -INFINITY, mm = sink ? fmaxf(m, s) : m, f = expf(m - mm);
        return f / (l * f + (sink ? expf(s - mm) : 0.0f));
    };
    auto store = [&](int i, float v) {  // element i of [G][vdim]
        const int h = i >> vshift, c = i & (vdim - 1);
        if (h >= live) return;
        if (a.gate) v *= 1.0f / (1.0f + expf(-Elem<T>::to_f(static_cast<const T *>(a.gate)[(size_t)t * a.gate_ld + (h0 + h) * vdim + c])));
        static_cast<T *>(a.out)[(size_t)t * a.out_ld + (h0 + h) * vdim + c] = Elem<T>::from_f(v * a.out_scale);
    };
    if (ctas == 1) {
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const int i = tid + e * kThreads;
            if (i < G * vdim) store(i, a.sigmoid ? out[e] : out[e] * factor(i >> vshift, out_m[e], out_l[e]));
        }
        return;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) last_one = atomicInc(a.tickets + item, ctas - 1) == (unsigned)(ctas - 1);
    __syncthreads();
    if (!last_one) return;
    __threadfence();
    // ---- the blocks from the scratch, first to last: [block][head] maxima and weights, then what Fold makes of them
    float *const ms = part, *const ls = ms + nblocks * G, *const of_new = ls + nblocks * G, *const of_old = sc;
    if (!a.sigmoid) {
        const int h = tid % G;
        for (int i = tid; i < nblocks * G; i += kThreads) ms[i] = __ldcg(all + (size_t)(i / G) * stride + h), ls[i] = __ldcg(all + (size_t)(i / G) * stride + G + h);
        __syncthreads();
        for (int i = tid; i < nblocks * G; i += kThreads) {
            float m = -INFINITY;
            for (int x = h; x < i; x += G) m = fmaxf(m, ms[x]);
            const Fold f(m, ms[i]);
            of_old[i] = f.of_old, of_new[i] = f.of_new;
        }
        __syncthreads();
        if (tid < G) {
            float m = -INFINITY, l = 0.0f;
            for (int x = tid; x < nblocks * G; x += G) m = fmaxf(m, ms[x]), l = fold(l, of_old[x], ls[x], of_new[x]);
            whole[tid] = factor(tid, m, l);
        }
        __syncthreads();
    }
    for (int i = tid; i < G * vdim; i += kThreads) {
        const int h = i >> vshift;
        float v = 0.0f;
        for (int s0 = 0; s0 < nblocks; s0 += 8) {  // (eight blocks' sums on their way at once)
            float p[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) p[s] = __ldcg(all + (size_t)min(s0 + s, nblocks - 1) * stride + 2 * G + i);
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (s0 + s < nblocks) v = a.sigmoid ? v + p[s] : fold(v, of_old[(s0 + s) * G + h], p[s], of_new[(s0 + s) * G + h]);
        }
        store(i, a.sigmoid ? v : v * whole[h]);
    }
}

template <typename T, int G> int launch_token_t(const TokenAttnArgs &args, const dim3 &grid, size_t smem, cudaStream_t st) {
    auto kern = token_attn_kernel<T, G>;
    if (smem > 48 * 1024) allow_smem(kern);
    launch_plain(kern, grid, dim3(kThreads), smem, st, args);
    return cuda_status("token_attention launch");
}

int heads_per_block(int heads, int kv_heads) {  // query heads that a CTA takes: 1, 2, 4 or 8
    const int group = heads / kv_heads;
    return group > 4 ? 8 : group > 2 ? 4 : group;
}

}  // namespace

size_t token_attention_part_floats(int heads, int kv_heads, int vdim) { return (size_t)kTokenParts * heads_per_block(heads, kv_heads) * (vdim + 2); }

// B200_ERR_UNSUPPORTED (no error text, nothing launched): fp32, head sizes that lanes or threads do not share evenly, no scratch, contexts whose blocks no CTA holds.
// The blocks are shared out evenly over kTokenCtas CTAs (two per SM); tokens whose blocks the scratch does not hold together go in several launches.
int launch_token_attention(int dtype, const TokenAttn &a, int tokens, cudaStream_t st) {
    if (tokens == 0) return B200_OK;
    if (dtype == B200_F32 || a.dim % 32 != 0 || a.dim > 128 || (a.vdim != 64 && a.vdim != 128) || !a.part || !a.tickets || !all_aligned16({a.k_pool, a.v_pool}))
        return B200_ERR_UNSUPPORTED;
    const int G = heads_per_block(a.heads, a.kv_heads), blocks = (a.heads / a.kv_heads + G - 1) / G, rows = a.kv_heads * blocks;
    auto keys_of = [&](int i) { return a.listed[i].w - first_key(a.listed[i].w, a.window, a.chunk) + 1; };
    auto blocks_of = [&](int keys) { return (keys + block_keys(keys) - 1) / block_keys(keys); };
    auto smem_of = [&](int per, int run) {
        return ((size_t)G * a.dim + (size_t)per * G + (size_t)kWarpsT * G * a.vdim + 3 * kWarpsT * G + G) * sizeof(float) + (run / kPageT + 2) * sizeof(int);
    };
    int longest = 1;
    for (int i = 0; i < tokens; ++i) longest = std::max(longest, keys_of(i));
    if (rows > 65535 || smem_of(std::max(block_keys(longest), kBlock), longest) > 110 * 1024) return B200_ERR_UNSUPPORTED;
    for (int i0 = 0, i1; i0 < tokens; i0 = i1) {
        long long all = 0;
        int per = kBlock, most = 1, keys = 1, run = 1;
        for (i1 = i0; i1 < tokens; ++i1) {
            const int n = keys_of(i1), m = std::max(most, blocks_of(n)), r = (int)((all + (long long)blocks_of(n) * rows + kTokenCtas - 1) / kTokenCtas);
            const bool fits = r >= m || (long long)(i1 - i0 + 1) * rows * m <= kTokenParts;
            if (i1 > i0 && !fits) break;
            all += (long long)blocks_of(n) * rows, most = m, run = fits ? r : m;
            per = std::max(per, block_keys(n)), keys = std::max(keys, n);
        }
        TokenAttnArgs args = {a, blocks, per, run, most};
        args.in.tokens += i0;
        const size_t smem = smem_of(per, std::min(keys, run * per));
        const dim3 grid(i1 - i0, rows, (most + run - 1) / run);
#define B200_TOKEN_G(T) (G == 1 ? launch_token_t<T, 1>(args, grid, smem, st) : G == 2 ? launch_token_t<T, 2>(args, grid, smem, st) \
                         : G == 4 ? launch_token_t<T, 4>(args, grid, smem, st) : launch_token_t<T, 8>(args, grid, smem, st))
        const int rc = dtype == B200_BF16 ? B200_TOKEN_G(__nv_bfloat16) : B200_TOKEN_G(__half);
#undef B200_TOKEN_G
        if (rc != B200_OK) return rc;
    }
    return B200_OK;
}

}  // namespace b200
