// attention_token.cu -- attention of decoded tokens over the paged key / value pool: one CTA per (token, key head, share of the keys), all query heads of the key
// head at once.  Covers the masks and scores of attention_chunked.cu and attention_scored.cu for 16-bit engines; those files keep a per-token kernel for the rest.
// Scores, weights and sums are fp32, two multiply-adds an instruction; the products of a key row and of a value row serve all query heads of their key head.
//
// What bounds it: round trips and instructions.  A CTA per (token, QUERY head) read, unpacked and addressed every key and value row once per query head and looked a
// row's page up in global memory before it could ask for the row: 36 thousand instructions for 513 keys of one head, half of the issue slots, and eight round trips
// one behind the other.  Here the pages of a share lie in shared memory, a lane has two key rows on their way and four value rows (the first requested before the
// weights are formed), and few tokens share out their keys over the device.  The last CTA of a token's shares to arrive (a counter that returns to zero by itself;
// nobody waits) adds them up in order.
// Measured (B200, us per launch in a decode step, one CTA per query head -> now; bf16, dim 128, 16 query heads of 4 key heads): 3 tokens of 1024 keys 40 -> 13,
// 16 tokens of 513 keys 17 -> 14, a step of 32 tokens of 1001 keys (two of these launches) 692 -> 655.  On the way: shares of 128 threads 26 for both; a share's
// four lanes each adding up all products and one thread per head combining the shares 18.
#include "hybrid_ops.cuh"

#include <algorithm>

namespace b200 {

namespace {

constexpr int kPageT = B200_KV_PAGE_SIZE;
constexpr int kThreads = 256, kWarpsT = kThreads / 32, kSlots = kThreads / 4;  // four lanes share a key row
constexpr int kRows = 4;                                                       // value rows of a thread on their way

struct TokenAttnArgs {
    TokenAttn in;
    int blocks;     // head blocks of G query heads per key head
    int share_max;  // keys of a share, at most
};

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
    const TokenAttn &a = args.in;
    extern __shared__ __align__(16) float sm[];
    const int4 token = a.tokens[blockIdx.x];  // {sequence, row, 1, position}: one access where row, position and sequence by turns were two behind one another
    const int t = token.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = a.heads / a.kv_heads, g = blockIdx.y / args.blocks, h0 = g * group + (blockIdx.y - g * args.blocks) * G, live = min(G, (g + 1) * group - h0);
    const int dim = a.dim, vdim = a.vdim;
    const int pos = token.w;
    int first = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    if (a.chunk > 0) first = max(first, pos - pos % a.chunk);
    const int nkeys = pos - first + 1, per = ((nkeys + (int)gridDim.z - 1) / (int)gridDim.z + 7) & ~7, shares = (nkeys + per - 1) / per;
    const int k0 = blockIdx.z * per, n = min(per, nkeys - k0);
    if (n <= 0) return;  // (a share that a short context leaves empty)

    float *const qs = sm, *const sc = qs + G * dim, *const part = sc + (size_t)args.share_max * G, *const red = part + kWarpsT * G * vdim;  // maxima and sums [2][warps][G]
    float *const whole = red + 2 * kWarpsT * G;                               // [G]: the share's maxima, then the factors of its sums
    int *const pages = reinterpret_cast<int *>(whole + G);
    __shared__ int last_one;
    const int page0 = (first + k0) / kPageT;
    for (int i = tid; i <= (first + k0 + n - 1) / kPageT - page0; i += kThreads) pages[i] = a.block_table[(size_t)token.x * a.mpps + page0 + i];
    if (tid < dim) {  // (dim <= the block's threads)
        const T *q = static_cast<const T *>(a.q) + ((size_t)t * a.heads + h0) * dim + tid;
#pragma unroll
        for (int h = 0; h < G; ++h) qs[h * dim + tid] = Elem<T>::to_f(q[min(h, live - 1) * dim]);
    }
    __syncthreads();
    auto row = [&](const void *pool, int j, int d) {  // key j of the share: its row in a pool of rows of d
        const int p = first + k0 + j;
        return static_cast<const T *>(pool) + (((size_t)pages[p / kPageT - page0] * a.kv_heads + g) * kPageT + p % kPageT) * d;
    };

    // ---- scores: two keys per lane group and round
    // The four lanes' parts of the 2 G products fold into one another: a lane ends with HQ heads of one key, whole (lane bit 1: which key, bit 0: which heads).
    constexpr int HQ = G >= 2 ? G / 2 : 1;
    const int hq = G >= 2 ? (lane & 1) * HQ : 0;
    float mx[HQ];
#pragma unroll
    for (int h = 0; h < HQ; ++h) mx[h] = -INFINITY;
    {
        const int sub = lane & 3, pieces = dim / 8;
        for (int j0 = 0; j0 + warp * 8 < n; j0 += 2 * kSlots) {  // (the same for all lanes of a warp: the shuffles take every one)
            float2 acc[2][G] = {};
            const T *kr[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) kr[u] = row(a.k_pool, min(j0 + (tid >> 2) + u * kSlots, n - 1), dim);
            for (int p0 = 0; p0 < pieces; p0 += 16) {
                uint4 raw[2][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int u = 0; u < 2; ++u) raw[u][i] = ld_v4(kr[u] + min(p0 + 4 * i + sub, pieces - 1) * 8);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (p0 + 4 * i >= pieces) break;  // (dim is a multiple of 32: the four lanes have a piece each, or none)
                    float2 f[2][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) unpack_pairs<T>(raw[u][i], f[u]);
#pragma unroll
                    for (int h = 0; h < G; ++h) {
                        const float4 *qp = reinterpret_cast<const float4 *>(qs + h * dim + (p0 + 4 * i + sub) * 8);
                        const float4 q0 = qp[0], q1 = qp[1];
                        const float2 q[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y), make_float2(q1.z, q1.w)};
#pragma unroll
                        for (int u = 0; u < 2; ++u)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[u][h] = fma2t(q[e], f[u][e], acc[u][h]);
                    }
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
    }
    // a thread's first value rows are on their way while the weights are formed
    const int vshift = 31 - __clz(vdim), tpr = vdim / 8, groups = kThreads >> (vshift - 3), kg = tid >> (vshift - 3), c0 = (tid & (tpr - 1)) * 8;
    uint4 raw[kRows];
    auto request = [&](int j) {
#pragma unroll
        for (int i = 0; i < kRows; ++i) raw[i] = ld_v4(row(a.v_pool, min(j + i * groups, n - 1), vdim) + c0);
    };
    request(kg);
    float sum = 0.0f;  // of head tid % G
    if (!a.sigmoid) {
#pragma unroll
        for (int h = 0; h < HQ; ++h) {
#pragma unroll
            for (int x = G >= 2 ? 2 : 1; x < 32; x <<= 1) mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], x));
            if (lane < (G >= 2 ? 2 : 1)) red[warp * G + hq + h] = mx[h];
        }
        __syncthreads();
        float m = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) m = fmaxf(m, red[w * G + tid % G]);
        const float top = m == -INFINITY ? 0.0f : m;  // (a share whose scores are all minus infinity has weights of zero, another may not)
        for (int i = tid; i < n * G; i += kThreads) {
            const float e = expf(sc[i] - top);
            sc[i] = e;
            sum += e;
        }
        if (tid < G) whole[tid] = m;
#pragma unroll
        for (int x = G; x < 32; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        if (lane < G) red[(kWarpsT + warp) * G + lane] = sum;
    }
    __syncthreads();

    // ---- weighted sum of the values
    float2 o[G][4] = {};
    for (int j = kg; j < n; j += kRows * groups) {
        uint4 now[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) now[i] = raw[i];
        if (j + kRows * groups < n) request(j + kRows * groups);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            if (j + i * groups >= n) break;
            float2 f[4];
            unpack_pairs<T>(now[i], f);
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
    __syncthreads();
    auto folded = [&](int i) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) v += part[(size_t)w * G * vdim + i];
        return v;
    };
    auto total = [&](int h) {
        float l = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarpsT; ++w) l += red[(kWarpsT + w) * G + h];
        return l;
    };
    const float *sink = a.sigmoid ? nullptr : a.sink;
    auto store = [&](int i, float v) {  // element i of [G][vdim], its sum over all keys
        const int h = i >> vshift, c = i & (vdim - 1);
        if (h >= live) return;
        if (a.gate) v *= 1.0f / (1.0f + expf(-Elem<T>::to_f(static_cast<const T *>(a.gate)[(size_t)t * a.gate_ld + (h0 + h) * vdim + c])));
        static_cast<T *>(a.out)[(size_t)t * a.out_ld + (h0 + h) * vdim + c] = Elem<T>::from_f(v * a.out_scale);
    };
    if (shares == 1) {
        if (!a.sigmoid) {
            if (tid < G) {  // the sink: a logit with no key and no value, counted once; it may be the largest
                const float m = whole[tid], l = total(tid), mm = sink ? fmaxf(m, sink[h0 + min(tid, live - 1)]) : m;
                const float f = expf(m - mm);
                whole[tid] = f / (l * f + (sink ? expf(sink[h0 + min(tid, live - 1)] - mm) : 0.0f));
            }
            __syncthreads();
        }
        for (int i = tid; i < G * vdim; i += kThreads) store(i, a.sigmoid ? folded(i) : folded(i) * whole[i >> vshift]);
        return;
    }
    // ---- this share to the scratch: [G] maxima, [G] sums, [G][vdim]
    const int item = blockIdx.x * gridDim.y + blockIdx.y, stride = G * (vdim + 2);
    float *const mine = a.part + ((size_t)item * gridDim.z + blockIdx.z) * stride;
    if (!a.sigmoid && tid < G) __stcg(mine + tid, whole[tid]), __stcg(mine + G + tid, total(tid));
    for (int i = tid; i < G * vdim; i += kThreads) __stcg(mine + 2 * G + i, folded(i));
    __threadfence();
    __syncthreads();
    if (tid == 0) last_one = atomicInc(a.tickets + item, shares - 1) == (unsigned)(shares - 1);
    __syncthreads();
    if (!last_one) return;
    __threadfence();
    const float *const all = a.part + (size_t)item * gridDim.z * stride;
    float *const factor = sc;  // [shares][G], then [G]: of every share's sums in the result
    if (!a.sigmoid) {
        // a thread per (share, head): its share's factor, and the head's sum over all of them (one thread per head, share by share, took 5 us of 16 shares)
        static_assert(kMaxTokenShares * 8 <= kThreads, "a thread per share and head");
        const int h = tid % G, s = tid / G;
        float m = -INFINITY, l = 0.0f, f = 0.0f;
        const float snk = sink ? sink[h0 + min(h, live - 1)] : -INFINITY;
        if (s < shares) factor[s * G + h] = m = __ldcg(all + (size_t)s * stride + h), l = __ldcg(all + (size_t)s * stride + G + h);
        __syncthreads();
        float top = snk;
#pragma unroll
        for (int x = 0; x < kMaxTokenShares; ++x)
            if (x < shares) top = fmaxf(top, factor[x * G + h]);
        f = expf(m - top), l *= f;
        __syncthreads();
        if (s < shares) factor[s * G + h] = l;
        __syncthreads();
        l = sink ? expf(snk - top) : 0.0f;
#pragma unroll
        for (int x = 0; x < kMaxTokenShares; ++x)
            if (x < shares) l += factor[x * G + h];
        __syncthreads();
        if (s < shares) factor[s * G + h] = f / l;
        __syncthreads();
    }
    for (int i = tid; i < G * vdim; i += kThreads) {
        float v = 0.0f;
        for (int s0 = 0; s0 < shares; s0 += 8) {  // (eight shares' sums on their way at once)
            float p[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) p[s] = __ldcg(all + (size_t)min(s0 + s, shares - 1) * stride + 2 * G + i);
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (s0 + s < shares) v = a.sigmoid ? v + p[s] : fmaf(factor[(s0 + s) * G + (i >> vshift)], p[s], v);
        }
        store(i, v);
    }
}

template <typename T, int G> int launch_token_t(const TokenAttnArgs &args, const dim3 &grid, size_t smem, cudaStream_t st) {
    auto kern = token_attn_kernel<T, G>;
    if (smem > 48 * 1024) allow_smem(kern);
    launch_plain(kern, grid, dim3(kThreads), smem, st, args);
    return cuda_status("token_attention launch");
}

}  // namespace

size_t token_attention_part_floats(int vdim) { return (size_t)kTokenShareCtas * 8 * (vdim + 2); }

// B200_ERR_UNSUPPORTED (no error text): fp32, head sizes that lanes or threads do not share evenly, no scratch, more keys a share than fit shared memory.
// Keys are shared out until kTokenShareCtas CTAs (two per SM) run, 64 of the longest window a share at least.
int launch_token_attention(int dtype, const TokenAttn &a, int tokens, int max_keys, cudaStream_t st) {
    if (tokens == 0) return B200_OK;
    if (dtype == B200_F32 || a.dim % 32 != 0 || a.dim > 256 || (a.vdim != 64 && a.vdim != 128 && a.vdim != 256) || !a.part || !a.tickets || !all_aligned16({a.k_pool, a.v_pool}))
        return B200_ERR_UNSUPPORTED;
    const int group = a.heads / a.kv_heads, G = group >= 8 ? 8 : group > 4 ? 8 : group > 2 ? 4 : group;
    TokenAttnArgs args = {a, (group + G - 1) / G, 0};
    const int ctas = tokens * a.kv_heads * args.blocks;
    const int shares = ctas < 1 ? 1 : std::max(1, std::min({kMaxTokenShares, kTokenShareCtas / ctas, (max_keys + 63) / 64}));
    args.share_max = std::max(((max_keys + shares - 1) / shares + 7) / 8 * 8, 2 * kMaxTokenShares);
    const size_t smem = ((size_t)G * a.dim + (size_t)args.share_max * G + (size_t)kWarpsT * G * a.vdim + 2 * kWarpsT * G + G) * sizeof(float) + (args.share_max / kPageT + 2) * sizeof(int);
    if (smem > 100 * 1024 || a.kv_heads * args.blocks > 65535) return B200_ERR_UNSUPPORTED;
    const dim3 grid(tokens, a.kv_heads * args.blocks, shares);
#define B200_TOKEN_G(T) (G == 1 ? launch_token_t<T, 1>(args, grid, smem, st) : G == 2 ? launch_token_t<T, 2>(args, grid, smem, st) \
                         : G == 4 ? launch_token_t<T, 4>(args, grid, smem, st) : launch_token_t<T, 8>(args, grid, smem, st))
    return dtype == B200_BF16 ? B200_TOKEN_G(__nv_bfloat16) : B200_TOKEN_G(__half);
#undef B200_TOKEN_G
}

}  // namespace b200
