// sampling.cu -- top-k over the vocabulary and top-k sampling for sm_100a.
// Reference: src/kernels/topk.cu:24-140 (+ includes/topk.cuh:9-42), src/kernels/sampling.cu:14-102.
//
// Top-k is two launches like the reference (B200_TOPK_BLOCKS partial lists per row, then a merge) but with
// -inf sentinels and a total order (value descending, ties -> lower id), so ids are bit-exact against a CPU
// partial sort.  A row of 32000 logits is 128 KB: the stage is latency-, not bandwidth-bound.
#include "common.cuh"

#include <curand_kernel.h>

namespace b200 {

constexpr int kTopkThreads = 256;
constexpr int kMaxK = B200_TOPK_MAX_K;

struct Cand {
    float v;
    int id;
};
__device__ __forceinline__ bool better(float v, int id, float v2, int id2) { return v > v2 || (v == v2 && id < id2); }

// the best of a warp's candidates in two warp reductions: the largest value (as an unsigned key in the values' order, both zeros alike), then the lowest id
// that has it.  The value handed back is that of the lane with the id, bit for bit
__device__ __forceinline__ Cand warp_best(Cand c) {
    const unsigned bits = __float_as_uint(c.v + 0.0f), key = bits & 0x80000000u ? ~bits : bits | 0x80000000u;
    const unsigned best = __reduce_max_sync(0xffffffffu, key);
    const int id = __reduce_min_sync(0xffffffffu, key == best ? c.id : INT_MAX);
    const unsigned owner = __ballot_sync(0xffffffffu, key == best && c.id == id);
    return Cand{__shfl_sync(0xffffffffu, c.v, __ffs(owner) - 1), id};
}

// sorted insertion into a thread-local list (descending).  The list always has kMaxK entries, whatever k is: an index that is not a constant would put it in
// local memory (11 us for 8 rows of 32000, of which the reads take 2)
__device__ __forceinline__ void insert(float (&lv)[kMaxK], int (&li)[kMaxK], float v, int id) {
    if (!better(v, id, lv[kMaxK - 1], li[kMaxK - 1])) return;
    lv[kMaxK - 1] = v, li[kMaxK - 1] = id;
#pragma unroll
    for (int i = kMaxK - 1; i > 0; --i) {
        if (better(lv[i], li[i], lv[i - 1], li[i - 1])) {
            const float tv = lv[i];
            const int ti = li[i];
            lv[i] = lv[i - 1], li[i] = li[i - 1];
            lv[i - 1] = tv, li[i - 1] = ti;
        }
    }
}

// k rounds of block arg-best over the heads of the thread-local lists; the winner pops its head.
// Thread 0 ends up with the block's top-k in out_v / out_i.
__device__ __forceinline__ void block_select(float (&lv)[kMaxK], int (&li)[kMaxK], int k, float *out_v, int *out_i, Cand *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int r = 0; r < k; ++r) {
        Cand c = warp_best(Cand{lv[0], li[0]});
        __syncthreads();
        if (lane == 0) red[warp] = c;
        __syncthreads();
        Cand b = lane < nwarp ? red[lane] : Cand{-INFINITY, INT_MAX};
        b = warp_best(b);  // every warp computes the same winner
        if (threadIdx.x == 0) out_v[r] = b.v, out_i[r] = b.id == INT_MAX ? -1 : b.id;
        if (li[0] == b.id && b.id != INT_MAX) {
#pragma unroll
            for (int i = 0; i < kMaxK - 1; ++i) lv[i] = lv[i + 1], li[i] = li[i + 1];
            lv[kMaxK - 1] = -INFINITY, li[kMaxK - 1] = INT_MAX;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kTopkThreads)
topk_stage1_kernel(const T *__restrict__ logits, int *__restrict__ tmp_ids, T *__restrict__ tmp_vals, int vocab, int k) {
    __shared__ Cand red[32];
    __shared__ float sv[kMaxK];
    __shared__ int si[kMaxK];
    const int row = blockIdx.y, blk = blockIdx.x;
    const int per = (vocab + B200_TOPK_BLOCKS - 1) / B200_TOPK_BLOCKS;
    const int lo = blk * per, hi = min(vocab, lo + per);
    float lv[kMaxK];
    int li[kMaxK];
#pragma unroll
    for (int i = 0; i < kMaxK; ++i) lv[i] = -INFINITY, li[i] = INT_MAX;
    pdl_wait();
    pdl_launch_dependents();  // the merge is small: it takes its place (and its random numbers) while this runs
    const T *p = logits + (size_t)row * vocab;
    constexpr int U = 16;  // loads in flight per thread: a block's share of 32000 logits is 16 per thread, one round trip instead of 16
    for (int base = lo + threadIdx.x; base < hi; base += U * kTopkThreads) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = Elem<T>::to_f(p[min(base + u * kTopkThreads, hi - 1)]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (base + u * kTopkThreads < hi) insert(lv, li, v[u], base + u * kTopkThreads);
    }
    block_select(lv, li, k, sv, si, red);
    __syncthreads();
    if (threadIdx.x < k) {
        const size_t o = ((size_t)row * B200_TOPK_BLOCKS + blk) * k + threadIdx.x;
        tmp_ids[o] = si[threadIdx.x];
        tmp_vals[o] = Elem<T>::from_f(sv[threadIdx.x]);
    }
}

// The first curand_uniform() of curand_init(seed, subsequence = row, offset = 0), XORWOW.  cuRAND reaches subsequence b by a serial product of bit
// matrices per set bit of b (53 us at 8 rows, more than the LM head before it).  Subsequences are 2^67 states apart, and a state is linear over GF(2)
// (xorshift with 160 bits of state, G. Marsaglia, "Xorshift RNGs", 2003): with x^(2^67 b) mod p(x) = sum_j c_j x^j, p the recurrence's characteristic
// polynomial, the state 2^67 b steps on is the XOR of the states j steps on with c_j = 1 (jump ahead by polynomials: H. Haramoto et al., "Efficient
// jump ahead for F2-linear random number generators", 2008): 160 plain steps, about 5 us in one thread, per non-zero digit of b in base 16.  The additive
// counter of the generator is 32 bits wide and comes back to itself after 2^67 steps.
// kJump[15 d + v - 1][n]: bits 32 n .. of the coefficients for b = v 16^d.
constexpr int kJumpDigits = 4;
__constant__ uint32_t kJump[15 * kJumpDigits][5] = {
    {0x26294934u, 0x77bbc248u, 0x1a87dad0u, 0x930052d4u, 0x947e6dd2u},
    {0x5f39c379u, 0x95e20ba6u, 0x20e9ff72u, 0x1244ce5eu, 0xe8fd228fu},
    {0xd34e34c8u, 0x63486aa2u, 0x7ff96712u, 0xb90b6c6fu, 0x02756bc3u},
    {0xa7474d19u, 0x37c549e0u, 0x140877d2u, 0x24c43924u, 0xcd52ebecu},
    {0x7d3f439fu, 0xf2102b15u, 0xaf1bed4bu, 0xf6f1cfecu, 0x1982ad53u},
    {0x355e3fb6u, 0x29467127u, 0x7954e427u, 0xd3a177ebu, 0x65a68842u},
    {0xe8f8402fu, 0x251607a4u, 0x973ac23cu, 0xb54f78fcu, 0x0e384edcu},
    {0xe0360ec5u, 0xb1c96c24u, 0xdbb91766u, 0x666ff5dcu, 0xf19a7e52u},
    {0xf4688790u, 0x150b7bd8u, 0xd8a4058bu, 0xa544e815u, 0x84f3cbe0u},
    {0x376a36a3u, 0x893d50f9u, 0x3cca775cu, 0x94188f5fu, 0x1f7c8c1cu},
    {0x6876703bu, 0xae8bcf58u, 0xeb4934b3u, 0xbe2cf977u, 0xe6c88e5au},
    {0xc7d2569fu, 0xcea9dca7u, 0x343a9caau, 0x9c4f3af0u, 0xaf3023c5u},
    {0x4860ac12u, 0x281a7616u, 0x95ec5753u, 0x3b99123du, 0x299eb019u},
    {0xc1e1cee4u, 0x8773de1cu, 0xef0edcaau, 0x957d6eccu, 0x6ca6ef04u},
    {0x0a8843f8u, 0x3c8b03b2u, 0x2a9df47du, 0xa3aee006u, 0xd33edbb5u},
    {0xfcc8f692u, 0x35aa698au, 0x04ebbf85u, 0x448304b0u, 0x082f3fd5u},
    {0x48c289bdu, 0xe851cf98u, 0x845ad581u, 0xfd70752au, 0x2c3e63f6u},
    {0x1e21ea90u, 0x66483ba4u, 0x367e8d5au, 0x354ec274u, 0xc46eebcfu},
    {0xe502f5b3u, 0x77859d31u, 0x97e1cbb3u, 0xea09047au, 0x61d5f37eu},
    {0x1cee85c5u, 0x5e20b31au, 0xae442891u, 0xda5c599eu, 0x2b5aa0ddu},
    {0x09979962u, 0xf7a2c5d6u, 0x82c38e48u, 0x80127a42u, 0xf08a08b1u},
    {0x5ec46d26u, 0xd29b6df8u, 0x199a9d07u, 0x338f779eu, 0xa948f8a9u},
    {0xb89326d0u, 0x5a8655a9u, 0xfb6e98f5u, 0x02102162u, 0x7e6fcf6fu},
    {0xcb2fec0eu, 0x515a7310u, 0x4f28da5au, 0x34eef0e3u, 0x84aaaa48u},
    {0x757560fbu, 0x0383e791u, 0xdff3e8acu, 0x40eed643u, 0x6576f7aau},
    {0xfe9fb37du, 0xa4b61dc1u, 0xac099770u, 0x4f3b098bu, 0x174cfea2u},
    {0xb67196a6u, 0x52d14ef3u, 0xf4b8b94du, 0x8dd71586u, 0x8c7c93b9u},
    {0xbe76bf2au, 0xafa4810au, 0x739ddda6u, 0x0afca9a7u, 0x38c9742fu},
    {0xa55bf292u, 0x2ad932b8u, 0x2a078539u, 0x84515a78u, 0x83ce2623u},
    {0x673c6826u, 0x7970589bu, 0x50c4b02eu, 0xf5833b5bu, 0xba027595u},
    {0xb3a15db4u, 0xc6df3330u, 0x1a8be751u, 0xf1e4b221u, 0x6bb61c05u},
    {0x133de1d0u, 0x361e4422u, 0xc6131fcfu, 0xd9719f45u, 0x9658a164u},
    {0x1cc3f658u, 0x7367a8cdu, 0x2de525a8u, 0x3d325bb2u, 0x11840690u},
    {0x19e2bee8u, 0xf8974218u, 0x4e65536au, 0xa2570336u, 0xe9b88082u},
    {0x9670b020u, 0xc8a19ceau, 0x6f9a91ddu, 0x88ff33feu, 0xfcacb8ceu},
    {0x27c4ed23u, 0x2ec72ef3u, 0x9e4baf39u, 0x9ef3a344u, 0xc8f4977au},
    {0x00f5736eu, 0xabfc9507u, 0xa647616eu, 0xb6902babu, 0xc732b131u},
    {0x7863644bu, 0x2a21ce84u, 0x112e86f1u, 0xed01ce0eu, 0xba143e84u},
    {0x5f388f5du, 0x8449c123u, 0x0a764122u, 0x56985ea6u, 0x1546a43du},
    {0x28b544d7u, 0x6d34c95fu, 0x159159a7u, 0x993487c7u, 0x43b9e8a5u},
    {0x35662364u, 0xf51d2ce2u, 0x304a7885u, 0x1c7fce4du, 0x918fab4au},
    {0xb6413ee8u, 0x465624d8u, 0xbef4cb2bu, 0x5e4f8afau, 0x7bca03cdu},
    {0x5d5db0edu, 0xcc749900u, 0x1f667c65u, 0xdef695d4u, 0x24433877u},
    {0xbc9909a5u, 0x75353d5eu, 0x09d6f85au, 0x0544302du, 0xbaf6e3b8u},
    {0x14c50bb1u, 0x659d7c53u, 0xdf8d6524u, 0x23f1cc03u, 0x93dfcf0au},
    {0x0e2cae2eu, 0xd1011279u, 0x58923768u, 0x2bf650bau, 0xc985bcdau},
    {0x213a286au, 0x6596b510u, 0x6fc10eaeu, 0x38a13547u, 0x11c7749eu},
    {0xcbac929eu, 0x0575f836u, 0x676f5c22u, 0xfd7e35afu, 0x6c6d186bu},
    {0x146281e7u, 0xa45b4452u, 0xafa8c695u, 0x74a0ac94u, 0x4b250e0au},
    {0x7cc3a30du, 0x7af6aba9u, 0xb76a95b5u, 0x7ede6bf3u, 0x73ca3ea2u},
    {0x0866032au, 0xcb8fbd43u, 0x434a2e25u, 0x76eaae6bu, 0x13033bc8u},
    {0x5bdf8040u, 0x819445feu, 0x8e1b4143u, 0x8fcbd027u, 0xb6d68447u},
    {0x2306bc52u, 0x790f3b4cu, 0x2fe473b9u, 0xbc81d7c0u, 0x093efe98u},
    {0xbbf96040u, 0x378d69edu, 0x818e3afdu, 0xc933a401u, 0xe1b3bd35u},
    {0xe56a37b5u, 0x7fbf623fu, 0xb65ee777u, 0x33ea8847u, 0xda382be9u},
    {0x5b985de7u, 0xbc7a8575u, 0xd49fdfc0u, 0xaceac3d0u, 0xabcc7c87u},
    {0xdb2cf4c2u, 0xb49a5412u, 0x5c88dea9u, 0xd999bf6cu, 0xffe7924eu},
    {0xa608a919u, 0xc837eb1du, 0xacb40874u, 0x30685f3eu, 0x5071b091u},
    {0x6dda9fe0u, 0x9173054bu, 0x9e61560au, 0x134264a2u, 0xccaaed2cu},
    {0x104ecff0u, 0x2d271e74u, 0x8406da7au, 0x5258916du, 0x7e87f982u},
};
__device__ __forceinline__ float first_uniform(unsigned long long seed, unsigned int row) {
    curandState_t state;
    const bool far = row >> (4 * kJumpDigits);
    curand_init(seed, far ? (unsigned long long)row : 0ull, 0ull, &state);
    if (!far) {
        for (int d = 0; row; ++d, row >>= 4) {
            const unsigned int digit = row & 15u;
            if (!digit) continue;
            uint32_t w[5], out[5] = {0u, 0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 5; ++e) w[e] = state.v[e];
            for (int n = 0; n < 5; ++n) {
                const uint32_t c = kJump[15 * d + digit - 1][n];
#pragma unroll
                for (int bit = 0; bit < 32; ++bit) {
                    const uint32_t take = 0u - ((c >> bit) & 1u);
#pragma unroll
                    for (int e = 0; e < 5; ++e) out[e] ^= w[e] & take;
                    const uint32_t t = w[0] ^ (w[0] >> 2);
                    w[0] = w[1], w[1] = w[2], w[2] = w[3], w[3] = w[4];
                    w[4] = (w[4] ^ (w[4] << 4)) ^ (t ^ (t << 1));
                }
            }
#pragma unroll
            for (int e = 0; e < 5; ++e) state.v[e] = out[e];
        }
    }
    return curand_uniform(&state);
}

// What one row draws from its k candidates; same arithmetic order as the reference kernel.
template <typename T>
__device__ __forceinline__ void draw_row(float uniform, const int *id, T *val, int *seq_len, uint8_t *finished, int *output_id, int k, int end_id, int vocab) {
    const float mx = Elem<T>::to_f(val[0]);
    for (int i = 0; i < k; ++i) val[i] = Elem<T>::from_f(expf(Elem<T>::to_f(val[i]) - mx));
    float sum = 0.0f;
    for (int i = 0; i < k; ++i) sum += Elem<T>::to_f(val[i]);
    float thr = uniform * sum;
    int chosen = id[0];
    for (int i = 0; i < k; ++i) {
        thr -= Elem<T>::to_f(val[i]);
        if (thr < 0.0f) {
            chosen = id[i];
            break;
        }
    }
    // an empty top-k slot (id -1 / INT_MAX: every candidate NaN or -inf, or vocab < k) must never reach the embedding gather of the next
    // step: the row ends instead (end_id when it is a valid token, else token 0)
    if (chosen < 0 || chosen == INT_MAX) chosen = (end_id >= 0 && end_id < vocab) ? end_id : 0;
    else chosen %= vocab;
    *output_id = chosen;
    if (!*finished) ++*seq_len;
    *finished = (uint8_t)(chosen == end_id);
}
struct DrawArgs {
    int *seq_len;
    uint8_t *finished;
    int *output_id;
    int step, end_id, vocab;
};

// DRAW: the row's sample is drawn from its candidates right here (the sampling tail of the engine: one launch less between the logits and the token).  The
// random number depends on the step and the row alone, so it is formed before the wait for the kernel in front.
template <typename T, bool DRAW>
__global__ void __launch_bounds__(64)
topk_stage2_kernel(const int *__restrict__ tmp_ids, const T *__restrict__ tmp_vals, int *final_ids, T *final_vals, int k, const DrawArgs draw) {
    __shared__ Cand red[32];
    __shared__ float sv[kMaxK];
    __shared__ int si[kMaxK];
    const int row = blockIdx.x;
    float lv[kMaxK];
    int li[kMaxK];
#pragma unroll
    for (int i = 0; i < kMaxK; ++i) lv[i] = -INFINITY, li[i] = INT_MAX;
    float uniform = 0.0f;
    if (DRAW && threadIdx.x == 0) uniform = first_uniform((unsigned long long)draw.step, (unsigned int)row);
    pdl_wait();
    if (!DRAW) pdl_launch_dependents();
    for (int i = threadIdx.x; i < B200_TOPK_BLOCKS * k; i += 64) {
        const int id = tmp_ids[(size_t)row * B200_TOPK_BLOCKS * k + i];
        if (id >= 0) insert(lv, li, Elem<T>::to_f(tmp_vals[(size_t)row * B200_TOPK_BLOCKS * k + i]), id);
    }
    block_select(lv, li, k, sv, si, red);
    if constexpr (DRAW) {
        static_assert(sizeof(T) == sizeof(float), "the candidates are drawn from as they are stored");
        if (threadIdx.x == 0)  // (it wrote sv and si)
            draw_row<float>(uniform, si, sv, draw.seq_len + row, draw.finished + row, draw.output_id + row, k, draw.end_id, draw.vocab);
    }
    __syncthreads();
    if (threadIdx.x < k) {
        final_ids[(size_t)row * k + threadIdx.x] = si[threadIdx.x];
        final_vals[(size_t)row * k + threadIdx.x] = Elem<T>::from_f(sv[threadIdx.x]);
    }
}

// one thread per batch row
template <typename T>
__global__ void sampling_kernel(const int *__restrict__ topk_id, T *topk_val, int *seq_len, uint8_t *finished, int *output_id,
                                int batch, int k, int step, int end_id, int vocab) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const float uniform = first_uniform((unsigned long long)step, (unsigned int)b);
    pdl_wait();
    if (b >= batch) return;
    draw_row<T>(uniform, topk_id + (size_t)b * k, topk_val + (size_t)b * k, seq_len + b, finished + b, output_id + b, k, end_id, vocab);
}

__global__ void xorwow_uniform_kernel(float *out, int n, unsigned long long seed) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    curandState_t state;
    curand_init(seed, (unsigned long long)b, 0ull, &state);
    out[b] = curand_uniform(&state);
}

// top-k over fp32 logits and the draw from it in two launches (b200_topk followed by b200_sampling: the same results)
int launch_topk_draw(const float *logits, int *tmp_ids, float *tmp_vals, int *final_ids, float *final_vals, int *seq_len, uint8_t *finished, int *output_id, int rows,
                     int vocab, int k, int step, int end_id, cudaStream_t st) {
    if (rows == 0) return B200_OK;
    launch_pdl(topk_stage1_kernel<float>, dim3(B200_TOPK_BLOCKS, rows), dim3(kTopkThreads), 0, st, true, logits, tmp_ids, tmp_vals, vocab, k);
    launch_pdl(topk_stage2_kernel<float, true>, dim3(rows), dim3(64), 0, st, true, (const int *)tmp_ids, (const float *)tmp_vals, final_ids, final_vals, k,
               DrawArgs{seq_len, finished, output_id, step, end_id, vocab});
    return cuda_status("topk + draw launch");
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_topk(const void *logits, int *tmp_ids, void *tmp_vals, int *final_ids, void *final_vals, int rows, int vocab, int k,
              int dtype, b200_stream_t stream) {
    B200_REQUIRE(logits && tmp_ids && tmp_vals && final_ids && final_vals, "topk: null pointer");
    B200_REQUIRE(rows >= 0 && vocab > 0, "topk: bad shape");
    B200_REQUIRE(k >= 1 && k <= B200_TOPK_MAX_K, "topk: k=%d outside [1, %d]", k, B200_TOPK_MAX_K);
    B200_REQUIRE(rows <= 65535, "topk: rows %d > 65535", rows);
    if (rows == 0) return B200_OK;
    cudaStream_t st = as_stream(stream);
    B200_DISPATCH_DTYPE(dtype, {
        launch_pdl(topk_stage1_kernel<T>, dim3(B200_TOPK_BLOCKS, rows), dim3(kTopkThreads), 0, st, true, (const T *)logits, tmp_ids,
                   (T *)tmp_vals, vocab, k);
        launch_pdl(topk_stage2_kernel<T, false>, dim3(rows), dim3(64), 0, st, true, (const int *)tmp_ids, (const T *)tmp_vals, final_ids,
                   (T *)final_vals, k, DrawArgs{});
    });
    return cuda_status("topk launch");
}

int b200_sampling(const int *topk_id, void *topk_val, int *seq_len, uint8_t *finished, int *output_id, int batch, int k, int step,
                  int end_id, int vocab, int dtype, b200_stream_t stream) {
    B200_REQUIRE(topk_id && topk_val && seq_len && finished && output_id, "sampling: null pointer");
    B200_REQUIRE(batch >= 0 && k >= 1 && vocab > 0, "sampling: bad shape");
    if (batch == 0) return B200_OK;
    B200_DISPATCH_DTYPE(dtype, launch_pdl(sampling_kernel<T>, dim3((batch + 31) / 32), dim3(32), 0, as_stream(stream), true, topk_id,
                                          (T *)topk_val, seq_len, finished, output_id, batch, k, step, end_id, vocab));
    return cuda_status("sampling launch");
}

int b200_xorwow_uniform(float *out, int n, unsigned long long seed, b200_stream_t stream) {
    B200_REQUIRE(out && n >= 0, "xorwow_uniform: bad argument");
    if (n == 0) return B200_OK;
    xorwow_uniform_kernel<<<(n + 31) / 32, 32, 0, as_stream(stream)>>>(out, n, seed);
    return cuda_status("xorwow_uniform launch");
}

}  // extern "C"
