// prompt_attn_tc.cu -- attention of prompt portions of the layer-list decoder on tcgen05 / TMEM: the chunked sink attention (attention_chunked.cu), the
// latent attention (attention_latent.cu) and the softmax form of the scored attention without a cap (attention_scored.cu; s loses r1 ln(1 + r2 (i - j))
// and slope (i - j)) at the sizes that fill its tiles; other sizes, short portions and fp32 engines keep those files' kernels.
//     s(i, j) = scale q_i . k_j over the visible j <= i (same block of `chunk` positions, or i - j < window);  out_i = sum_j p_ij v_j, p the softmax
//     with one more logit `sink` in the denominator
// The mma.sync kernels reach a tenth of the tensor rate: operands go through registers, two CTAs per SM hide little of it.  Here one CTA takes the 64
// tokens of a tile x TWO heads that share their keys (any two latent heads; two query heads of one kv head) as the 128 rows of an MMA, so a key page is
// read from memory once for both:
//   * producer warp: one page of 64 keys or values per ring stage (page-table look-up, one TMA box per 64 columns, 128-byte swizzle), in the order the
//     products take them (K0 K1 V0 K2 V1 ...); latent layers have their values in the first DV columns of the key rows: one tile serves both products;
//   * MMA warp: S = Q K^T (128 x 64, two TMEM buffers: the next page's scores are formed while the softmax works) and O += P V, V the MN-major operand,
//     O in TMEM for the whole loop;
//   * WARPS softmax warps: WARPS / 4 threads share a row; lazy rescale: O is scaled only when the running maximum grows by more than 2^8 (see
//     context_attn_tc.cu, whose loop this follows); the sink is the initial maximum and sum; value rows past the tile's last query are zeroed, since a page's
//     unwritten rows may hold anything and 0 * NaN would reach the accumulator.
// A step is a chain (scores, TMEM read, row maximum, exponentials, P, product): two CTAs per SM fill each other's waits (not for latent rows, which are too
// large, nor for logits with a penalty).
// Measured against the mma.sync kernels, us per layer: chunked 175 -> 63 (4096 tokens, 16 heads of 128), latent 244 -> 80 (3085 tokens in two prompts, 16
// heads, rank 192 + 64), scored with a distance penalty and a window of 1024 116 -> 79 (2911 tokens in three prompts, 16 heads of 128).
#include "hybrid_ops.cuh"

#include <cuda.h>
#include <algorithm>

namespace b200 {

namespace {

constexpr int kPage = B200_KV_PAGE_SIZE;   // keys per tile
constexpr int kQRows = 128;                // 64 tokens x 2 heads
constexpr int kQBox = kQRows * 128;        // bytes of 64 columns of Q or of P
constexpr int kKBox = kPage * 128;         // bytes of 64 columns of a key / value page
constexpr float kLog2eP = 1.4426950408889634f;
constexpr float kRescale = 8.0f;           // log2 domain
constexpr int kMaxPenalty = 8192;          // longest window with a distance penalty (its table is in shared memory)

struct PromptAttn {
    const void *q, *qr;        // latent: q [heads, t_pad, DV], qr [tokens, heads, DK - DV];  chunked: q [tokens, heads * DK]
    const float *sink;         // [heads] or NULL
    const void *gate;          // chunked: [tokens, gate_ld] or NULL
    void *out;                 // latent: [heads, t_pad, DV];  chunked: [tokens, heads * DV]
    const int *tiles, *block_table;
    int n_tiles, mpps, heads, group, kv_heads, t_pad, gate_ld, window, chunk, is_bf16;  // group: query heads per kv head (latent: all share)
    float scale;
    // scored layers: out rows `out_ld` apart, scaled; what the distance i - j takes off a logit: r1[h] ln(1 + r2[h] d) (d < pen_len) + slope[h] d
    int out_ld, pen_len;
    float out_scale;
    const float *dist_r1, *dist_r2, *slope;
    WaitGuard wait;
};

__device__ __forceinline__ uint32_t pa_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void pa_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void pa_expect(uint32_t bar, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ void pa_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void pa_tma(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void pa_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pa_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pa_commit(uint32_t bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void pa_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pa_ld16(uint32_t addr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                   "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void pa_st16(uint32_t addr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void pa_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pa_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float pa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 128-byte-swizzled operands (8-row atoms of 1024 bytes): K-major, and MN-major with `box` bytes between groups of 64 columns
__device__ __forceinline__ uint64_t pa_desc(uint32_t addr, uint32_t box) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(box >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint32_t pa_idesc(bool bf16, int n, bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kQRows >> 4) << 24);
}

template <int DK, int DV, bool LATENT> struct PaShape {
    static constexpr int kWarps = LATENT ? 16 : 8;                               // softmax warps
    static constexpr int kStages = 3;
    static constexpr int kStage = DK / 64 * kKBox;                               // bytes of a ring stage: a key page, or a value page (DV == DK)
    static constexpr int kCtas = LATENT ? 1 : 2;                                 // per SM
    static constexpr int kTmem = DV + 2 * kPage <= 256 ? 256 : 512;
    static constexpr size_t kSmem = 1024 + (size_t)(DK / 64) * kQBox + (size_t)kStages * kStage + kQBox + 256 + 2 * kQRows * (kWarps / 4) * sizeof(float);
};

template <typename T, int DK, int DV, bool LATENT, bool BIASED>
__global__ void __launch_bounds__(PaShape<DK, DV, LATENT>::kWarps * 32 + 64, PaShape<DK, DV, LATENT>::kCtas)
prompt_attn_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const PromptAttn p) {
    using Sh = PaShape<DK, DV, LATENT>;
    constexpr int WARPS = Sh::kWarps, WPR = WARPS / 4, ST = Sh::kStages, SC = kPage / WPR, OC = DV / WPR;  // keys / value columns per thread
    static_assert(SC % 16 == 0 && OC % 16 == 0, "TMEM is read 16 columns at a time");
    static_assert(LATENT || DK == DV, "a ring stage holds a key or a value page");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *sQ = smem, *ring = sQ + (DK / 64) * kQBox, *sP = ring + ST * Sh::kStage;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sP + kQBox);
    const uint32_t q_full = pa_u32(bars), full0 = q_full + 8, empty0 = full0 + 8 * ST, s_full0 = empty0 + 8 * ST, s_free0 = s_full0 + 16, p_ready = s_free0 + 16, pv_done = p_ready + 8, drain = pv_done + 8;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 16);
    float *red = reinterpret_cast<float *>(bars + 32);  // [2][128][WPR]
    float *pen = red + 2 * kQRows * WPR;                // [2][pen_len] (BIASED): the penalty of either head in base-2 units

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 tile = reinterpret_cast<const int4 *>(p.tiles)[p.n_tiles - 1 - blockIdx.x];  // later tiles see more keys: first
    const int seq = tile.x, row0 = tile.y, rows = tile.z, pos0 = tile.w;
    const int h0 = 2 * blockIdx.y, last = pos0 + rows - 1;
    // pages that hold a key some row of the tile sees
    int lo = 0;
    if (p.window > 0) lo = max(0, pos0 - p.window + 1);
    if (p.chunk > 0) lo = max(lo, pos0 / p.chunk * p.chunk);
    const int page0 = lo / kPage, n = last / kPage + 1 - page0;
    // ring items in the order the products take them: K0 K1 V0 K2 V1 ... (latent: every page once)
    auto k_item = [&](int j) { return LATENT ? j : (j == 0 ? 0 : 2 * j - 1); };
    auto v_item = [&](int j) { return LATENT ? j : (j + 1 < n ? 2 * j + 2 : 2 * j + 1); };

    if (warp == WARPS && lane == 0) {
        cta_gave_up() = 0;
        pa_init(q_full, WARPS);
        for (int s = 0; s < ST; ++s) {
            pa_init(full0 + 8 * s, 1);
            pa_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            pa_init(s_full0 + 8 * b, 1);
            pa_init(s_free0 + 8 * b, WARPS);
        }
        pa_init(p_ready, WARPS);
        pa_init(pv_done, 1);
        pa_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pa_u32(tmem_slot)), "r"((uint32_t)Sh::kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pa_before();
    __syncthreads();
    pa_after();
    const uint32_t tmem = *tmem_slot;  // columns: S0 [0, 64) S1 [64, 128) O [128, 128 + DV)
    // a wait that runs out ends all of the CTA's: no more copies, no more products; the softmax warps go through their tiles (they meet at named barriers)
    // and store NaN
    auto wait = [&](uint32_t bar, uint32_t parity) { return mbar_wait_guarded(bar, parity, p.wait, kWaitPromptAttn); };

    if (warp == WARPS) {
        // ================================================= producer
        if (lane == 0) {
            const int *bt = p.block_table + (size_t)seq * p.mpps + page0;
            int i = 0;
            bool live = true;
            for (; i < (LATENT ? n : 2 * n); ++i) {
                const int s = i % ST;
                const bool value = !LATENT && i > 0 && (i == 2 * n - 1 || (i & 1) == 0);
                const int j = LATENT ? i : (i == 0 ? 0 : (value ? (i == 2 * n - 1 ? n - 1 : i / 2 - 1) : (i + 1) / 2));
                const int row = LATENT ? __ldg(bt + j) * kPage : (__ldg(bt + j) * p.kv_heads + h0 / p.group) * kPage;
                live = wait(empty0 + 8 * s, ((i / ST) & 1) ^ 1);
                if (!live) break;
                const uint32_t d = pa_u32(ring + s * Sh::kStage), bar = full0 + 8 * s;
                pa_expect(bar, Sh::kStage);
#pragma unroll
                for (int c = 0; c < DK / 64; ++c) pa_tma(d + c * kKBox, value ? &tmV : &tmK, 64 * c, row, bar);
            }
            // the CTA stays until its last copies have landed and, if all is well, their stages have been released
            for (int j = max(0, i - ST); j < i; ++j) {
                if (!mbar_drain(full0 + 8 * (j % ST), (j / ST) & 1)) break;
                if (live) live = wait(empty0 + 8 * (j % ST), (j / ST) & 1);
            }
        }
    } else if (warp == WARPS + 1) {
        // ================================================= MMA issuer: one thread
        if (lane == 0) {
            const uint32_t id_qk = pa_idesc(p.is_bf16 != 0, kPage, false), id_pv = pa_idesc(p.is_bf16 != 0, DV, true);
            auto scores = [&](int j) -> bool {
                const int i = k_item(j), s = i % ST, sb = j & 1;
                if (!wait(full0 + 8 * s, (i / ST) & 1) || !wait(s_free0 + 8 * sb, ((j >> 1) & 1) ^ 1)) return false;
                pa_after();
                const uint32_t aq = pa_u32(sQ), bk = pa_u32(ring + s * Sh::kStage);
#pragma unroll
                for (int k = 0; k < DK / 16; ++k)
                    pa_mma(tmem + (uint32_t)(sb * kPage), pa_desc(aq + (k / 4) * kQBox + (k % 4) * 32, 16), pa_desc(bk + (k / 4) * kKBox + (k % 4) * 32, 16), id_qk, k > 0 ? 1u : 0u);
                if (!LATENT) pa_commit(empty0 + 8 * s);  // (a latent page still serves as the values)
                pa_commit(s_full0 + 8 * sb);
                return true;
            };
            bool live = wait(q_full, 0) && scores(0);
            for (int j = 0; live && j < n; ++j) {
                if (j + 1 < n && !scores(j + 1)) break;
                const int i = v_item(j), s = i % ST;
                if (!LATENT && !wait(full0 + 8 * s, (i / ST) & 1)) break;
                if (!wait(p_ready, j & 1)) break;
                pa_after();
                const uint32_t ap = pa_u32(sP), bv = pa_u32(ring + s * Sh::kStage);
#pragma unroll
                for (int k = 0; k < kPage / 16; ++k)
                    pa_mma(tmem + 2 * kPage, pa_desc(ap + k * 32, 16), pa_desc(bv + k * 16 * 128, kKBox), id_pv, (j > 0 || k > 0) ? 1u : 0u);
                pa_commit(empty0 + 8 * s);
                pa_commit(pv_done);
            }
            pa_commit(drain);  // no product reads shared memory or writes TMEM when the CTA leaves
            mbar_drain(drain, 0);
        }
    } else {
        // ================================================= softmax + epilogue: row = head half x token; WPR threads per row
        const int quarter = warp & 3, cg = warp >> 2, row = quarter * 32 + lane;
        const int head = h0 + (row >> 6), tok = row & 63, pos = pos0 + tok;
        const bool live = tok < rows;
        // ---- Q into shared memory (swizzled): this row's pieces are dealt to its WPR threads
        {
            const T *src = nullptr, *src_r = nullptr;
            if constexpr (LATENT) {
                src = static_cast<const T *>(p.q) + ((size_t)head * p.t_pad + row0 + tok) * DV;
                src_r = static_cast<const T *>(p.qr) + ((size_t)(row0 + tok) * p.heads + head) * (DK - DV);
            } else {
                src = static_cast<const T *>(p.q) + ((size_t)(row0 + tok) * p.heads + head) * DK;
            }
#pragma unroll 8
            for (int c = cg; c < DK / 8; c += WPR) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (live) v = LATENT && c >= DV / 8 ? ld_v4(src_r + (c - DV / 8) * 8) : ld_v4(src + c * 8);
                *reinterpret_cast<uint4 *>(sQ + (c >> 3) * kQBox + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = v;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) pa_arrive(q_full);
        }
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t o_addr = lane_addr + (uint32_t)(2 * kPage + cg * OC);
        const float sl2 = p.scale * kLog2eP;
        const float slope = BIASED && p.slope ? p.slope[head] * kLog2eP : 0.0f;
        const float *my_pen = pen + (row >> 6) * p.pen_len;
        const bool has_pen = BIASED && p.dist_r1 != nullptr;
        if (has_pen) {
            for (int i = threadIdx.x; i < 2 * p.pen_len; i += WARPS * 32) {
                const int hh = h0 + (i >= p.pen_len), d = i >= p.pen_len ? i - p.pen_len : i;
                pen[i] = p.dist_r1[hh] * kLog2eP * log1pf(p.dist_r2[hh] * (float)d);
            }
            asm volatile("bar.sync 5, %0;" ::"r"(WARPS * 32) : "memory");
        }
        const float sink = p.sink ? p.sink[head] * kLog2eP : 0.0f;
        float m_run = p.sink ? sink : -1e30f, m_use = m_run, l = 0.0f;
        // visible keys of this row: [first, pos]
        int first = 0;
        if (p.window > 0) first = max(first, pos - p.window + 1);
        if (p.chunk > 0) first = max(first, pos / p.chunk * p.chunk);
        // the tile's rows all see keys [first_all, pos0]: pages inside need no mask
        int first_all = 0;
        if (p.window > 0) first_all = max(first_all, last - p.window + 1);
        if (p.chunk > 0) first_all = max(first_all, last / p.chunk * p.chunk);
        for (int j = 0; j < n; ++j) {
            const int sb = j & 1, kp = (page0 + j) * kPage, k0 = kp + cg * SC;
            uint32_t r[SC];
            (void)wait(s_full0 + 8 * sb, (j >> 1) & 1);
            pa_after();
#pragma unroll
            for (int c = 0; c < SC; c += 16) pa_ld16(lane_addr + (uint32_t)(sb * kPage + cg * SC + c), r + c);
            pa_wait_ld();
            pa_before();
            __syncwarp();
            if (lane == 0) pa_arrive(s_free0 + 8 * sb);
            float mloc = -INFINITY;
            if constexpr (BIASED) {  // the logits in base-2 units
#pragma unroll
                for (int e = 0; e < SC; ++e) {
                    const int d = pos - (k0 + e);
                    float v = fmaf(-slope, (float)d, __uint_as_float(r[e]) * sl2);
                    if (has_pen) v -= my_pen[min(max(d, 0), p.pen_len - 1)];
                    r[e] = __float_as_uint(v);
                }
            }
            if (kp < first_all || kp + kPage - 1 > pos0) {
#pragma unroll
                for (int e = 0; e < SC; ++e) {
                    if (k0 + e < first || k0 + e > pos) r[e] = 0xff800000u;  // -inf
                    mloc = fmaxf(mloc, __uint_as_float(r[e]));
                }
            } else {
#pragma unroll
                for (int e = 0; e < SC; ++e) mloc = fmaxf(mloc, __uint_as_float(r[e]));
            }
            float *rx = red + ((size_t)(j & 1) * kQRows + row) * WPR;
            rx[cg] = BIASED ? mloc : mloc * sl2;  // scale > 0
            asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "r"(WPR * 32) : "memory");
#pragma unroll
            for (int c = 0; c < WPR; ++c) m_run = fmaxf(m_run, rx[c]);
            if (j == 0) {
                m_use = m_run;  // the first tile overwrites the accumulator
                l = p.sink && cg == 0 ? pa_ex2(sink - m_use) : 0.0f;
            } else {
                const bool need = m_run - m_use > kRescale;
                if (__any_sync(0xffffffffu, need)) {
                    const float corr = need ? pa_ex2(m_use - m_run) : 1.0f;
                    if (need) m_use = m_run;
                    l *= corr;
                    (void)wait(pv_done, (j - 1) & 1);
                    pa_after();
#pragma unroll
                    for (int c = 0; c < OC; c += 16) {
                        uint32_t acc[16];
                        pa_ld16(o_addr + c, acc);
                        pa_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) acc[e] = __float_as_uint(__uint_as_float(acc[e]) * corr);
                        pa_st16(o_addr + c, acc);
                    }
                    pa_wait_st();
                    pa_before();
                }
            }
            uint4 packed[SC / 8];
#pragma unroll
            for (int q = 0; q < SC / 8; ++q) {
                float pf[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    pf[u] = BIASED ? pa_ex2(__uint_as_float(r[8 * q + u]) - m_use) : pa_ex2(fmaf(__uint_as_float(r[8 * q + u]), sl2, -m_use));
                    l += pf[u];
                }
                packed[q] = pack16<T>(pf);
            }
            if (j > 0) (void)wait(pv_done, (j - 1) & 1);  // the previous product has read P
            unsigned char *prow = sP + row * 128;
#pragma unroll
            for (int q = 0; q < SC / 8; ++q) *reinterpret_cast<uint4 *>(prow + (((cg * (SC / 8) + q) ^ (row & 7)) << 4)) = packed[q];
            // value rows past the tile's last query: cleared by the threads of rows 0 .. 63 (the scores have been formed: a shared tile may go too)
            if (row < kPage && kp + row > last) {
                const int i = v_item(j);
                (void)wait(full0 + 8 * (i % ST), (i / ST) & 1);
                unsigned char *v = ring + (i % ST) * Sh::kStage + row * 128;
                for (int c = cg; c < DV / 8; c += WPR) *reinterpret_cast<uint4 *>(v + (c >> 3) * kKBox + ((c & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) pa_arrive(p_ready);
        }
        float *rx = red + ((size_t)(n & 1) * kQRows + row) * WPR;
        rx[cg] = l;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "r"(WPR * 32) : "memory");
        float sum = 0.0f;
#pragma unroll
        for (int c = 0; c < WPR; ++c) sum += rx[c];
        const float inv = LATENT ? 1.0f / sum : p.out_scale / sum;
        const bool lost = !wait(pv_done, (n - 1) & 1) || cta_gave_up();  // (set before anything that was formed without having waited is handed on)
        pa_after();
#pragma unroll
        for (int c = 0; c < OC; c += 16) {
            uint32_t acc[16];
            pa_ld16(o_addr + c, acc);
            pa_wait_ld();
            if (live) {
                const int col = cg * OC + c;
                float f[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] = lost ? __int_as_float(0x7fc00000) : __uint_as_float(acc[e]) * inv;
                T *dst;
                if constexpr (LATENT) {
                    dst = static_cast<T *>(p.out) + ((size_t)head * p.t_pad + row0 + tok) * DV + col;
                } else {
                    dst = static_cast<T *>(p.out) + (size_t)(row0 + tok) * p.out_ld + head * DV + col;
                    if (p.gate) {
                        const T *gz = static_cast<const T *>(p.gate) + (size_t)(row0 + tok) * p.gate_ld + head * DV + col;
                        float z[16];
                        unpack16<T>(ld_v4(gz), z);
                        unpack16<T>(ld_v4(gz + 8), z + 8);
#pragma unroll
                        for (int e = 0; e < 16; ++e) f[e] = f[e] / (1.0f + expf(-z[e]));
                    }
                }
                st_v4(dst, pack16<T>(f));
                st_v4(dst + 8, pack16<T>(f + 8));
            }
        }
    }

    pa_before();
    __syncthreads();
    if (warp == WARPS + 1) {
        pa_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)Sh::kTmem) : "memory");
    }
}

// the pool as a matrix of `cols`-wide rows in boxes of one page x 64 columns.  Its row count is not known here: the block table names the rows that are
// asked for, and those exist
bool pa_map(CUtensorMap *map, const void *ptr, int cols, bool bf16) {
    return tile_map(map, ptr, (size_t)1 << 30, cols, kPage, bf16);
}

template <typename T, int DK, int DV, bool LATENT, bool BIASED>
int pa_launch(PromptAttn p, const void *k_pool, const void *v_pool, bool bf16, cudaStream_t st) {
    CUtensorMap tmK, tmV;
    p.wait = wait_guard();
    if (!pa_map(&tmK, k_pool, DK, bf16) || !pa_map(&tmV, v_pool, LATENT ? DK : DV, bf16)) {
        set_error("prompt attention: cuTensorMapEncodeTiled failed");
        return B200_ERR_CUDA;
    }
    using Sh = PaShape<DK, DV, LATENT>;
    auto kern = prompt_attn_tc_kernel<T, DK, DV, LATENT, BIASED>;
    // (logits with a penalty: one CTA per SM.  Two ran only while the launches of this path overlapped, an order that stopped for a reason not found and was
    // taken back with them; the form has not been shown sound by itself)
    const size_t smem = std::max<size_t>(Sh::kSmem + 2 * p.pen_len * sizeof(float), BIASED ? 120 * 1024 : 0);
    allow_smem(reinterpret_cast<const void *>(kern), std::max<size_t>(Sh::kSmem + (BIASED ? 2 * (kMaxPenalty + 64) * sizeof(float) : 0), BIASED ? 120 * 1024 : 0));
    launch_plain(kern, dim3(p.n_tiles, p.heads / 2), dim3(Sh::kWarps * 32 + 64), smem, st, tmK, tmV, p);
    return cuda_status("prompt attention (tcgen05) launch");
}

}  // namespace

// B200_ERR_UNSUPPORTED (no error text, nothing launched): types, sizes and alignments that keep the mma.sync kernels
int launch_chunked_attention_tc(int dtype, const void *q, const void *k_pool, const void *v_pool, const float *sink, const void *gate, int gate_ld, void *out,
                                const int *tiles, int n_tiles, const int *block_table, int mpps, int heads, int kv_heads, int dim, float scale, int chunk, cudaStream_t st) {
    if ((dtype != B200_BF16 && dtype != B200_F16) || dim != 128 || heads / kv_heads % 2 != 0 || !(scale > 0.0f)) return B200_ERR_UNSUPPORTED;
    if (!all_aligned16({q, k_pool, v_pool, gate, out, tiles}) || (gate && gate_ld % 8 != 0)) return B200_ERR_UNSUPPORTED;
    if (n_tiles == 0) return B200_OK;
    PromptAttn p = {};
    p.q = q, p.sink = sink, p.gate = gate, p.gate_ld = gate_ld, p.out = out, p.tiles = tiles, p.n_tiles = n_tiles, p.block_table = block_table, p.mpps = mpps;
    p.heads = heads, p.group = heads / kv_heads, p.kv_heads = kv_heads, p.chunk = chunk, p.scale = scale, p.is_bf16 = dtype == B200_BF16;
    p.out_ld = heads * dim, p.out_scale = 1.0f;
    return dtype == B200_BF16 ? pa_launch<__nv_bfloat16, 128, 128, false, false>(p, k_pool, v_pool, true, st) : pa_launch<__half, 128, 128, false, false>(p, k_pool, v_pool, false, st);
}

int launch_scored_attention_tc(int dtype, const void *q, const void *k_pool, const void *v_pool, const float *dist_r1, const float *dist_r2, const void *gate, int gate_ld,
                               void *out, int out_ld, float out_scale, const int *tiles, int n_tiles, const int *block_table, int mpps, int heads, int kv_heads, int dim, int vdim,
                               float scale, int window, int sigmoid, ScoredOptions opt, cudaStream_t st) {
    if ((dtype != B200_BF16 && dtype != B200_F16) || dim != 128 || vdim != 128 || sigmoid || opt.softcap > 0.0f || heads / kv_heads % 2 != 0 || !(scale > 0.0f)) return B200_ERR_UNSUPPORTED;
    if (dist_r1 && !(window > 0 && window <= kMaxPenalty)) return B200_ERR_UNSUPPORTED;
    if (!all_aligned16({q, k_pool, v_pool, gate, out, tiles}) || (gate && gate_ld % 8 != 0) || out_ld % 8 != 0) return B200_ERR_UNSUPPORTED;
    if (n_tiles == 0) return B200_OK;
    PromptAttn p = {};
    p.q = q, p.sink = opt.sink, p.gate = gate, p.gate_ld = gate_ld, p.out = out, p.out_ld = out_ld, p.out_scale = out_scale, p.tiles = tiles, p.n_tiles = n_tiles;
    p.block_table = block_table, p.mpps = mpps, p.heads = heads, p.group = heads / kv_heads, p.kv_heads = kv_heads, p.window = window, p.chunk = opt.chunk, p.scale = scale;
    p.is_bf16 = dtype == B200_BF16, p.dist_r1 = dist_r1, p.dist_r2 = dist_r2, p.slope = opt.slope, p.pen_len = dist_r1 ? window + 64 : 0;
    const bool bf = dtype == B200_BF16;
    if (dist_r1 || opt.slope)
        return bf ? pa_launch<__nv_bfloat16, 128, 128, false, true>(p, k_pool, v_pool, true, st) : pa_launch<__half, 128, 128, false, true>(p, k_pool, v_pool, false, st);
    return bf ? pa_launch<__nv_bfloat16, 128, 128, false, false>(p, k_pool, v_pool, true, st) : pa_launch<__half, 128, 128, false, false>(p, k_pool, v_pool, false, st);
}

int launch_latent_attention_tc(int dtype, const void *ql, const void *qr, const void *pool, const float *sink, void *ol, const int *tiles, int n_tiles,
                               const int *block_table, int mpps, int t_pad, int heads, int kv_rank, int rot_dim, float scale, int window, cudaStream_t st) {
    if ((dtype != B200_BF16 && dtype != B200_F16) || rot_dim != 64 || (kv_rank != 128 && kv_rank != 192 && kv_rank != 256) || heads % 2 != 0 || !(scale > 0.0f)) return B200_ERR_UNSUPPORTED;
    if (!all_aligned16({ql, qr, pool, ol, tiles})) return B200_ERR_UNSUPPORTED;
    if (n_tiles == 0) return B200_OK;
    PromptAttn p = {};
    p.q = ql, p.qr = qr, p.sink = sink, p.out = ol, p.tiles = tiles, p.n_tiles = n_tiles, p.block_table = block_table, p.mpps = mpps;
    p.heads = heads, p.group = heads, p.kv_heads = 1, p.t_pad = t_pad, p.window = window, p.scale = scale, p.is_bf16 = dtype == B200_BF16;
    const bool bf = dtype == B200_BF16;
    switch (kv_rank) {
        case 128: return bf ? pa_launch<__nv_bfloat16, 192, 128, true, false>(p, pool, pool, true, st) : pa_launch<__half, 192, 128, true, false>(p, pool, pool, false, st);
        case 192: return bf ? pa_launch<__nv_bfloat16, 256, 192, true, false>(p, pool, pool, true, st) : pa_launch<__half, 256, 192, true, false>(p, pool, pool, false, st);
        default: return bf ? pa_launch<__nv_bfloat16, 320, 256, true, false>(p, pool, pool, true, st) : pa_launch<__half, 320, 256, true, false>(p, pool, pool, false, st);
    }
}

}  // namespace b200
