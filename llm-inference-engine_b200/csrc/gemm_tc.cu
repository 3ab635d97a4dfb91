// gemm_tc.cu -- tcgen05 / TMEM tensor-core GEMM for sm_100a: D[i,j] = sum_k A[i,k] * B[j,k], both operands K-major.
//
// Serves launchLinearGemm (reference src/kernels/linear.cu:10-87) with W packed [N,K] beyond the decode kernels' 16 tokens: A = x [M,K], B = W [N,K], C[i,j].
//
// Structure (one persistent CTA per SM, 192 threads, warp-specialised):
//   warp 0   TMA producer: cp.async.bulk.tensor 2-D tiles (128B swizzle) of A and B into a ring of smem stages, mbarrier tx counts
//   warp 1   MMA issuer: one elected lane issues tcgen05.mma.cta_group::1.kind::f16 (128 x BN x 16 per instruction, fp32
//            accumulate in TMEM), tcgen05.commit releases the smem stage / publishes the accumulator
//   warp 2-5 epilogue: tcgen05.ld the accumulator (each warp owns its 32-lane TMEM quarter), convert, store; double-buffered
//            accumulators so the epilogue of tile t overlaps the MMAs of tile t+1
// What bounds it: the operand rows that a tile loads -- L2 to shared memory at 75 bytes a nanosecond and SM -- and, with few rows, the round trip of a ring of
// stages.  So few tokens take narrow tiles (up to 128 tokens and N = 2048: 16 columns on 128 SMs), and where a narrow tile would load the tokens' rows too often or
// walk too long a k (N = 4096, K = 11008), two CTAs of a cluster share a tile's k: each leaves its sums in its shared memory and adds up its part of the columns of
// both, in rank order (deterministic; no memory traffic).  plan_tiles weighs the forms.
#include "gemm_tc.cuh"

#include <cuda.h>  // CUtensorMap
#include <algorithm>

namespace b200 {

constexpr int kBM = 128;   // UMMA M
constexpr int kBK = 64;    // K elements per stage = one 128-byte swizzle row of a 16-bit type
constexpr int kUmmaK = 16; // K per tcgen05.mma for 16-bit inputs
constexpr int kTcThreads = 192;
constexpr int kMaxStages = 24;
constexpr int kATileBytes = kBM * kBK * 2;
constexpr size_t kRingBytes = 200 * 1024;  // of stages, at most
constexpr size_t kTcExtra = 1024 /*alignment slack*/ + (2 * kMaxStages + 4) * 8 + 16;
constexpr size_t kTcSmem = kRingBytes + kATileBytes + kTcExtra;  // of a CTA, at most (a product reads 128 rows of A from a stage that may hold fewer)

struct GemmTcParams {
    void *C;
    int ldc;
    int rowsA, rowsB;
    int tilesA, tilesB, kb_total;
    int splits;    // CTAs of a cluster that share the k of one tile (then a CTA has one tile), or 1: tiles are dealt round-robin
    int bn;        // UMMA N: rows of B per tile, multiple of 16, <= 256
    int a_rows;    // rows of A that a stage loads: all 128, or fewer where A has fewer (what lies below them in a stage fills accumulator rows that nobody stores)
    int stages;
    int is_bf16;
    int acc_stride;  // TMEM columns between the two accumulators: bn, or 256 above 128 columns (power-of-two placement)
    unsigned int tmem_cols;
    // SwiGLU epilogue (gate_up linear of the prefill path, launchLinearGemm + launchSiluAndMul in one kernel): B = W [2I, K] with the gate
    // rows first; tile tb multiplies gate rows [hw tb, +hw) AND up rows [I + hw tb, +hw) as one N = 2 hw tile (two TMA boxes into one
    // B stage), the epilogue reads both halves of the accumulator and writes silu(gate) * up: C [rowsA, I], rowsB = I.  0: plain GEMM.
    int swiglu_inter;
    int swiglu_hw;  // gate (and up) columns per tile: bn = 2 * swiglu_hw (a multiple of 16 up to 128)
    // Grouped GEMM (mixture of experts): every tile of a_rows rows of A (32, 64 or 128) belongs to ONE expert, tile_expert[ta]; B = the experts' weights stacked
    // [experts * rowsB, K], so tile (ta, tb) multiplies B rows [tile_expert[ta] * rowsB + tb * bn, +bn).  Only the first *n_live row
    // tiles hold rows (a device-side count): those are dealt, and no others.  NULL: plain.
    const int *tile_expert;
    const int *n_live;
    int act;        // b200_act_t applied to the result before it is stored, -1: none (plain and grouped GEMM, not the SwiGLU epilogue)
    const float *scale;  // of every row of B (fp32, NULL: none): the sums are multiplied by it, before anything else
    int finish;     // 1: the result is rounded and takes `bias` (bias_act) before its activation (plain GEMM, A = activations)
    const float *bias;
    WaitGuard wait;
};

// A CTA's pieces of work: k-blocks [kb0, kb1) of output tiles.
struct Seg {
    int ta, tb, kb0, kb1;
};
struct SegIter {
    const GemmTcParams &p;
    int item, tilesA, tiles;
    __device__ SegIter(const GemmTcParams &pp) : p(pp), item(blockIdx.x / pp.splits), tilesA(pp.tile_expert ? *pp.n_live : pp.tilesA), tiles(tilesA * pp.tilesB) {}
    __device__ bool next(Seg &s) {
        if (item >= tiles) return false;
        const int rank = blockIdx.x % p.splits;
        s.ta = item % tilesA, s.tb = item / tilesA, s.kb0 = p.kb_total * rank / p.splits, s.kb1 = p.kb_total * (rank + 1) / p.splits;
        item += gridDim.x / p.splits;
        return true;
    }
};

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t s_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A stage's copies, two or three boxes at column c of their matrices, and what its barrier expects of them; yes == 0: nothing.
__device__ __forceinline__ void tma_stage(uint32_t yes, uint32_t bar, uint32_t bytes, int c, uint32_t da, const CUtensorMap *ma, int ra, uint32_t db, const CUtensorMap *mb, int rb) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %0, 0;\n\t@p bra DONE_%=;\n\t"
        "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n\t"
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%4], [%5, {%3, %6}], [%1];\n\t"
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%7], [%8, {%3, %9}], [%1];\n\t"
        "DONE_%=:\n\t}" ::"r"(yes), "r"(bar), "r"(bytes), "r"(c), "r"(da), "l"(ma), "r"(ra), "r"(db), "l"(mb), "r"(rb)
        : "memory");
}
__device__ __forceinline__ void tma_stage(uint32_t yes, uint32_t bar, uint32_t bytes, int c, uint32_t da, const CUtensorMap *ma, int ra, uint32_t db, const CUtensorMap *mb, int rb,
                                          uint32_t dc, int rc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %0, 0;\n\t@p bra DONE_%=;\n\t"
        "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %2;\n\t"
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%4], [%5, {%3, %6}], [%1];\n\t"
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%7], [%8, {%3, %9}], [%1];\n\t"
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%10], [%8, {%3, %11}], [%1];\n\t"
        "DONE_%=:\n\t}" ::"r"(yes), "r"(bar), "r"(bytes), "r"(c), "r"(da), "l"(ma), "r"(ra), "r"(db), "l"(mb), "r"(rb), "r"(dc), "r"(rc)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_commit_if(uint32_t yes, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %0, 0;\n\t@p bra DONE_%=;\n\t"
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t"
        "DONE_%=:\n\t}" ::"r"(yes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 lanes x 16 consecutive fp32 columns -> 16 registers per thread (thread t = lane base + t)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row atoms of 1024 bytes (SBO), descriptor version 1 (sm_100),
// layout type 2 (SWIZZLE_128B) in bits 61..63; LBO is unused for swizzled K-major layouts (canonical value 1).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// kind::f16 instruction descriptor: fp32 accumulate, A/B both K-major, no negate / sparsity / saturation.
__device__ __forceinline__ uint32_t instr_desc_f16(bool bf16, int m, int n) {
    uint32_t d = 0;
    d |= 1u << 4;                      // D format: F32
    d |= (bf16 ? 1u : 0u) << 7;        // A format
    d |= (bf16 ? 1u : 0u) << 10;       // B format
    d |= (uint32_t)(n >> 3) << 17;     // N / 8
    d |= (uint32_t)(m >> 4) << 24;     // M / 16
    return d;
}

template <typename T> __device__ __forceinline__ void store_row16(T *dst, const uint32_t (&r)[16], int valid) {
    // dst: 16 consecutive outputs of one row (32 bytes for 16-bit T); valid = number of in-range columns
    if (valid >= 16 && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
        float f[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(r[e]);
        st_v4(dst, pack16<T>(f));
        st_v4(dst + 8, pack16<T>(f + 8));
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e)
            if (e < valid) dst[e] = Elem<T>::from_f(__uint_as_float(r[e]));
    }
}

// the numbers of 16 consecutive columns, the first n0 of `cols` (past the last: the last)
__device__ __forceinline__ void columns16(const float *p, int n0, int cols, float (&b)[16]) {
    if ((reinterpret_cast<size_t>(p + n0) & 15) == 0 && n0 + 16 <= cols) {
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(p + n0 + e));
            b[e] = v.x, b[e + 1] = v.y, b[e + 2] = v.z, b[e + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) b[e] = __ldg(p + min(n0 + e, cols - 1));
    }
}
__device__ __forceinline__ void scale16(uint32_t (&r)[16], const float *scale, int n0, int cols) {
    float b[16];
    columns16(scale, n0, cols, b);
#pragma unroll
    for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * b[e]);
}

// an activation (-1: none) of 16 numbers, the choice outside of them
__device__ __forceinline__ void act16(float (&v)[16], int act) {
    if (act == B200_ACT_RELU2) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = act_apply(v[e], B200_ACT_RELU2);
    } else if (act == B200_ACT_RELU) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = act_apply(v[e], B200_ACT_RELU);
    } else if (act == B200_ACT_SILU) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = act_apply(v[e], B200_ACT_SILU);
    } else if (act >= 0) {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = act_apply(v[e], B200_ACT_GELU_TANH);
    }
}

// bias_act on 16 consecutive outputs of one row, the first of them column n0 of `cols`.  The choice of the activation stands outside the columns (inside, an
// epilogue outlasted the products it should hide behind: a layer of 3085 rows with a biased up projection of 8192 columns 638 us, now 572), the biases come in 16-byte loads where they can.
template <typename T> __device__ __forceinline__ void finish16(uint32_t (&r)[16], const float *bias, int n0, int cols, int act) {
    float v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = round_to<T>(__uint_as_float(r[e]));
    if (bias) {
        float b[16];
        columns16(bias, n0, cols, b);
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] += b[e];
    }
    act16(v, act);
#pragma unroll
    for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(v[e]);
}

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {  // the same shared-memory offset in CTA `rank` of the cluster
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Output columns [c0, c1) (steps of 16, counted from the tile's first) of row `row` of tile (ta, tb), from accumulator columns that `get` fetches.
template <typename T, typename GET> __device__ __forceinline__ void finish_tile(const GemmTcParams &p, int ta, int row, int tb, int c0, int c1, GET get) {
    T *C = reinterpret_cast<T *>(p.C);
    const int i = row < p.a_rows ? ta * p.a_rows + row : p.rowsA;  // (accumulator rows below A's: nobody's)
    if (p.swiglu_inter) {
        // gate in accumulator columns [0, hw), up in [hw, 2 hw): both rounded to T first (the reference's linear writes a T
        // tensor that launchSiluAndMul reads back, src/kernels/silu_and_mul.cu:6-41), same expression as silu_and_mul_kernel
        const int hw = p.swiglu_hw;
        for (int c = c0; c < c1; c += 16) {
            uint32_t g[16], u[16];
            get(c, g);
            get(hw + c, u);
            if (p.scale) scale16(g, p.scale, tb * hw + c, p.rowsB), scale16(u, p.scale + p.swiglu_inter, tb * hw + c, p.rowsB);
            const int valid = min(16, p.rowsB - (tb * hw + c));
            if (i < p.rowsA && valid > 0) {
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float gf = round_to<T>(__uint_as_float(g[e])), uf = round_to<T>(__uint_as_float(u[e]));
                    g[e] = __float_as_uint((gf / (1.0f + expf(-gf))) * uf);
                }
                store_row16<T>(C + (size_t)i * p.ldc + tb * hw + c, g, valid);
            }
        }
        return;
    }
    const int j0 = tb * p.bn;
    for (int c = c0; c < c1; c += 16) {
        uint32_t r[16];
        get(c, r);
        if (p.scale) scale16(r, p.scale, j0 + c, p.rowsB);
        if (p.finish) {
            finish16<T>(r, p.bias, j0 + c, p.rowsB, p.act);
        } else {
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[e]);
            act16(v, p.act);
#pragma unroll
            for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(v[e]);
        }
        const int valid = min(16, p.rowsB - (j0 + c));
        if (i < p.rowsA && valid > 0) store_row16<T>(C + (size_t)i * p.ldc + j0 + c, r, valid);
    }
}

// Rows that a product multiplies: 64 where a tile has no more.  (With 128 for everybody, tokens of a small batch kept the tensor cores at work on rows of nothing until the
// board's power limit took the clock down: a 70B-shaped layer over 21 tokens, run back to back, 342 us at 1545 MHz where 128 weights' rows by 24 tokens took 333.)
__device__ __forceinline__ int mma_rows(const GemmTcParams &p) { return p.a_rows <= kBM / 2 ? kBM / 2 : kBM; }
// the tile's row in a lane of an accumulator's quarter q: 32 of them each, or (64 rows) 16 in the lower half
__device__ __forceinline__ int acc_row(const GemmTcParams &p, int q, int lane) { return p.a_rows > kBM / 2 ? q * 32 + lane : lane < 16 ? q * 16 + lane : kBM; }

// what a wait that ran out leaves of those columns
template <typename T> __device__ __forceinline__ void lose_tile(const GemmTcParams &p, int ta, int row, int tb, int c0, int c1) {
    const int i = ta * p.a_rows + row, j0 = tb * (p.swiglu_inter ? p.swiglu_hw : p.bn);
    if (row >= p.a_rows || i >= p.rowsA) return;
    for (int c = j0 + c0; c < min(j0 + c1, p.rowsB); ++c) reinterpret_cast<T *>(p.C)[(size_t)i * p.ldc + c] = Elem<T>::from_f(__uint_as_float(0x7fc00000u));
}

template <typename T>
__global__ void __launch_bounds__(kTcThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmTcParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // carve: stages x [A tile | B tile] (1024-byte aligned), then barriers, then the TMEM base address
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int b_tile_bytes = p.bn * kBK * 2;
    const int a_tile_bytes = p.a_rows * kBK * 2, stage_bytes = a_tile_bytes + b_tile_bytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)p.stages * stage_bytes);
    const uint32_t full0 = s_u32(bars), empty0 = full0 + 8 * kMaxStages;
    const uint32_t tfull0 = empty0 + 8 * kMaxStages, tempty0 = tfull0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kMaxStages + 4);
    const uint32_t drain = tempty0 + 24;  // (behind the TMEM slot)
    __shared__ __align__(16) volatile int gave_up[8];  // the producer: {yes, -, its stage and phase then}; the issuer or the epilogue: {yes, -, -, -}

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
        for (int s = 0; s < p.stages; ++s) {
            bar_init(full0 + 8 * s, 1);
            bar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            bar_init(tfull0 + 8 * a, 1);
            bar_init(tempty0 + 8 * a, 4);  // one arrive per epilogue warp
        }
        bar_init(drain, 1);
        gave_up[0] = gave_up[4] = p.wait.clocks == 0, gave_up[2] = 0, gave_up[3] = 1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    pdl_wait();               // everything below reads (x) or overwrites (C) tensors of the previous kernel
    pdl_launch_dependents();

    // A wait that runs out: the producer copies no more, the issuer hands nothing on (so that the others' waits run out in turn), and all of the CTA's tiles are NaN in the
    // end.  The loops run on, and nothing that they need lives beyond them: an exit that hangs on a wait, or a stage counter that is read again at the end, takes
    // the uniform registers from them.  Against waits without a limit, us: 2048 x 2048 of 94 tokens 6.8 -> 7.5 (with exits from the loops 9.6 to 10.7), K = 4096, N = 4096
    // of 94 11.8 -> 12.4, K = 11008, N = 4096 of 267 36.0 -> 36.7.
    const uint32_t flag = s_u32(const_cast<const int *>(gave_up));
    if (warp == 0) {
        // ================================================= TMA producer
        if (elect_one()) {
            SegIter si(p);
            Seg sg;
            int s = 0;  // (stage and phase by counting: a remainder and a quotient per k-block were a third of what a narrow tile's block took)
            uint32_t ph = 1, left = p.wait.clocks;
            while (si.next(sg)) {
                const int ta = sg.ta, tb = sg.tb;
                const int brow = (p.tile_expert ? p.tile_expert[ta] * p.rowsB : 0) + tb * p.bn;
                for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
                    mbar_wait_near(empty0 + 8 * s, ph, left, flag, (uint32_t)s, ph);
                    const uint32_t sa = s_u32(smem + (size_t)s * stage_bytes), sb = sa + a_tile_bytes, bar = full0 + 8 * s;
                    if (p.swiglu_inter)  // box = hw rows: the gate rows, then the up rows of the same columns
                        tma_stage(left, bar, stage_bytes, kb * kBK, sa, &tmA, ta * p.a_rows, sb, &tmB, tb * p.swiglu_hw, sb + p.swiglu_hw * kBK * 2, p.swiglu_inter + tb * p.swiglu_hw);
                    else
                        tma_stage(left, bar, stage_bytes, kb * kBK, sa, &tmA, ta * p.a_rows, sb, &tmB, brow);
                    if (++s == p.stages) s = 0, ph ^= 1;
                }
            }
            if (left) gave_up[2] = s, gave_up[3] = (int)ph;
        }
    } else if (warp == 1) {
        // ================================================= MMA issuer
        const uint32_t idesc = instr_desc_f16(p.is_bf16 != 0, mma_rows(p), p.bn);
        SegIter si(p);
        Seg sg;
        int s = 0, t = 0;
        uint32_t ph = 0, left = p.wait.clocks;
        auto wait = [&](uint32_t bar, uint32_t parity) { mbar_wait_near(bar, parity, left, flag + 16, 0, 0); };
        const bool issuer = elect_one();
        for (; issuer && si.next(sg); ++t) {
            const int acc = t & 1;
            wait(tempty0 + 8 * acc, ((t >> 1) & 1) ^ 1);  // the epilogue has drained this accumulator
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(acc * p.acc_stride);
            for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
                wait(full0 + 8 * s, ph);
                tc_fence_after();
                {
                    const uint32_t sa = s_u32(smem + (size_t)s * stage_bytes);
                    const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + a_tile_bytes);
#pragma unroll
                    for (int k = 0; k < kBK / kUmmaK; ++k) {
                        // advancing K inside the 128-byte swizzle row: +32 bytes = +2 in the (>>4) start-address field
                        tc_mma_f16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > sg.kb0 || k > 0) ? 1u : 0u);
                    }
                    tc_commit_if(left, empty0 + 8 * s);                          // smem stage reusable once these MMAs have read it
                    if (kb == sg.kb1 - 1) tc_commit_if(left, tfull0 + 8 * acc);  // accumulator complete
                }
                if (++s == p.stages) s = 0, ph ^= 1;
            }
        }
    } else {
        // ================================================= epilogue (warps 2..5 -> TMEM lane quarters 2,3,0,1)
        const int q = warp & 3;
        SegIter si(p);
        Seg sg;
        int t = 0;
        uint32_t left = p.wait.clocks;
        for (; si.next(sg); ++t) {
            const int acc = t & 1;
            mbar_wait_near(tfull0 + 8 * acc, (t >> 1) & 1, left, flag + 16, 0, 0);
            __syncwarp();
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * p.acc_stride);
            auto fetch = [&](int c, uint32_t (&r)[16]) {
                tc_ld16(taddr + c, r);
                tc_wait_ld();
            };
            if (p.splits > 1) {  // this CTA's part of the sums, [column][row], where its stages were
                float *mine = reinterpret_cast<float *>(smem) + q * 32 + lane;
                for (int c = 0; c < p.bn; c += 16) {
                    uint32_t r[16];
                    fetch(c, r);
#pragma unroll
                    for (int e = 0; e < 16; ++e) mine[(size_t)(c + e) * kBM] = __uint_as_float(r[e]);
                }
            } else {
                finish_tile<T>(p, sg.ta, acc_row(p, q, lane), sg.tb, 0, p.swiglu_inter ? p.swiglu_hw : p.bn, fetch);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(tempty0 + 8 * acc);
        }
    }
    int lost = 0;
    if (p.splits > 1) {
        // every CTA of the cluster adds up its part of the tile's columns, and stays until the others have read what it holds
        __syncthreads();
        cluster_sync_all();
        const int tile = blockIdx.x / p.splits, rank = blockIdx.x % p.splits;
        for (int x = 0; x < p.splits; ++x) {
            int a, b;
            asm volatile("ld.shared::cluster.s32 %0, [%2];\n\tld.shared::cluster.s32 %1, [%2 + 16];" : "=r"(a), "=r"(b) : "r"(in_cta(flag, (uint32_t)x)) : "memory");
            lost |= a | b;
        }
        if (warp >= 2) {
            const int q = warp & 3, cols = (p.swiglu_inter ? p.swiglu_hw : p.bn) / p.splits;
            const uint32_t at = s_u32(smem) + (uint32_t)(q * 32 + lane) * 4;
            finish_tile<T>(p, tile % p.tilesA, acc_row(p, q, lane), tile / p.tilesA, rank * cols, (rank + 1) * cols, [&](int c, uint32_t (&r)[16]) {
                float v[16];
                for (int x = 0; x < p.splits; ++x) {
                    const uint32_t from = in_cta(at + (uint32_t)c * kBM * 4, (uint32_t)x);
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        float f;
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(from + (uint32_t)e * kBM * 4) : "memory");
                        v[e] = x == 0 ? f : v[e] + f;
                    }
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(v[e]);
            });
        }
        cluster_sync_all();
    }

    tc_fence_before();
    __syncthreads();
    if (lost | gave_up[0] | gave_up[4]) {  // the CTA stays until its copies have landed and its products have read them, and its tiles are NaN
        uint32_t left = kWaitClocks;
        if (warp == 0 && elect_one()) {  // (stages before the producer's last one in its round, the others in the round before)
            for (int i = 0; i < p.stages; ++i) mbar_wait_near(full0 + 8 * i, (uint32_t)(i < gave_up[2] ? gave_up[3] ^ 1 : gave_up[3]), left, flag + 16, 0, 0);
            if (p.wait.word) {
                *reinterpret_cast<volatile unsigned int *>(p.wait.word) = kWaitGemm;
                __threadfence_system();
            }
        } else if (warp == 1 && elect_one()) {  // (the same thread as above)
            tc_commit(drain);
            mbar_wait_near(drain, 0, left, flag + 16, 0, 0);
        } else if (warp >= 2) {
            const int cols = (p.swiglu_inter ? p.swiglu_hw : p.bn) / p.splits, c0 = blockIdx.x % p.splits * cols;
            SegIter si(p);
            Seg sg;
            while (si.next(sg)) lose_tile<T>(p, sg.ta, acc_row(p, warp & 3, lane), sg.tb, c0, c0 + cols);
        }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------ CTA pairs (prefill shapes)
// The same product with TWO SMs on one 256-row tile (tcgen05.mma.cta_group::2): each CTA of a cluster of two stages its own 128 rows of A and HALF
// of the tile's B rows, and one instruction of the leader reads both halves -- per flop half the shared-memory writes and reads of B.  That traffic,
// not the tensor pipe, is what the one-CTA form pays for (power as well as time: these launches run under the board's power cap).
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer (leader only), warps 2..9 epilogue of the CTA's own 128 rows (two warps per TMEM lane quarter,
// one per half of the columns: a launch ends on an epilogue that nothing overlaps).  Every byte that either CTA loads is counted on the leader's
// `full` barrier; `empty` and `tfull` are arrived at in both CTAs by multicast commits; both CTAs' epilogues release the leader's `tempty`.
// Columns: the first n_wide column tiles are p.bn wide, the rest bn2: the last wave is cut so that it fills the pairs (choose_widths).
// Measured: see pair_takes.
struct GemmPairParams {
    void *C;
    int ldc, rowsA, rowsB, kb_total, tilesA, tilesB;
    int bn, bn2, n_wide;
    int stages, is_bf16;
    int swiglu_inter;  // as above: gate rows come from the leader's half of B, up rows from its peer's; tile widths count both
    const float *scale;  // of every row of B, as above
    int finish, act;   // finish: bias_act on the result, as above
    const float *bias;
    WaitGuard wait;
};
constexpr int kPairThreads = 320;
constexpr int kPairStageBytes = 2 * kATileBytes;  // 128 rows of A, up to 128 rows of B

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(c0), "r"(c1), "r"(leader_bar)
                 : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_commit_leader(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <typename T>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmB2, const GemmPairParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)p.stages * kPairStageBytes);
    const uint32_t full0 = s_u32(bars), empty0 = full0 + 8 * kMaxStages, tfull0 = empty0 + 8 * kMaxStages, tempty0 = tfull0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kMaxStages + 4);
    const uint32_t drain = tempty0 + 24;  // (behind the TMEM slot)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
        for (int s = 0; s < p.stages; ++s) {
            bar_init(full0 + 8 * s, 1);
            bar_init(empty0 + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            bar_init(tfull0 + 8 * a, 1);
            bar_init(tempty0 + 8 * a, 16);  // eight epilogue warps of either CTA
        }
        bar_init(drain, 1);
        cta_gave_up() = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers are initialised and its TMEM is allocated
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    pdl_wait();
    pdl_launch_dependents();

    const int tilesA = p.tilesA, tiles = tilesA * p.tilesB;
    // a wait that runs out: no more copies, no more products, NaN for the tiles that are left, and the other CTA's waits on them run out in turn
    auto wait = [&](uint32_t bar, uint32_t parity) { return mbar_wait_guarded(bar, parity, p.wait, kWaitGemmPair); };
    auto width_of = [&](int tb) { return tb < p.n_wide ? p.bn : p.bn2; };
    auto col_of = [&](int tb) {  // first output column (SwiGLU: half of a tile's width are output columns)
        const int c = tb < p.n_wide ? tb * p.bn : p.n_wide * p.bn + (tb - p.n_wide) * p.bn2;
        return p.swiglu_inter ? c >> 1 : c;
    };

    if (warp == 0) {
        // ================================================= TMA producer: this CTA's rows of A, its half of the B rows
        if (elect_one()) {
            int it = 0, s = 0;
            uint32_t ph = 1;
            bool live = true;
            for (int item = pair; live && item < tiles; item += pairs) {
                const int ta = item % tilesA, tb = item / tilesA, w = width_of(tb);
                const int arow = ta * 2 * kBM + (int)rank * kBM;
                const int brow = p.swiglu_inter ? (rank ? p.swiglu_inter : 0) + col_of(tb) : col_of(tb) + (int)rank * (w >> 1);
                const CUtensorMap *mb = tb < p.n_wide ? &tmB : &tmB2;
                for (int kb = 0; kb < p.kb_total; ++kb, ++it) {
                    live = wait(empty0 + 8 * s, ph);
                    if (!live) break;
                    const uint32_t sa = s_u32(smem + (size_t)s * kPairStageBytes), bar = in_cta(full0 + 8 * s, 0);
                    if (rank == 0) bar_expect_tx(full0 + 8 * s, (uint32_t)(2 * (kATileBytes + (w >> 1) * kBK * 2)));
                    tma_load_2d_pair(sa, &tmA, kb * kBK, arow, bar);
                    tma_load_2d_pair(sa + kATileBytes, mb, kb * kBK, brow, bar);
                    if (++s == p.stages) s = 0, ph ^= 1;
                }
            }
            // The leader's last commits arrive at `empty` of both CTAs and nobody refills those stages: each CTA waits for its own here, since the
            // closing cluster barrier does not order them and a late one would land in the shared memory of whatever runs on this SM next
            for (int i = max(0, it - p.stages); live && i < it; ++i) live = wait(empty0 + 8 * (i % p.stages), (i / p.stages) & 1);
            // (given up: both CTAs' copies are counted here, and the peer stays until the leader has seen them land)
            for (int i = max(0, it - p.stages); !live && rank == 0 && i < it; ++i)
                if (!mbar_drain(full0 + 8 * (i % p.stages), (i / p.stages) & 1)) break;
        }
    } else if (warp == 1) {
        // ================================================= MMA issuer: the leader, for both
        if (rank == 0 && elect_one()) {
            int s = 0, t = 0;
            uint32_t ph = 0;
            bool live = true;
            for (int item = pair; live && item < tiles; item += pairs, ++t) {
                const uint32_t idesc = instr_desc_f16(p.is_bf16 != 0, 2 * kBM, width_of(item / tilesA));
                const int acc = t & 1;
                live = wait(tempty0 + 8 * acc, ((t >> 1) & 1) ^ 1);
                if (!live) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * 256);
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    live = wait(full0 + 8 * s, ph);
                    if (!live) break;
                    tc_fence_after();
                    const uint32_t sa = s_u32(smem + (size_t)s * kPairStageBytes);
                    const uint64_t da = smem_desc_sw128(sa), db = smem_desc_sw128(sa + kATileBytes);
#pragma unroll
                    for (int k = 0; k < kBK / kUmmaK; ++k) tc_mma_f16_pair(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit_pair(empty0 + 8 * s);
                    if (kb == p.kb_total - 1) tc_commit_pair(tfull0 + 8 * acc);
                    if (++s == p.stages) s = 0, ph ^= 1;
                }
            }
            tc_commit_leader(drain);  // no product reads either CTA's shared memory when the pair leaves
            mbar_drain(drain, 0);
        }
    } else {
        // ================================================= epilogue: TMEM lane quarter q, one half of the columns
        const int q = warp & 3, half = (warp - 2) >> 2;
        T *C = reinterpret_cast<T *>(p.C);
        int t = 0;
        bool live = true;
        for (int item = pair; item < tiles; item += pairs, ++t) {
            const int ta = item % tilesA, tb = item / tilesA, w = width_of(tb), acc = t & 1, col0 = col_of(tb);
            live = live && __all_sync(0xffffffffu, wait(tfull0 + 8 * acc, (t >> 1) & 1));
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 256);
            const int i = ta * 2 * kBM + (int)rank * kBM + q * 32 + lane;
            const int out_w = p.swiglu_inter ? w >> 1 : w;               // output columns of the tile, a multiple of 16
            const int mid = (out_w >> 5) << 4;                            // this warp's share: [0, mid) or [mid, out_w), in steps of 16
            for (int c = half ? mid : 0; c < (half ? out_w : mid); c += 16) {
                uint32_t g[16];
                tc_ld16(taddr + c, g);
                const int valid = min(16, p.rowsB - (col0 + c));
                if (p.swiglu_inter) {
                    uint32_t u[16];
                    tc_ld16(taddr + out_w + c, u);
                    tc_wait_ld();
                    if (p.scale) scale16(g, p.scale, col0 + c, p.rowsB), scale16(u, p.scale + p.swiglu_inter, col0 + c, p.rowsB);
#pragma unroll
                    for (int e = 0; e < 16; ++e) {  // (the same expression and roundings as the one-CTA epilogue)
                        const float gf = round_to<T>(__uint_as_float(g[e])), uf = round_to<T>(__uint_as_float(u[e]));
                        g[e] = __float_as_uint((gf / (1.0f + expf(-gf))) * uf);
                    }
                } else {
                    tc_wait_ld();
                    if (p.scale) scale16(g, p.scale, col0 + c, p.rowsB);
                    if (p.finish) finish16<T>(g, p.bias, col0 + c, p.rowsB, p.act);
                }
                if (!live) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) g[e] = 0x7fc00000u;
                }
                if (i < p.rowsA && valid > 0) store_row16<T>(C + (size_t)i * p.ldc + col0 + c, g, valid);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta(tempty0 + 8 * acc, 0)) : "memory");
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other may still read its shared memory or arrive at its barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// ------------------------------------------------------------------ host side
static unsigned int pow2_cols(int c) {
    unsigned int v = 32;
    while ((int)v < c) v <<= 1;
    return v;
}

// Column tiles of a pair launch: n_wide tiles of bn columns, the rest bn2 wide.  Tiles are dealt to the pairs in order, wide ones first, so pair 0 has
// the most work; its load (columns, and what a tile costs beside its columns) is what a choice is judged by.  Widths are steps of 32 MMA columns.
struct PairWidths { int bn, bn2, n_wide, n_tiles; long long cost; };
static PairWidths choose_widths(int tiles_a, int cols, int pairs) {  // cols: MMA columns (SwiGLU: gate and up together)
    constexpr int kTileCost = 24;
    auto load = [&](int n1, int w1, int n2, int w2) {
        const long long wide = (long long)tiles_a * n1, all = wide + (long long)tiles_a * n2;
        const long long c1 = (wide + pairs - 1) / pairs, c = (all + pairs - 1) / pairs;
        return c1 * (w1 + kTileCost) + (c - c1) * (w2 + kTileCost);
    };
    const int most = (cols + 255) / 256, back = std::max(1, (2 * pairs + tiles_a - 1) / tiles_a);
    PairWidths best = {256, 256, most, most, load(most, 256, 0, 0)};
    for (int n1 = std::max(0, most - 1 - back); n1 < most; ++n1)
        for (int w2 = 224; w2 >= 64; w2 -= 32) {
            const int n2 = (cols - n1 * 256 + w2 - 1) / w2;
            const long long c = load(n1, 256, n2, w2);
            if (c < best.cost) best = {256, w2, n1, n1 + n2, c};
        }
    return best;
}

// Tiles of the one-CTA form: the width and the number of CTAs per tile whose estimate is smallest, in nanoseconds.  A k-block costs its operand rows, but never less
// than the issue of its copies and products (130); a wave ends on an epilogue; the weights come from memory at 6500 bytes a nanosecond.  Two CTAs on one tile's k pay
// an exchange of 4.5 us: K = 11008, N = 4096 of 17 / 128 tokens 64 columns on two CTAs 20.5 / 23.1 us, 32 columns on one 24.1 / 26.0 (four CTAs: 22.0 / 23.6, and
// behind two everywhere else).  Swept on a B200 (us, widths 16 to 256): K = 4096, N = 4096 of 128 tokens 32 columns 12.3, 64 14.0, 128 17.8; K = 2048, N = 6208 of 94:
// 48 8.4, 128 10.7; K = 8192, N = 10240 of 400: 144 (two waves) 80, 192 89, 256 112; K = N = 8192 of 1084: 256 115, 192 131.
// Against what was here (128 x 128 and wider tiles; up to 128 tokens the weights' rows as the tile's 128, their sums shared out through memory), us: 17 / 64 / 128 /
// 267 / 600 tokens: K = 2048, N = 2048 12.1 / 17.6 / 28.4 / 13.0 / 14.4, K = 4096, N = 12288 25.8 / 31.4 / 40.4 / 35.4 / 57.1, K = 11008, N = 4096
// 22.9 / 27.6 / 36.4 / 54.9 / 62.3.
struct TilePlan {
    int bn, splits;
    double ns;
};
// tiles_a row tiles that load `rows` rows each; only: this many CTAs per tile (0: any)
static TilePlan plan_tiles(int tiles_a, int rows, int cols, int K, int sms, int step, int only = 0) {
    const int kb = (K + kBK - 1) / kBK, widest = std::min(256, (cols + step - 1) / step * step);
    TilePlan best = {widest, 1, 1e30};
    for (int splits : {1, 2}) {
        if (only && splits != only) continue;
        for (int bn = widest; bn >= step * splits; bn -= step) {
            if (bn % (step * splits)) continue;
            const long long tiles = (long long)tiles_a * ((cols + bn - 1) / bn);
            if (splits > 1 && (tiles * splits > sms || kb < 4 * splits)) break;  // (narrower: more of them)
            const int stages = std::min(kMaxStages, (int)(kRingBytes / ((rows + bn) * kBK * 2)));
            if (splits > 1 && stages * (rows + bn) * kBK * 2 < 4 * bn * kBM) continue;  // (the exchange lies where the stages were)
            const long long waves = (tiles * splits + sms - 1) / sms;
            double ns = waves * ((kb + splits - 1) / splits * std::max(130.0, 1.1 * (rows + bn)) + 600) + (splits > 1 ? 4500 : 0);
            ns = std::max(ns, cols * (double)K * 2 / 6500) + 0.05 * ns;
            if (ns < best.ns) best = {bn, splits, ns};
        }
    }
    return best;
}

// CTA pairs where their estimate (1.5 ns per column and k-block of the busiest pair) is smaller: large launches whose row tiles of 256 are nearly full.  A pair loads
// half of a tile's B rows per CTA, which counts where all SMs load all the time (7B at 2048 tokens, all eight linears: 1235 us on one-CTA tiles, 1158 on pairs);
// few waves of narrow tiles waste less (K = 2048, N = 6208 of 267 tokens: 15.1 on pairs, 12.2 here).
static bool pair_takes(int M, int cols, int K, int sms, const TilePlan &one) {
    const int t256 = (M + 2 * kBM - 1) / (2 * kBM), pairs = sms / 2;
    if (M <= kBM || cols < 256 || t256 * ((cols + 255) / 256) * 2 < pairs) return false;
    return choose_widths(t256, cols, pairs).cost * ((K + kBK - 1) / kBK) * 1.5 + 600 < one.ns;
}

// the launch itself: `rows` rows of A, `cols` of B
static int launch_pair(GemmPairParams &p, const void *x, const void *w, int rows, int cols, int K, cudaStream_t st) {
    const bool bf16 = p.is_bf16;
    const size_t smem = (size_t)p.stages * kPairStageBytes + kTcExtra + 16;
    CUtensorMap tmA, tmB, tmB2;
    if (!tile_map(&tmA, x, rows, K, kBM, bf16) || !tile_map(&tmB, w, cols, K, p.bn / 2, bf16) || !tile_map(&tmB2, w, cols, K, p.bn2 / 2, bf16)) {
        set_error("gemm_tc pair: cuTensorMapEncodeTiled failed (rows %d/%d, K %d)", rows, cols, K);
        return B200_ERR_CUDA;
    }
    const int grid = 2 * std::min(p.tilesA * p.tilesB, sm_count() / 2);
    auto launch = [&](auto kern) {
        allow_smem(reinterpret_cast<const void *>(kern), smem);
        launch_pdl_cluster(kern, dim3(grid), dim3(kPairThreads), smem, st, true, 2u, tmA, tmB, tmB2, p);
    };
    if (bf16) launch(gemm_tc_pair_kernel<__nv_bfloat16>);
    else launch(gemm_tc_pair_kernel<__half>);
    return cuda_status("gemm_tc pair launch");
}

struct Finish {
    int on, act;
    const float *bias, *scale;
};
static int launch_gemm_pair(const void *x, const void *w, void *y, int M, int N, int K, int dtype, int swiglu_inter, const Finish &fin, cudaStream_t st) {
    const bool bf16 = dtype == B200_BF16;
    const int cols = swiglu_inter ? 2 * swiglu_inter : N, sms = sm_count(), pairs = sms / 2;
    GemmPairParams p = {};
    p.C = y, p.ldc = swiglu_inter ? swiglu_inter : N, p.rowsA = M, p.rowsB = p.ldc;
    p.kb_total = (K + kBK - 1) / kBK, p.is_bf16 = bf16 ? 1 : 0, p.swiglu_inter = swiglu_inter;
    p.tilesA = (M + 2 * kBM - 1) / (2 * kBM);
    const PairWidths pw = choose_widths(p.tilesA, cols, pairs);
    p.bn = pw.bn, p.bn2 = pw.bn2, p.n_wide = pw.n_wide, p.tilesB = pw.n_tiles;
    p.finish = fin.on, p.act = fin.act, p.bias = fin.bias, p.scale = fin.scale;
    p.stages = 6, p.wait = wait_guard();
    return launch_pair(p, x, w, M, cols, K, st);
}

static int launch_gemm_tc_impl(const void *x, const void *w, void *y, int M, int N, int K, int dtype, int swiglu_inter, const Finish &fin, cudaStream_t st) {
    if (dtype != B200_BF16 && dtype != B200_F16) return B200_ERR_UNSUPPORTED;
    if (M < 1 || K % 8 != 0 || K < kBK || !aligned16(x) || !aligned16(w) || !y) return B200_ERR_UNSUPPORTED;
    const bool bf16 = dtype == B200_BF16;
    if (swiglu_inter && swiglu_inter < 128) return B200_ERR_UNSUPPORTED;
    const int sms = sm_count(), cols = swiglu_inter ? 2 * swiglu_inter : N;
    const int a_rows = std::min(kBM, (M + 7) / 8 * 8), tiles_a = (M + kBM - 1) / kBM;
    TilePlan plan = plan_tiles(tiles_a, a_rows, cols, K, sms, 16);
    // Whether two CTAs add up a tile's k is the plain linear's choice for SwiGLU too (the same bits); its widths, and pairs in place of whole tiles, are its own.
    const bool split = plan.splits > 1 && !pair_takes(M, cols, K, sms, plan);
    if (swiglu_inter) plan = plan_tiles(tiles_a, a_rows, cols, K, sms, 32, split ? plan.splits : 1);
    if (!split && pair_takes(M, cols, K, sms, plan)) return launch_gemm_pair(x, w, y, M, N, K, dtype, swiglu_inter, fin, st);
    GemmTcParams p = {};
    p.C = y, p.is_bf16 = bf16 ? 1 : 0;
    p.swiglu_inter = swiglu_inter;
    p.finish = fin.on, p.act = fin.on ? fin.act : -1, p.bias = fin.bias, p.scale = fin.scale;
    p.wait = wait_guard();
    p.kb_total = (K + kBK - 1) / kBK;
    p.rowsA = M, p.rowsB = p.ldc = swiglu_inter ? swiglu_inter : N;  // (SwiGLU: I output columns; the MMA tile is hw gate + hw up rows)
    p.bn = plan.bn, p.splits = plan.splits, p.swiglu_hw = swiglu_inter ? plan.bn / 2 : 0;
    p.a_rows = a_rows;
    p.tilesA = tiles_a, p.tilesB = (cols + p.bn - 1) / p.bn;
    const int tiles = p.tilesA * p.tilesB, grid = p.splits > 1 ? tiles * p.splits : std::min(tiles, sms);
    p.acc_stride = p.bn > 128 ? 256 : p.bn;
    p.tmem_cols = pow2_cols(p.acc_stride + p.bn);
    const int stage_bytes = (p.a_rows + p.bn) * kBK * 2;
    p.stages = std::min(kMaxStages, (int)(kRingBytes / stage_bytes));
    const size_t smem = (size_t)p.stages * stage_bytes + (kATileBytes - p.a_rows * kBK * 2) + kTcExtra;

    CUtensorMap tmA, tmB;
    if (!tile_map(&tmA, x, M, K, p.a_rows, bf16) || !tile_map(&tmB, w, cols, K, swiglu_inter ? p.swiglu_hw : p.bn, bf16)) {
        set_error("gemm_tc: cuTensorMapEncodeTiled failed (rows %d/%d, K %d)", M, cols, K);
        return B200_ERR_CUDA;
    }
    auto launch = [&](auto kern) {
        allow_smem(reinterpret_cast<const void *>(kern), kTcSmem);
        launch_pdl_cluster(kern, dim3(grid), dim3(kTcThreads), smem, st, true, (unsigned)p.splits, tmA, tmB, p);
    };
    if (bf16) launch(gemm_tc_kernel<__nv_bfloat16>);
    else launch(gemm_tc_kernel<__half>);
    return cuda_status("gemm_tc launch");
}

int launch_gemm_tc(const void *x, const void *w, void *y, int M, int N, int K, int dtype, cudaStream_t st, const float *row_scale) {
    return launch_gemm_tc_impl(x, w, y, M, N, K, dtype, 0, Finish{0, -1, nullptr, row_scale}, st);
}

int launch_gemm_tc_act(const void *x, const void *w, void *y, int M, int N, int K, const float *bias, int act, int dtype, cudaStream_t st) {
    return launch_gemm_tc_impl(x, w, y, M, N, K, dtype, 0, Finish{1, act, bias, nullptr}, st);
}

// act[M, inter] = silu(x . Wgate^T) * (x . Wup^T), w = [2 * inter, K] (gate rows, then up rows): the gate_up linear and launchSiluAndMul in one
// kernel; the [M, 2 * inter] intermediate is never written.  B200_ERR_UNSUPPORTED: use the two launchers.
int launch_gemm_tc_swiglu(const void *x, const void *w, void *act, int M, int inter, int K, int dtype, cudaStream_t st, const float *row_scale) {
    return launch_gemm_tc_impl(x, w, act, M, inter, K, dtype, inter, Finish{0, -1, nullptr, row_scale}, st);
}

// c[row, :] = act?(a[row, :] . W_e^T) with e = tile_expert[row / tile]: the experts' up or down projection as ONE launch.  a [max_rows, K]
// (rows grouped by expert, every expert padded to whole tiles of `tile` rows: 32, 64 or 128), w [experts * N, K], c [max_rows, N]; *n_live row
// tiles are live, of which the launch expects the even share (every expert pads half a tile).  (Tiles of 256 rows on CTA pairs: 64 us where
// 128 take 48, 16384 rows of 32 experts, 2048 x 512.)
int launch_gemm_tc_grouped(const void *a, const void *w, void *c, int max_rows, int N, int K, int experts, const int *tile_expert,
                           const int *n_live, int act, int dtype, cudaStream_t st, int tile) {
    if (dtype != B200_BF16 && dtype != B200_F16) return B200_ERR_UNSUPPORTED;
    if (max_rows < tile || max_rows % tile != 0 || K % 8 != 0 || K < kBK || N < 16 || !aligned16(a) || !aligned16(w) || !c) return B200_ERR_UNSUPPORTED;
    const bool bf16 = dtype == B200_BF16;
    const int sms = sm_count(), most = max_rows / tile, likely = std::max(1, most - experts / 2);
    GemmTcParams p = {};
    p.C = c, p.ldc = N, p.splits = 1, p.is_bf16 = bf16 ? 1 : 0;
    p.act = act, p.tile_expert = tile_expert, p.n_live = n_live, p.wait = wait_guard();
    p.kb_total = (K + kBK - 1) / kBK;
    p.rowsA = max_rows, p.rowsB = N;
    p.a_rows = tile, p.tilesA = most;
    p.bn = plan_tiles(likely, tile, N, K, sms, 16, 1).bn;
    p.tilesB = (N + p.bn - 1) / p.bn;
    const int grid = std::min(most * p.tilesB, sms);
    p.acc_stride = p.bn > 128 ? 256 : p.bn;
    p.tmem_cols = pow2_cols(p.acc_stride + p.bn);
    const int stage_bytes = (p.a_rows + p.bn) * kBK * 2;
    p.stages = std::min(kMaxStages, (int)(kRingBytes / stage_bytes));
    const size_t smem = (size_t)p.stages * stage_bytes + (kATileBytes - p.a_rows * kBK * 2) + kTcExtra;
    CUtensorMap tmA, tmB;
    if (!tile_map(&tmA, a, max_rows, K, p.a_rows, bf16) || !tile_map(&tmB, w, experts * N, K, p.bn, bf16)) {
        set_error("gemm_tc grouped: cuTensorMapEncodeTiled failed (rows %d, experts %d x %d, K %d)", max_rows, experts, N, K);
        return B200_ERR_CUDA;
    }
    auto launch = [&](auto kern) {
        allow_smem(reinterpret_cast<const void *>(kern), kTcSmem);
        launch_pdl(kern, dim3(grid), dim3(kTcThreads), smem, st, true, tmA, tmB, p);
    };
    if (bf16) launch(gemm_tc_kernel<__nv_bfloat16>);
    else launch(gemm_tc_kernel<__half>);
    return cuda_status("gemm_tc grouped launch");
}

}  // namespace b200
