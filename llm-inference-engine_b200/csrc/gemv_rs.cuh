// gemv_rs.cuh -- the decode-shaped linear for 1..16 tokens with the ACTIVATIONS STATIONARY IN REGISTERS: y[M,N] = x[M,K] * W^T, W packed [N,K], dense
// 16-bit, FP8-e4m3 (W8A16) or INT4-g128 (W4A16).  Reference: launchLinearGemm (src/kernels/linear.cu:10-87) at the decode shapes of
// src/layers/self_attention.cpp:79-86,131-138 and src/layers/ffn.cpp:105-139.
//
// Bound: HBM -- every weight byte once per call -- if nothing on the SM is slower.  gemv_mma.cuh keeps the activations in shared memory and reads them
// again for every 8 or 16 weight rows: at 16 tokens three times the shared-memory traffic of FP8 weights and six times that of INT4, behind a staging
// pass that every launch waits for.  Here a compute warp owns ONE slice of k for the whole launch and holds all tokens' activations of it as
// mma.sync A fragments (4 or 8 registers per block of 32 k), so the stream of weights is all that shared memory carries:
//   * one persistent CTA per SM: 16 compute warps (the k split), a TMA-producer warp, a reducer warp; a unit of work is 8 (dense) or 16 weight rows, a
//     ring stage is a whole unit (one bulk copy per row), so a launch has one hand-off per unit and no tail longer than one;
//   * the ring is filled before griddepcontrol.wait; the fragments come straight from global memory (L2) in 16-byte pieces, all in flight at once:
//     k is permuted inside each 32-k block (quantised: 128-k group) alike for A and B, so a lane's 8 consecutive k are its fragments of two k-steps;
//   * rows longer than the slices reach (K > 4096) go in parts, the reducer adding the parts' tiles in shared memory.
// The reducer adds the 16 warps' tiles in a fixed order (deterministic), applies the FP8 row scale / SwiGLU and stores, or pushes the tensor-parallel
// partial, as in gemv_mma.cuh.
// Measured, 4 layers of 7B size, us per decode step (the kernels before -> now): dense 2 tokens 430 -> 370, 8: 435 -> 375, 16 ragged 517 -> 447;
// FP8 2: 328 -> 263, 4: 382 -> 261, 8: 388 -> 280, 16 ragged 520 -> 382; INT4 2: 383 -> 273, 4: 433 -> 276, 8: 573 -> 296, 16: 617 -> 451.  The gate / up
// linear of 16 FP8 tokens (90 MB): 41 -> 25 us.  FP8, a lane's k as two sixteens 64 apart (before -> now, us per launch, 1 / 8 / 16
// tokens): K = 4096, N = 4096 4.9 / 6.0 / 8.5 -> 4.8 / 5.4 / 7.3, N = 12288 9.7 / 11.1 / 14.4 -> 9.5 / 10.5 / 13.4, K = 11008, N = 4096 9.7 / 11.5 / 19.7 -> 9.5 / 10.5 / 17.2,
// K = 8192, N = 7168 11.3 / 13.1 / 19.6 -> 11.3 / 12.0 / 17.3; the steps above, 16 ragged FP8 382 -> 351.  (As consecutive eights, in 8-byte reads of the weights: 1 token 1 to 3 %
// slower than before, 16 tokens 7.8 / 13.8 / 18.3 / 18.5.)  A norm on the fragments in front of the product was slower than a norm kernel: every CTA redid all rows
// (16 dense tokens 490 against 449).
#pragma once
#include "gemv_mma.cuh"

namespace b200 {

constexpr int kRsMaxStages = 12;
constexpr size_t kRsSmem = 226 * 1024;  // dynamic shared memory of a CTA, at most
constexpr int kRsBlocks = 8;            // 32-k blocks of a part that a warp holds (4 registers each at up to 8 tokens, 8 above)
// Dense weights: a unit is 8 rows, the activations are the MMA's A operand (16 tokens), the weights its B.  Quantised weights: a unit is 16 rows and the
// weights are A -- up to 8 tokens fill B, more take a second one, the dequantised rows serve both -- so that what a unit costs beside its weights
// (waits, hand-off, addresses: two thirds of the instructions of an INT4 unit of 8 rows) is paid half as often.
__host__ __device__ constexpr int rs_rows(bool dense) { return dense ? kMmaRows : 16; }
// fp32 values of one warp's tile: [16 tokens][8 rows]; quantised [8 NT tokens][16 rows + 4]: the lanes' stores fall on different banks
__host__ __device__ constexpr int rs_tile(bool dense, int nt) { return dense ? 16 * kMmaRows : 8 * nt * 20; }

struct RsGeom {
    int part_k, parts;  // k per part (a multiple of 128)
    int row_stride;     // bytes between the rows of a stage
    int stage_bytes, stages;
    int max_units;      // units of the busiest CTA
    WaitGuard wait;
};

// 8 activations of T in k order -> the A fragments' halves: dense as they are; quantised formats in f16, INT4 with the pairs its dequantisation makes
template <typename T, int FMT> __device__ __forceinline__ uint4 rs_fragment(const uint4 raw) {
    if constexpr (FMT == WF_DENSE) {
        return raw;
    } else {
        float q[8], o[8];
        unpack16<T>(raw, q);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[FMT == WF_INT4 ? ((j & 3) * 2 + (j >> 2)) : j] = q[j];
        return pack16<__half>(o);
    }
}

// NT 1: M <= 8, 2: M <= 16
template <typename T, int FMT, bool kSwiGLU, int NT>
__global__ void __launch_bounds__(kMmaThreads, 1)
gemv_rs_kernel(const GemvArgs a, const RsGeom geo) {
    constexpr int NB = kRsBlocks;
    static_assert(NB % 4 == 0, "four blocks are one quantisation group");
    constexpr bool kDense = FMT == WF_DENSE;
    constexpr int R = rs_rows(kDense), TILE = rs_tile(kDense, NT), VALS = kDense ? 128 : 128 * NT;
    extern __shared__ __align__(128) unsigned char smem[];

    const int K = a.K, N = a.N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    auto bytes_of = [&](int k) -> size_t { return kDense ? (size_t)k * 2 : (FMT == WF_FP8 ? (size_t)k : (size_t)k / 2); };
    const size_t row_bytes = bytes_of(K);
    const int units = kSwiGLU ? (a.inter + R / 2 - 1) / (R / 2) : (N + R - 1) / R;
    const int stages = geo.stages, parts = geo.parts;
    const int gid = blockIdx.x, total = gridDim.x;
    const int my_units = gid < units ? (units - gid + total - 1) / total : 0;
    const int my_items = my_units * parts;

    unsigned char *ring = smem;
    size_t off = (size_t)stages * geo.stage_bytes;
    const uint32_t full0 = smem_u32(smem + off), empty0 = full0 + kRsMaxStages * 8, ready0 = empty0 + kRsMaxStages * 8, free0 = ready0 + 16;
    off += (size_t)(2 * kRsMaxStages + 4) * 8;
    float *tiles = reinterpret_cast<float *>(smem + off);  // [parity][warp][TILE]
    off += (size_t)2 * kMmaWarps * TILE * sizeof(float);
    float *outacc = reinterpret_cast<float *>(smem + off);  // [unit][VALS], parts > 1 only
    const uint32_t ring_u32 = smem_u32(ring);

    // Whatever stops in the CTA, the reducer's wait for the next tile runs out, and that ends all other waits: the compute warps run through what they have
    // (their barriers count on it), the producer stops, and what the reducer stores from then on is NaN.  Only the reducer keeps the time: the limit inside
    // every wait made the loops' code larger and a decode step 1 to 3 % slower.
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        while (!mbar_try(bar, parity))
            if (cta_gave_up()) return false;
        return true;
    };
    auto unit_row = [&](int u, int r) -> int { return kSwiGLU ? ((r & 1) ? a.inter : 0) + (R / 2) * u + (r >> 1) : R * u + r; };
    auto row_ok = [&](int u, int r) -> bool { return kSwiGLU ? ((R / 2) * u + (r >> 1) < a.inter) : (R * u + r < N); };

    if (warp == kMmaWarps) {
        // ================================================= producer warp: order (part, unit); lane 0 arms the stage, lanes 0..R-1 copy one row each
        int item = 0, un = 0, p = 0, s = 0;
        auto issue_next = [&]() {
            const int u = gid + un * total, k0 = p * geo.part_k;
            const uint32_t bytes = (uint32_t)bytes_of(min(geo.part_k, K - k0)), bar = full0 + s * 8;
            const bool mine = lane < R && row_ok(u, lane);
            const unsigned nrows = __popc(__ballot_sync(0xffffffffu, mine));
            if (lane == 0) mbar_expect_tx(bar, bytes * nrows);
            __syncwarp();
            if (mine)
                bulk_g2s(ring_u32 + s * geo.stage_bytes + lane * geo.row_stride,
                         reinterpret_cast<const unsigned char *>(a.w) + (size_t)unit_row(u, lane) * row_bytes + bytes_of(k0), bytes, bar);
            ++item;
            if (++un == my_units) un = 0, ++p;
            if (++s == stages) s = 0;
        };
        if (lane == 0) {
            cta_gave_up() = 0;
            for (int i = 0; i < stages; ++i) {
                mbar_init(full0 + i * 8, 1);
                mbar_init(empty0 + i * 8, kMmaWarps);
            }
            for (int b = 0; b < 2; ++b) {
                mbar_init(ready0 + b * 8, kMmaWarps);
                mbar_init(free0 + b * 8, 1);
            }
            fence_mbar_init();
        }
        __syncwarp();
        while (item < stages && item < my_items) issue_next();  // the weights do not depend on the previous kernel
        __syncthreads();                                         // publishes the barriers
        pdl_wait();  // (nothing here reads what the kernel in front writes: the limit of the waits below starts when it is done)
        int e_s = 0, e_ph = 0;
        while (item < my_items) {
            if (!__all_sync(0xffffffffu, wait(empty0 + e_s * 8, e_ph))) break;
            if (++e_s == stages) e_s = 0, e_ph ^= 1;
            fence_proxy_async();
            issue_next();
        }
        // the CTA stays until its last copies have landed, whether or not somebody still waits for them
        for (int i = max(0, item - stages); i < item; ++i)
            if (!mbar_drain(full0 + i % stages * 8, (i / stages) & 1)) break;
        return;
    }
    if (warp > kMmaWarps) {
        // ================================================= reducer: lane l finishes 4 consecutive rows of one token of the tile
        __syncthreads();
        pdl_wait();  // (y may be what the previous kernel reads)
        const unsigned int push_flag = a.push.n > 0 ? tp_flag(a.push.epoch, a.push.seq) : 0u;
        const int m0 = lane * 4 / R, r0 = lane * 4 % R;
        int h = 0;
        for (int p = 0; p < parts; ++p) {
            for (int un = 0; un < my_units; ++un, ++h) {
                const int u = gid + un * total, b = h & 1;
                float s8[4];
                if constexpr (FMT == WF_FP8) {  // requested before the wait: the latency hides behind the compute warps
#pragma unroll
                    for (int i = 0; i < 4; ++i) s8[i] = (p + 1 == parts && row_ok(u, r0 + i)) ? __ldg(reinterpret_cast<const float *>(a.scales) + unit_row(u, r0 + i)) : 1.0f;
                }
                const bool lost = !mbar_wait_guarded(ready0 + b * 8, (h >> 1) & 1, geo.wait, kWaitGemvRs) || cta_gave_up();  // (set before whatever the warps hand over without having waited)
                constexpr int PASSES = VALS / 128;
                float4 sums[PASSES];
#pragma unroll
                for (int q = 0; q < PASSES; ++q) {
                    const float *slot = tiles + (size_t)b * kMmaWarps * TILE + (kDense ? lane * 4 : (m0 + 8 * q) * 20 + r0);
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int w2 = 0; w2 < kMmaWarps; ++w2) {  // fixed order: deterministic
                        const float4 o = *reinterpret_cast<const float4 *>(slot + (size_t)w2 * TILE);
                        v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
                    }
                    sums[q] = v;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(free0 + b * 8);
#pragma unroll
                for (int q = 0; q < PASSES; ++q) {
                    float4 v = sums[q];
                    const int m = m0 + 8 * q;
                    if (parts > 1) {  // accumulate across the parts (part order: deterministic)
                        float4 *acc = reinterpret_cast<float4 *>(outacc + (size_t)un * VALS + q * 128 + lane * 4);
                        if (p > 0) {
                            const float4 o = *acc;
                            v.x += o.x, v.y += o.y, v.z += o.z, v.w += o.w;
                        }
                        if (p + 1 < parts) {
                            *acc = v;
                            continue;
                        }
                    }
                    if (m >= a.M) continue;
                    if (lost) v.x = v.y = v.z = v.w = __int_as_float(0x7fc00000);
                    float o[4] = {v.x, v.y, v.z, v.w};
                    if constexpr (FMT == WF_FP8) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[i] *= s8[i];
                    }
                    if constexpr (kSwiGLU) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int j = (R / 2) * u + (r0 >> 1) + i;  // rows (r0 + 2i, r0 + 2i + 1) = (gate_j, up_j)
                            if (j < a.inter) {
                                // the un-fused reference stores gate / up in T before SiLU reads them
                                const float gt = round_to<T>(o[2 * i]), up = round_to<T>(o[2 * i + 1]);
                                const float sv = (gt / (1.0f + expf(-gt))) * up;
                                if (a.y_f32) reinterpret_cast<float *>(a.y)[(size_t)m * a.inter + j] = sv;
                                else reinterpret_cast<T *>(a.y)[(size_t)m * a.inter + j] = Elem<T>::from_f(sv);
                            }
                        }
                    } else if (a.push.n > 0) {
                        // tensor-parallel partial: this lane's four consecutive rows are two LL words = one 16-byte store per peer
                        if (row_ok(u, r0 + 3) && (N & 3) == 0) {
                            tp_push_quad<T>(a.push, push_flag, (size_t)m * N + R * u + r0, o);
                        } else {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
                                if (row_ok(u, r0 + 2 * i + 1)) tp_push_pair<T>(a.push, push_flag, (size_t)m * N + R * u + r0 + 2 * i, o[2 * i], o[2 * i + 1]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (row_ok(u, r0 + i)) {
                                const size_t idx = (size_t)m * N + R * u + r0 + i;
                                if (a.y_f32) reinterpret_cast<float *>(a.y)[idx] = o[i];
                                else reinterpret_cast<T *>(a.y)[idx] = Elem<T>::from_f(o[i]);
                            }
                    }
                }
            }
        }
        return;
    }

    // ===================================================== compute warps
    const T *x = reinterpret_cast<const T *>(a.x);
    uint4 av[NB], bv[NT == 2 ? NB : 1];
    int k0w = 0, nb = 0;  // this warp's slice of the part: first k, blocks
    auto slice = [&](int p) {
        const int pk0 = p * geo.part_k, pk = min(geo.part_k, K - pk0);
        constexpr int step = kDense ? 1 : 4;  // quantised: whole groups of 128 k
        const int n = pk / (32 * step), first = n * warp / kMmaWarps, last = n * (warp + 1) / kMmaWarps;
        nb = (last - first) * step;
        k0w = pk0 + min(first, n - 1) * step * 32;  // (a warp without blocks multiplies some live row's weights by zeros)
    };
    slice(0);
    __syncthreads();
    pdl_wait();

    const int ngroups_k = FMT == WF_INT4 ? K / 128 : 0;
    constexpr int NG = NB / 4;
    // the k of a lane's 8 activations of block j, counted from the slice: the block's t-th eight (dense), or 8 of the 32 k of a group that the lane's pieces of 16 bytes
    // of a weight row hold: consecutive ones (INT4, one piece), or two times 16, 64 apart (FP8; with 32 in a row there too a load of activations met 16 lines of the
    // first-level cache instead of 8, which is what 16 tokens waited for: see the file's header)
    auto k_of = [&](int j) -> int { return kDense ? 32 * j + 8 * t : FMT == WF_FP8 ? 64 * (j >> 1) + 16 * t + 8 * (j & 1) : 128 * (j >> 2) + 32 * t + 8 * (j & 3); };
    // INT4 parameters of the slice's groups.  A warp needs 16 rows x 2 groups of them per unit -- 2-byte and 1-byte loads a round trip to L2 away,
    // several units' worth of streaming.  So its 32 lanes fetch TWO units at once (lane: unit lane / 16 of the batch, row lane % 16), a batch ahead of
    // the one in use, and a unit's scales and zero points reach their lanes by shuffles.
    struct QBatch {
        uint32_t z, s[NG];  // zero points, a byte per group; scales (the bits of T)
    };
    auto load_qbatch = [&](int un0) -> QBatch {
        QBatch q = {};
        if constexpr (FMT == WF_INT4) {
            const int u = gid + min(un0 + (lane >> 4), my_units - 1) * total;
            const int row = min(unit_row(u, lane & 15), N - 1);
            const size_t gi = (size_t)row * ngroups_k + k0w / 128;
#pragma unroll
            for (int j = 0; j < NG; ++j)
                if (4 * j < nb) {
                    q.z |= (uint32_t)__ldg(reinterpret_cast<const uint8_t *>(a.zeros) + gi + j) << (8 * j);
                    q.s[j] = (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(a.scales) + gi + j);
                }
        }
        return q;
    };

    int s = 0, ph = 0, h = 0;
    for (int p = 0; p < parts; ++p) {
        if (p > 0) slice(p);
        const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
        // ---- this part's activations of the slice: tokens g and g + 8
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            av[j] = zero4;
            if (j < nb && g < a.M) av[j] = ld_v4(x + (size_t)g * K + k0w + k_of(j));
            if constexpr (NT == 2) {
                bv[j] = zero4;
                if (j < nb && g + 8 < a.M) bv[j] = ld_v4(x + (size_t)(g + 8) * K + k0w + k_of(j));
            }
        }
        if (p == 0) pdl_launch_dependents();
        if constexpr (!kDense) {
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                av[j] = rs_fragment<T, FMT>(av[j]);
                if constexpr (NT == 2) bv[j] = rs_fragment<T, FMT>(bv[j]);
            }
        }
        const int wk = k0w - p * geo.part_k, top = max(nb - 1, 0);
        QBatch qcur = {}, qnxt = {};
        if (FMT == WF_INT4 && my_units > 0) qcur = load_qbatch(0), qnxt = load_qbatch(2);
        for (int un = 0; un < my_units; ++un, ++h) {
            // dense: [token g (+8)][row 2t (+1)], two chains; quantised: [row g (+8)][token 2t (+1)], acc2: tokens 8 .. 15
            float acc[4] = {}, acc2[4] = {};
            (void)wait(full0 + s * 8, ph);
            uint32_t za = 0, zb = 0;
            const int src = (un & 1) * 16 + g;  // the lane that fetched row g of this unit
            if constexpr (FMT == WF_INT4) {
                if (un > 0 && (un & 1) == 0) qcur = qnxt, qnxt = load_qbatch(un + 2);
                za = __shfl_sync(0xffffffffu, qcur.z, src), zb = __shfl_sync(0xffffffffu, qcur.z, src + 8);
            }
            const unsigned char *wrow = ring + (size_t)s * geo.stage_bytes + (size_t)g * geo.row_stride + bytes_of(wk) + bytes_of(k_of(0));
            if constexpr (kDense) {
#pragma unroll
                for (int j0 = 0; j0 < NB; j0 += 4) {
                    if (j0 >= nb) break;
                    uint4 wq[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) wq[i] = *reinterpret_cast<const uint4 *>(wrow + (size_t)min(j0 + i, top) * 64);  // past the slice: A is zero
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 b = NT == 2 ? bv[j0 + i] : zero4, &q = av[j0 + i];
                        float(&c)[4] = (i & 1) ? acc2 : acc;
                        if constexpr (std::is_same<T, __nv_bfloat16>::value) {
                            mma_bf16(c, q.x, b.x, q.y, b.y, wq[i].x, wq[i].y);
                            mma_bf16(c, q.z, b.z, q.w, b.w, wq[i].z, wq[i].w);
                        } else {
                            mma_f16f16(c, q.x, b.x, q.y, b.y, wq[i].x, wq[i].y);
                            mma_f16f16(c, q.z, b.z, q.w, b.w, wq[i].z, wq[i].w);
                        }
                    }
                }
            } else {
                const unsigned char *wrow8 = wrow + 8 * geo.row_stride;
#pragma unroll
                for (int q = 0; q < NG; ++q) {
                    if (4 * q >= nb) break;
                    // this lane's 32 weights of rows g and g + 8 in the group
                    constexpr int PIECES = FMT == WF_FP8 ? 2 : 1;
                    uint32_t wa[4 * PIECES], wb[4 * PIECES];
#pragma unroll
                    for (int i = 0; i < PIECES; ++i) {
                        *reinterpret_cast<uint4 *>(wa + 4 * i) = *reinterpret_cast<const uint4 *>(wrow + 64 * (PIECES * q + i));
                        *reinterpret_cast<uint4 *>(wb + 4 * i) = *reinterpret_cast<const uint4 *>(wrow8 + 64 * (PIECES * q + i));
                    }
                    float c0[4] = {}, c1[4] = {};  // two chains: the k-steps of the first tokens, or (16 tokens) the first and the second eight
                    uint32_t zpa = 0, nza = 0, zpb = 0, nzb = 0;
                    if constexpr (FMT == WF_INT4) {
                        mma_int4_consts((za >> (8 * q)) & 0xffu, zpa, nza);
                        mma_int4_consts((zb >> (8 * q)) & 0xffu, zpb, nzb);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t e[4], f[4];
                        if constexpr (FMT == WF_INT4) {
                            mma_deq_int4(wa[i], zpa, nza, e);
                            mma_deq_int4(wb[i], zpb, nzb, f);
                        } else {
#pragma unroll
                            for (int y = 0; y < 4; ++y) {
                                e[y] = mma_e4m3x2_to_f16x2(wa[2 * i + (y >> 1)] >> (16 * (y & 1)));
                                f[y] = mma_e4m3x2_to_f16x2(wb[2 * i + (y >> 1)] >> (16 * (y & 1)));
                            }
                        }
                        const uint4 &x0 = av[4 * q + i];
                        mma_f16f16(c0, e[0], f[0], e[1], f[1], x0.x, x0.y);
                        if constexpr (NT == 2) {
                            const uint4 &x1 = bv[4 * q + i];
                            mma_f16f16(c1, e[0], f[0], e[1], f[1], x1.x, x1.y);
                            mma_f16f16(c0, e[2], f[2], e[3], f[3], x0.z, x0.w);
                            mma_f16f16(c1, e[2], f[2], e[3], f[3], x1.z, x1.w);
                        } else {
                            mma_f16f16(c1, e[2], f[2], e[3], f[3], x0.z, x0.w);
                        }
                    }
                    float sa = 1.0f, sb = 1.0f;  // the group's scales of rows g and g + 8
                    if constexpr (FMT == WF_INT4) {
                        const unsigned short lo = (unsigned short)__shfl_sync(0xffffffffu, qcur.s[q], src), hi = (unsigned short)__shfl_sync(0xffffffffu, qcur.s[q], src + 8);
                        sa = Elem<T>::to_f(*reinterpret_cast<const T *>(&lo)), sb = Elem<T>::to_f(*reinterpret_cast<const T *>(&hi));
                    }
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const float sc = y < 2 ? sa : sb;
                        acc[y] = fmaf(sc, NT == 2 ? c0[y] : c0[y] + c1[y], acc[y]);
                        if constexpr (NT == 2) acc2[y] = fmaf(sc, c1[y], acc2[y]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + s * 8);  // this warp has left the stage
            if (++s == stages) s = 0, ph ^= 1;
            // ---- hand this warp's tile of the (part, unit) to the reducer (double-buffered slot)
            const int b = h & 1;
            if (h >= 2) (void)wait(free0 + b * 8, ((h >> 1) - 1) & 1);
            float *slot = tiles + ((size_t)b * kMmaWarps + warp) * TILE;
            if constexpr (kDense) {
                *reinterpret_cast<float2 *>(slot + g * R + 2 * t) = make_float2(acc[0] + acc2[0], acc[1] + acc2[1]);
                if constexpr (NT == 2) *reinterpret_cast<float2 *>(slot + (g + 8) * R + 2 * t) = make_float2(acc[2] + acc2[2], acc[3] + acc2[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int at = (2 * t + (e & 1)) * 20 + g + 8 * (e >> 1);
                    slot[at] = acc[e];
                    if constexpr (NT == 2) slot[8 * 20 + at] = acc2[e];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(ready0 + b * 8);
        }
    }
}

// host side ----------------------------------------------------------------------------------------------------------
inline size_t gemv_rs_fixed_smem(const RsGeom &g, bool dense, int nt) {
    return (size_t)(2 * kRsMaxStages + 4) * 8 + (size_t)2 * kMmaWarps * rs_tile(dense, nt) * 4 + (g.parts > 1 ? (size_t)g.max_units * (dense ? 128 : 128 * nt) * 4 : 0);
}
inline bool gemv_rs_geometry(int M, int K, int max_units, int fmt, RsGeom *out) {
    if (M < 1 || M > 16 || K % 128 != 0) return false;
    const int groups = K / 128;
    // quantised slices are whole groups of 128 k, dense ones whole blocks of 32: either way a part has at most 16 x 8 blocks
    RsGeom g = {};
    g.parts = (groups * 4 + kMmaWarps * kRsBlocks - 1) / (kMmaWarps * kRsBlocks);
    g.part_k = (groups + g.parts - 1) / g.parts * 128;
    g.parts = (K + g.part_k - 1) / g.part_k;
    g.max_units = max_units;
    const size_t bytes = fmt == WF_DENSE ? (size_t)g.part_k * 2 : (fmt == WF_FP8 ? (size_t)g.part_k : (size_t)g.part_k / 2);
    // rows of a stage 64 bytes apart modulo 128: the 16-byte reads of the eight lanes of a phase -- two rows' four pieces, 64 bytes of each -- fall on different banks
    g.row_stride = (int)((bytes + 127) / 128 * 128) + 64;
    g.stage_bytes = rs_rows(fmt == WF_DENSE) * g.row_stride;
    const size_t budget = kRsSmem, fixed = gemv_rs_fixed_smem(g, fmt == WF_DENSE, M > 8 ? 2 : 1);
    if (fixed + (size_t)2 * g.stage_bytes > budget) return false;
    g.wait = wait_guard();
    g.stages = (int)((budget - fixed) / g.stage_bytes);
    if (g.stages > kRsMaxStages) g.stages = kRsMaxStages;
    *out = g;
    return true;
}

template <typename T, int FMT, bool SW, int NT>
static int launch_gemv_rs_inst(const GemvArgs &a, const RsGeom &g, int grid, cudaStream_t st) {
    auto kern = gemv_rs_kernel<T, FMT, SW, NT>;
    const size_t smem = gemv_rs_fixed_smem(g, FMT == WF_DENSE, NT) + (size_t)g.stages * g.stage_bytes;
    if (!allow_smem(reinterpret_cast<const void *>(kern), kRsSmem)) return cuda_status("gemv_rs cudaFuncSetAttribute");
    launch_pdl(kern, dim3(grid), dim3(kMmaThreads), smem, st, true, a, g);
    return cuda_status("gemv_rs launch");
}

// B200_ERR_UNSUPPORTED (no error text): shapes it does not take, a tensor-parallel reduce or a norm in front.
template <typename T>
static int launch_gemv_rs_t(const GemvArgs &a, int fmt, bool swiglu, cudaStream_t st) {
    if (a.M < 1 || a.M > 16 || a.K % 128 != 0 || !aligned16(a.w) || !aligned16(a.x) || a.tp.world > 1 || a.norm) return B200_ERR_UNSUPPORTED;
    if (fmt == WF_INT4 && a.group != 128) return B200_ERR_UNSUPPORTED;
    if (swiglu && a.inter % 8 != 0) return B200_ERR_UNSUPPORTED;
    if (a.push.n > 0 && a.N % 2 != 0) return B200_ERR_UNSUPPORTED;
    const int R = rs_rows(fmt == WF_DENSE), units = swiglu ? (a.inter + R / 2 - 1) / (R / 2) : (a.N + R - 1) / R;
    const int grid = std::max(1, std::min(sm_count(), units));
    RsGeom g = {};
    if (!gemv_rs_geometry(a.M, a.K, (units + grid - 1) / grid, fmt, &g) ) return B200_ERR_UNSUPPORTED;
#define B200_RS_GO(FMTC, SW) (a.M > 8 ? launch_gemv_rs_inst<T, FMTC, SW, 2>(a, g, grid, st) : launch_gemv_rs_inst<T, FMTC, SW, 1>(a, g, grid, st))
    if (fmt == WF_DENSE) return swiglu ? B200_RS_GO(WF_DENSE, true) : B200_RS_GO(WF_DENSE, false);
    if (fmt == WF_FP8) return swiglu ? B200_RS_GO(WF_FP8, true) : B200_RS_GO(WF_FP8, false);
    if (fmt == WF_INT4) return swiglu ? B200_RS_GO(WF_INT4, true) : B200_RS_GO(WF_INT4, false);
#undef B200_RS_GO
    return B200_ERR_UNSUPPORTED;
}

}  // namespace b200
