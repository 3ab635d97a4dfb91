"""The linears' tensor-core kernels at the edges of their tiles: the register-stationary GEMV (csrc/gemv_rs.cuh: one to sixteen tokens, every weight
format, k slices that do not divide evenly, rows past the last unit, several parts) and the CTA-pair GEMM (csrc/gemm_tc.cu: rows past the last
256-row tile, column tiles of two widths, k past the last stage), against the product in 64 bits; and the sampler's random numbers."""
import math

import pytest
import torch

import util

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
b200 = util.b200()
# one rounding of the result to the output type; the sums themselves are fp32 (2^-24 per term of up to 16384 random signs: below a tenth of it)
ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def close(got, want, dtype, what):
    scale = want.abs().max()
    err = (got.double() - want).abs() - ROUND[dtype] * want.abs()
    assert not torch.isnan(got).any(), what
    assert float(err.max() / scale) < 2e-4, (what, float(err.max() / scale))  # 2e-4 of the largest: sums of up to 16384 products in fp32


def quantised(gen, n, k, fmt, dtype):
    """-> (codes, scales, zeros, dense weights in 64 bits)."""
    if fmt == "fp8":
        q = torch.randn(n, k, generator=gen, device=DEV).to(torch.float8_e4m3fn)
        s = torch.rand(n, generator=gen, device=DEV) + 0.5
        return q.view(torch.uint8), s, None, q.to(torch.float32).double() * s.double()[:, None]
    codes = torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8)
    s = (torch.rand(n, k // 128, generator=gen, device=DEV) + 0.5).to(dtype)
    z = torch.randint(0, 16, (n, k // 128), generator=gen, device=DEV, dtype=torch.uint8)
    q = torch.stack((codes & 15, codes >> 4), -1).reshape(n, k // 128, 128).double()
    return codes, s, z, ((q - z.double()[..., None]) * s.double()[..., None]).reshape(n, k)


@pytest.mark.parametrize("fmt", ["dense", "fp8", "int4"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("m", [1, 2, 3, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("k,n", [(128, 64), (384, 72), (2176, 1187 * 8), (4096, 40), (4224, 1184), (8192, 264), (11008, 2376), (14336, 8)])
def test_linear_of_few_tokens(fmt, dtype, m, k, n):
    gen = torch.Generator(device=DEV).manual_seed(m * 1000 + k + n)
    x = torch.randn(m, k, generator=gen, device=DEV).to(dtype)
    if fmt == "dense":
        w = torch.randn(n, k, generator=gen, device=DEV).to(dtype)
        got, dense = b200.linear(x, w), w.double()
    else:
        w, s, z, dense = quantised(gen, n, k, fmt, dtype)
        got = b200.linear(x, w, w_format=b200.W_FP8 if fmt == "fp8" else b200.W_INT4, scales=s, zeros=z, group=128, N=n)
    close(got, x.double() @ dense.T, dtype, (fmt, m, k, n))


@pytest.mark.parametrize("n", [1, 7, 9, 1185])
def test_linear_of_few_tokens_and_odd_rows(n):
    """Row counts that are no multiple of a unit: the last unit's missing rows are neither fetched nor stored."""
    gen = torch.Generator(device=DEV).manual_seed(n)
    x, w = torch.randn(6, 512, generator=gen, device=DEV).bfloat16(), torch.randn(n, 512, generator=gen, device=DEV).bfloat16()
    out = torch.full((6 * n + 64,), 7.0, dtype=torch.bfloat16, device=DEV)
    b200.linear(x, w, out=out[:6 * n].view(6, n))
    close(out[:6 * n].view(6, n), x.double() @ w.double().T, torch.bfloat16, n)
    assert bool((out[6 * n:] == 7.0).all())


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("k,n", [(128, 1), (512, 7), (1408, 296), (1536, 2369), (1664, 4738), (3072, 31), (3200, 297)])
def test_fp32_rows_of_a_few_tokens(m, k, n):
    """csrc/gemv_sr.cuh: rows that are no whole number of a warp's slots, row counts around the SMs and their warps, odd ones, and the lengths it leaves alone."""
    gen = torch.Generator(device=DEV).manual_seed(m + k + n)
    x, w = torch.randn(m, k, generator=gen, device=DEV), torch.randn(n, k, generator=gen, device=DEV)
    out = torch.full((m * n + 64,), 7.0, device=DEV)
    got = b200.linear(x, w, out=out[:m * n].view(m, n))
    # chains of at most k / 128 products a lane, then the lanes: each rounding 2^-24 of the terms' sizes
    assert bool(((got.double() - x.double() @ w.double().T).abs() <= (k / 128 + 8) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
    assert bool((out[m * n:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("m,k,n", [(1, 128, 1), (8, 640, 31), (3, 1920, 2369), (8, 2176, 4743), (2, 4096, 17), (5, 4096, 4737), (8, 4224, 2384), (1, 8320, 4743), (6, 8192, 16),
                                   (6, 11008, 24), (7, 11008, 24), (2, 28672, 48), (3, 28672, 48)])
def test_int4_weights_streamed_into_registers(dtype, m, k, n):
    """csrc/gemv_qd.cuh: every zero point of a byte, activations with a mean or tiny (2^-12), odd group counts per warp and warps without groups, rows past the
    last unit, activations that only just fit (or no longer do)."""
    gen = torch.Generator(device=DEV).manual_seed(m + k + n)
    q, s, _, _ = quantised(gen, n, k, "int4", dtype)
    s *= 2.0 ** -11  # the largest result, 28672 products of 270 and activations of mean 4, stays below 65504
    z = torch.randint(0, 256, (n, k // 128), generator=gen, device=DEV, dtype=torch.uint8)
    z[::2] &= 15
    codes = torch.stack((q & 15, q >> 4), -1).reshape(n, k // 128, 128).double()
    dense = ((codes - z.double()[..., None]) * s.double()[..., None]).reshape(n, k)
    for mean, scale in ((4.0, 1.0), (0.0, 2.0 ** -12)):
        x = ((torch.randn(m, k, generator=gen, device=DEV) + mean) * scale).to(dtype)
        out = torch.full((m * n + 64,), 7.0, dtype=dtype, device=DEV)
        got = b200.linear(x, q, w_format=b200.W_INT4, scales=s, zeros=z, group=128, N=n, out=out[:m * n].view(m, n)).double()
        # one rounding of the result; fp32 sums: 2^-24 of the terms' sizes for each of a group's 8 products, the groups' and the warps' sums (28672 k: 14 + 16)
        x16 = x.half().double()  # the activations as the tensor cores take them
        bound = ROUND[dtype] * (x16 @ dense.T).abs() + 38 * 2.0 ** -24 * x16.abs() @ ((codes - z.double()[..., None]).abs() * s.double()[..., None]).reshape(n, k).T + 2.0 ** -24
        assert bool(((got - x16 @ dense.T).abs() <= bound).all()), (mean, float(((got - x16 @ dense.T).abs() / bound).max()))
        assert bool((out[m * n:] == 7.0).all())


@pytest.mark.parametrize("fmt", ["int4", "fp8"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("k", [128, 640, 1152, 1920, 2048, 2176, 3968, 4096, 4224, 4352, 5120, 7168, 8192, 8832, 11008, 12416, 14336, 28672])
def test_quantised_token_has_the_same_bits_beside_any_others(fmt, dtype, k):
    """1 to 8 tokens, and 9 to 16.  INT4 of up to 8: whichever form of csrc/gemv_qd.cuh holds their activations, or csrc/gemv_rs.cuh where none does (11008 k from 7
    tokens on, 28672 from 3 on)."""
    for n in (17, 300, 4743):
        gen = torch.Generator(device=DEV).manual_seed(k + n)
        x = torch.randn(16, k, generator=gen, device=DEV).to(dtype)
        q, s, z, _ = quantised(gen, n, k, fmt, dtype)
        s *= 2.0 ** -8
        run = lambda t: b200.linear(t.contiguous(), q, w_format=b200.W_INT4 if fmt == "int4" else b200.W_FP8, scales=s, zeros=z, group=128, N=n)  # noqa: B023,E731
        for first, most in ((1, 8), (9, 16)):
            every = run(x[:most])
            for m in range(first, most):
                assert torch.equal(run(x[:m]), every[:m]), (n, m)
            assert torch.equal(run(x[most - first:most]), every[most - first:]), (n, first)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("k", [128, 640, 1024, 1152, 1536, 1920, 2048, 2176, 2688, 3072, 3200, 4096, 5120, 11008])
def test_dense_token_has_the_same_bits_beside_any_others(dtype, k):
    """2 to 16 tokens, in csrc/gemv_qd.cuh (to 3072 k, one token too) and in csrc/gemv_rs.cuh."""
    for n in (17, 300, 4743):
        gen = torch.Generator(device=DEV).manual_seed(k + n)
        x, w = (torch.randn(r, k, generator=gen, device=DEV).to(dtype) for r in (16, n))
        all16 = b200.linear(x, w)
        for m in range(1 if k <= 3072 else 2, 16):
            assert torch.equal(b200.linear(x[:m].contiguous(), w), all16[:m]), (n, m)
        assert torch.equal(b200.linear(x[5:].contiguous(), w), all16[5:]), n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("hidden", [1024, 2048, 3072, 4096])
def test_logits_of_a_row_have_the_same_bits_beside_any_others(dtype, hidden):
    """The head's fp32 logits, norm in front, of 2 to 16 rows, and of 17 to 24, whose last pass has 1 to 8 rows (one row has a kernel of its own)."""
    gen = torch.Generator(device=DEV).manual_seed(hidden)
    vocab, k = 1003, 5
    x, gamma, head = (torch.randn(*s, generator=gen, device=DEV).to(dtype) for s in ((24, hidden), (hidden,), (vocab, hidden)))
    code = {torch.bfloat16: b200.BF16, torch.float16: b200.F16}[dtype]
    engine = b200.Decoder(b200.DecoderConfig(hidden, hidden // 128, hidden // 128, 128, 256, 1, 64, 24, code, b200.W_DENSE, 128, 1e-6, 128, 10000.0, 1, 0), DEV)

    def logits(rows):
        b = len(rows)
        z = lambda *s, dtype=torch.int32: torch.zeros(*s, dtype=dtype, device=DEV)  # noqa: E731
        bufs = dict(logits=z(b, vocab, dtype=torch.float32), tmp_ids=z(b, b200.TOPK_BLOCKS, k), tmp_vals=z(b, b200.TOPK_BLOCKS, k, dtype=torch.float32),
                    topk_ids=z(b, k), topk_vals=z(b, k, dtype=torch.float32), seq_len=z(b), finished=z(b, dtype=torch.uint8), output_id=z(b))
        engine.lm_head_topk_sample(rows.clone(), gamma, head, bufs, k, 7, 2)
        return bufs["logits"]

    all16 = logits(x[:16])
    for m in (2, 3, 7, 8, 9, 12, 15):
        assert torch.equal(logits(x[:m]), all16[:m]), m
    all24 = logits(x)
    assert torch.equal(all24[:16], all16) and torch.equal(logits(x[:19])[16:], all24[16:19])


@pytest.mark.parametrize("k", [128, 512, 1024, 1408, 1536, 1664, 2048, 2688, 3072, 4096])
def test_fp32_token_has_the_same_bits_beside_any_others(k):
    """1 to 4 tokens, in csrc/gemv_sr.cuh (to 1536 k) and in csrc/gemv.cuh; and a decode step, whose linears norm their tokens: hidden size k, one layer."""
    for n in (17, 300, 4743):
        gen = torch.Generator(device=DEV).manual_seed(k + n)
        x, w = torch.randn(4, k, generator=gen, device=DEV), torch.randn(n, k, generator=gen, device=DEV)
        all4 = b200.linear(x, w)
        for m in (1, 2, 3):
            assert torch.equal(b200.linear(x[:m].contiguous(), w), all4[:m]), (n, m)
        assert torch.equal(b200.linear(x[3:].contiguous(), w), all4[3:]), n
    gen = torch.Generator(device=DEV).manual_seed(k)
    r = lambda *s: torch.randn(*s, generator=gen, device=DEV) / math.sqrt(s[-1])  # noqa: E731
    heads, inter = k // 128, k + 128
    layer = dict(g1=r(k) + 1, g2=r(k) + 1, qkv=r(3 * heads * 128, k), o=r(k, heads * 128), gate_up=r(2 * inter, k), down=r(k, inter))
    x, cache = torch.randn(4, k, generator=gen, device=DEV), torch.randn(2, 1, 4, heads, 64, 128, generator=gen, device=DEV)
    got = []
    for m in (4, 1, 2, 3):
        dec = b200.Decoder(b200.DecoderConfig(k, heads, heads, 128, inter, 1, 64, m, b200.F32, b200.W_DENSE, 128, 1e-6, 128, 10000.0, 1, 0), DEV)
        dec.set_layer(0, layer)
        hidden = x[:m].clone()
        dec.step(hidden, cache[0, :, :m].contiguous(), cache[1, :, :m].contiguous(), 33)
        got.append(hidden)
    for y in got[1:]:
        assert torch.equal(y, got[0][:len(y)]), len(y)


@pytest.mark.parametrize("m", [1, 2, 4])
@pytest.mark.parametrize("k", [512, 1024, 1408, 1536])
def test_fp32_sums_round_no_more_often_than_they_need(m, k):
    """csrc/gemv_sr.cuh's distance from 64 bits over 8192 rows.  A sum of j random terms has variance j (a term's: 1); rounding it adds s^2 j, s^2 = 2^-46 / 12 times
    the mean of 1 / mantissa^2 (0.541 for mantissas spread over their logarithm).  A lane's four chains: slots of four products (1 + 2 + 3 + 4), which join one
    another (4 (2 + .. + S) for S = k / 512); then four chains to one (2 additions of a half, one of all: twice k over all lanes) and five rounds over the
    lanes (k each).  One chain of k / 128 products (1 + .. + k / 128) instead comes out 1.05 times as far at 1408 and 1536 k.  Sums of normal products have
    mantissas a little nearer to 1 than that (6 % more, measured): 8 % are allowed."""
    pieces = k // 128
    chains = sum(10 if s + 4 <= pieces else sum(range(1, pieces - s + 1)) for s in range(0, pieces, 4)) + sum(min(4 * i, pieces) for i in range(2, (pieces + 3) // 4 + 1))
    model = math.sqrt(2.0 ** -46 / 12 * 0.541 * (128 * chains / k + 2 + 5))
    gen = torch.Generator(device=DEV).manual_seed(m + k)
    x, w = torch.randn(m, k, generator=gen, device=DEV), torch.randn(8192, k, generator=gen, device=DEV)
    want = x.double() @ w.double().T
    assert float((b200.linear(x, w).double() - want).norm() / want.norm()) < 1.08 * model


@pytest.mark.parametrize("fmt,n", [("dense", 192000), ("fp8", 152064), ("int4", 290000)])
def test_linear_whose_sums_leave_no_ring(fmt, n):
    """Vocabulary-sized outputs of rows of 8192 k, 16 tokens: sizes that stay with the kernel whose activations are in shared memory (csrc/gemv_mma.cuh), and
    (INT4) that neither takes at once: two passes of eight tokens."""
    m, k, step = 16, 8192, 16000
    gen = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(m, k, generator=gen, device=DEV).bfloat16()
    kw = {}
    if fmt == "dense":
        w = torch.empty(n, k, dtype=torch.bfloat16, device=DEV).normal_(generator=gen)
    elif fmt == "fp8":
        w = torch.randint(0, 0x70, (n, k), generator=gen, device=DEV, dtype=torch.uint8) | (torch.randint(0, 2, (n, k), generator=gen, device=DEV, dtype=torch.uint8) << 7)
        kw = dict(w_format=b200.W_FP8, scales=torch.rand(n, generator=gen, device=DEV) + 0.5, N=n)
    else:
        w = torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8)
        kw = dict(w_format=b200.W_INT4, scales=(torch.rand(n, k // 128, generator=gen, device=DEV) + 0.5).bfloat16(),
                  zeros=torch.randint(0, 16, (n, k // 128), generator=gen, device=DEV, dtype=torch.uint8), group=128, N=n)
    got = b200.linear(x, w, **kw)
    for r in range(0, n, step):
        part = w[r:r + step]
        if fmt == "fp8":
            part = part.view(torch.float8_e4m3fn).to(torch.float32) * kw["scales"][r:r + step, None]
        elif fmt == "int4":
            q = torch.stack((part & 15, part >> 4), -1).reshape(len(part), k // 128, 128).float() - kw["zeros"][r:r + step, :, None].float()
            part = (q * kw["scales"][r:r + step, :, None].float()).reshape(len(part), k)
        close(got[:, r:r + step], x.double() @ part.double().T, torch.bfloat16, (fmt, r))


@pytest.mark.parametrize("fmt", ["dense", "fp8", "int4"])
@pytest.mark.parametrize("batch", [1, 2, 5, 8, 9, 16])
def test_few_tokens_match_the_same_rows_in_a_larger_batch(fmt, batch):
    """Layers of up to 16 tokens (streamed weights; one dense token: norms inside the linears) against the same rows in a batch of 17: rows agree to the
    roundings of the layer's 16-bit intermediates."""
    gen = torch.Generator(device=DEV).manual_seed(3)
    h, heads, kv, d, inter, rows = 1024, 8, 2, 128, 1408, 17

    def lin(n, k):
        if fmt == "dense":
            return (torch.randn(n, k, generator=gen, device=DEV) / math.sqrt(k)).bfloat16()
        q, s, z, _ = quantised(gen, n, k, fmt, torch.bfloat16)
        return (q, s / math.sqrt(k), None) if fmt == "fp8" else (q, (s.float() / (5 * math.sqrt(k))).bfloat16(), z)

    def vec(n):
        return (1 + 0.2 * torch.randn(n, generator=gen, device=DEV)).bfloat16()

    layers = [dict(g1=vec(h), g2=vec(h), o_bias=vec(h), qkv_bias=vec((heads + 2 * kv) * d), qkv=lin((heads + 2 * kv) * d, h), o=lin(h, heads * d),
                   gate_up=lin(2 * inter, h), down=lin(h, inter)) for _ in range(2)]
    wf = {"dense": b200.W_DENSE, "fp8": b200.W_FP8, "int4": b200.W_INT4}[fmt]
    x = (2 * torch.randn(rows, h, generator=gen, device=DEV)).bfloat16()
    k0, v0 = (torch.randn(2, rows, kv, 64, d, generator=gen, device=DEV).bfloat16() for _ in range(2))

    def step(n):
        dec = b200.Decoder(b200.DecoderConfig(h, heads, kv, d, inter, 2, 64, n, b200.BF16, wf, 128, 1e-6, d, 10000.0, 1, 0), DEV)
        for i, w in enumerate(layers):
            dec.set_layer(i, w)
        hidden, kc, vc = x[:n].clone(), k0[:, :n].contiguous(), v0[:, :n].contiguous()
        dec.step(hidden, kc, vc, 33)
        torch.cuda.synchronize()
        return hidden.double()

    want, got = step(rows)[:batch], step(batch)
    # per row: two layers of 16-bit intermediates summed in another order
    rel = (got - want).norm(dim=-1) / want.norm(dim=-1)
    assert float(rel.max()) < 1.5e-2, rel


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("m,k,n", [(256, 64, 9728), (250, 72, 9728), (512, 136, 4928), (769, 200, 4096), (1000, 1024, 4096), (1084, 320, 5136), (2048, 128, 4096),
                                   (2047, 88, 2056), (4096, 64, 264), (129, 4096, 12288)])
def test_linear_of_prompts(dtype, m, k, n):
    """Pairs of CTAs on 256-row tiles where they serve: rows and columns past the last tile, two tile widths, a last stage that is mostly padding."""
    gen = torch.Generator(device=DEV).manual_seed(m + k + n)
    x, w = torch.randn(m, k, generator=gen, device=DEV).to(dtype), torch.randn(n, k, generator=gen, device=DEV).to(dtype)
    out = torch.full((m * n + 64,), 7.0, dtype=dtype, device=DEV)
    b200.linear(x, w, out=out[:m * n].view(m, n))
    close(out[:m * n].view(m, n), x.double() @ w.double().T, dtype, (m, k, n))
    assert bool((out[m * n:] == 7.0).all())


@pytest.mark.parametrize("k", [64, 384, 448, 1024])
def test_pairs_leave_nothing_under_way(k):
    """Launches of CTA pairs whose k blocks are fewer than, as many as and more than the ring's stages, each with kernels behind it that hold barriers in the
    same shared memory: an arrival that outlived its CTA would complete a phase of theirs too early.  Every launch gives the first one's bits."""
    gen = torch.Generator(device=DEV).manual_seed(k)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()  # noqa: E731
    x, w, few, odd = rand(512, k), rand(9728, k), rand(6, 2048), rand(200, 2048)
    w2 = rand(1024, 2048)
    first = None
    for _ in range(200):
        got = (b200.linear(x, w), b200.linear(few, w2), b200.linear(odd, w2))
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(got, first))
    for (a, b), got in zip(((x, w), (few, w2), (odd, w2)), first):
        close(got, a.double() @ b.double().T, torch.bfloat16, k)


@pytest.mark.parametrize("m,k,inter", [(256, 64, 4864), (1000, 200, 2752), (2048, 128, 2688), (1084, 72, 5000), (300, 512, 1408)])
def test_swiglu_of_prompts_is_the_two_launchers(m, k, inter):
    """Gate and up halves of a tile come from the two CTAs of a pair: bit-identical to the linear followed by silu-and-mul."""
    gen = torch.Generator(device=DEV).manual_seed(m + inter)
    x, w = torch.randn(m, k, generator=gen, device=DEV).bfloat16(), torch.randn(2 * inter, k, generator=gen, device=DEV).bfloat16()
    want = b200.silu_and_mul(b200.linear(x, w).view(m, 2, inter))
    assert torch.equal(b200.linear_swiglu(x, w), want)


@pytest.mark.parametrize("step", [1, 77, 123456])
def test_sampled_ids_use_the_generators_own_numbers(step):
    """Rows 0 .. 299 (all low digits of the subsequence, alone and together) and rows past 2^16: the ids that cuRAND's own first numbers give."""
    for rows in (300, 65536 + 40):
        gen = torch.Generator(device=DEV).manual_seed(step)
        k = 8
        ids = torch.arange(rows * k, dtype=torch.int32, device=DEV).reshape(rows, k)
        vals = torch.sort(torch.randn(rows, k, generator=gen, device=DEV), -1, descending=True).values.contiguous()
        u = b200.xorwow_uniform(rows, step, DEV)
        weights = torch.exp(vals - vals[:, :1])
        total = torch.zeros(rows, device=DEV)
        for i in range(k):
            total = total + weights[:, i]
        left, want, done = u * total, ids[:, 0].clone(), torch.zeros(rows, dtype=torch.bool, device=DEV)
        margin = torch.full((rows,), 9.0, device=DEV)
        for i in range(k):
            left = left - weights[:, i]
            margin = torch.minimum(margin, left.abs())
            hit = (left < 0) & ~done
            want = torch.where(hit, ids[:, i], want)
            done |= hit
        seq, fin = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.zeros(rows, dtype=torch.uint8, device=DEV)
        got = b200.sampling(ids, vals.clone(), seq, fin, step, -1, rows * k)
        clear = margin > 1e-5  # (a draw on the edge of two candidates may fall on either side of an ulp of exp)
        assert bool((got == want)[clear].all()) and float(clear.float().mean()) > 0.99
