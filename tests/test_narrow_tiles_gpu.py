"""The tcgen05 linears of 17 tokens and more (csrc/gemm_tc.cu, plan_tiles): narrow tiles, rows that fill no tile, a tile's k shared by two CTAs, and quantised prompts on
exact FP8 codes with the rows' scales on the sums.  Against float64; a sum of k products of 16-bit numbers is off by the rounding of the result (half a unit of the
type) and by fp32 sums (2^-23 per addition of the running sum, far less in practice: k 2^-24 of the products' root sum of squares is allowed)."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
m = importlib.import_module("llm-inference-engine_b200")
DEV = "cuda"


def rand(gen, *shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, generator=gen, device=DEV) * scale).to(dtype)


def close(got, x, w, dtype):
    want = x.double() @ w.double().T
    norm = x.double().norm(dim=1)[:, None] * w.double().norm(dim=1)[None]
    bound = 0.51 * torch.finfo(dtype).eps * want.abs() + x.shape[1] ** 0.5 * 2.0 ** -23 * norm
    assert ((got.double() - want).abs() <= bound).all(), float(((got.double() - want).abs() / bound).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [17, 24, 25, 64, 65, 127, 128, 129, 200, 256, 257, 300])  # (64 | 65: rows of a product)
@pytest.mark.parametrize("K,N", [(64, 16), (72, 40), (2048, 2056), (1000, 4104), (4096, 1024)])
def test_tiles(dtype, M, K, N):
    gen = torch.Generator(device=DEV).manual_seed(M * 7 + K + N)
    x, w = rand(gen, M, K, dtype=dtype), rand(gen, N, K, dtype=dtype, scale=K ** -0.5)
    close(m.linear(x, w), x, w, dtype)


@pytest.mark.parametrize("M,K,N", [(17, 11008, 4096), (128, 11008, 4096), (129, 8200, 2048), (40, 16392, 1000), (256, 28672, 1024)])
def test_two_ctas_share_a_tile(M, K, N):
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = rand(gen, M, K), rand(gen, N, K, scale=K ** -0.5)
    got = m.linear(x, w)
    close(got, x, w, torch.bfloat16)
    for _ in range(5):
        assert torch.equal(m.linear(x, w), got)  # (added in rank order: the same every time)
    bias = torch.randn(N, generator=gen, device=DEV)
    assert torch.equal(m.linear_act(x, w, bias, 3), torch.relu(got.float() + bias).bfloat16())


# the last two: sizes at which the plain linear's widths leave two CTAs a tile and the SwiGLU ending's would have taken a CTA pair, which adds k up in one chain
@pytest.mark.parametrize("M,K,inter", [(200, 11008, 2048), (150, 16384, 512), (300, 8192, 1000), (257, 5120, 2376), (257, 16384, 2320)])
def test_swiglu_sums_in_the_same_order(M, K, inter):
    gen = torch.Generator(device=DEV).manual_seed(M + K)
    x, w = rand(gen, M, K), rand(gen, 2 * inter, K, scale=K ** -0.5)
    assert torch.equal(m.linear_swiglu(x, w), m.silu_and_mul(m.linear(x, w).view(M, 2, inter)))


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("T", [48, 49, 128, 129, 300])
def test_fp8_prompts_keep_their_scales_in_32_bits(dtype, T):
    """One layer whose linears are FP8 against the same layer on dense weights of the codes' own values and a scale of one: with scales that are powers of two the
    products are the same numbers, so both differ by the order of their sums only; with any scales a prompt agrees with itself fed sixteen tokens at a time."""
    h, heads, kv, inter, d = 512, 4, 2, 768, 128
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    gen = torch.Generator(device=DEV).manual_seed(T)

    def engine(fmt, power):
        g = torch.Generator(device=DEV).manual_seed(3)
        code = m.BF16 if dt == torch.bfloat16 else m.F16
        dec = m.Decoder(m.DecoderConfig(h, heads, kv, d, inter, 1, 320, 1, code, m.W_FP8 if fmt == "fp8" else m.W_DENSE, 128, 1e-6, d, 10000.0, 1, 0), DEV)
        layer = {"g1": torch.ones(h, device=DEV, dtype=dt), "g2": torch.ones(h, device=DEV, dtype=dt)}
        for name, n, k in (("qkv", (heads + 2 * kv) * d, h), ("o", h, heads * d), ("gate_up", 2 * inter, h), ("down", h, inter)):
            codes = torch.randn(n, k, generator=g, device=DEV).to(torch.float8_e4m3fn)
            scale = 2.0 ** torch.randint(-7, -4, (n,), generator=g, device=DEV) if power else torch.rand(n, generator=g, device=DEV) * 0.03 + 0.02
            layer[name] = (codes.view(torch.uint8), scale.float(), None) if fmt == "fp8" else (codes.float() * scale[:, None]).to(dt)
        dec.set_layer(0, layer)
        return dec, layer

    hidden = rand(gen, T, h, dtype=dt)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731

    def run(dec, cuts):
        k, v = (torch.zeros(1, 5, kv, 64, d, device=DEV, dtype=dt) for _ in range(2))
        table = torch.arange(5, dtype=torch.int32, device=DEV).reshape(1, 5)
        out, at = [], 0
        for n in cuts:
            x = hidden[at:at + n].clone()
            dec.prefill_paged(x, k, v, table, i32(n), i32(at), i32(at + n), n)
            out.append(x)
            at += n
        return torch.cat(out).double()

    u = torch.finfo(dt).eps
    same, (dense, _) = engine("fp8", True), engine("dense", True)
    a, b = run(same[0], [T]), run(dense, [T])
    assert (a - b).norm() <= 2 * u * b.norm()
    anyscale, _ = engine("fp8", False)
    a, b = run(anyscale, [T]), run(anyscale, [16] * (T // 16) + ([T % 16] if T % 16 else []))
    assert (a - b).norm() <= 4 * u * b.norm()


def fp8_scales(n, dt, gen):
    """Scales that a rounding to 16 bits moves by a quarter to a half of its unit."""
    u = torch.finfo(dt).eps
    return ((1 + u * (torch.randint(0, 64, (n,), generator=gen, device=DEV) + 0.25 + 0.25 * torch.rand(n, generator=gen, device=DEV))) * 0.03).float()


# the large layer: QKV of 151 MB in 16 bits, which leaves the passes at 65 tokens, gate-up of 411 MB, at 81
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,size", [(T, (512, 4, 2, 768)) for T in (48, 49, 128, 129, 300)] + [(T, (8192, 64, 4, 12544)) for T in (64, 65, 80, 81)])
def test_fp8_scales_are_not_rounded(dtype, T, size):
    """The value rows that a prompt leaves in the cache are one FP8 linear's outputs.  Its inputs are made +-1 (a norm of +-1 rows), so that the codes' sums are exact
    in fp32 and the only roundings are the product's with the scale and the result's: half a unit of the type and 2^-23.  Scales folded into rounded 16-bit weights
    break that bound.  The whole layer agrees with the same prompt sixteen tokens at a time."""
    (h, heads, kv, inter), d = size, 128
    gen = torch.Generator(device=DEV).manual_seed(T)
    code = m.BF16 if dtype == torch.bfloat16 else m.F16
    dec = m.Decoder(m.DecoderConfig(h, heads, kv, d, inter, 1, 320, 1, code, m.W_FP8, 128, 1e-6, d, 10000.0, 1, 0), DEV)
    layer = {"g1": torch.ones(h, device=DEV, dtype=dtype), "g2": torch.ones(h, device=DEV, dtype=dtype)}
    for name, n, k in (("qkv", (heads + 2 * kv) * d, h), ("o", h, heads * d), ("gate_up", 2 * inter, h), ("down", h, inter)):
        layer[name] = (torch.randn(n, k, generator=gen, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8), fp8_scales(n, dtype, gen), None)
    dec.set_layer(0, layer)
    x = torch.randint(0, 2, (T, h), generator=gen, device=DEV).to(dtype) * 2 - 1
    k, v, k2, v2 = (torch.zeros(1, 5, kv, 64, d, device=DEV, dtype=dtype) for _ in range(4))
    i32 = lambda *a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    table = torch.arange(5, dtype=torch.int32, device=DEV).reshape(1, 5)
    whole, parts = x.clone(), x.clone()
    dec.prefill_paged(whole, k, v, table, i32(T), i32(0), i32(T), T)
    for a in range(0, T, 16):
        n = min(16, T - a)
        dec.prefill_paged(parts[a:a + n], k2, v2, table, i32(n), i32(a), i32(a + n), n)
    assert (whole.double() - parts.double()).norm() <= 4 * torch.finfo(dtype).eps * parts.double().norm()
    got = v[0].permute(0, 2, 1, 3).reshape(-1, kv * d)[:T].double()
    codes, scales, _ = layer["qkv"]
    codes, scales = codes[(heads + kv) * d:].view(torch.float8_e4m3fn).double(), scales[(heads + kv) * d:].double()
    want = (x.double() @ codes.T) * scales
    bound = (0.5 * torch.finfo(dtype).eps + 2.0 ** -22) * want.abs() + torch.finfo(dtype).tiny

    def broken(rows):
        return float(((rows - want).abs() > bound).double().mean())

    folded = (x.double() @ (codes * scales[:, None]).to(dtype).double().T).to(dtype).double()
    assert broken(folded) > 0.05  # (so many outputs are more than that bound off with folded scales: 0.15 of fp16, more of bf16)
    assert broken(got) == 0.0, broken(got)
