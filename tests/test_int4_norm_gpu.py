"""One INT4 token with its residual add and RMSNorm inside the linear (csrc/gemv_qd.cuh, NORM) against two tokens of the same engine, whose norm is a kernel: the
first token's hidden row and cache rows agree in every bit, for rows shorter and longer than the norm kernel's threads and for every form of the linear (K of 256 to
8192), from a first layer without a residual to layers with one."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
m = importlib.import_module("llm-inference-engine_b200")
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("h,inter", [(256, 384), (1024, 1408), (2048, 2688), (4096, 512), (4224, 256), (5120, 640), (8192, 256)])
def test_same_bits_as_the_norm_kernel(dtype, h, inter):
    heads, d, layers = max(h // 512, 1), 128, 3
    gen = torch.Generator(device=DEV).manual_seed(h)
    code = m.BF16 if dtype == torch.bfloat16 else m.F16

    def weight(n, k):
        return (torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8),
                (torch.rand(n, k // 128, generator=gen, device=DEV) * 0.1 / k ** 0.5 + 0.17 / k ** 0.5).to(dtype), torch.randint(7, 9, (n, k // 128), generator=gen, device=DEV, dtype=torch.uint8))

    weights = [{"g1": (torch.randn(h, generator=gen, device=DEV) * 0.1 + 1).to(dtype), "g2": (torch.randn(h, generator=gen, device=DEV) * 0.1 + 1).to(dtype), "qkv": weight(3 * heads * d, h),
                "o": weight(h, heads * d), "gate_up": weight(2 * inter, h), "down": weight(h, inter)} for _ in range(layers)]
    x = torch.randn(1, h, generator=gen, device=DEV).to(dtype)
    out = []
    for batch in (1, 2):
        dec = m.Decoder(m.DecoderConfig(h, heads, heads, d, inter, layers, 64, batch, code, m.W_INT4, 128, 1e-6, d, 10000.0, 1, 0), DEV)
        for i, w in enumerate(weights):
            dec.set_layer(i, w)
        hidden = x.repeat(batch, 1).contiguous()
        k, v = (torch.zeros(layers, batch, heads, 64, d, device=DEV, dtype=dtype) for _ in range(2))
        dec.step(hidden, k, v, 1)
        out.append((hidden[0].clone(), k[:, 0].clone(), v[:, 0].clone()))
    assert not bool(torch.isnan(out[0][0]).any())
    for a, b in zip(*out):
        assert torch.equal(a, b)
