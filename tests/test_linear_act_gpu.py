"""A linear's ending (b200_linear_act): bias and activation in the linear's kernel give every bit of the linear and the pass over its stored rows (in torch: a
rounded row, an fp32 bias added, the activation in fp32, rounded).  Sizes on both sides of each kernel's range: rows of 1, 8, 9, 16 | 17, 128 | 129 and more, short
and long k, columns that do not fill a tile, and biases that start on no 16-byte boundary."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
m = importlib.import_module("llm-inference-engine_b200")

ACTS = {-1: lambda v: v, 0: lambda v: torch.relu(v) ** 2, 3: torch.relu}  # exact in fp32; the others (SiLU, tanh GELU) are compared with a unit in the last place


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("M,K,N", [(1, 256, 40), (1, 4096, 136), (8, 2048, 1000), (9, 2048, 2064), (16, 3072, 24), (16, 8192, 520), (17, 512, 256), (128, 128, 384),
                                   (129, 64, 16), (200, 512, 1000), (1030, 256, 2056), (2300, 128, 4104)])
def test_ending_is_the_pass(dtype, M, K, N):
    gen = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, generator=gen, device="cuda").to(dtype)
    w = (torch.randn(N, K, generator=gen, device="cuda") / K ** 0.5).to(dtype)
    bias = torch.randn(N + 1, generator=gen, device="cuda")[1:]
    row = m.linear(x, w).float()
    for b in (None, bias):
        for act, fn in ACTS.items():
            want = fn(row + b if b is not None else row).to(dtype)
            assert torch.equal(m.linear_act(x, w, b, act), want), (act, b is None)
        v = row + b if b is not None else row
        for act, fn in ((1, torch.nn.functional.silu), (2, lambda z: torch.nn.functional.gelu(z, approximate="tanh"))):
            want = fn(v.double())
            eps = torch.finfo(dtype).eps  # half a unit of the type's rounding, and some of fp32 in the exponential or the tangent
            assert ((m.linear_act(x, w, b, act).double() - want).abs() <= 0.51 * eps * want.abs() + 4e-6 * (1 + v.abs().double())).all(), act


def test_refusals():
    x, w = torch.zeros(2, 64, device="cuda"), torch.zeros(8, 64, device="cuda")
    for act in (-2, 4, 5):
        with pytest.raises(Exception):
            m.linear_act(x, w, None, act)
