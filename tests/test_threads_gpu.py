"""Threads that call with different sizes: what one of them launches does not depend on what another launched before."""
import threading

import pytest
import torch

import util

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
b200 = util.b200()


@pytest.mark.parametrize("m", [1, 2, 16])
@pytest.mark.parametrize("fmt", ["dense", "fp8", "int4"])
def test_linears_of_two_threads(fmt, m):
    """A large linear, a small one of the same kernel from a thread that has not called before, the large one again."""
    gen = torch.Generator(device=DEV).manual_seed(m)

    def linear(k, n):
        x = torch.randn(m, k, generator=gen, device=DEV).bfloat16()
        if fmt == "dense":
            w = torch.randn(n, k, generator=gen, device=DEV).bfloat16()
            return lambda: b200.linear(x, w)
        if fmt == "fp8":
            w, s = torch.randn(n, k, generator=gen, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8), torch.ones(n, device=DEV)
            return lambda: b200.linear(x, w, w_format=b200.W_FP8, scales=s, N=n)
        w = torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8)
        s, z = torch.ones(n, k // 128, device=DEV).bfloat16(), torch.full((n, k // 128), 8, device=DEV, dtype=torch.uint8)
        return lambda: b200.linear(x, w, w_format=b200.W_INT4, scales=s, zeros=z, group=128, N=n)

    large, small, failed = linear(4096, 4096), linear(128, 64), []

    def other():
        try:
            small()
        except b200.B200Error as e:
            failed.append(e)

    want = large()
    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert not failed and torch.equal(large(), want)
