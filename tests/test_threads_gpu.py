"""Threads that call with different sizes, and threads whose first call this is: what one of them launches depends on no other call."""
import threading

import pytest
import torch

import util

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
b200 = util.b200()


@pytest.mark.parametrize("m", [1, 2, 16, 200])
@pytest.mark.parametrize("fmt", ["dense", "fp8", "int4"])
def test_linears_of_two_threads(fmt, m):
    """A large linear, a small one of the same kernel from a thread that has not called before, the large one again."""
    if fmt != "dense" and m > 16:
        pytest.skip("linears of quantised weights are the engine's at prompt sizes")
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


def test_a_thread_that_begins_with_attention():
    """Prompt attention as the first call of a thread: the tensor maps want a context, which such a thread has not got yet."""
    gen = torch.Generator(device=DEV).manual_seed(7)
    h, hkv, n, d = 4, 2, 200, 128
    q, k, v = (torch.randn(1, x, n, d, generator=gen, device=DEV).bfloat16() for x in (h, hkv, hkv))
    one = lambda x: torch.tensor([x], dtype=torch.int32, device=DEV)
    pad, length = torch.zeros(n, dtype=torch.int32, device=DEV), one(n)
    call = lambda: b200.context_attention(q, k[None], v[None], pad, length, length, 0, n, d**-0.5)
    want, got, failed = call(), [], []

    def other():
        try:
            got.append(call())
        except b200.B200Error as e:
            failed.append(e)

    t = threading.Thread(target=other)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not failed and torch.equal(got[0], want)
