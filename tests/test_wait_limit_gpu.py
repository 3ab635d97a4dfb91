"""Waits inside kernels that run out (csrc/common.cuh, WaitGuard): the kernel returns, what it could not form is NaN, the next call says so, and after the
word is cleared the same call gives what it gave before.  The limit of zero that brings this about takes nothing out of the kernels: every wait still
ends, only earlier, and a CTA stays until its own copies and products are done."""
import ctypes
import math

import pytest
import torch

import util

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
b200 = util.b200()
GEMV, PAIR, PROMPT, PROBE, GEMM = 1, 2, 3, 4, 5


@pytest.fixture(autouse=True)
def word_cleared():
    assert b200.wait_error() == 0
    yield
    b200.lib().b200_wait_limit(2 ** 32 - 1)
    torch.cuda.synchronize()
    b200.wait_error(clear=True)


def run_out(call, code):
    """One launch whose waits run out at once."""
    torch.cuda._sleep(5_000_000)  # (the launch has returned before its kernel starts)
    b200.lib().b200_wait_limit(0)
    out = call()
    b200.lib().b200_wait_limit(2 ** 32 - 1)
    torch.cuda.synchronize()
    assert b200.wait_error() == code
    with pytest.raises(b200.B200Error, match="ran out"):
        call()
    torch.cuda.synchronize()
    assert b200.wait_error(clear=True) == code and b200.wait_error() == 0
    return out


def test_a_barrier_that_nothing_arrives_at():
    """The limit is some thousand clocks; the kernel returns and its code comes back, once, from every call until it is cleared."""
    lib = b200.lib()
    lib.b200_wait_limit(5000)
    b200.check(lib.b200_wait_probe(b200.stream()))
    lib.b200_wait_limit(2 ** 32 - 1)
    torch.cuda.synchronize()
    assert b200.wait_error() == PROBE
    x, w = torch.ones(4, 256, device=DEV).bfloat16(), torch.ones(64, 256, device=DEV).bfloat16()
    for _ in range(2):
        with pytest.raises(b200.B200Error, match="wait probe ran out"):
            b200.linear(x, w)
    assert b200.wait_error(clear=True) == PROBE
    assert bool((b200.linear(x, w) == 256).all())


def streamed(fmt, m, k, n):
    """A linear's call."""
    gen = torch.Generator(device=DEV).manual_seed(k + n + m)
    x = torch.randn(m, k, generator=gen, device=DEV).bfloat16()
    kw = {}
    if fmt == "dense":
        w = torch.randn(n, k, generator=gen, device=DEV).bfloat16()
    elif fmt == "fp8":
        w = torch.randn(n, k, generator=gen, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8)
        kw = dict(w_format=b200.W_FP8, scales=torch.ones(n, device=DEV), N=n)
    else:
        w = torch.randint(0, 256, (n, k // 2), generator=gen, device=DEV, dtype=torch.uint8)
        kw = dict(w_format=b200.W_INT4, scales=torch.ones(n, k // 128, device=DEV).bfloat16(), zeros=torch.full((n, k // 128), 8, device=DEV, dtype=torch.uint8), group=128, N=n)
    return lambda: b200.linear(x, w, **kw)


@pytest.mark.parametrize("fmt,m,k,n", [("fp8", m, k, n) for m in (2, 13) for k, n in ((256, 40), (2048, 4736), (8192, 2400))]
                         + [("int4", 13, k, n) for k, n in ((256, 40), (2048, 4736), (8192, 2400))] + [("int4", 8, 11008, 2400)]
                         + [("dense", m, k, n) for m in (2, 13) for k, n in ((3200, 40), (4096, 4736), (8192, 2400))])
def test_streaming_gemv(fmt, m, k, n):
    call = streamed(fmt, m, k, n)
    want = call()
    got = run_out(call, GEMV)
    assert bool(torch.isnan(got).all())
    assert torch.equal(call(), want) and not bool(torch.isnan(want).any())


@pytest.mark.parametrize("fmt,m,k,n", [("int4", m, k, n) for m in (1, 2, 8) for k, n in ((256, 40), (2048, 4736), (8192, 2400))]
                         + [("dense", m, k, n) for m in (1, 2, 13) for k, n in ((256, 40), (2048, 4736), (3072, 2400))])
def test_linears_without_a_wait(fmt, m, k, n):
    """The limit is no choice between kernels: a linear that streams into registers waits for no barrier, whatever the limit."""
    call = streamed(fmt, m, k, n)
    want = call()
    b200.lib().b200_wait_limit(0)
    got = call()
    b200.lib().b200_wait_limit(2 ** 32 - 1)
    torch.cuda.synchronize()
    assert b200.wait_error() == 0
    assert torch.equal(got, want) and not bool(torch.isnan(want).any())


@pytest.mark.parametrize("m,k,n", [(512, 64, 4928), (2048, 128, 4096)])
def test_pair_gemm(m, k, n):
    gen = torch.Generator(device=DEV).manual_seed(k + n + m)
    x, w = (torch.randn(r, k, generator=gen, device=DEV).bfloat16() for r in (m, n))
    for call in (lambda: b200.linear(x, w), lambda: b200.linear_swiglu(x, w)):
        want = call()
        got = run_out(call, PAIR)
        assert bool(torch.isnan(got).all())
        assert torch.equal(call(), want) and not bool(torch.isnan(want).any())


@pytest.mark.parametrize("m,k,n", [(17, 64, 16), (94, 2048, 2048), (300, 2048, 512), (100, 512, 64000), (17, 11008, 4096), (256, 28672, 1024)])
def test_one_cta_gemm(m, k, n):
    """Tiles of their own, one and several a CTA, and (the last two) tiles whose k two CTAs share."""
    gen = torch.Generator(device=DEV).manual_seed(k + n + m)
    x, w = (torch.randn(r, k, generator=gen, device=DEV).bfloat16() for r in (m, n))
    bias = torch.randn(n, generator=gen, device=DEV)
    calls = [lambda: b200.linear(x, w), lambda: b200.linear_act(x, w, bias, 3)]  # (a rectifier would make a number of NaN)
    if m > 128 and n >= 256:
        calls.append(lambda: b200.linear_swiglu(x, w))
    for call in calls:
        want = call()
        got = run_out(call, GEMM)
        assert bool(torch.isnan(got).all())
        assert torch.equal(call(), want) and not bool(torch.isnan(want).any())


@pytest.mark.parametrize("m,k,n", [(94, 2048, 2048), (100, 512, 64000), (300, 4096, 12288), (17, 11008, 4096), (256, 28672, 1024)])
def test_one_cta_gemm_that_gives_up_halfway(m, k, n):
    """Limits of the order of what a launch waits for, so that some CTAs give up with copies and products under way: what a CTA stores is either right or NaN, and the
    next call is what it was."""
    gen = torch.Generator(device=DEV).manual_seed(k + n + m)
    x, w = (torch.randn(r, k, generator=gen, device=DEV).bfloat16() for r in (m, n))
    want = b200.linear(x, w)
    for clocks in (1, 300, 1000, 2000, 4000, 8000, 2 ** 31 - 1):
        b200.lib().b200_wait_limit(clocks)
        got = b200.linear(x, w)
        b200.lib().b200_wait_limit(2 ** 32 - 1)
        torch.cuda.synchronize()
        code = b200.wait_error(clear=True)
        lost = torch.isnan(got)
        assert code in (0, GEMM) and bool((lost | (got == want)).all())
        assert bool(lost.any()) == (code == GEMM) and (clocks < 2 ** 30 or code == 0)
        assert torch.equal(b200.linear(x, w), want)


@pytest.mark.parametrize("window", [0, 100])
def test_prompt_attention(window):
    """Two prompts of 200 and 70 tokens, four query heads on two kv heads of 128; with a window also the distance penalty."""
    gen = torch.Generator(device=DEV).manual_seed(window)
    heads, kv, d = 4, 2, 128
    q = torch.randn(270, heads, d, generator=gen, device=DEV).bfloat16()
    pools = [torch.randn(6, kv, 64, d, generator=gen, device=DEV).bfloat16() for _ in range(2)]
    table = torch.tensor([[0, 1, 2, 3], [4, 5, 0, 0]], dtype=torch.int32, device=DEV)
    tiles = torch.tensor([[0, t, min(64, 200 - t), t] for t in range(0, 200, 64)] + [[1, 200 + t, min(64, 70 - t), t] for t in range(0, 70, 64)],
                         dtype=torch.int32, device=DEV)
    r1, r2 = (torch.rand(heads, generator=gen, device=DEV) + 0.2 for _ in range(2))
    ptr = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731

    def call():
        out = torch.zeros(270, heads * d, device=DEV).bfloat16()
        b200.check(b200.lib().b200_scored_attention_tiles_paged(ptr(q), ptr(pools[0]), ptr(pools[1]), None, ptr(r1 if window else None), ptr(r2 if window else None), None, 0,
                                                                ptr(out), heads * d, 1.0, ptr(tiles), len(tiles), ptr(table), 4, heads, kv, d, d, 1 / math.sqrt(d), window, 0,
                                                                b200.BF16, b200.stream()))
        return out

    want = call()
    got = run_out(call, PROMPT)
    assert bool(torch.isnan(got).all())
    assert torch.equal(call(), want) and not bool(torch.isnan(want).any())
