"""The sampler's jump polynomials (csrc/sampling.cu, kJump) from the recurrence alone.  A XORWOW state is five 32-bit words under a linear map over GF(2)
(G. Marsaglia, "Xorshift RNGs", 2003); its characteristic polynomial p comes out of any one bit's sequence (Berlekamp-Massey), and the coefficients that carry a
state 2^67 b steps on are those of x^(2^67 b) mod p (H. Haramoto et al., "Efficient jump ahead for F2-linear random number generators", 2008)."""
import os
import random
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-inference-engine_b200", "csrc", "sampling.cu")
MASK = 0xFFFFFFFF


def step(s):
    t = s[0] ^ (s[0] >> 2)
    return (*s[1:], (s[4] ^ (s[4] << 4)) & MASK ^ (t ^ (t << 1)) & MASK)


def characteristic():
    """p as an integer, bit i the coefficient of x^i."""
    s, bits = (1, 2, 3, 4, 0x12345), []
    for _ in range(700):
        bits.append(s[0] & 1)
        s = step(s)
    c, b, length, gap = 1, 1, 0, 1
    for n, bit in enumerate(bits):
        if sum((c >> i & 1) & bits[n - i] for i in range(length + 1)) & 1:
            c, old = c ^ b << gap, c
            if 2 * length <= n:
                length, b, gap = n + 1 - length, old, 0
        gap += 1
    assert length == 160
    return sum((c >> i & 1) << length - i for i in range(length + 1))


P = characteristic()


def mul(a, b):
    r = 0
    while b:
        if b & 1:
            r ^= a
        b >>= 1
        a <<= 1
        if a >> 160 & 1:
            a ^= P
    return r


def jump(s, poly):
    """The state whose step count is that of x^n = poly mod p: the sum of the states j steps on with a coefficient."""
    out = [0] * 5
    for j in range(160):
        if poly >> j & 1:
            out = [a ^ b for a, b in zip(out, s)]
        s = step(s)
    return tuple(out)


def test_a_jump_is_that_many_steps():
    rng = random.Random(1)
    s = tuple(rng.getrandbits(32) for _ in range(5))
    for n in (1, 159, 160, 161, 1000):
        x, base, e, t = 1, 2, n, s
        while e:
            x, base, e = mul(x, base) if e & 1 else x, mul(base, base), e >> 1
        for _ in range(n):
            t = step(t)
        assert jump(s, x) == t, n


def test_the_table():
    text = open(SOURCE).read()
    table = text[text.index("kJump[15 * kJumpDigits][5] = {"):]
    rows = re.findall(r"\{(0x[0-9a-f]{8}u(?:, 0x[0-9a-f]{8}u){4})\}", table[:table.index("};")])
    got = [sum(int(w.strip(" u"), 16) << 32 * i for i, w in enumerate(r.split(","))) for r in rows]
    base = 2
    for _ in range(67):  # x^(2^67)
        base = mul(base, base)
    want = []
    for _ in range(4):
        acc = 1
        for _ in range(15):
            acc = mul(acc, base)
            want.append(acc)
        base = mul(acc, base)
    assert got == want
