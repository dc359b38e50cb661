"""The three-limb Goldilocks DFT (csrc/dft_goldilocks.cuh) emulated with big
integers: every value stays within the bounds its limbs and shifts need, at
inputs on the ends of their range and at random ones, and the results are the
DFT's."""
import random

import pytest

P = 2**64 - 2**32 + 1
EPS = 2**32 - 1
ONE = 2**64
BIAS_MID, BIAS_OUT, BIAS_I = 5, 28, 16
LO, HI = -(2**32) + 1, 2**65 - 1  # inputs: unreduced products


def shift(x, s, k):
    q, r = divmod(s, 32)
    assert 0 <= x < 2 ** (96 - r), "a shifted value leaves three limbs"
    y = x << r
    y0, y1, y2 = y & EPS, (y >> 32) & EPS, y >> 64
    if q == 0:
        assert k == 0
        out = y0 + (y1 << 32) + y2 * EPS
    elif q == 1:
        out = ((y0 + y1) << 32) - (y1 + y2) + (k << r)
    else:
        assert k == 0 and y2 < EPS
        out = (y0 << 32) - (y0 + y1 + (y2 << 32))
    assert (out - ((x - k * ONE) << s)) % P == 0
    assert abs(out) < 2 * ONE
    return out


def radix4(a, b, c, d, inv, nb=False, nc=False, nd=False):
    s0, d0 = (a - c, a + c) if nc else (a + c, a - c)
    s1 = b - d if nb != nd else b + d
    d1 = b + BIAS_I * ONE + (d if nb != nd else -d)
    i1 = shift(d1, 48, BIAS_I)
    add = lambda x, y, neg: x - y if neg else x + y  # noqa: E731
    return add(s0, s1, nb), add(d0, i1, nb != inv), add(s0, s1, not nb), add(d0, i1, nb == inv)


def root_pow(logr, k, inv):
    e = 39 * (64 >> logr) * k % 192
    return (192 - e) % 192 if inv else e


def twiddle(x, e):
    return x if e % 96 == 0 else shift(x, e % 96, 0)


def dft(v, logr, inv):
    if logr == 1:
        a = v[0] + BIAS_MID * P
        return [a + v[1], a - v[1]]
    if logr == 2:
        return list(radix4(v[0] + BIAS_MID * P, *v[1:], inv))
    m = 1 << (logr - 2)
    u = [list(radix4(v[j] + (BIAS_MID if j else BIAS_OUT) * P, v[j + m], v[j + 2 * m], v[j + 3 * m], inv))
         for j in range(m)]
    out = [0] * (4 * m)
    for k in range(4):
        e = [root_pow(logr, j * k, inv) if j else 0 for j in range(m)]
        w = [u[0][k]] + [twiddle(u[j][k], e[j]) for j in range(1, m)]
        if m == 2:
            out[k], out[k + 4] = (w[0] - w[1], w[0] + w[1]) if e[1] >= 96 else (w[0] + w[1], w[0] - w[1])
        else:
            out[k], out[k + 4], out[k + 8], out[k + 12] = radix4(*w, inv, *[x >= 96 for x in e[1:]])
    return out


def fold(x):
    assert 0 <= x < 2**71
    r = (x & (ONE - 1)) + (x >> 64) * EPS
    r = (r & (ONE - 1)) + (r >> 64) * EPS
    assert 0 <= r < ONE, "the fold carries twice"
    return r


@pytest.mark.parametrize("logr", [1, 2, 3, 4])
@pytest.mark.parametrize("inv", [False, True])
def test_three_limb_dft(logr, inv):
    rng = random.Random(logr * 2 + inv)
    n = 1 << logr
    w = pow(7, (P - 1) // n, P)
    if inv:
        w = pow(w, P - 2, P)
    pools = [lambda: rng.choice([LO, HI, 0]), lambda: rng.randrange(LO, HI),
             lambda: rng.choice([0, 1, P - 1, P, ONE - 1, 2**32, 2**63])]
    for it in range(600):
        v = [pools[it % 3]() for _ in range(n)]
        out = [fold(x) for x in dft(v, logr, inv)]
        if it < 60:
            for k in range(n):
                assert (out[k] - sum(v[j] * pow(w, j * k, P) for j in range(n))) % P == 0


def test_product_reduction_bounds():
    """reduce3 leaves (-2^32, 2^65) and fold_small one word for any 128-bit
    product, with an addend too."""
    rng = random.Random(5)
    ends = [0, 1, 2**32 - 1, 2**32, P - 1, P, ONE - 1, ONE - 2**32]
    for it in range(3000):
        a, b, c = ([rng.choice(ends) for _ in range(3)] if it % 2 else [rng.randrange(ONE) for _ in range(3)])
        x = a * b + c
        assert x < 2**128
        lo, h0, h1 = x & (ONE - 1), (x >> 64) & EPS, x >> 96
        r = lo + h0 * EPS - h1
        assert -(2**32) < r < 2 * ONE
        x2 = r >> 64
        assert x2 in (-1, 0, 1)
        word = (r & (ONE - 1)) + x2 * EPS
        assert 0 <= word < ONE and (word - x) % P == 0
