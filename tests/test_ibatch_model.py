"""CPU model of the interval-batched FP64 operator's arithmetic (csrc/sg_ibatch.cu).

Replays, with Python integers, how one pair's contribution is formed: 60-bit fixed-point operands under
power-of-two scales, six signed 10-bit digits, digit products summed per weight (each sum an integer
that FP32 holds exactly), 64-bit combination of digits and real / imaginary parts, and the two half sums
in t. Bounds: every accumulator within 2^24, the 64-bit combination within 2^63, and the result against
extended-precision values within 2^-52 of the sum of the absolute products (FP64's own rounding level).
"""
import math

import numpy as np
import pytest

BIAS = 512 * sum(1 << (10 * i) for i in range(6))


def fixed(v, scale):
    """The kernel's ib_fixed: trunc(|v| 2^(59 - scale)) with v's sign, offset by the digits' bias."""
    m, e = math.frexp(abs(v))
    m53, below = int(m * (1 << 53)), scale - e
    assert v == 0 or below >= 0
    f = (m53 << 6) >> below if v else 0
    return BIAS - f if v < 0 else BIAS + f


def digits(f):
    return [(f >> 50) - 512] + [((f >> (10 * (5 - s))) & 1023) - 512 for s in range(1, 6)]


def exponent(values):
    return max((math.frexp(v)[1] for v in values if v), default=0)


def combine(rows, cols):
    """64-bit combination (units of 2^-56 of the scales) of digit vectors rows[k], cols[k]."""
    D = [sum(r[i] * c[d - i] for r, c in zip(rows, cols) for i in range(d + 1)) for d in range(6)]
    assert max(abs(v) for v in D) <= 1 << 24
    hi = (D[0] << 20) + (D[1] << 10) + D[2]
    lo = (D[3] << 20) + (D[4] << 10) + D[5]
    return (hi << 18) + ((lo + 2048) >> 12)


def test_digits_reproduce_fixed_point():
    rng = np.random.default_rng(1)
    for v in list(rng.standard_normal(200) * 10.0 ** rng.integers(-9, 1, 200)) + [0.0, 1 - 2.0 ** -53, -(1 - 2.0 ** -53), 2.0 ** -59]:
        f = fixed(float(v), max(0, math.frexp(v)[1]))
        d = digits(f)
        assert all(-512 <= x <= 512 for x in d) and sum(x << (10 * (5 - s)) for s, x in enumerate(d)) == f - BIAS


@pytest.mark.parametrize("bs,coefs,spread", [(1, 2, 1.0), (7, 4, 1.0), (30, 4, 1e-3), (32, 4, 1.0), (32, 2, 1e-6)])
def test_pair_contribution_is_fp64_grade(bs, coefs, spread):
    rng = np.random.default_rng(bs + coefs)
    C = rng.standard_normal((coefs, bs, bs, 2)) * 10.0 ** -np.arange(coefs)[:, None, None, None]
    C *= spread ** rng.random((1, 1, bs, 1))       # columns of very different size
    u = rng.standard_normal((bs, 2)) * spread ** rng.random((bs, 1))
    if bs == 32:  # largest digits everywhere: the accumulators' and the combination's worst case
        C[:], u[:] = 1 - 2.0 ** -53, 1 - 2.0 ** -53
    t = float(rng.random())
    eb = [exponent(C[:, :, n2].ravel()) for n2 in range(bs)]
    ea = [max(exponent(C[:, n1, n2].ravel()) - eb[n2] for n2 in range(bs)) for n1 in range(bs)]
    ec = max(exponent(u[n2]) + eb[n2] for n2 in range(bs))
    half = [[[digits(fixed(float(w * u[n2, p]), ec - eb[n2])) for n2 in range(bs)] for p in range(2)] for w in (1.0, t * t)]
    for n1 in range(min(bs, 4)):
        parity = []
        for odd in range(2):
            w = {}
            for part in range(2):       # Re, Im of C
                rows = [digits(fixed(float(C[c, n1, n2, part]), ea[n1] + eb[n2])) for c in range(odd, coefs, 2) for n2 in range(bs)]
                for p in range(2):      # Re, Im of u
                    w[part, p] = combine(rows, [x for h in range(coefs // 2) for x in half[h][p]])
            pair = (w[0, 0] - w[1, 1], w[0, 1] + w[1, 0])
            assert all(abs(v) < 1 << 63 for v in pair)
            parity.append([math.ldexp(float(v), ea[n1] + ec - 56) for v in pair])
        got = np.array([parity[0][p] + t * parity[1][p] for p in range(2)])
        q = np.longdouble(t) ** np.arange(coefs)[:, None, None]
        L = (q * C[:, n1].astype(np.longdouble)).sum(0)
        ul = u.astype(np.longdouble)
        want = np.array([(L[:, 0] * ul[:, 0] - L[:, 1] * ul[:, 1]).sum(), (L[:, 0] * ul[:, 1] + L[:, 1] * ul[:, 0]).sum()])
        size = float((np.abs(L).sum(1) * np.abs(ul).sum(1)).sum())
        assert np.abs(got - want).max() <= 2.0 ** -52 * size + 2.0 ** -55 * math.ldexp(1.0, ea[n1] + ec)
