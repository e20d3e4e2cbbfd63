"""CPU model of the interval-batched FP64 operator's arithmetic (csrc/sg_ibatch.cu).

Replays, with Python integers, how one pair's contribution is formed: 63-bit fixed-point operands under
power-of-two scales, seven signed 9-bit digits, digit products summed per weight (each sum an integer
that FP32 holds exactly), 64-bit combination of digits and real / imaginary parts, powers of t and the
rotation from 31-bit words. Bounds: every accumulator within 2^24, every 64-bit sum within 2^63, and the
result against extended-precision values within 2^-52 of the sum of the absolute products (FP64's own
rounding level) plus two of the kernel's last places.
"""
import math

import numpy as np
import pytest

BITS, DIGITS = 9, 7
BIAS = sum(1 << (BITS * i + BITS - 1) for i in range(DIGITS))


def fixed(v, scale):
    """The kernel's ib_fixed: trunc(|v| 2^(62 - scale)) with v's sign."""
    m, e = math.frexp(abs(v))
    m53, below = int(m * (1 << 53)), scale - e
    assert v == 0 or below >= 0
    f = (m53 << 9) >> below if v else 0
    return -f if v < 0 else f


def digits(f):
    f += BIAS
    assert f >= 0
    top = f >> (BITS * (DIGITS - 1))
    return [top - 256] + [((f >> (BITS * (DIGITS - 1 - s))) & 511) - 256 for s in range(1, DIGITS)]


def exponent(values):
    return max((math.frexp(v)[1] for v in values if v), default=0)


def s64(v):
    assert -(1 << 63) <= v < 1 << 63
    return v


def s32(v):
    assert -(1 << 31) <= v < 1 << 31
    return v


def split(v):
    return s32(v >> 31), v & 0x7FFFFFFF


def split_signed(v):
    h = (v + (1 << 30)) >> 31
    return s32(h), s32(v - (h << 31))


def mul(a, b, c):
    mid = s64(a[0] * b[1] + a[1] * b[0] + (1 << 30))
    return s64(a[0] * b[0] + c + (mid >> 31))


def combine(rows, cols):
    """64-bit combination (units of 2^-55 of the scales) of digit vectors rows[k], cols[k]."""
    D = [sum(r[i] * c[d - i] for r, c in zip(rows, cols) for i in range(d + 1)) for d in range(DIGITS)]
    assert max(abs(v) for v in D) <= 1 << 24 and max(abs(D[0]), abs(D[1])) < 1 << 22
    low = round((D[5] + D[6] / 512) / 64)
    assert abs(low) < 1 << 22
    w = s32(low + s32(D[4] * 8))
    return s64(w + (D[3] << 12) + (D[2] << 21) + (D[1] << 30) + (s32(D[0] << 7) << 32))


def test_digits_reproduce_fixed_point():
    rng = np.random.default_rng(1)
    for v in list(rng.standard_normal(200) * 10.0 ** rng.integers(-9, 1, 200)) + [0.0, 1 - 2.0 ** -53, -(1 - 2.0 ** -53),
                                                                                 2.0 ** -62]:
        f = fixed(float(v), max(0, math.frexp(v)[1]))
        d = digits(f)
        assert all(-256 <= x <= 256 for x in d) and sum(x << (BITS * (DIGITS - 1 - s)) for s, x in enumerate(d)) == f


def test_accumulators_stay_exact_for_the_largest_digits():
    """All digits at their largest magnitude: 7 x 30 products of 2^16 per accumulator, within 2^24."""
    worst = [[-256] * DIGITS] * 30
    D = [sum(r[i] * c[d - i] for r, c in zip(worst, worst) for i in range(d + 1)) for d in range(DIGITS)]
    assert max(D) == 7 * 30 * 65536 <= 1 << 24


@pytest.mark.parametrize("bs,coefs,spread", [(1, 2, 1.0), (7, 4, 1.0), (29, 4, 1e-3), (30, 4, 1.0), (30, 2, 1e-6)])
def test_pair_contribution_is_fp64_grade(bs, coefs, spread):
    rng = np.random.default_rng(bs + coefs)
    C = rng.standard_normal((coefs, bs, bs, 2)) * 10.0 ** -np.arange(coefs)[:, None, None, None]
    C *= spread ** rng.random((1, 1, bs, 1))       # columns of very different size
    x = rng.standard_normal((bs, 2)) * spread ** rng.random((bs, 1))
    if bs == 30 and coefs == 4:  # the 64-bit sums' worst case
        C[:], x[:] = 1 - 2.0 ** -53, 1 - 2.0 ** -53
    m = rng.integers(-3, 4, bs)
    phi, t = float(rng.uniform(0, 6.28)), float(rng.random())
    z = [1.0 + 0.0j]  # e^{i m phi} in FP64 by repeated multiplication, the values both sides use
    for _ in range(3):
        z.append(z[-1] * complex(math.cos(phi), math.sin(phi)))
    cs = {a: (split_signed(int(z[a].real * 2 ** 61)), split_signed(int(z[a].imag * 2 ** 61))) for a in range(4)}
    phase = np.array([z[abs(a)] if a >= 0 else z[-a].conjugate() for a in m]).astype(np.clongdouble)
    tw = split_signed(int(t * 2 ** 62))
    eb = [exponent(C[:, :, n2].ravel()) for n2 in range(bs)]
    ea = [max(exponent(C[:, n1, n2].ravel()) - eb[n2] for n2 in range(bs)) for n1 in range(bs)]
    ec = max(exponent(x[n2]) + eb[n2] for n2 in range(bs))

    def rotate(p, q, mm, sign, half):
        """(p + i q) e^{i sign mm phi} from words; half: half of it."""
        (ch, cl), (sh, sl) = cs[abs(mm)]
        if (mm < 0) != (sign < 0):
            sh, sl = -sh, -sl
        out = []
        for (a, b, g) in ((split(p), split(q), -1), (split(q), split(p), 1)):
            mid = s64(a[0] * cl + a[1] * ch + b[0] * g * sl + b[1] * g * sh + (1 << (30 if half else 29)))
            hh = a[0] * ch + b[0] * g * sh
            out.append(s64(hh + (mid >> 31)) if half else s64(2 * hh + (mid >> 30)))
        return out

    u = [rotate(fixed(float(x[n, 0]), ec - eb[n]), fixed(float(x[n, 1]), ec - eb[n]), int(m[n]), 1, True) for n in range(bs)]
    cols = [[digits(u[n][p]) for n in range(bs)] for p in range(2)]
    xl = (x[:, 0] + 1j * x[:, 1]).astype(np.clongdouble)
    ul = xl * phase
    for n1 in range(min(bs, 4)):
        acc = [0, 0]
        for c in range(coefs - 1, -1, -1):
            rows = [[digits(fixed(float(C[c, n1, n2, part]), ea[n1] + eb[n2])) for n2 in range(bs)] for part in range(2)]
            w = {(part, p): combine(rows[part], cols[p]) for part in range(2) for p in range(2)}
            e = (s64(w[0, 0] - w[1, 1]), s64(w[0, 1] + w[1, 0]))
            acc = list(e) if c == coefs - 1 else [mul(split(acc[p]), tw, e[p]) for p in range(2)]
        out = rotate(acc[0], acc[1], int(m[n1]), -1, False)
        unit = math.ldexp(1.0, ea[n1] + ec + 1 - 55)
        got = complex(out[0] * unit, out[1] * unit)
        L = ((np.longdouble(t) ** np.arange(coefs))[:, None, None] * C[:, n1].astype(np.longdouble)).sum(0)
        L = L[:, 0] + 1j * L[:, 1]
        want = (L * ul).sum() * phase[n1].conjugate()
        size = float((np.abs(L) * np.abs(ul)).sum())
        assert abs(got - complex(want)) <= 2.0 ** -52 * size + 2 * unit
