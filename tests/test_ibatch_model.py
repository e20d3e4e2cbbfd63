"""CPU model of the interval-batched FP64 operator's arithmetic (csrc/sg_ibatch.cu).

Replays, with Python integers, how one pair's contribution is formed, for both digit sizes (9 bits up to
blocksize 30, 8 bits up to 48): fixed-point operands under power-of-two scales, seven signed digits, digit
products of real and imaginary parts summed per weight in FP32, 64-bit combination of digits, powers of t
and the rotation from 31-bit words. Bounds: exact accumulators within 2^24, every 64-bit sum within 2^63,
and the result against extended-precision values within 2^-52 of the sum of the absolute products (FP64's
own rounding level) plus two of the kernel's last places (8-bit digits: plus one for every pair of operands,
each cut at half a place).
"""
import math

import numpy as np
import pytest

DIGITS = 7
MAGIC_LIMIT = 1 << 22


class Form:
    def __init__(self, bits, up, unit, jobs, maxb, exact, whole, low):
        self.bits, self.up, self.unit, self.jobs, self.maxb, self.exact, self.whole, self.low = (
            bits, up, unit, jobs, maxb, exact, whole, low)
        self.bias = sum(1 << (bits * i + bits - 1) for i in range(DIGITS))


# weights that are exact in FP32 whatever the digits; units of the whole weights; factors of the others
SMALL = Form(9, 9, 55, 7, 30, 4, (1 << 39, 1 << 30, 1 << 21, 1 << 12, 8), (2.0 ** -6, 2.0 ** -15))
LARGE = Form(8, 2, 54, 8, 48, 8, (1 << 40, 1 << 32, 1 << 24, 1 << 16, 1 << 8, 1), (2.0 ** -8, 2.0 ** -16))


def fixed(v, scale, up):
    """The kernel's ib_fixed: trunc(|v| 2^(53 + up - scale)) with v's sign."""
    m, e = math.frexp(abs(v))
    m53, below = int(m * (1 << 53)), scale - e
    assert v == 0 or below >= 0
    f = (m53 << up) >> below if v else 0
    return -f if v < 0 else f


def digits(f, q):
    f += q.bias
    assert f >= 0
    half, mask = 1 << (q.bits - 1), (1 << q.bits) - 1
    top = f >> (q.bits * (DIGITS - 1))
    return [top - half] + [((f >> (q.bits * (DIGITS - 1 - s))) & mask) - half for s in range(1, DIGITS)]


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


def combine(rows, cols, q):
    """64-bit combination (units of 2^-unit of the scales) of digit vectors rows[k], cols[k]."""
    D = [sum(r[i] * c[d - i] for r, c in zip(rows, cols) for i in range(DIGITS) if 0 <= d - i < DIGITS)
         for d in range(q.jobs)]
    assert max(abs(v) for v in D[:q.exact]) <= 1 << 24 and abs(D[0]) < MAGIC_LIMIT
    D = [int(np.float32(v)) for v in D]
    n = len(q.whole)
    low = np.float32(D[n]) * np.float32(q.low[0]) + np.float32(D[n + 1]) * np.float32(q.low[1])
    assert abs(low) < MAGIC_LIMIT
    # the least whole weight and the rest share a word whose offset leaves room for 2^28
    small = int(np.rint(low)) + q.whole[-1] * D[n - 1]
    assert abs(small) < 1 << 28
    return s64(small + sum(u * d for u, d in zip(q.whole[:-1], D)))


@pytest.mark.parametrize("q", [SMALL, LARGE])
def test_digits_reproduce_fixed_point(q):
    rng = np.random.default_rng(1)
    half = 1 << (q.bits - 1)
    for v in list(rng.standard_normal(200) * 10.0 ** rng.integers(-9, 1, 200)) + [0.0, 1 - 2.0 ** -53, -(1 - 2.0 ** -53),
                                                                                 2.0 ** -62]:
        f = fixed(float(v), max(0, math.frexp(v)[1]), q.up)
        for g in (f, -f):
            d = digits(g, q)
            assert all(-half <= x <= half for x in d) and sum(x << (q.bits * (DIGITS - 1 - s)) for s, x in enumerate(d)) == g


@pytest.mark.parametrize("q", [SMALL, LARGE])
def test_accumulators_for_the_largest_digits(q):
    """All digits at their largest magnitude: which weights are exact, and the smallest one below 2^22."""
    top = (1 << (q.bits - 1)) ** 2
    sums = [2 * q.maxb * min(d + 1, DIGITS, 2 * DIGITS - 1 - d) * top for d in range(q.jobs)]
    assert all(v <= 1 << 24 for v in sums[:q.exact]) and sums[0] < MAGIC_LIMIT
    assert all(v < 1 << 25 for v in sums)


@pytest.mark.parametrize("bs,coefs,spread", [(1, 2, 1.0), (7, 4, 1.0), (29, 4, 1e-3), (30, 4, 1.0), (30, 2, 1e-6),
                                             (31, 2, 1e-3), (48, 4, 1.0), (47, 4, 1e-6)])
def test_pair_contribution_is_fp64_grade(bs, coefs, spread):
    q = SMALL if bs <= 30 else LARGE
    rng = np.random.default_rng(bs + coefs)
    C = rng.standard_normal((coefs, bs, bs, 2)) * 10.0 ** -np.arange(coefs)[:, None, None, None]
    C *= spread ** rng.random((1, 1, bs, 1))       # columns of very different size
    x = rng.standard_normal((bs, 2)) * spread ** rng.random((bs, 1))
    if bs == q.maxb and coefs == 4:  # the 64-bit sums' worst case
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
    ex = [exponent(x[n2]) for n2 in range(bs)]
    ec = max(e + b for e, b in zip(ex, eb))

    def rotate(p, r, mm, sign, half):
        """(p + i r) e^{i sign mm phi} from words; half: half of it."""
        (ch, cl), (sh, sl) = cs[abs(mm)]
        if (mm < 0) != (sign < 0):
            sh, sl = -sh, -sl
        out = []
        for (a, b, g) in ((split(p), split(r), -1), (split(r), split(p), 1)):
            mid = s64(a[0] * cl + a[1] * ch + b[0] * g * sl + b[1] * g * sh + (1 << (30 if half else 29)))
            hh = a[0] * ch + b[0] * g * sh
            out.append(s64(hh + (mid >> 31)) if half else s64(2 * hh + (mid >> 30)))
        return out

    u = []
    for n in range(bs):  # words of the element's own scale, rotated, then moved to the column's
        w = rotate(fixed(float(x[n, 0]), ex[n], 9), fixed(float(x[n, 1]), ex[n], 9), int(m[n]), 1, True)
        u.append([v >> min(63, ec - ex[n] - eb[n] + 9 - q.up) for v in w])
    re, im = [digits(v[0], q) for v in u], [digits(v[1], q) for v in u]
    xl = (x[:, 0] + 1j * x[:, 1]).astype(np.clongdouble)
    ul = xl * phase
    for n1 in range(min(bs, 4)):
        acc = [0, 0]
        for c in range(coefs - 1, -1, -1):
            f = [[fixed(float(C[c, n1, n2, part]), ea[n1] + eb[n2], q.up) for n2 in range(bs)] for part in range(2)]
            cr, ci, cn = [[digits(v, q) for v in w] for w in (f[0], f[1], [-v for v in f[1]])]
            e = (combine(cn + cr, im + re, q), combine(cr + ci, im + re, q))
            acc = list(e) if c == coefs - 1 else [mul(split(acc[p]), tw, e[p]) for p in range(2)]
        out = rotate(acc[0], acc[1], int(m[n1]), -1, False)
        unit = math.ldexp(1.0, ea[n1] + ec + 1 - q.unit)
        got = complex(out[0] * unit, out[1] * unit)
        L = ((np.longdouble(t) ** np.arange(coefs))[:, None, None] * C[:, n1].astype(np.longdouble)).sum(0)
        L = L[:, 0] + 1j * L[:, 1]
        want = (L * ul).sum() * phase[n1].conjugate()
        size = float((np.abs(L) * np.abs(ul)).sum())
        places = 2 + (bs * coefs if q is LARGE else 0)
        assert abs(got - complex(want)) <= 2.0 ** -52 * size + places * unit
