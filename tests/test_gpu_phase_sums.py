"""The far-field particle sum and the near-field kernel against direct FP64 evaluation at the edges of their
tiles: chunks of 32 particles, blocks of 128 azimuths, tiles of two (one right-hand side) and four columns,
every m_max with a kernel of its own (0 .. 4) and the general one, phases up to and beyond the range of the
table-driven sine.

Bounds: a phase of x rad carries the rounding of x itself on both sides, 2^-52 |x|; sums of N such terms
stay within 2^-52 (|x|_max + N^(1/2) + 8) of the sum's 2-norm size N^(1/2).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,m_max,nk,na,side", [(1, 1, 0, 1, 1, 1e3), (31, 1, 1, 3, 127, 1e4), (32, 2, 2, 2, 128, 1e4),
                                                  (33, 3, 3, 3, 129, 1e5), (65, 1, 3, 2, 130, 1e6), (40, 16, 4, 2, 33, 1e4),
                                                  (34, 5, 5, 2, 40, 1e4), (33, 1, 3, 2, 20, 1e12)])
def test_far_field_sum(n, R, m_max, nk, na, side, gpu_context):
    import torch
    rng = np.random.default_rng(n + R)
    m = np.concatenate([np.arange(-m_max, m_max + 1), rng.integers(-m_max, m_max + 1, 6)]).astype(np.int32)
    B = len(m)
    xy = rng.uniform(0, side, (n, 2))
    c = rng.standard_normal((n, B, R)) + 1j * rng.standard_normal((n, B, R))
    S = rng.standard_normal((B, 2, nk)) + 1j * rng.standard_normal((B, 2, nk))
    kp, al = rng.uniform(0, 0.0114, nk), rng.uniform(-1, 7, na)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xy, c, kp, S, al)]
    out = torch.full((R, 2, nk, na), float("nan"), dtype=torch.complex128, device="cuda")
    gpu_context.farfield_sum_dev(n, d[0].data_ptr(), B, R, d[1].data_ptr(), m_max, m, nk, d[2].data_ptr(), d[3].data_ptr(),
                                 na, d[4].data_ptr(), out.data_ptr())
    u = np.cos(al)[:, None] * xy[:, 0] + np.sin(al)[:, None] * xy[:, 1]
    x = kp[:, None, None] * u
    ref = np.einsum("kai,ibr,bpk,ba->rpka", np.exp(-1j * x), c, S, np.exp(1j * np.outer(m, al)), optimize=True)
    err = np.linalg.norm(out.cpu().numpy() - ref)
    assert err <= 2.0 ** -52 * (np.abs(x).max() + np.sqrt(n * B) + 8) * 2 * np.sqrt(n * B) * np.sqrt(ref.size) * 2


@pytest.mark.parametrize("n,nk,na,field,size", [(1, 2, 2, 0, 1e3), (33, 9, 31, 1, 1e4), (70, 40, 8192, 0, 1e3),
                                                (5, 3, 17, 0, 1e12)])
def test_near_field(n, nk, na, field, size, gpu_context):
    import torch
    rng = np.random.default_rng(n + nk)
    k, omega = 0.0114, 0.0114
    p = rng.uniform(-size, size, (3, n))
    p[2] = rng.uniform(0, 300, n)
    kp = np.sort(rng.uniform(0, 0.016, nk)) - 1e-3j / size * (np.arange(nk) % 2)
    kz = np.sqrt(k ** 2 - kp ** 2 + 0j)
    kz = np.where(kz.imag < 0, -kz, kz)
    al = np.sort(rng.uniform(0, 6.3, na))
    g = rng.standard_normal((2, nk, na)) + 1j * rng.standard_normal((2, nk, na))
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (p, kp.astype(complex), kz, al, g)]
    out = torch.full((3, n), float("nan"), dtype=torch.complex128, device="cuda")
    gpu_context.pwe_field_dev(field, n, d[0][0].data_ptr(), d[0][1].data_ptr(), d[0][2].data_ptr(), nk, d[1].data_ptr(),
                              d[2].data_ptr(), na, d[3].data_ptr(), d[4].data_ptr(), k, omega, out.data_ptr())
    wa, wk = np.zeros(na), np.zeros(nk, complex)
    wa[1:] += np.diff(al) / 2
    wa[:-1] += np.diff(al) / 2
    wk[1:] += np.diff(kp) / 2
    wk[:-1] += np.diff(kp) / 2
    ca, sa = np.cos(al), np.sin(al)
    if field == 0:
        q = [-sa * g[0] + ca * (kz / k)[:, None] * g[1], ca * g[0] + sa * (kz / k)[:, None] * g[1], -(kp / k)[:, None] * g[1]]
    else:
        q = [-kz[:, None] * ca * g[0] - k * sa * g[1], -kz[:, None] * sa * g[0] + k * ca * g[1], kp[:, None] * g[0]]
        q = [v / omega for v in q]
    u = np.outer(p[0], ca) + np.outer(p[1], sa)
    ref, bound = np.zeros((3, n), complex), np.zeros(3)
    for j in range(nk):
        x = kp[j] * u
        for c in range(3):
            f = wk[j] * kp[j] * wa * q[c][j]
            ref[c] += (np.exp(1j * x) @ f) * np.exp(1j * kz[j] * p[2])
            bound[c] += np.abs(f).sum() * (np.abs(x).max() + 12) * np.exp(np.abs(x.imag).max())
    assert (np.abs(out.cpu().numpy() - ref).max(1) <= 2.0 ** -51 * bound).all()
