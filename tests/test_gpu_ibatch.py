"""The interval-batched FP64 operator (csrc/sg_ibatch.cu) against a direct FP64 evaluation.

Random tables on a coarse grid, so that intervals hold from one to many tiles of pairs; block sizes and
right-hand-side counts at the edges of the kernel's tiles (rows in groups of 8, 64 complex columns,
16 right-hand sides per launch), particles just above the smallest count that takes the path. Bound
1e-13: a row sums n * blocksize <= 4000 products, each side rounds at 2^-53 of its partial sums.
"""
import numpy as np
import pytest
import scipy.interpolate

pytestmark = pytest.mark.gpu

RES = 40.0


def _system(ctx, n, bs, kind, seed, l_values=None):
    rng = np.random.default_rng(seed)
    xy = rng.uniform(0, 900.0, (n, 2))
    m = rng.integers(-3, 4, bs) if bs <= 30 else rng.integers(-4, 5, bs)
    rho = np.arange(-3 * RES, 900.0 * 1.5 + 4 * RES, RES)
    table = rng.standard_normal((len(rho), bs, bs)) + 1j * rng.standard_normal((len(rho), bs, bs))
    table *= 10.0 ** -rng.uniform(0, 3, bs)[None, None, :]   # columns of different size
    up, un = np.divmod(np.arange(n * bs), bs)
    ctx.set_particles(xy, up, un, bs, m)
    ctx.set_lookup(kind, table, rho[0], RES)
    return xy, m, rho, table


def _direct(xy, m, rho, table, kind, x):
    d = xy[:, None] - xy[None]
    r = np.sqrt((d ** 2).sum(-1))
    phi = np.arctan2(d[..., 1], d[..., 0])
    if kind == "cubic_hermite":
        k = np.floor((r - rho[0]) / RES).astype(int)
        t = ((r - rho[0]) / RES - k)[..., None, None]
        a, b, c, e = (table[k + q] for q in (-1, 0, 1, 2))
        w = b + t * (0.5 * (c - a) + t * (0.5 * (2 * a - 5 * b + 4 * c - e) + t * 0.5 * (-a + 3 * b - 3 * c + e)))
    else:
        w = scipy.interpolate.interp1d(rho, table, kind=kind, axis=0)(r)
    w = w * np.exp(1j * (m[None, :] - m[:, None]) * phi[..., None, None])
    return np.einsum("ijab,jbr->iar", w, x)


@pytest.mark.parametrize("n,bs,R,kind", [(32, 1, 1, "linear"), (33, 30, 1, "cubic"), (40, 6, 3, "cubic_hermite"),
                                         (47, 30, 16, "cubic"), (64, 17, 17, "linear"), (65, 30, 64, "cubic"),
                                         (101, 30, 2, "linear"), (35, 9, 13, "cubic"), (34, 31, 1, "cubic"),
                                         (50, 48, 3, "cubic"), (65, 48, 1, "linear"), (33, 36, 16, "cubic_hermite"),
                                         (40, 47, 21, "linear")])
def test_matches_direct_evaluation(n, bs, R, kind, gpu_context):
    xy, m, rho, table = _system(gpu_context, n, bs, kind, 100 * n + bs)
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))) * 10.0 ** -rng.uniform(0, 3, (1, bs, 1))
    y = gpu_context.coupling_matvec(x.reshape(n * bs, R), 0).reshape(n, bs, R)
    ref = _direct(xy, m, rho, table, kind, x)
    for r in range(R):
        assert np.linalg.norm(y[..., r] - ref[..., r]) <= 1e-13 * np.linalg.norm(ref[..., r])


@pytest.mark.parametrize("bs", [30, 48])
def test_largest_digit_sums(bs, gpu_context):
    """Equal operands with all mantissa bits set: digit sums beyond 2^22, which the kernel converts one by one."""
    n = 40
    xy, m, rho, table = _system(gpu_context, n, bs, "linear", 21)
    table[:] = (1 - 2.0 ** -53) * (1 + 1j)
    gpu_context.set_particles(xy, *np.divmod(np.arange(n * bs), bs), bs, 0 * m)
    gpu_context.set_lookup("linear", table, rho[0], RES)
    x = np.full((n, bs, 1), (1 - 2.0 ** -53) * (1 - 1j))
    y = gpu_context.coupling_matvec(x.reshape(n * bs, 1), 0).reshape(n, bs, 1)
    ref = _direct(xy, 0 * m, rho, table, "linear", x)
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)


def test_scales_and_zero_columns(gpu_context):
    """Right-hand sides of any magnitude (exact powers of two scale exactly), zero ones stay zero."""
    n, bs = 50, 30
    _system(gpu_context, n, bs, "cubic", 7)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(n * bs) + 1j * rng.standard_normal(n * bs)
    y = gpu_context.coupling_matvec(x, 0)
    X = np.stack([x * 2.0 ** e for e in (-900, -60, 0, 60, 900)] + [0 * x], axis=1)
    Y = gpu_context.coupling_matvec(np.ascontiguousarray(X), 0)
    for q, e in enumerate((-900, -60, 0, 60, 900)):
        assert np.linalg.norm(Y[:, q] * 2.0 ** -e - y) <= 1e-15 * np.linalg.norm(y)
    assert not Y[:, 5].any()


def test_workspace_chunks_agree(gpu_context):
    """A problem larger than the workspace runs in chunks of tiles and equals its single columns."""
    n, bs, R = 420, 30, 16
    _system(gpu_context, n, bs, "linear", 11)
    rng = np.random.default_rng(5)
    X = rng.standard_normal((n * bs, R)) + 1j * rng.standard_normal((n * bs, R))
    Y = gpu_context.coupling_matvec(X, 0)
    for r in (0, 9, 15):
        y = gpu_context.coupling_matvec(np.ascontiguousarray(X[:, r]), 0)
        assert np.linalg.norm(Y[:, r] - y) <= 1e-14 * np.linalg.norm(y)


def test_not_a_number_reaches_every_receiver(gpu_context):
    """Device calls do not check their input: a NaN in one emitter's column gives NaN in that column only."""
    import torch
    n, bs = 60, 30
    _system(gpu_context, n, bs, "cubic", 13)
    x = torch.randn(n * bs, 2, dtype=torch.complex128, device="cuda")
    x[17, 1] = float("nan")
    y = torch.zeros_like(x)
    gpu_context.coupling_matvec_dev(x.data_ptr(), y.data_ptr(), 2, 0)
    torch.cuda.synchronize()
    assert torch.isnan(y[:, 1]).all() and torch.isfinite(y[:, 0].real).all()
