"""The interval-batched operators (csrc/sg_ibatch.cu, sg_ibatch32.cu) at the edges of their number ranges, against a
direct FP64 evaluation.
"""
import numpy as np
import pytest

from smuthi_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def batched(gpu_context):
    gpu_context.fp64_set_kernel(1)
    yield
    gpu_context.fp64_set_kernel()


def _line(n, step, res, bs, seed, scale=1.0):
    """Particles on a line, `step` apart, and a smooth random table on a grid from zero."""
    rng = np.random.default_rng(seed)
    xy = np.stack([step * np.arange(n), np.zeros(n)], 1)
    m = rng.integers(-3, 4, bs)
    rho = res * np.arange(int(np.ceil(step * n / res)) + 4)
    table = np.exp(1j * rho[:, None, None] * rng.uniform(0.1, 1.0, (bs, bs))) * rng.standard_normal((bs, bs)) * scale
    x = rng.standard_normal((n, bs)) + 1j * rng.standard_normal((n, bs))
    return xy, m, table, x


def _linear(xy, m, table, res, x):
    d = xy[:, None] - xy[None]
    s = np.sqrt((d ** 2).sum(-1)) / res
    k = np.floor(s).astype(int)
    t = (s - k)[..., None, None]
    w = table[k] + t * (table[k + 1] - table[k])
    w = w * np.exp(1j * (m[None, :] - m[:, None]) * np.arctan2(d[..., 1], d[..., 0])[..., None, None])
    return np.einsum("ijab,jb->ia", w, x), s - k


def _upload(ctx, xy, m, table, res, bs):
    ctx.set_particles(xy, *np.divmod(np.arange(len(xy) * bs), bs), bs, m)
    ctx.set_lookup("linear", table, 0.0, res)


@pytest.mark.parametrize("bs", [30, 48])
def test_fraction_just_below_one(bs, gpu_context):
    """Distances that fall a rounding error short of a grid point: t within 2^-32 of one. Bound as in
    test_gpu_ibatch.py: n * blocksize <= 3100 products, each side rounds at 2^-53 of its partial sums."""
    n, res = 64, 0.1
    xy, m, table, x = _line(n, 0.3, res, bs, 1)
    ref, t = _linear(xy, m, table, res, x)
    assert (t > 1 - 2.0 ** -32).sum() > 1000
    _upload(gpu_context, xy, m, table, res, bs)
    y = gpu_context.coupling_matvec(x.reshape(-1), _lib.SG_FP64).reshape(n, bs)
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("precision,R,tol", [(_lib.SG_FP64, 1, 1e-13), (_lib.SG_FP32, 16, 4e-6)])
def test_zero_column_of_a_small_table(precision, R, tol, gpu_context):
    """A table far below one with a multipole that couples to nothing: its part of x, which is not small, must not set
    the scale of the products. Bounds as in test_gpu_ibatch.py and test_gpu_ibatch32.py."""
    n, bs, res = 40, 30, 1.0
    xy, m, table, x = _line(n, 7.3, res, bs, 2, 1e-9)
    table[:, :, 3] = 0
    ref, _ = _linear(xy, m, table, res, x)
    _upload(gpu_context, xy, m, table, res, bs)
    if precision == _lib.SG_FP32:
        assert gpu_context.fp32_batched(R, take=True)[0]
    y = gpu_context.coupling_matvec(np.repeat(x.reshape(-1, 1), R, axis=1), precision)
    for r in range(R):
        assert np.linalg.norm(y[:, r] - ref.reshape(-1)) <= tol * np.linalg.norm(ref)
    table[:] = 0
    _upload(gpu_context, xy, m, table, res, bs)
    if precision == _lib.SG_FP32:
        assert gpu_context.fp32_batched(R, take=True)[0]
    assert not gpu_context.coupling_matvec(np.repeat(x.reshape(-1, 1), R, axis=1), precision).any()


@pytest.mark.parametrize("e", [-1000, -1015, -1030, -1060])
def test_subnormal_vectors(e, gpu_context):
    """x in and below the last binades of FP64: the result scales with it, up to the rounding of each pair's
    contribution and of their sum to a multiple of 2^-1074 (and FP64's own)."""
    n, bs, res = 40, 30, 1.0
    xy, m, table, x = _line(n, 7.3, res, bs, 3)
    x = np.round(np.stack([x.real, x.imag], -1) * 2.0 ** 10) / 2.0 ** 10  # exact multiples of 2^(e - 10)
    _upload(gpu_context, xy, m, table, res, bs)
    big = gpu_context.coupling_matvec((x[..., 0] + 1j * x[..., 1]).reshape(-1), _lib.SG_FP64)
    x = np.ldexp(x, e)
    y = gpu_context.coupling_matvec((x[..., 0] + 1j * x[..., 1]).reshape(-1), _lib.SG_FP64)
    for got, want in ((y.real, big.real), (y.imag, big.imag)):
        got = np.ldexp(np.ldexp(got, 600), -e - 600)
        assert (np.abs(got - want) <= 1e-13 * np.abs(big).max() + np.ldexp(n, -1074 - e)).all()


def test_table_beyond_fp32(gpu_context):
    """Coefficients too large for FP32 give no finite numbers, as with the other FP32 operators."""
    n, bs, res, R = 40, 30, 1.0, 16
    xy, m, table, x = _line(n, 7.3, res, bs, 2, 1e50)
    _upload(gpu_context, xy, m, table, res, bs)
    x = np.repeat(x.reshape(-1, 1), R, axis=1)
    assert gpu_context.fp32_batched(R, take=True)[0]
    assert not np.isfinite(gpu_context.coupling_matvec(x, _lib.SG_FP32)).any()
    gpu_context.fp32_set_kernel(R, 0, 8)
    assert not np.isfinite(gpu_context.coupling_matvec(x, _lib.SG_FP32)).any()


@pytest.mark.parametrize("n,bs,R", [(512, 4, 16), (513, 4, 16), (1024, 4, 16), (1025, 4, 17), (3100, 3, 35), (5001, 2, 16)])
def test_fp32_sums_in_chunks(n, bs, R, gpu_context):
    """Systems of one to twenty chunks of tiles, groups of 16 right-hand sides with a remainder. Bound: 2.5e-6 of
    the operands and products as in test_gpu_ibatch32.py, and sums over about 1024 pairs (sqrt(1024) 2^-24)."""
    res = 40.0
    rng = np.random.default_rng(n)
    xy = rng.uniform(0, 2500.0, (n, 2))
    m = rng.integers(-3, 4, bs)
    table = rng.standard_normal((100, bs, bs)) + 1j * rng.standard_normal((100, bs, bs))
    x = rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))
    _upload(gpu_context, xy, m, table, res, bs)
    assert gpu_context.fp32_batched(R, take=True)[0]
    y = gpu_context.coupling_matvec(x.reshape(n * bs, R), _lib.SG_FP32).reshape(n, bs, R)
    rows = rng.choice(n, 40, replace=False)
    d = xy[rows, None] - xy[None]
    s = np.sqrt((d ** 2).sum(-1)) / res
    k = np.floor(s).astype(int)
    w = table[k] + (s - k)[..., None, None] * (table[k + 1] - table[k])
    w = w * np.exp(1j * (m[None, :] - m[:, None]) * np.arctan2(d[..., 1], d[..., 0])[..., None, None])
    ref = np.einsum("ijab,jbr->iar", w, x)
    for r in range(R):
        assert np.linalg.norm(y[rows, :, r] - ref[..., r]) <= 4.4e-6 * np.linalg.norm(ref[..., r])


def _launches(ctx, x, precision):
    before = ctx.launch_count()
    y = ctx.coupling_matvec(x, precision)
    return y, ctx.launch_count() - before


@pytest.mark.parametrize("n,bs,R,kind", [(101, 30, 16, "linear"), (64, 30, 19, "cubic"), (50, 48, 3, "cubic"), (33, 7, 1, "linear")])
def test_chunks_of_the_workspace(n, bs, R, kind, gpu_context):
    """A workspace far below the contributions: many chunks of tiles, with edges inside intervals, groups of right-hand
    sides and a remainder. Bound as in test_gpu_ibatch.py."""
    from test_gpu_ibatch import _direct, _system
    xy, m, rho, table = _system(gpu_context, n, bs, kind, 100 * n + bs)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))
    ref = _direct(xy, m, rho, table, kind, x)
    try:
        for workspace in (1, 300_000, 1_000_000):
            gpu_context.batched_memory(0, workspace)
            y, launches = _launches(gpu_context, x.reshape(n * bs, R), _lib.SG_FP64)
            assert launches >= 2 * n * n * bs * R * 16 // max(workspace, 128 * bs * 16)
            y = y.reshape(n, bs, R)
            for r in range(R):
                assert np.linalg.norm(y[..., r] - ref[..., r]) <= 1e-13 * np.linalg.norm(ref[..., r])
    finally:
        gpu_context.batched_memory()


@pytest.mark.parametrize("precision,R,tol", [(_lib.SG_FP64, 2, 1e-13), (_lib.SG_DF64, 2, 1e-12), (_lib.SG_FP32, 16, 2e-5)])
def test_memory_that_cannot_be_had(precision, R, tol, gpu_context):
    """Wherever an allocation of the batched operators fails, from the first to the last, the product comes from
    another kernel; what fits takes them again. Bounds as elsewhere (double-float 1e-12, FP32 kernels 2e-5)."""
    from test_gpu_ibatch import _direct, _system
    n, bs = 110, 30
    xy, m, rho, table = _system(gpu_context, n, bs, "linear", 5)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))
    ref = _direct(xy, m, rho, table, "linear", x)
    x, ref = x.reshape(n * bs, R), ref.reshape(n * bs, R)
    try:
        seen = set()
        for limit in list(np.geomspace(1e3, 1e9, 60).astype(np.int64)) + [0]:
            gpu_context.batched_memory(limit)
            if precision == _lib.SG_FP32:
                gpu_context.fp32_batched(R, take=True)
            for _ in range(2):
                y, launches = _launches(gpu_context, x, precision)
                assert np.linalg.norm(y - ref) <= tol * np.linalg.norm(ref)
            seen.add(launches if precision == _lib.SG_FP32 else y.tobytes())  # FP64-grade products repeat exactly
        assert len(seen) == 2, "both routes were taken"
    finally:
        gpu_context.batched_memory()


def test_autotuner_without_memory(gpu_context):
    """The FP32 autotuner drops the batched operator where it does not fit, and keeps the others."""
    from test_gpu_ibatch import _direct, _system
    n, bs, R = 330, 30, 16
    xy, m, rho, table = _system(gpu_context, n, bs, "linear", 6)
    x = np.random.default_rng(n).standard_normal((n * bs, R)) + 0j
    try:
        gpu_context.batched_memory(1000)
        y = gpu_context.coupling_matvec(x, _lib.SG_FP32)
        assert gpu_context.fp32_batched(R) == (False, -1.0) and gpu_context.fp32_autotune(R)[0] >= 0
        ref = _direct(xy, m, rho, table, "linear", x.reshape(n, bs, R)).reshape(n * bs, R)
        assert np.linalg.norm(y - ref) <= 2e-5 * np.linalg.norm(ref)
    finally:
        gpu_context.batched_memory()
