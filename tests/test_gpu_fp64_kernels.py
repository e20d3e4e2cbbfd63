"""The kernels of FP64-grade products, each fixed in turn (sg_fp64_set_kernel), against a direct FP64 evaluation, and the
rule that chooses between them.

Bounds: 1e-13 for the FP64 kernels (n * blocksize <= 10000 products, each side rounds at 2^-53 of its partial sums), 1e-12
for double-float (48 bits).
"""
import numpy as np
import pytest

from smuthi_gb300 import _lib
from test_gpu_ibatch import _direct, _system

pytestmark = pytest.mark.gpu

BATCHED = [(32, 1, 1, "linear"), (33, 30, 1, "cubic"), (40, 6, 3, "cubic_hermite"), (47, 30, 16, "cubic"), (64, 17, 17, "linear"),
           (65, 30, 64, "cubic"), (101, 30, 2, "linear"), (35, 9, 13, "cubic"), (34, 31, 1, "cubic"), (50, 48, 3, "cubic"),
           (65, 48, 1, "linear"), (33, 36, 16, "cubic_hermite"), (40, 47, 21, "linear")]


@pytest.fixture
def ctx(gpu_context):
    yield gpu_context
    gpu_context.fp64_set_kernel()


def _check(ctx, n, bs, R, kind, precision, tol):
    xy, m, rho, table = _system(ctx, n, bs, kind, 100 * n + bs)
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))) * 10.0 ** -rng.uniform(0, 3, (1, bs, 1))
    y = ctx.coupling_matvec(x.reshape(n * bs, R), precision).reshape(n, bs, R)
    ref = _direct(xy, m, rho, table, kind, x)
    for r in range(R):
        assert np.linalg.norm(y[..., r] - ref[..., r]) <= tol * np.linalg.norm(ref[..., r])


@pytest.mark.parametrize("n,bs,R,kind", BATCHED)
def test_batched(n, bs, R, kind, ctx):
    ctx.fp64_set_kernel(1)
    _check(ctx, n, bs, R, kind, _lib.SG_FP64, 1e-13)


# with partial sums (fewer particles than half the blocks in flight) and without, one to three rows per lane, tiles of 1
# to 16 right-hand sides
@pytest.mark.parametrize("n,bs,kind", [(8, 30, "cubic"), (20, 96, "linear"), (60, 30, "linear"), (310, 16, "cubic"), (100, 48, "cubic_hermite"),
                                       (33, 17, "cubic")])
@pytest.mark.parametrize("R", [1, 2, 4, 8, 13, 16])
@pytest.mark.parametrize("precision,tol", [(_lib.SG_FP64, 1e-13), (_lib.SG_DF64, 1e-12)])
def test_per_receiver(n, bs, kind, R, precision, tol, ctx):
    ctx.fp64_set_kernel(2)
    _check(ctx, n, bs, R, kind, precision, tol)


@pytest.mark.parametrize("n,res,R,batched", [(32, 1.0, 1, False), (40, 0.5, 2, False), (100, 50.0, 1, True), (100, 0.2, 1, False),
                                             (250, 1.0, 1, True), (64, 40.0, 16, True)])
@pytest.mark.parametrize("precision", [_lib.SG_FP64, _lib.SG_DF64])
def test_choice(n, res, R, batched, precision, ctx):
    """Few pairs per interval: the per-receiver FP64 kernel, for double-float products too; many: the batched one. Both
    repeat exactly, so the product shows which one ran."""
    rng = np.random.default_rng(n)
    bs = 6
    xy = rng.uniform(0, 25.0 * np.sqrt(n), (n, 2))
    up, un = np.divmod(np.arange(n * bs), bs)
    ctx.set_particles(xy, up, un, bs, rng.integers(-1, 2, bs))
    rows = int(25.0 * np.sqrt(2 * n) / res) + 4
    table = rng.standard_normal((rows, bs, bs)) + 1j * rng.standard_normal((rows, bs, bs))
    ctx.set_lookup("linear", table, 0.0, res)
    x = rng.standard_normal((n * bs, R)) + 1j * rng.standard_normal((n * bs, R))
    y = ctx.coupling_matvec(x, precision)
    ctx.fp64_set_kernel(1 if batched else 2)
    assert np.array_equal(y, ctx.coupling_matvec(x, _lib.SG_FP64))
    ctx.fp64_set_kernel(2 if batched else 1)
    other = ctx.coupling_matvec(x, _lib.SG_FP64)
    assert not np.array_equal(y, other) and np.linalg.norm(y - other) <= 1e-13 * np.linalg.norm(other)


def test_kernel_is_validated(ctx):
    for kernel in (-1, 3):
        with pytest.raises(_lib.SmuthiGB300Error) as e:
            ctx.fp64_set_kernel(kernel)
        assert e.value.code == _lib.SG_ERR_ARG
