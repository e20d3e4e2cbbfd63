"""The interval-batched FP32 operator (csrc/sg_ibatch32.cu) against a direct FP64 evaluation.

Random tables on a coarse grid; blocksizes at the edges of the kernel's chunks of eight, passes and padded
sizes, right-hand-side counts around its groups of 16, one to many tiles per interval. Bound 4e-6 of the
result's norm: operands split at 2^-23, a dropped product of 2^-24 and at most 18 truncating accumulations of
2^-23 (2.5e-6 together), FP32 sums over at most 200 pairs (sqrt(200) 2^-24).
"""
import numpy as np
import pytest

from test_gpu_ibatch import _direct, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bs,R,kind", [(32, 1, 16, "linear"), (33, 30, 17, "cubic"), (64, 17, 64, "cubic_hermite"),
                                         (200, 30, 16, "linear"), (50, 48, 16, "cubic"), (35, 33, 33, "linear"),
                                         (65, 8, 32, "cubic"), (40, 47, 20, "cubic")])
def test_matches_direct_evaluation(n, bs, R, kind, gpu_context):
    from smuthi_gb300 import _lib
    xy, m, rho, table = _system(gpu_context, n, bs, kind, 100 * n + bs)
    assert gpu_context.fp32_batched(R, take=True)[0]
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, bs, R)) + 1j * rng.standard_normal((n, bs, R))) * 10.0 ** -rng.uniform(0, 3, (1, bs, 1))
    x *= 2.0 ** np.resize([0, 100, -100], R)   # columns are scaled one by one
    y = gpu_context.coupling_matvec(x.reshape(n * bs, R), _lib.SG_FP32).reshape(n, bs, R)
    ref = _direct(xy, m, rho, table, kind, x)
    for r in range(R):
        assert np.linalg.norm(y[..., r] - ref[..., r]) <= 4e-6 * np.linalg.norm(ref[..., r])


def test_zero_and_not_a_number_columns(gpu_context):
    import torch
    from smuthi_gb300 import _lib
    n, bs = 60, 30
    _system(gpu_context, n, bs, "cubic", 13)
    gpu_context.fp32_batched(16, take=True)
    x = torch.randn(n * bs, 16, dtype=torch.complex128, device="cuda")
    x[17, 1], x[40, 2], x[:, 3] = float("nan"), float("inf"), 0
    y = torch.zeros_like(x)
    gpu_context.coupling_matvec_dev(x.data_ptr(), y.data_ptr(), 16, _lib.SG_FP32)
    torch.cuda.synchronize()
    assert torch.isnan(y[:, 1]).all() and torch.isnan(y[:, 2]).all() and not y[:, 3].any()
    assert torch.isfinite(torch.view_as_real(y[:, 4:])).all()


def test_refused_where_it_does_not_apply(gpu_context):
    from smuthi_gb300 import _lib
    _system(gpu_context, 31, 6, "linear", 1)
    for n, bs, R in ((31, 6, 16), (40, 6, 15), (40, 31, 16), (40, 49, 16)):
        _system(gpu_context, n, bs, "linear", 1)
        with pytest.raises(_lib.SmuthiGB300Error) as e:
            gpu_context.fp32_batched(R, take=True)
        assert e.value.code == _lib.SG_ERR_ARG
