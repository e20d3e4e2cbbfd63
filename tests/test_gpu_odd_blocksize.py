"""FP32 products of odd blocksizes, whose coefficient columns are not multiples of 16 bytes.

The pair-symmetric FP32 kernel copies such columns in bulk and does not take them; the autotuner must choose among the
others. Bound 2e-5, as for the FP32 kernels elsewhere."""
import numpy as np
import pytest

from smuthi_gb300 import _lib
from test_gpu_ibatch import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bs", [(20, 3), (40, 17), (33, 31), (40, 49), (20, 63)])
@pytest.mark.parametrize("R", [1, 8, 16])
def test_fp32_products(n, bs, R, gpu_context):
    _system(gpu_context, n, bs, "cubic", n + bs)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n * bs, R)) + 1j * rng.standard_normal((n * bs, R))
    y = gpu_context.coupling_matvec(x, _lib.SG_FP32)
    assert gpu_context.fp32_autotune(R)[0] not in (2, 3)
    ref = gpu_context.coupling_matvec(x, _lib.SG_FP64)
    assert np.linalg.norm(y - ref) <= 2e-5 * np.linalg.norm(ref)
    for variant in (2, 3):
        with pytest.raises(_lib.SmuthiGB300Error) as e:
            gpu_context.fp32_set_kernel(R, variant, 4 if R > 1 else 1)
        assert e.value.code == _lib.SG_ERR_ARG
