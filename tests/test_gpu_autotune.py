"""The FP32 autotuner and the interval-batched operator: it is timed only where it may be chosen, that is for right-hand
side counts for which a tensor-core kernel has won, and its choice is the faster of the two."""
import numpy as np
import pytest

from smuthi_gb300 import _lib
from test_gpu_ibatch import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(300, 24), (300, 48), (300, 128), (300, 16), (40, 16), (700, 16), (300, 32)])
def test_batched_operator_is_timed_where_it_may_win(n, R, gpu_context):
    ctx = _lib.Context(0)
    _system(ctx, n, 30, "cubic", n)
    x = np.random.default_rng(n).standard_normal((n * 30, R)) + 0j
    y = ctx.coupling_matvec(x, _lib.SG_FP32)
    variant, _, *times = ctx.fp32_autotune(R)
    taken, ms = ctx.fp32_batched(R)
    assert min(t for t in times if t >= 0) == (times[0], times[1], times[2], times[2], times[3], times[4])[variant]
    if variant < 4:
        assert (taken, ms) == (False, -1.0)
    else:
        assert ms > 0 and taken == (ms < times[variant - 1])
    ref = ctx.coupling_matvec(x, _lib.SG_FP64)
    assert np.linalg.norm(y - ref) <= 2e-5 * np.linalg.norm(ref)
    ctx.close()
