"""Operator products under stream capture: after an uncaptured product, a captured one is replayed on new inputs and has
to equal the uncaptured product of the same inputs, whatever else the context computed in between.

FP64-grade products repeat to the order of their sums only where the captured call may take another kernel (1e-12, the
sums of at most 100 * 30 products); FP32 ones within twice the bound of test_gpu_ibatch32.py.
"""
import numpy as np
import pytest

from smuthi_gb300 import _lib
from test_gpu_ibatch import _system

pytestmark = pytest.mark.gpu

TOL = {_lib.SG_FP64: 1e-12, _lib.SG_DF64: 1e-12, _lib.SG_FP32: 8e-6}


def _product(ctx, x, precision):
    import torch
    y = torch.full_like(x, float("nan"))
    ctx.coupling_matvec_dev(x.data_ptr(), y.data_ptr(), x.shape[1], precision, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return y


def _capture(ctx, x, precision, mode="global"):
    import torch
    y = torch.full_like(x, float("nan"))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        ctx.coupling_matvec_dev(x.data_ptr(), y.data_ptr(), x.shape[1], precision,
                                torch.cuda.current_stream().cuda_stream)
    return graph, y


def _vector(rows, R, seed):
    import torch
    return torch.randn(rows, R, dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _close(y, ref, tol):
    import torch
    return bool(torch.linalg.vector_norm(y - ref) <= tol * torch.linalg.vector_norm(ref))


# 20 particles: below the batched operators; 100 and 420: they apply; blocksize 49: too large for them
@pytest.mark.parametrize("n,bs", [(20, 30), (100, 30), (420, 6), (40, 49), (60, 48)])
@pytest.mark.parametrize("R", [1, 16, 19])
@pytest.mark.parametrize("precision", [_lib.SG_FP64, _lib.SG_DF64, _lib.SG_FP32])
def test_replay_after_a_warm_up(n, bs, R, precision, gpu_context):
    import torch
    _system(gpu_context, n, bs, "cubic", n + bs)
    x = _vector(n * bs, R, 1)
    _product(gpu_context, x, precision)
    graph, y = _capture(gpu_context, x, precision)
    # products that use, and grow, the buffers of the context (those that the FP32 kernels share stay as they are for a
    # captured FP32 product)
    for p in (_lib.SG_FP64, _lib.SG_DF64) + ((_lib.SG_FP32,) if precision != _lib.SG_FP32 else ()):
        _product(gpu_context, _vector(n * bs, 32, 2), p)
    for seed in (3, 4):
        x.copy_(_vector(n * bs, R, seed))
        ref = _product(gpu_context, x.clone(), precision)
        y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert _close(y, ref, TOL[precision])


@pytest.mark.parametrize("n,R0,R,precision", [(100, 16, 1, _lib.SG_FP64), (100, 16, 8, _lib.SG_DF64), (100, 1, 3, _lib.SG_DF64),
                                              (330, 1, 16, _lib.SG_FP64), (20, 16, 1, _lib.SG_FP64)])
def test_other_counts_than_the_warm_up(n, R0, R, precision, gpu_context):
    """A captured product of another number of right-hand sides than the products before it."""
    import torch
    _system(gpu_context, n, 30, "linear", n)
    _product(gpu_context, _vector(n * 30, R0, 1), precision)
    x = _vector(n * 30, R, 5)
    graph, y = _capture(gpu_context, x, precision, "relaxed")
    ref = _product(gpu_context, x.clone(), precision)
    for _ in range(2):
        y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert _close(y, ref, TOL[precision])


def test_discarded_capture(gpu_context):
    """A captured product that is never replayed leaves nothing behind that a second one would rely on."""
    import torch
    _system(gpu_context, 100, 30, "linear", 9)
    x = _vector(3000, 3, 5)
    _product(gpu_context, x, _lib.SG_FP64)
    for p in (_lib.SG_DF64, _lib.SG_FP64):
        first, _ = _capture(gpu_context, x, p, "relaxed")
        del first
        graph, y = _capture(gpu_context, x, p, "relaxed")
        graph.replay()
        torch.cuda.synchronize()
        assert _close(y, _product(gpu_context, x, _lib.SG_FP64), 1e-12)


def test_captured_batched_fp32(gpu_context):
    """The interval-batched FP32 operator in a graph, fixed by the caller, with a remainder of a group of 16."""
    import torch
    _system(gpu_context, 600, 30, "linear", 10)
    x = _vector(18000, 20, 5)
    assert gpu_context.fp32_batched(20, take=True)[0]
    _product(gpu_context, x, _lib.SG_FP32)
    graph, y = _capture(gpu_context, x, _lib.SG_FP32)
    x.copy_(_vector(18000, 20, 6))
    ref = _product(gpu_context, x.clone(), _lib.SG_FP64)
    graph.replay()
    torch.cuda.synchronize()
    assert _close(y, ref, 4e-6)
