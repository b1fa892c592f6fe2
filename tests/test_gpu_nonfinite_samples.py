"""Samples with a NaN or infinite coordinate among ordinary ones: they lie in no Gaussian (-1 and
weight 0), and nothing of theirs reaches a gradient.  Gradients against the oracle's FP64 adjoint
over the other samples, with the tolerances of test_gpu_rasterizer."""
import numpy as np
import pytest

from test_gpu_rasterizer import assert_grads_close, oracle_backward, run_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("path,mode", [("plain", "auto"), ("plain", "tensor_core"), ("tensor_core", "auto")])
def test_samples_that_are_no_points(cuda, orc, path, mode, bad):
    from bvh_diff_gaussian_rasterization import _C
    means, scales, rots, values, weights = orc.mixture_small(seed=7, P=2000)
    samples = orc.grid_centres(32).copy()
    S = samples.shape[0]
    samples[100, 1] = bad
    samples[S // 2] = bad
    samples[S - 1, 2] = bad
    fin = np.isfinite(samples).all(1)
    rng = np.random.default_rng(71)
    gout, gw = (rng.normal(size=S).astype(np.float32) for _ in range(2))
    _C.set_eval_path(path)
    _C.set_backward_mode(mode)  # before the forward, which prepares for it
    try:
        got, out, outw, conics = run_backward(cuda, (means, scales, rots, values, weights, samples), gout, gw, mode)
    finally:
        _C.set_eval_path("plain")
        _C.set_backward_mode("auto")
    assert (out[~fin] == -1.0).all() and (outw[~fin] == 0.0).all()
    assert (outw[fin] > 0.0).any()
    ref = oracle_backward(orc, (means, scales, rots, values, weights, samples[fin]), out[fin], outw[fin], conics,
                          gout[fin], gw[fin])
    assert all(np.isfinite(g).all() for g in got)
    assert_grads_close(got, ref)


def test_order_of_the_other_samples(cuda, orc):
    """An infinite coordinate does not count among the bounds of the Morton grid."""
    import ctypes

    import gvc_native
    import torch
    from test_gpu_rasterizer import T
    pts = np.random.default_rng(72).random((20_000, 3)).astype(np.float32)
    pts[7, 0], pts[11], pts[13, 2] = np.inf, -np.inf, np.nan
    ctx = gvc_native.Context()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    d = T(pts, cuda)
    ctx.call("gvc_build_bvh", gvc_native.ptr(d), pts.shape[0], 0, 0, st)
    perm = torch.empty(pts.shape[0], dtype=torch.int32, device=cuda)
    keys = torch.empty(pts.shape[0], dtype=torch.int32, device=cuda)
    ctx.call("gvc_debug_sample_order", gvc_native.ptr(perm), gvc_native.ptr(keys), st)
    _, skeys, order = orc.morton30_points(pts)
    np.testing.assert_array_equal(perm.cpu().numpy(), order)
    np.testing.assert_array_equal(keys.cpu().numpy().view(np.uint32), skeys)
