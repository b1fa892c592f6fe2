"""A backward takes (out, W) as its caller hands them in: changed in place after the forward of an
evaluation path that keeps no copy of them, they are read as they are then."""
import numpy as np
import pytest
import torch

from test_gpu_rasterizer import T, assert_grads_close, oracle_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["deterministic", "tensor_core"])
def test_outputs_changed_in_place(cuda, orc, mode):
    from bvh_diff_gaussian_rasterization import _C
    a = orc.mixture_small(seed=3, P=2000)
    samples = orc.grid_centres(32)
    rng = np.random.default_rng(81)
    up = [rng.normal(size=samples.shape[0]).astype(np.float32) for _ in range(2)]
    _C.set_eval_path("tensor_core")
    _C.set_backward_mode(mode)
    try:
        t = [T(x, cuda) for x in a]
        _C.build_bvh(T(samples, cuda), False, False)
        out, outw, conics = _C.rasterize_gaussians(*t, 1.0, 0, 0, 0, 1, 1, 1, -1.0, False, False)
        out.mul_(0.5)
        outw.copy_(torch.where(outw > 0.5, outw, torch.zeros_like(outw)))
        g = _C.rasterize_gaussians_backward(t[0], t[1], t[2], conics, t[3], t[4], out, outw, 1.0, 0, 0, 0, 1, 1, 1,
                                            -1.0, T(up[0], cuda), T(up[1], cuda), False, False)
        _C.check_status()
    finally:
        _C.set_eval_path("plain")
        _C.set_backward_mode("auto")
    ref = oracle_backward(orc, tuple(a) + (samples,), out.cpu().numpy(), outw.cpu().numpy(),
                          conics.cpu().numpy().reshape(-1, 6), *up)
    assert_grads_close([x.cpu().numpy() for x in g], ref)
