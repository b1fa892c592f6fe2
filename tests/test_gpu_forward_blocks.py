"""The forward kernels (fwd_points.cu, fwd_blocks.cu, cta.cu) at the sizes where they can go
wrong: both sides of the rule for sparse samples (S * S < 360000 P), of whole blocks per warp
(530432 samples) and, with the tensor-core backward selected, of 32 rows per warp (below
100000), a CTA per block and whole blocks (from 500000); a last block of one row; Gaussian
trees of one leaf, of partial nodes on each level (8, 256, 8192 leaves) and of several levels.

Against the oracle's FP64 forward at the GPU's conics and boxes, with the tolerance of
test_gpu_rasterizer."""
import numpy as np
import pytest

import gvc_native
from test_gpu_rasterizer import compare_forward, gpu_preprocess, run_forward

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda):
    return gvc_native.Context()


@pytest.mark.parametrize("mode,P,S", [
    ("auto", 1, 1), ("auto", 1, 599), ("auto", 1, 600), ("auto", 1000, 18973), ("auto", 1000, 18974),
    ("auto", 8, 2049), ("auto", 9, 4127), ("auto", 257, 20_001), ("auto", 8193, 65_537), ("auto", 40, 530_431),
    ("auto", 40, 530_433), ("auto", 8193, 300),
    ("tensor_core", 1, 1), ("tensor_core", 2, 129), ("tensor_core", 257, 99_999), ("tensor_core", 257, 100_001),
    ("tensor_core", 40, 499_999), ("tensor_core", 40, 500_001), ("tensor_core", 8193, 300)])
def test_sizes_match_oracle(ctx, cuda, orc, mode, P, S):
    from bvh_diff_gaussian_rasterization import _C
    means, scales, rots, values, weights = orc.mixture_small(seed=P, P=P)
    scales = (scales * (2.0 if P < 1000 else 1.0)).astype(np.float32)
    rng = np.random.default_rng(S)
    pts = rng.random((S, 3)).astype(np.float32)
    near = rng.integers(0, P, S // 2 + 1)
    pts[:near.size] = means[near] + rng.normal(size=(near.size, 3)) * scales[near]
    _C.set_backward_mode(mode)
    try:
        out, outw, conics = run_forward(cuda, means, scales, rots, values, weights, pts)
    finally:
        _C.set_backward_mode("auto")
    gc = conics.cpu().numpy().reshape(-1, 6)
    _, gb = gpu_preprocess(ctx, cuda, means, scales, rots, weights)
    ro, rw = orc.forward(means, values, weights, gc.astype(np.float64), gb, pts)
    compare_forward(out.cpu().numpy(), outw.cpu().numpy(), ro, rw, 2e-5, 2e-5)
    assert (ro != -1).any()


@pytest.mark.parametrize("path", ["plain", "tensor_core"])
def test_one_order_of_sums(cuda, orc, path):
    """With the tensor-core backward selected a sample's sums are the same bits whatever kernel
    the number of samples selects: 38400 samples alone (32 rows per warp), and followed by
    copies of the last corner, which sort behind them and leave their blocks as they are, up to
    a CTA per block and up to a warp per block."""
    from bvh_diff_gaussian_rasterization import _C
    means, scales, rots, values, weights = orc.mixture_small(seed=3, P=3000)
    n = 128 * 300
    pts = np.random.default_rng(5).random((n, 3)).astype(np.float32)
    pts[0], pts[1] = 0.0, 1.0
    got = []
    _C.set_backward_mode("tensor_core")
    _C.set_eval_path(path)
    try:
        for more in (0, 70_000, 480_000):
            all_pts = np.concatenate([pts, np.ones((more, 3), np.float32)])
            out, outw, _ = run_forward(cuda, means, scales, rots, values, weights, all_pts)
            got.append((out[:n].cpu().numpy(), outw[:n].cpu().numpy()))
    finally:
        _C.set_backward_mode("auto")
        _C.set_eval_path("plain")
    assert (got[0][1] > 0).any()
    for out, outw in got[1:]:
        np.testing.assert_array_equal(out, got[0][0])
        np.testing.assert_array_equal(outw, got[0][1])
