"""The Gaussian-owned backward (bwd_gauss.cu) at the sizes where it can go wrong: partial
chunks of 16 rows, partial level-1 nodes of 128, one and several tree levels, the three
ways of sharing warps (fewer than 4736 Gaussians, up to 100000, more), a shared list of
chunks that overflows, and boxes discarded by the power-window test.

Gradients against the oracle's FP64 adjoint at the GPU forward's own outputs, with the
tolerances of test_gpu_rasterizer; contributing pairs counted by the kernels against an
FP64 count, where only pairs within 1e-3 of the -14 floor or 1e-6 of a box face may differ
(the powers are FP32 evaluations of forms whose condition here is below 1e4)."""
import numpy as np
import pytest
import torch

from test_gpu_rasterizer import T, assert_grads_close, oracle_backward, run_backward

pytestmark = pytest.mark.gpu


def mixture(orc, P, scale, seed):
    means, scales, rots, values, weights = orc.mixture_small(seed=seed, P=P)
    return means, (scales * (scale / 0.02)).astype(np.float32), rots, values, weights


def upstream(S, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=S).astype(np.float32), rng.normal(size=S).astype(np.float32)


@pytest.mark.parametrize("P,S,scale", [(1, 1, 0.1), (1, 15, 0.1), (2, 16, 0.1), (3, 17, 0.1), (5, 127, 0.1),
                                       (5, 128, 0.1), (7, 129, 0.1), (300, 4097, 0.05), (64, 300_001, 0.05),
                                       (4735, 8193, 0.02), (4736, 8191, 0.02)])
def test_sizes_match_oracle(cuda, orc, P, S, scale):
    means, scales, rots, values, weights = mixture(orc, P, scale, seed=P)
    rng = np.random.default_rng(S)
    pts = rng.random((S, 3)).astype(np.float32)
    near = rng.integers(0, P, S // 2 + 1)
    pts[:near.size] = means[near] + rng.normal(size=(near.size, 3)) * scale
    case = (means, scales, rots, values, weights, pts.astype(np.float32))
    gout, gw = upstream(S, S + 1)
    got, out, outw, conics = run_backward(cuda, case, gout, gw)
    assert_grads_close(got, oracle_backward(orc, case, out, outw, conics, gout, gw))


@pytest.mark.parametrize("P", [100_000, 100_003])
def test_shared_walks_match_oracle(cuda, orc, P):
    """Four Gaussians per warp, the last warp partly empty; eight wide Gaussians meet every one
    of 1875 chunks, more than their warps can list, and walk by themselves."""
    means, scales, rots, values, weights = mixture(orc, P, 0.01, seed=9)
    wide = np.linspace(0, P - 1, 8).astype(int)
    scales[wide] = 0.3
    S = 30_000
    pts = np.random.default_rng(10).random((S, 3)).astype(np.float32)
    gout, gw = upstream(S, 11)
    got, out, outw, conics = run_backward(cuda, (means, scales, rots, values, weights, pts), gout, gw)
    sel = np.unique(np.concatenate([wide, wide[:-1] + 1, np.random.default_rng(12).choice(P, 2000, replace=False)]))
    sub = (means[sel], scales[sel], rots[sel], values[sel], weights[sel], pts)
    ref = oracle_backward(orc, sub, out, outw, conics[sel], gout, gw)
    assert_grads_close([g.reshape(P, -1)[sel] for g in got], [r.reshape(len(sel), -1) for r in ref])


@pytest.mark.parametrize("P,aspect", [(200, 1.0), (200, 30.0), (6000, 5.0)])
def test_no_contributing_pair_is_culled(cuda, orc, P, aspect):
    from bvh_diff_gaussian_rasterization import _C
    means, scales, rots, values, weights = mixture(orc, P, 0.03, seed=21)
    scales[:, 0] *= aspect ** 0.5
    scales[:, 1] /= aspect ** 0.5
    weights = (0.3 + 0.7 * weights).astype(np.float32)
    S = 20_011
    pts = (means[np.random.default_rng(22).integers(0, P, S)] +
           np.random.default_rng(23).normal(size=(S, 3)) * 0.02).astype(np.float32)
    gout, gw = upstream(S, 24)
    _C.set_count_pairs(True)
    try:
        _, out, outw, conics = run_backward(cuda, (means, scales, rots, values, weights, pts), gout, gw)
        st = _C.stats()
    finally:
        _C.set_count_pairs(False)
    _, _, bb = orc.preprocess(means, scales, rots, weights)
    x = T(pts, cuda).double()
    mu, C, b = T(means, cuda).double(), T(conics.astype(np.float64), cuda), T(bb.astype(np.float64), cuda)
    ok = T(outw > 0.01, cuda)
    lo_n = hi_n = lo_all = hi_all = 0
    for i in range(0, P, 50):
        d = x[None] - mu[i:i + 50, None]
        c = C[i:i + 50, None]
        p = -0.5 * (c[..., 0] * d[..., 0] ** 2 + c[..., 3] * d[..., 1] ** 2 + c[..., 5] * d[..., 2] ** 2) - (
            c[..., 1] * d[..., 0] * d[..., 1] + c[..., 2] * d[..., 0] * d[..., 2] + c[..., 4] * d[..., 1] * d[..., 2])

        def count(e, f, rows):
            inside = ((x[None] >= b[i:i + 50, None, :3] - e) & (x[None] <= b[i:i + 50, None, 3:] + e)).all(2)
            return int((inside & (p >= -14.0 * (1 + f)) & rows).sum())

        lo_n += count(-1e-6, -1e-3, ok)
        hi_n += count(1e-6, 1e-3, ok)
        lo_all += count(-1e-6, -1e-3, torch.ones_like(ok))
        hi_all += count(1e-6, 1e-3, torch.ones_like(ok))
    assert lo_n <= st["bwd_contributing"] <= hi_n
    assert lo_all <= st["fwd_contributing"] <= hi_all
    assert hi_n < st["bwd_rows"]
