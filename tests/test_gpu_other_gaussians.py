"""The tensor-core backward of Gaussians that are not the last forward's, though as many: another
forward (of a second mixture, or of moved parameters) came between, and the candidate log is its
own.  Gradients against the oracle's FP64 adjoint with the tolerances of test_gpu_rasterizer;
copies of the same arrays read the log all the same."""
import numpy as np
import pytest

from test_gpu_candlog import modes
from test_gpu_rasterizer import T, assert_grads_close, oracle_backward

pytestmark = pytest.mark.gpu


def forward(_C, t):
    return _C.rasterize_gaussians(*t, 1.0, 0, 0, 0, 1, 1, 1, -1.0, False, False)


def backward(_C, t, fwd, up):
    out, outw, conics = fwd
    means, scales, rots, values, weights = t
    g = _C.rasterize_gaussians_backward(means, scales, rots, conics, values, weights, out, outw, 1.0, 0, 0, 0, 1, 1, 1,
                                        -1.0, *up, False, False)
    _C.check_status()
    return [x.cpu().numpy() for x in g]


@pytest.mark.parametrize("path", ["plain", "tensor_core"])
@pytest.mark.parametrize("other", ["mixture", "moved"])
def test_backward_after_another_forward(cuda, orc, path, other):
    a = orc.mixture_small(seed=0, P=4096)
    b = orc.mixture_small(seed=1, P=4096) if other == "mixture" else ((a[0] + np.float32(0.05)),) + tuple(a[1:])
    samples = orc.grid_centres(48)
    rng = np.random.default_rng(61)
    up_np = [rng.normal(size=samples.shape[0]).astype(np.float32) for _ in range(2)]
    with modes(path) as _C:
        ta, tb = [T(x, cuda) for x in a], [T(x, cuda) for x in b]
        up = [T(u, cuda) for u in up_np]
        _C.build_bvh(T(samples, cuda), False, False)
        fa = forward(_C, ta)
        fb = forward(_C, tb)
        # the first one's, the last one's (whose records the call before replaced), the first's again
        got = [(a, fa, backward(_C, ta, fa, up)), (b, fb, backward(_C, tb, fb, up)), (a, fa, backward(_C, ta, fa, up))]
    for mix, (out, outw, conics), g in got:
        ref = oracle_backward(orc, tuple(mix) + (samples,), out.cpu().numpy(), outw.cpu().numpy(),
                              conics.cpu().numpy().reshape(-1, 6), *up_np)
        assert_grads_close(g, ref)


def test_copies_of_the_same_gaussians_read_the_log(cuda, orc):
    a = orc.mixture_small(seed=2, P=4096)
    samples = orc.grid_centres(48)
    rng = np.random.default_rng(62)
    up_np = [rng.normal(size=samples.shape[0]).astype(np.float32) for _ in range(2)]
    with modes() as _C:
        ta = [T(x, cuda) for x in a]
        _C.build_bvh(T(samples, cuda), False, False)
        _C.set_count_pairs(True)
        try:
            fa = forward(_C, ta)
            g = backward(_C, [x.clone() for x in ta], fa, [T(u, cuda) for u in up_np])
            st = _C.stats()
        finally:
            _C.set_count_pairs(False)
    assert st["bwd_node_visits"] == 0
    assert_grads_close(g, oracle_backward(orc, tuple(a) + (samples,), fa[0].cpu().numpy(), fa[1].cpu().numpy(),
                                          fa[2].cpu().numpy().reshape(-1, 6), *up_np))


def test_copies_under_capture(cuda, orc):
    """A backward of copies is captured after one of the forward's own arrays has grown its buffers."""
    import torch
    a = orc.mixture_small(seed=3, P=4096)
    samples = orc.grid_centres(48)
    rng = np.random.default_rng(63)
    up = [T(rng.normal(size=samples.shape[0]).astype(np.float32), cuda) for _ in range(2)]
    with modes() as _C:
        ta = [T(x, cuda) for x in a]
        _C.build_bvh(T(samples, cuda), False, False)
        out, outw, conics = forward(_C, ta)

        def run(t):
            return _C.rasterize_gaussians_backward(t[0], t[1], t[2], conics, t[3], t[4], out, outw, 1.0, 0, 0, 0, 1, 1, 1,
                                                   -1.0, *up, False, False)
        want = run(ta)
        copies = [x.clone() for x in ta]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run(copies)
        graph.replay()
        _C.check_status()
        # the atomics' order alone differs
        for g, w in zip(got, want):
            assert (g - w).abs().max() <= 1e-4 * w.abs().max()
