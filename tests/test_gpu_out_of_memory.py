"""A forward that finds no device memory half way: it reports GVC_ERR_CUDA, once, and the context
works on."""
import ctypes
import gc

import numpy as np
import pytest
import torch

import gvc_native
from test_gpu_rasterizer import T, assert_grads_close, oracle_backward

pytestmark = pytest.mark.gpu

p = gvc_native.ptr
ONE, BG = ctypes.c_float(1.0), ctypes.c_float(-1.0)
MODES = [1, 3]  # Gaussian-owned sums, tensor-core sums


class Calls:
    """A context with one forward done, and one of four million Gaussians that finds no memory."""

    def __init__(self, cuda, orc, mode):
        self.a = orc.mixture_small(seed=5, P=3000)
        self.samples = orc.grid_centres(24)
        self.S = self.samples.shape[0]
        self.st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        self.ctx = gvc_native.Context()
        self.ctx.set_option(gvc_native.OPT_BWD_MODE, mode)
        self.dev = cuda
        self.ta = [T(x, cuda) for x in self.a]
        self.d_s = T(self.samples, cuda)
        self.ctx.call("gvc_build_bvh", p(self.d_s), self.S, 0, 0, self.st)
        self.outs = self.forward(self.ta)
        self.ctx.sync_status(self.st.value)
        self.fail()

    def outputs(self, n):
        return [torch.empty(k, device=self.dev) for k in (self.S, self.S, 6 * n)]

    def forward(self, t, outs=None):
        n = t[0].shape[0]
        outs = outs or self.outputs(n)
        self.ctx.call("gvc_rasterize_gaussians", n, *[p(x) for x in t], ONE, None, BG, 0, 0, *[p(o) for o in outs],
                      self.st)
        return outs

    def fail(self):
        n = 4_000_000
        t = [torch.rand((n, k), device=self.dev) * 0.01 + 0.01 for k in (3, 3, 4, 1, 1)]
        outs = self.outputs(n)
        gc.collect()  # contexts of earlier tests: what they free later would be found by the call
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        # the boxes (128 MB) and the sort's arrays fit, the records (320 MB) do not
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (340 << 20), dtype=torch.uint8, device=self.dev)
        try:
            with pytest.raises(gvc_native.GvcError, match="out of memory") as e:
                self.forward(t, outs)
            assert e.value.code == 2
        finally:
            del hold
            torch.cuda.empty_cache()


@pytest.mark.parametrize("mode", MODES)
def test_forward_after_a_failed_one(cuda, orc, mode):
    c = Calls(cuda, orc, mode)
    again = c.forward(c.ta)
    c.ctx.sync_status(c.st.value)
    assert all(torch.equal(x, y) for x, y in zip(again, c.outs))


@pytest.mark.parametrize("mode", MODES)
def test_backward_after_a_failed_forward(cuda, orc, mode):
    """Of the forward before it: what the failed one left (the order of more Gaussians) is not used."""
    c = Calls(cuda, orc, mode)
    rng = np.random.default_rng(91)
    up = [rng.normal(size=c.S).astype(np.float32) for _ in range(2)]
    d_up = [T(u, cuda) for u in up]
    means, scales, rots, values, weights = c.ta
    out, outw, conics = c.outs
    grads = [torch.empty((3000, k), device=cuda) for k in (3, 3, 4, 1, 1)]
    c.ctx.call("gvc_rasterize_gaussians_backward", 3000, p(means), p(scales), p(rots), p(conics), p(values),
               p(weights), p(out), p(outw), ONE, None, BG, p(d_up[0]), p(d_up[1]), 0, 0, *[p(g) for g in grads], c.st)
    c.ctx.sync_status(c.st.value)
    ref = oracle_backward(orc, tuple(c.a) + (c.samples,), out.cpu().numpy(), outw.cpu().numpy(),
                          conics.cpu().numpy().reshape(-1, 6), *up)
    assert_grads_close([g.cpu().numpy() for g in grads], ref)
