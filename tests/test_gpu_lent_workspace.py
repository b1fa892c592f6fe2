"""A context lent a workspace for training samples keeps the buffers of its own: a mesh sampler
that has grown to its sizes stays capturable afterwards (an allocation ends a capture)."""
import ctypes

import numpy as np
import pytest
import torch

import gvc_native

pytestmark = pytest.mark.gpu


def test_sampler_capturable_after_a_lent_workspace(cuda, orc):
    pts, tets = orc.jittered_tet_mesh(n=12, seed=4)
    C, N, B, S = tets.shape[0], 20_000, 2, 5000
    q = np.random.default_rng(5).random((N, 3)).astype(np.float32)
    d_pts = torch.from_numpy(np.ascontiguousarray(pts, np.float32)).to(cuda)
    d_tets = torch.from_numpy(np.ascontiguousarray(tets, np.int32)).to(cuda)
    d_vals = torch.from_numpy(orc.blob_field(pts).astype(np.float64)).to(cuda)
    d_q = torch.from_numpy(q).to(cuda)
    out = [torch.zeros(N, dtype=torch.float64, device=cuda) for _ in range(2)]
    batches = torch.empty((B, S, 3), device=cuda)
    gt = torch.empty((B, S), device=cuda)
    size = gvc_native.lib().gvc_training_workspace(C, B, S, 1)
    work = torch.empty(size, dtype=torch.uint8, device=cuda)
    ctx = gvc_native.Context()
    p = gvc_native.ptr

    def st():
        return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def sample(dst):
        ctx.call("gvc_sample_tets", pts.shape[0], p(d_pts), C, p(d_tets), p(d_vals), N, p(d_q), p(dst), None, st())

    sample(out[0])
    ctx.call("gvc_training_samples_in", pts.shape[0], p(d_pts), C, p(d_tets), p(d_vals), B, S, ctypes.c_uint64(1),
             p(batches), p(gt), p(work), size, st())
    ctx.sync_status(st().value)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sample(out[1])
    graph.replay()
    ctx.sync_status(st().value)
    assert (out[0] != -1.0).any()
    assert torch.equal(out[0], out[1])
