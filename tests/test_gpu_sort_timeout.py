"""A sort whose look-back runs out (a block's count that nothing publishes) over an order that held
no indices: the timeout is reported, what gathers by the order stays within the arrays, and the
context sorts on."""
import ctypes

import numpy as np
import pytest
import torch

import gvc_native
from test_gpu_rasterizer import T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 12_288, 20_001])
def test_order_stays_in_range(cuda, orc, n):
    pts = np.random.default_rng(n).random((n, 3)).astype(np.float32)
    d = T(pts, cuda)
    ctx = gvc_native.Context()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    perm = torch.empty(n, dtype=torch.int32, device=cuda)
    slots = torch.empty((n, 4), device=cuda)
    p = gvc_native.ptr
    ctx.call("gvc_debug_sort_timeout", n, p(d), p(perm), p(slots), st)
    with pytest.raises(gvc_native.GvcError) as e:
        ctx.sync_status(st.value)
    assert e.value.code == gvc_native.GVC_ERR_TIMEOUT
    order = perm.cpu().numpy()
    assert order.min() >= 0 and order.max() < n
    got = slots.cpu().numpy()
    np.testing.assert_array_equal(got[:, 3].copy().view(np.int32), order)
    np.testing.assert_array_equal(got[:, :3], pts[order])
    # cleared, and a sort whose blocks all run is right
    ctx.sync_status(st.value)
    keys = torch.empty(n, dtype=torch.int32, device=cuda)
    ctx.call("gvc_build_bvh", p(d), n, 0, 0, st)
    ctx.call("gvc_debug_sample_order", p(perm), p(keys), st)
    ctx.sync_status(st.value)
    _, skeys, want = orc.morton30_points(pts)
    np.testing.assert_array_equal(perm.cpu().numpy(), want)
    np.testing.assert_array_equal(keys.cpu().numpy().view(np.uint32), skeys)
