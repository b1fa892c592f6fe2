"""Morton sort on both sides of the one-CTA kernel's limit (8192), of its rounds of 1024 and of
a warp, with equal keys among them: keys and stable order equal the oracle's."""
import numpy as np
import pytest

import gvc_native
from test_gpu_rasterizer import gpu_lbvh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda):
    return gvc_native.Context()


@pytest.mark.parametrize("kind", ["rand", "dup"])
@pytest.mark.parametrize("n", [31, 1023, 1024, 1025, 7169, 8192, 8193])
def test_small_sort_bit_exact(ctx, cuda, orc, n, kind):
    rng = np.random.default_rng(n)
    c = rng.random((n, 3)).astype(np.float32)
    if kind == "dup":
        c = c[rng.integers(0, max(n // 50, 1), n)]
    boxes = np.concatenate([c - 0.01, c + 0.01], 1).astype(np.float32)
    keys, perm, left, right, node_boxes = gpu_lbvh(ctx, cuda, boxes)
    k, p, l, r, nb = orc.lbvh_build(boxes)
    np.testing.assert_array_equal(keys, k)
    np.testing.assert_array_equal(perm, p)
    np.testing.assert_array_equal(left, l)
    np.testing.assert_array_equal(right, r)
    np.testing.assert_array_equal(node_boxes, nb)
