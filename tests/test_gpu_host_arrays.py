"""Host arrays of the mesh samplers: sizes on both sides of the 1 MB pinned chunks and of the
shares of their copying threads, several Python threads at once, and the checks on the device
against those on the host (_check_cells) over the forms that they accept and refuse."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,ns", [(np.uint8, 1), (np.uint8, 87_381), (np.uint8, 87_382), (np.float32, 262_144),
                                      (np.float32, 262_145), (np.float64, 131_073), (np.float32, 1_500_001)])
def test_copied_whole(cuda, orc, dtype, ns):
    from gpu_mesh_sampling import gpu_sample
    rng = np.random.default_rng(ns)
    dims = np.array([65, 33, 17])
    vals = (rng.random(dims.prod()) * 200).astype(dtype)
    q = (rng.random((ns, 3)) * 1.1 - 0.05).astype(np.float32)
    args = (dims, np.zeros(3, np.float32), (1.0 / (dims - 1)).astype(np.float32), vals, q)
    ref, valid = orc.sample_uniform(*args)
    want = orc.cast_sampled(ref, valid, dtype)
    got = [None] * 3

    def one(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = gpu_sample(*args)
    threads = [threading.Thread(target=one, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g in got:
        np.testing.assert_array_equal(g, want)


def _mesh(orc, kinds):
    pts, conn, types, offs = orc.mixed_cell_mesh(n=5, seed=1, kinds=kinds)
    return pts, np.asarray(conn, np.int64), np.asarray(types, np.int64), np.asarray(offs, np.int64)


def _set(a, i, v):
    a = a.copy()
    a[i] = v
    return a


FORMS = {
    "as given": lambda p, c, t, o: (c, t, o),
    "narrow types": lambda p, c, t, o: (c.astype(np.int32), t.astype(np.uint8), o.astype(np.int32)),
    "lists": lambda p, c, t, o: (c.tolist(), t.tolist(), o.tolist()),
    "strided": lambda p, c, t, o: (np.repeat(c, 2)[::2], np.repeat(t, 2)[::2], np.repeat(o, 2)[::2]),
    "no last offset": lambda p, c, t, o: (c, t, o[:-1]),
    "ids in front": lambda p, c, t, o: (np.concatenate([[0, 1], c]), t, o + 2),
    "bad ids in front": lambda p, c, t, o: (np.concatenate([[-1, 10 ** 6], c]), t, o + 2),
    "wide id": lambda p, c, t, o: (_set(c, 3, c[3] + 2 ** 32), t, o),
    "id too large": lambda p, c, t, o: (_set(c, -1, p.shape[0]), t, o),
    "negative id": lambda p, c, t, o: (_set(c, 0, -1), t, o),
    "unknown type": lambda p, c, t, o: (c, _set(_set(t, 7, 11), 9, -4), o),
    "type 16": lambda p, c, t, o: (c, _set(t, -1, 16), o),
    "wrong count": lambda p, c, t, o: (c, _set(t, 4, 3), o),
    "long last cell": lambda p, c, t, o: (np.concatenate([c, [0]]), t, o),
    "offset off": lambda p, c, t, o: (c, t, _set(o, 5, o[5] + 1)),
    "negative offset": lambda p, c, t, o: (c, t, o - 1),
    "few offsets": lambda p, c, t, o: (c, t, o[:3]),
    "no cells": lambda p, c, t, o: (c[:0], t[:0], o[:0]),
}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("kinds", [(10,), (12, 13, 14, 10)])
def test_checks_match_host(cuda, orc, kinds, form):
    from gpu_mesh_sampling import _gpu_mesh_sampling as M
    pts, conn, types, offs = _mesh(orc, kinds)
    vals = orc.blob_field(pts).astype(np.float64)
    q = np.random.default_rng(0).random((500, 3)).astype(np.float32)
    c, t, o = FORMS[form](pts, conn, types, offs)

    def host():
        """The checks on the host; tetrahedra alone as four ids per cell."""
        hc, ht, ho = M._check_cells(c, t, o)
        if ht.size and np.all(ht == 10):
            return M.sample_meshu_cells(pts, hc[ho[:, None] + np.arange(4)], vals, q)[0]
        return M.sample_meshu_mixed(pts, c, t, o, vals, q)[0]

    try:
        want = host()
    except RuntimeError as e:
        with pytest.raises(RuntimeError) as got:
            M.sample_meshu(pts, c, t, o, vals, q)
        assert str(got.value) == str(e)
        return
    np.testing.assert_array_equal(M.sample_meshu(pts, c, t, o, vals, q), want)
    with pytest.raises(RuntimeError, match="one entry per point") if len(t) else pytest.raises(RuntimeError):
        M.sample_meshu(pts, c, t, o, vals[:-1], q)


def test_training_refuses_wide_ids(cuda, orc):
    from gpu_mesh_sampling import sample_training_batches
    pts, tets = orc.jittered_tet_mesh(n=3, seed=1)
    vals = orc.blob_field(pts).astype(np.float64)
    for bad in (tets.max() + 1, -1, int(tets[5, 1]) + 2 ** 32):
        with pytest.raises(RuntimeError, match="outside the point array"):
            sample_training_batches(pts, _set(tets.astype(np.int64), (5, 1), bad), vals, 1, 100)
