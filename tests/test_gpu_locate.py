"""Point location by the wide tree (mesh.cu) where it can go wrong: the plane pre-test at
scales, offsets and shapes that shift its rounding (quantised and sliver tetrahedra, a mesh
far from the origin, ranges where the planes are left out), sample counts on both sides of
the samples-per-warp rule with partial warps, runs of samples that jump across the mesh, NaN
samples, and points on vertices and edges.  Cell ids and values equal the oracle's bit for
bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,offset,squash,ns", [
    (1.0, 0.0, 1.0, 1), (1.0, 0.0, 1.0, 31), (1.0, 0.0, 1.0, 8289), (1.0, 0.0, 1.0, 132_609),
    (1e-3, 5.0, 1.0, 132_607), (1e6, -3e5, 1.0, 20_000), (1.0, 0.0, 1e-4, 140_000), (1e-20, 0.0, 1.0, 20_000),
    (1e-34, 0.0, 1.0, 5000), (1e9, 0.0, 1e-7, 20_000)])
def test_tets_match_oracle(cuda, orc, scale, offset, squash, ns):
    from gpu_mesh_sampling._gpu_mesh_sampling import sample_meshu_cells
    pts, tets = orc.jittered_tet_mesh(n=17, seed=7)
    vals = orc.blob_field(pts).astype(np.float64)
    pts = (pts.astype(np.float64) * scale * np.array([1.0, 1.0, squash]) + offset).astype(np.float32)
    rng = np.random.default_rng(ns)
    lo, hi = pts.min(0).astype(np.float64), pts.max(0).astype(np.float64)
    q = (lo + rng.random((ns, 3)) * (hi - lo) * 1.02 - 0.01 * (hi - lo)).astype(np.float32)
    k = ns // 10
    q[:k] = pts[rng.integers(0, pts.shape[0], k)]
    a, b = tets[rng.integers(0, tets.shape[0], k), :2].T
    q[k:2 * k] = ((pts[a].astype(np.float64) + pts[b]) * 0.5).astype(np.float32)
    q[2 * k:2 * k + 3] = np.nan
    out, cell = sample_meshu_cells(pts, tets, vals, q)
    ref, rcell = orc.sample_tets(pts, tets, vals, q)
    np.testing.assert_array_equal(cell, rcell)
    np.testing.assert_array_equal(out, ref)


def test_scattered_samples_match_oracle(cuda, orc):
    """Two hundred samples per side of a fine mesh: every run spans much of it."""
    from gpu_mesh_sampling._gpu_mesh_sampling import sample_meshu_cells, sample_meshu_mixed
    pts, tets = orc.jittered_tet_mesh(n=40, seed=9)
    vals = orc.blob_field(pts).astype(np.float64)
    q = np.random.default_rng(1).random((200, 3)).astype(np.float32)
    q = np.repeat(q, 700, 0)[np.random.default_rng(2).permutation(140_000)]  # equal keys, far from the next
    ref, rcell = orc.sample_tets(pts, tets, vals, q)
    out, cell = sample_meshu_cells(pts, tets, vals, q)
    np.testing.assert_array_equal(cell, rcell)
    np.testing.assert_array_equal(out, ref)
    C = tets.shape[0]
    out, cell = sample_meshu_mixed(pts, tets.reshape(-1).astype(np.int64), np.full(C, 10), np.arange(C + 1) * 4, vals, q)
    np.testing.assert_array_equal(cell, rcell)
    np.testing.assert_array_equal(out, ref)
