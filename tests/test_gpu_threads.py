"""Several Python threads in the entry points that share a context per device: meshes of different
kinds and sizes, so that one call's buffers are too small for the next, and 3-NN sets, each on the
thread's own stream or all on the default one.  Every thread gets what it gets alone."""
import threading

import numpy as np
import pytest
import torch

from test_gpu_rasterizer import T

pytestmark = pytest.mark.gpu


def together(jobs, rounds):
    """Runs every job `rounds` times, one thread each, started together; the results by job."""
    got, errors = [[] for _ in jobs], []
    start = threading.Barrier(len(jobs))

    def one(i):
        try:
            start.wait()
            for _ in range(rounds):
                got[i].append(jobs[i]())
        except Exception as e:  # reported by the main thread
            errors.append(e)
    threads = [threading.Thread(target=one, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return got


@pytest.mark.parametrize("own_streams", [False, True])
def test_mesh_samplers(cuda, orc, own_streams):
    from gpu_mesh_sampling import gpu_sampleu
    meshes = []
    for n, kinds in ((3, (10,)), (9, (12, 13, 14, 10)), (14, (10,)), (6, (12,))):
        pts, conn, types, offs = orc.mixed_cell_mesh(n=n, seed=n, kinds=kinds)
        q = np.random.default_rng(n).random((3000 * n, 3)).astype(np.float32)
        meshes.append((pts, conn, types, offs, orc.blob_field(pts).astype(np.float64), q))
    want = [gpu_sampleu(*m) for m in meshes]

    def job(m):
        def run():
            if not own_streams:
                return gpu_sampleu(*m)
            with torch.cuda.stream(torch.cuda.Stream()):
                return gpu_sampleu(*m)
        return run
    for g, w in zip(together([job(m) for m in meshes], 6), want):
        assert (w != -1.0).any()
        for x in g:
            np.testing.assert_array_equal(x, w)


def test_nearest(cuda):
    from simple_knn._C import distCUDA2
    sets = [T(np.random.default_rng(n).random((n, 3)).astype(np.float32), cuda) for n in (700, 9000, 30_000, 120_000)]
    want = [distCUDA2(s).clone() for s in sets]
    torch.cuda.synchronize()
    got = together([lambda s=s: distCUDA2(s) for s in sets], 6)
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert all(torch.equal(x, w) for x in g)
