"""The framework's workloads as timed cases: what a program that uses it has it compute.

A training program (train.py of the reference project, which runs unchanged on these
packages) spends its time in one step: index the step's sample points (build_bvh), evaluate
the mixture at them (forward) and its adjoint (backward).  Around that it renders whole
grids for evaluation, computes initial scales (distCUDA2), and makes its targets by sampling
volumes and meshes.  The families below are those calls:

  step     build_bvh + forward + backward through GaussianRasterizer and autograd; the loss
           is the caller's own, so its gradients with respect to both outputs are inputs
  render   build_bvh + forward without gradients, on a grid in storage order
  nearest  distCUDA2
  uniform  gpu_sample: host arrays in, host array out
  cells    gpu_sampleu: host arrays in, host array out (tetrahedra, or hexahedra and wedges)
  batches  sample_training_batches: mesh on the host, batches on the device

Mixtures ("mix"):
  uniform    means U[0,1]^3, log-scales N(log s, 0.3), random rotations, w = sigmoid(N(0,1)),
             s = 0.02 at 4096 Gaussians and the same coverage at other counts
  lattice    the start of a fit: distinct points of a 256^3 lattice, isotropic scales of a
             3-nearest-neighbour distance with the soft cap of 0.02, no rotation, w = 0.1
  fitted     the same points later on: scales spread by N(0, 0.3), rotated, w of sigmoid(N(-1,1))
  clustered  256 clusters of deviation 0.05, log-scales N(log 0.004, 0.4); half the samples
             uniform, half near the means
Sample orders ("order"): "random"; "morton" (the training program sorts each batch); "grid".
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gaussian-volume-compression_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)


def listed():
    return [
        # the small mixture at the cell centres of a 64^3 grid, library defaults: a step whose
        # kernels are short, so launches and host work count
        {"name": "step_small", "family": "step", "mix": "uniform", "P": 4096, "S": 64 ** 3, "order": "grid",
         "backward": "auto", "evaluate": "plain", "gaussian_bvh": False},
        # the training program as it stands (library defaults): one Morton-sorted batch of 128^3
        # points on a mixture in mid-fit
        {"name": "step_train", "family": "step", "mix": "fitted", "P": 300_000, "S": 128 ** 3, "order": "morton",
         "backward": "auto", "evaluate": "plain", "gaussian_bvh": False},
        # the first steps of a structured-volume fit, with the tensor-core backward
        {"name": "step_fit", "family": "step", "mix": "lattice", "P": 200_000, "S": 4_000_000, "order": "random",
         "backward": "tensor_core", "evaluate": "plain", "gaussian_bvh": False},
        # the large evaluation, the benchmark's own configuration
        {"name": "step_large", "family": "step", "mix": "clustered", "P": 2_000_000, "S": 16_000_000,
         "order": "random", "backward": "tensor_core", "evaluate": "plain", "gaussian_bvh": False},
        # a large mixture with the library defaults, sizes that fill no tile
        {"name": "step_ragged", "family": "step", "mix": "clustered", "P": 999_983, "S": 3_999_971,
         "order": "random", "backward": "auto", "evaluate": "plain", "gaussian_bvh": False},
        # the rasterizer's Gaussian-BVH switch (sample-side sums)
        {"name": "step_gaussian_bvh", "family": "step", "mix": "clustered", "P": 200_000, "S": 1_000_000,
         "order": "random", "backward": "auto", "evaluate": "plain", "gaussian_bvh": True},
        # tensor cores in both directions
        {"name": "step_tensor", "family": "step", "mix": "fitted", "P": 500_000, "S": 1_500_000, "order": "morton",
         "backward": "auto", "evaluate": "tensor_core", "gaussian_bvh": False},
        # evaluation of a compressed volume: the whole 256^3 grid in storage order, no gradients
        {"name": "render_grid", "family": "render", "mix": "fitted", "P": 500_000, "S": 256 ** 3, "order": "grid",
         "backward": "auto", "evaluate": "plain", "gaussian_bvh": False},
        # initial scales of a large point cloud
        {"name": "nearest", "family": "nearest", "mix": "clustered", "P": 2_000_000},
        # targets out of a structured volume
        {"name": "sample_uniform", "family": "uniform", "n": 256, "S": 4_000_000, "dtype": "float32"},
        # targets out of a tetrahedral mesh
        {"name": "sample_cells", "family": "cells", "n": 40, "S": 2_000_000, "kind": "tets"},
        # a training run's batches out of a tetrahedral mesh
        {"name": "training_batches", "family": "batches", "n": 64, "batches": 12, "S": 128 ** 3},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]; odd more often than not."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.6:
        v |= 1
    return max(lo, min(hi, v))


def draw(rng):
    family = rng.choice(["step"] * 8 + ["render"] * 2 + ["nearest", "uniform", "cells", "batches"])
    if family in ("step", "render"):
        mix = rng.choice(["uniform", "lattice", "fitted", "clustered", "clustered"])
        c = {"family": family, "mix": mix, "P": 0, "S": 0, "order": rng.choice(["random", "morton", "grid"]),
             "backward": "auto", "evaluate": "plain", "gaussian_bvh": False}
        if mix == "clustered":
            # the clusters' scales do not shrink with the count: from 20k Gaussians up
            c["P"], c["order"] = _spread(rng, 20_000, 1_500_000), "random"
        else:
            c["P"] = _spread(rng, 512, 1_000_000)
        if family == "step":
            how = rng.choice(["default", "default", "tensor_core", "tensor_core", "both", "gaussian_bvh"])
            c["S"] = _spread(rng, 13_824, 8_000_000 if how == "tensor_core" else 3_000_000)
            if how == "tensor_core":
                c["backward"] = "tensor_core"
            elif how == "both":
                c["evaluate"] = "tensor_core"
            elif how == "gaussian_bvh":
                c["gaussian_bvh"] = True
                c["P"] = min(c["P"], 500_000)
        else:
            c["S"] = _spread(rng, 13_824, 16_000_000)
            c["evaluate"] = rng.choice(["plain", "plain", "tensor_core"])
        if c["order"] == "grid":
            c["S"] = max(2, int(round(c["S"] ** (1.0 / 3.0)))) ** 3
        return c
    if family == "nearest":
        return {"family": "nearest", "mix": rng.choice(["uniform", "lattice", "clustered"]),
                "P": _spread(rng, 512, 3_000_000)}
    if family == "uniform":
        return {"family": "uniform", "n": _spread(rng, 32, 320), "S": _spread(rng, 20_000, 8_000_000),
                "dtype": rng.choice(["float32", "float64", "uint16", "uint8"])}
    if family == "cells":
        kind = rng.choice(["tets", "hexes", "mixed"])
        return {"family": "cells", "n": _spread(rng, 6, 48), "S": _spread(rng, 20_000, 2_000_000), "kind": kind}
    return {"family": "batches", "n": _spread(rng, 8, 64), "batches": rng.randint(1, 12),
            "S": _spread(rng, 20_000, 128 ** 3)}


# ---- inputs ------------------------------------------------------------------------------

def _generator(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _spacing_scale(P):
    """sqrt of the mean of the three smallest squared distances of P uniform points."""
    return 0.7525 * P ** (-1.0 / 3.0)


def _scale_of(mix, P):
    if mix == "clustered":
        return 0.004
    if mix == "uniform":
        return 0.02 * (4096.0 / P) ** (1.0 / 3.0)
    s = _spacing_scale(P)
    r = math.sqrt(3.0) * s
    return s * 0.02 * math.tanh(r / 0.02) / r


def _means(mix, P, g):
    if mix == "clustered":
        centres = torch.rand(256, 3, generator=g, device="cuda")
        label = torch.randint(0, 256, (P,), generator=g, device="cuda")
        return (centres[label] + 0.05 * torch.randn(P, 3, generator=g, device="cuda")).clamp(0, 1).contiguous()
    if mix == "uniform":
        return torch.rand(P, 3, generator=g, device="cuda")
    n = 256
    at = torch.randperm(n ** 3, generator=g, device="cuda")[:P]
    return (torch.stack([at % n, (at // n) % n, at // (n * n)], 1).float() / (n - 1)).contiguous()


def _mixture(mix, P, g):
    """(means [P,3], scales [P,3], rotations [P,4], values [P,1], weights [P,1]), activated."""
    means = _means(mix, P, g)
    spread = {"clustered": 0.4, "uniform": 0.3, "fitted": 0.3, "lattice": 0.0}[mix]
    scales = torch.exp(spread * torch.randn(P, 3, generator=g, device="cuda")) * _scale_of(mix, P)
    values = torch.rand(P, 1, generator=g, device="cuda")
    if mix == "lattice":
        rots = torch.zeros(P, 4, device="cuda")
        rots[:, 0] = 1.0
        weights = torch.full((P, 1), 0.1, device="cuda")
    else:
        rots = torch.nn.functional.normalize(torch.randn(P, 4, generator=g, device="cuda"))
        weights = torch.sigmoid(torch.randn(P, 1, generator=g, device="cuda") - (1.0 if mix == "fitted" else 0.0))
    return means, scales, rots, values, weights


def _part_bits(v, bits):
    out = torch.zeros_like(v)
    for b in range(bits):
        out |= ((v >> b) & 1) << (3 * b)
    return out


def _morton(points, bits):
    q = (points.clamp(0, 1) * float(2 ** bits - 1)).to(torch.int64)
    return _part_bits(q[:, 0], bits) | (_part_bits(q[:, 1], bits) << 1) | (_part_bits(q[:, 2], bits) << 2)


def _samples(case, means, scales, g):
    S = case["S"]
    if case["order"] == "grid":
        n = int(round(S ** (1.0 / 3.0)))
        c = (torch.arange(n, dtype=torch.float32, device="cuda") + 0.5) / n
        z, y, x = torch.meshgrid(c, c, c, indexing="ij")
        return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1).contiguous()
    if case["mix"] == "clustered":
        half = S // 2
        j = torch.randint(0, means.shape[0], (S - half,), generator=g, device="cuda")
        near = means[j] + torch.randn(S - half, 3, generator=g, device="cuda") * scales[j]
        pts = torch.cat([torch.rand(half, 3, generator=g, device="cuda"), near])
    else:
        pts = torch.rand(S, 3, generator=g, device="cuda")
    if case["order"] == "morton":
        pts = pts[torch.argsort(_morton(pts, 21))]
    return pts.contiguous()


def _field(case, seed):
    """Inputs of a step or a render: parameters, sample points and upstream gradients (those of
    an L1 loss averaged over the samples, with a small regulariser on the weights)."""
    g = _generator(seed)
    params = _mixture(case["mix"], case["P"], g)
    pts = _samples(case, params[0], params[1], g)
    S = pts.shape[0]
    g_cells = torch.sign(torch.rand(S, generator=g, device="cuda") - 0.5) / S
    g_weights = 0.1 * torch.randn(S, generator=g, device="cuda") / S
    return params, pts, g_cells, g_weights


def _grid_points(n, jitter, g):
    """Vertices of an n^3 cell grid on [0,1]^3, the inner ones moved by up to jitter cells."""
    h = 1.0 / n
    c = torch.arange(n + 1, dtype=torch.float64, device="cuda") * h
    z, y, x = torch.meshgrid(c, c, c, indexing="ij")
    p = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    inner = ((p > 0.5 * h) & (p < 1 - 0.5 * h)).all(1, keepdim=True)
    move = (torch.rand(p.shape, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * jitter * h
    return (p + inner * move).float()


def _corners(n):
    """[n^3, 8] vertex ids of the grid's cells in VTK hexahedron order, and its (i, j, k)."""
    at = torch.arange(n ** 3, device="cuda")
    i, j, k = at % n, (at // n) % n, at // (n * n)
    m = n + 1

    def v(a, b, c):
        return (k + c) * m * m + (j + b) * m + (i + a)

    return torch.stack([v(0, 0, 0), v(1, 0, 0), v(1, 1, 0), v(0, 1, 0),
                        v(0, 0, 1), v(1, 0, 1), v(1, 1, 1), v(0, 1, 1)], 1), (i, j, k)


# the six tetrahedra of a hexahedron along its diagonal 0-6, in VTK hexahedron vertices
_TETS = [[0, 1, 2, 6], [0, 1, 5, 6], [0, 3, 2, 6], [0, 3, 7, 6], [0, 4, 5, 6], [0, 4, 7, 6]]
# the two wedges of a hexahedron split along its 1-3 diagonal
_WEDGES = [[0, 1, 3, 4, 5, 7], [1, 2, 3, 5, 6, 7]]


def _mesh(case, seed):
    """Point positions, a smooth point field, and per grid cell its hexahedron's vertices."""
    g = _generator(seed)
    n = case["n"]
    pts = _grid_points(n, 0.2, g)
    c = torch.rand(16, 3, generator=g, device="cuda", dtype=torch.float64)
    p = pts.double()
    vals = torch.zeros(p.shape[0], dtype=torch.float64, device="cuda")
    for b in range(16):
        vals += torch.exp(-0.5 * ((p - c[b]) ** 2).sum(1) / (0.1 + 0.01 * b) ** 2)
    hexes, ijk = _corners(n)
    return g, pts, vals, hexes, ijk


def _is_wedge(case, ijk):
    """Every third column of a mixed mesh is split into wedges."""
    if case["kind"] != "mixed":
        return torch.zeros_like(ijk[0], dtype=torch.bool)
    return (ijk[0] + ijk[1]) % 3 == 0


def _query_points(S, g):
    """Points over a slightly larger box than the mesh: a few per cent lie outside."""
    return (torch.rand(S, 3, generator=g, device="cuda") * 1.02 - 0.01).contiguous()


def _cells_inputs(case, seed):
    g, pts, vals, hexes, ijk = _mesh(case, seed)
    q = _query_points(case["S"], g)
    if case["kind"] == "tets":
        conn = torch.stack([hexes[:, t] for t in _TETS], 1).reshape(-1)
        types = torch.full((conn.numel() // 4,), 10, dtype=torch.int64, device="cuda")
        sizes = torch.full_like(types, 4)
    else:
        wedge = _is_wedge(case, ijk)
        count = torch.where(wedge, 2, 1)
        types = torch.repeat_interleave(torch.where(wedge, 13, 12), count)
        sizes = torch.where(types == 13, 6, 8)
        rows = torch.repeat_interleave(torch.arange(hexes.shape[0], device="cuda"), count)
        second = torch.cat([torch.zeros(1, dtype=torch.bool, device="cuda"), rows[1:] == rows[:-1]])
        full = hexes[rows]
        w0, w1 = torch.tensor(_WEDGES[0], device="cuda"), torch.tensor(_WEDGES[1], device="cuda")
        six = torch.where(second[:, None], full[:, w1], full[:, w0])
        padded = torch.where((types == 13)[:, None], torch.cat([six, six[:, :2]], 1), full)
        conn = padded[torch.arange(8, device="cuda")[None] < sizes[:, None]]
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(sizes, 0)])
    return pts, conn, types, offsets, vals, q


def _volume(case, seed):
    """An n^3 point field (x fastest) in the case's type, its grid, and points to sample."""
    g = _generator(seed)
    n = case["n"]
    t = torch.arange(n, dtype=torch.float32, device="cuda") / (n - 1)
    k = torch.randint(1, 9, (6, 3), generator=g, device="cuda").float()
    ph = torch.rand(6, generator=g, device="cuda") * 6.28
    v = torch.zeros(n, n, n, device="cuda")
    for m in range(6):
        v += torch.cos(6.2831853 * (k[m, 2] * t[:, None, None] + k[m, 1] * t[None, :, None] +
                                    k[m, 0] * t[None, None, :]) + ph[m]) / (1 + m)
    v = (v - v.min()) / (v.max() - v.min())
    top = {"uint8": 255.0, "uint16": 65535.0}.get(case["dtype"])
    v = v if top is None else torch.round(v * top)
    return v.reshape(-1), _query_points(case["S"], g)


def prepare(case, seed):
    family = case["family"]
    if family in ("step", "render"):
        from bvh_diff_gaussian_rasterization import GaussianRasterizationSettings, GaussianRasterizer
        params, pts, g_cells, g_weights = _field(case, seed)
        settings = GaussianRasterizationSettings(
            volume_mins=(0.0, 0.0, 0.0), volume_maxes=(1.0, 1.0, 1.0), cell_count=pts.shape[0], bg=-1.0,
            scale_modifier=1.0, use_gaussian_bvh=bool(case["gaussian_bvh"]), debug=False)
        state = {"rasterizer": GaussianRasterizer(settings), "samples": pts}
        if family == "step":
            params = [p.requires_grad_(True) for p in params]
            state["upstream"] = (g_cells, g_weights)
        state["params"] = list(params)
    elif family == "nearest":
        state = {"points": _means(case["mix"], case["P"], _generator(seed))}
    elif family == "uniform":
        v, q = _volume(case, seed)
        n = case["n"]
        state = {"args": (np.array([n, n, n], dtype=np.int64), np.zeros(3, np.float32),
                          np.full(3, 1.0 / (n - 1), np.float32),
                          v.cpu().numpy().astype(case["dtype"]), q.cpu().numpy())}
    elif family == "cells":
        state = {"args": tuple(x.cpu().numpy() for x in _cells_inputs(case, seed))}
    else:
        _, pts, vals, hexes, _ = _mesh(case, seed)
        tets = torch.stack([hexes[:, t] for t in _TETS], 1).reshape(-1, 4)
        state = {"mesh": tuple(x.cpu().numpy() for x in (pts, tets, vals)), "seed": int(seed)}
    state["case"] = dict(case)
    return state


# ---- one pass ----------------------------------------------------------------------------

def run(state):
    case = state["case"]
    family = case["family"]
    if family in ("step", "render"):
        from bvh_diff_gaussian_rasterization import _C
        # the program's choice of kernels (per device, kept by the library)
        _C.set_eval_path(case["evaluate"])
        _C.set_backward_mode(case["backward"])
        r = state["rasterizer"]
        means, scales, rots, values, weights = state["params"]
        r.build_bvh(state["samples"], use_gaussian_bvh=bool(case["gaussian_bvh"]))
        if family == "render":
            with torch.no_grad():
                cells, cell_weights = r(means, scales, rots, values, weights)
            return {"cells": cells, "weights": cell_weights}
        cells, cell_weights = r(means, scales, rots, values, weights)
        grads = torch.autograd.grad((cells, cell_weights), state["params"], state["upstream"])
        names = ("d_means", "d_scales", "d_rotations", "d_values", "d_weights")
        return {"cells": cells.detach(), "weights": cell_weights.detach(), **dict(zip(names, grads))}
    if family == "nearest":
        from simple_knn._C import distCUDA2
        return distCUDA2(state["points"])
    if family == "uniform":
        from gpu_mesh_sampling import gpu_sample
        return gpu_sample(*state["args"])
    if family == "cells":
        from gpu_mesh_sampling import gpu_sampleu
        return gpu_sampleu(*state["args"])
    from gpu_mesh_sampling import sample_training_batches
    pts, tets, vals = state["mesh"]
    samples, gt = sample_training_batches(pts, tets, vals, case["batches"], case["S"], seed=state["seed"])
    return {"samples": samples, "targets": gt}


# ---- the work of a pass --------------------------------------------------------------------

def _pairs(case):
    """Expected contributing (sample, Gaussian) pairs: the volume in which a Gaussian counts is
    the part of its ellipsoid of power -14 inside its box, about 480 s^3 at the weights of a
    fitted mixture (counted at 2M x 16M) and the box of 223 s^3 at w = 0.1."""
    s = _scale_of(case["mix"], case["P"])
    spread = {"clustered": 0.4, "uniform": 0.3, "fitted": 0.3, "lattice": 0.0}[case["mix"]]
    v = (223.0 if case["mix"] == "lattice" else 480.0) * s ** 3 * math.exp(4.5 * spread * spread)
    return case["P"] * case["S"] * min(1.0, v)


def work(case):
    family = case["family"]
    if family in ("step", "render"):
        P, S = case["P"], case["S"]
        # 28 operations and one exponential (8 in kind) of a contributing pair forward, 64 and one backward
        byts, flops = 12.0 * S + 48.0 * P + 8.0 * S, 36.0 * _pairs(case)
        if family == "step":
            byts, flops = byts + 8.0 * S + 48.0 * P, flops + 72.0 * _pairs(case)
        return {"bytes": byts, "flops": flops}
    if family == "nearest":
        # three neighbours: each point against the three it keeps
        return {"bytes": 16.0 * case["P"], "flops": 3 * 8.0 * case["P"]}
    if family == "uniform":
        size = np.dtype(case["dtype"]).itemsize
        return {"bytes": size * float(case["n"]) ** 3 + (12.0 + size) * case["S"], "flops": 30.0 * case["S"]}
    cells = float(case["n"]) ** 3
    points = (case["n"] + 1.0) ** 3
    if family == "cells":
        # connectivity, types and offsets as 64-bit whole numbers
        per = {"tets": 6 * (4 + 2) * 8.0, "hexes": (8 + 2) * 8.0, "mixed": (28 / 3 + 8 / 3) * 8.0}[case["kind"]]
        return {"bytes": per * cells + 20.0 * points + (12.0 + 8.0) * case["S"], "flops": 150.0 * case["S"]}
    total = float(case["batches"]) * case["S"]
    return {"bytes": 6 * 32.0 * cells + 20.0 * points + 16.0 * total, "flops": 150.0 * total}


# ---- the same in 64 bits -------------------------------------------------------------------

def _rotation64(q):
    r, x, y, z = q.unbind(1)
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y)], 1),
        torch.stack([2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x)], 1),
        torch.stack([2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], 1)], 1)


def _conic64(scales, rots):
    R = _rotation64(rots)
    M = R * scales[:, None, :]
    cov = M @ M.transpose(1, 2)
    eps = 1e-5 * torch.diagonal(cov, dim1=1, dim2=2).abs().max(1).values
    return torch.linalg.inv(cov + eps[:, None, None] * torch.eye(3, dtype=cov.dtype, device=cov.device))


def _boxes64(means, scales, rots, weights):
    """The box of the corners mean +- m s_k R[k] (R's rows), m = sqrt(-2 ln(1e-3 / w)), rounded
    to 32 bits as the candidate test has it; a weight under 1e-3 leaves the mean."""
    R = _rotation64(rots)
    m = torch.sqrt(torch.clamp_min(-2.0 * torch.log(1e-3 / weights), 0.0))
    half = (R.abs() * (scales * m[:, None])[:, :, None]).sum(1)
    return (means - half).float().double(), (means + half).float().double()


def _tiles64(pts, lo, hi, rows, most):
    """(tile, Gaussian) index pairs whose boxes overlap, in pieces of at most about `most` pairs,
    for tiles of `rows` consecutive points."""
    T = pts.shape[0] // rows
    t = pts.view(T, rows, 3)
    tlo, thi = t.amin(1).float(), t.amax(1).float()
    glo, ghi = lo.float(), hi.float()
    P = lo.shape[0]
    step = max(1, int(2e8 // P))
    for a in range(0, T, step):
        b = min(T, a + step)
        hit = torch.ones(b - a, P, dtype=torch.bool, device=pts.device)
        for ax in range(3):
            hit &= (tlo[a:b, None, ax] <= ghi[None, :, ax]) & (thi[a:b, None, ax] >= glo[None, :, ax])
        pair = hit.nonzero()
        for c in range(0, pair.shape[0], most):
            yield pair[c:c + most, 0] + a, pair[c:c + most, 1]


def _field64(case, seed, gradients):
    params, pts32, g_cells, g_weights = _field(case, seed)
    means, scales, rots, values, weights = [p.detach().double() for p in params]
    values, weights = values[:, 0], weights[:, 0]
    S, rows, most = pts32.shape[0], 256, 200_000
    # points in spatial order, padded to whole tiles with copies of the last one
    order = torch.argsort(_morton(pts32, 10))
    pad = (-S) % rows
    full = torch.cat([order, order[-1:].expand(pad)])
    pts = pts32[full].double()
    T = pts.shape[0] // rows
    x = pts.view(T, rows, 3)
    scales.requires_grad_(gradients)
    rots.requires_grad_(gradients)
    conic = _conic64(scales, rots)
    C = conic.detach()
    lo, hi = _boxes64(means, scales.detach(), rots.detach(), weights)
    W = torch.zeros(T, rows, dtype=torch.float64, device=pts.device)
    V = torch.zeros_like(W)

    def pair_terms(ti, gi):
        p = x[ti]
        d = p - means[gi][:, None, :]
        inside = ((p >= lo[gi][:, None, :]) & (p <= hi[gi][:, None, :])).all(2)
        c = C[gi]
        power = -0.5 * (c[:, 0, 0, None] * d[..., 0] ** 2 + c[:, 1, 1, None] * d[..., 1] ** 2 +
                        c[:, 2, 2, None] * d[..., 2] ** 2 + 2 * c[:, 0, 1, None] * d[..., 0] * d[..., 1] +
                        2 * c[:, 0, 2, None] * d[..., 0] * d[..., 2] + 2 * c[:, 1, 2, None] * d[..., 1] * d[..., 2])
        e = torch.where(inside & (power >= -14.0) & (power <= 0.0), torch.exp(power), torch.zeros_like(power))
        return d, e

    for ti, gi in _tiles64(pts, lo, hi, rows, most):
        _, e = pair_terms(ti, gi)
        we = weights[gi][:, None] * e
        W.index_add_(0, ti, we)
        V.index_add_(0, ti, we * values[gi][:, None])
    valid = W > 0.01
    out = torch.where(valid, V / torch.where(valid, W, torch.ones_like(W)), torch.full_like(W, -1.0))
    outw = torch.where(valid, W, torch.zeros_like(W))

    def caller(t):
        r = torch.empty(S, dtype=torch.float64, device=t.device)
        r[order] = t.reshape(-1)[:S]
        return r

    result = {"cells": caller(out), "weights": caller(outw)}
    if not gradients:
        return result
    live = valid.clone()
    live.view(-1)[S:] = False
    gc = g_cells[full].double().view(T, rows)
    gw = g_weights[full].double().view(T, rows)
    zero = torch.zeros_like(W)
    dV = torch.where(live, gc / torch.where(valid, W, torch.ones_like(W)), zero)
    dW = torch.where(live, gw - dV * out, zero)
    P = means.shape[0]
    sums = {k: torch.zeros(P, *s, dtype=torch.float64, device=pts.device)
            for k, s in (("v", ()), ("w", ()), ("m", (3,)), ("c", (3, 3)))}
    for ti, gi in _tiles64(pts, lo, hi, rows, most):
        d, e = pair_terms(ti, gi)
        a = dV[ti] * e
        s = a * values[gi][:, None] + dW[ti] * e
        sums["v"].index_add_(0, gi, weights[gi] * a.sum(1))
        sums["w"].index_add_(0, gi, s.sum(1))
        first = torch.einsum("kr,kra->ka", s, d)
        second = torch.einsum("kra,krb->kab", s[..., None] * d, d)
        sums["m"].index_add_(0, gi, weights[gi][:, None] * torch.einsum("kab,kb->ka", C[gi], first))
        sums["c"].index_add_(0, gi, -0.5 * weights[gi][:, None, None] * second)
    d_scales, d_rots = torch.autograd.grad(conic, (scales, rots), sums["c"])
    result.update({"d_means": sums["m"], "d_scales": d_scales, "d_rotations": d_rots,
                   "d_values": sums["v"][:, None], "d_weights": sums["w"][:, None]})
    return result


def _nearest64(pts):
    p = pts.double()
    n = p.shape[0]
    out = torch.empty(n, dtype=torch.float64, device=p.device)
    step = max(1, int(1e8 // n))
    for a in range(0, n, step):
        b = min(n, a + step)
        d = torch.zeros(b - a, n, dtype=torch.float64, device=p.device)
        for ax in range(3):
            d += (p[a:b, None, ax] - p[None, :, ax]) ** 2
        d[torch.arange(b - a, device=p.device), torch.arange(a, b, device=p.device)] = math.inf
        out[a:b] = d.topk(3, dim=1, largest=False).values.mean(1)
    return out


def _uniform64(case, seed):
    v, q = _volume(case, seed)
    n = case["n"]
    v = v.to(getattr(torch, case["dtype"])).double().view(n, n, n)
    f = q.double() / float(np.float32(1.0 / (n - 1)))
    inside = ((f >= 0) & (f <= n - 1)).all(1)
    i = f.floor().long().clamp(0, n - 2)
    t = f - i
    out = torch.zeros(q.shape[0], dtype=torch.float64, device=q.device)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                w = ((t[:, 0] if dx else 1 - t[:, 0]) * (t[:, 1] if dy else 1 - t[:, 1]) *
                     (t[:, 2] if dz else 1 - t[:, 2]))
                out += w * v[i[:, 2] + dz, i[:, 1] + dy, i[:, 0] + dx]
    return torch.where(inside, out, torch.full_like(out, -1.0))


def _newton64(wedge, x, p):
    """Shape functions of the parametric place of p in the cells with vertices x ([K, 8 or 6, 3])
    and whether that place is inside."""
    K = p.shape[0]
    u = torch.full((K, 3), 0.5, dtype=torch.float64, device=p.device)
    if wedge:
        u[:, :2] = 1.0 / 3.0

    def shape(u):
        r, s, t = u.unbind(1)
        if wedge:
            tri = torch.stack([1 - r - s, r, s], 1)
            dr = torch.tensor([-1.0, 1.0, 0.0], dtype=torch.float64, device=p.device).expand(K, 3)
            ds = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device=p.device).expand(K, 3)
        else:
            tri = torch.stack([(1 - r) * (1 - s), r * (1 - s), r * s, (1 - r) * s], 1)
            dr = torch.stack([s - 1, 1 - s, s, -s], 1)
            ds = torch.stack([r - 1, -r, r, 1 - r], 1)
        a, b = (1 - t)[:, None], t[:, None]
        N = torch.cat([tri * a, tri * b], 1)
        dN = torch.stack([torch.cat([dr * a, dr * b], 1), torch.cat([ds * a, ds * b], 1), torch.cat([-tri, tri], 1)], 2)
        return N, dN

    for _ in range(16):
        N, dN = shape(u)
        f = torch.einsum("kn,kna->ka", N, x) - p
        J = torch.einsum("knb,kna->kab", dN, x)
        u = u - torch.linalg.solve(J, f[:, :, None])[:, :, 0].clamp(-2, 2)
    N, _ = shape(u)
    e = 1e-9
    there = ((torch.einsum("kn,kna->ka", N, x) - p).abs() < 1e-12).all(1)  # converged
    inside = there & (u >= -e).all(1) & (u[:, 2] <= 1 + e)
    inside &= (u[:, 0] + u[:, 1] <= 1 + e) if wedge else (u[:, :2] <= 1 + e).all(1)
    return N, inside


def _tet64(x, p):
    """Barycentric weights of p in the tetrahedra x [K, 4, 3] and whether it is inside."""
    A = torch.stack([x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]], 2)
    l = torch.linalg.solve(A, (p - x[:, 0])[:, :, None])[:, :, 0]
    N = torch.cat([1 - l.sum(1, keepdim=True), l], 1)
    return N, (N >= -1e-12).all(1)


def _cells64(case, seed):
    """Every query against the cells of the 27 grid cells about its own; the first that holds it."""
    g, pts32, vals, hexes, ijk = _mesh(case, seed)
    q = _query_points(case["S"], g).double()
    pts = pts32.double()
    n = case["n"]
    wedge = _is_wedge(case, ijk)
    out = torch.full((q.shape[0],), -1.0, dtype=torch.float64, device=q.device)
    own = (q * n).floor().long().clamp(-1, n)
    todo = torch.ones(q.shape[0], dtype=torch.bool, device=q.device)
    shifts = sorted([(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)], key=lambda s: sum(map(abs, s)))
    for sh in shifts:
        c = own + torch.tensor(sh, device=q.device)
        rows = (todo & ((c >= 0) & (c < n)).all(1)).nonzero()[:, 0]
        cell = (c[rows, 2] * n + c[rows, 1]) * n + c[rows, 0]
        if case["kind"] == "tets":
            parts = [(None, t) for t in _TETS]
        else:
            parts = [(False, list(range(8)))] + [(True, w) for w in _WEDGES]
        for is_wedge, which in parts:
            keep = todo[rows] if is_wedge is None else todo[rows] & (wedge[cell] == is_wedge)
            r, k = rows[keep], cell[keep]
            for a in range(0, r.shape[0], 1_000_000):
                ra, va = r[a:a + 1_000_000], hexes[k[a:a + 1_000_000]][:, which]
                N, inside = _tet64(pts[va], q[ra]) if is_wedge is None else _newton64(is_wedge, pts[va], q[ra])
                out[ra[inside]] = (N * vals[va]).sum(1)[inside]
                todo[ra[inside]] = False
    return out


def exact(case, seed):
    family = case["family"]
    if family in ("step", "render"):
        # beyond this the tiles of all pairs take longer than a comparison is worth
        if case["P"] * case["S"] > 5e12 or _pairs(case) > 6e8:
            return None
        return _field64(case, seed, family == "step")
    if family == "nearest":
        return _nearest64(_means(case["mix"], case["P"], _generator(seed))) if case["P"] <= 300_000 else None
    if family == "uniform":
        return _uniform64(case, seed) if case["dtype"].startswith("float") else None
    if family == "cells":
        return _cells64(case, seed)
    # the points are drawn by the library itself, and the targets are taken at them
    return None
