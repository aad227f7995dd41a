"""Performance cases of the framework: what its users run, through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a user's program holds before
the call (meshes as PLC handles, plans, batches, device tensors), ``run`` makes one
pass, ``work`` says what a pass cannot do without, and ``exact`` gives the outputs in
64 bits from plain torch and numpy.

Families (``kind``):

* ``voxelize`` — the reference binding's call ``voxelize(plc, resolution, mode, pad)``:
  a mesh on the host in, a NumPy grid out (bit-exact FP64 distances).
* ``voxelize_ex`` — the same with options: FP64 or mixed precision, occupancy and
  distances together, the nearest-feature checkpoint.
* ``batch`` — many meshes of uneven size in one pipeline (data preparation).
* ``fit`` — a step of an optimisation of the mesh's vertices through the
  differentiable distance field: forward, loss, backward.
* ``predicates`` — orient3d and insphere signs of device-resident query streams.
* ``sizing`` — a background sizing field evaluated at device-resident queries.
* ``intake`` — a surface file's way in: STL image to PLC, self-intersection check,
  simplification.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cybermeshgenerator_gb300 as cm
from cybermeshgenerator_gb300 import torch_sdf
from cybermeshgenerator_gb300 import workloads as W

#: point-triangle distance evaluations below which exact() is affordable
_EXACT_PAIRS = 2e10


# --------------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest useful call: a coarse preview of an 80-triangle body; launches,
        # synchronisations and host work are all there is
        dict(name="sdf_smallest", kind="voxelize", mesh="ico", a=1, b=0, resolution=16, pad=1,
             mode="sdf"),
        # the ordinary small call: a 1280-triangle jittered icosphere on a 64^3 grid
        dict(name="sdf_icosphere_64", kind="voxelize", mesh="ico", a=3, b=0, resolution=58, pad=3,
             mode="sdf"),
        # occupancy of a large CAD-like mesh (axis-aligned box and a 262k-triangle torus)
        dict(name="occupancy_box_torus_256", kind="voxelize", mesh="boxtorus", a=512, b=256,
             resolution=254, pad=1, mode="occupancy"),
        # the largest ordinary call: a 65k-triangle scanned surface at 256 cells, the
        # reference's FP64 distances, as the default entry returns them
        dict(name="sdf_surface_256", kind="voxelize", mesh="sh", a=256, b=128, resolution=254,
             pad=1, mode="sdf"),
        # the same surface in mixed precision with occupancy: the headline workload
        dict(name="mixed_surface_256", kind="voxelize_ex", mesh="sh", a=256, b=128, resolution=254,
             pad=1, precision="mixed", near=False),
        # occupancy, FP64 distance and nearest feature of many separate bodies on an
        # odd-sized grid (most cells far from small triangles)
        dict(name="nearest_field_135", kind="voxelize_ex", mesh="field", a=160, b=3, resolution=131,
             pad=2, precision="fp64", near=True),
        # data preparation: 24 meshes of 80 to 130k triangles at 32^3 to 192^3, mixed
        dict(name="batch_24", kind="batch", count=24, max_subdiv=5, max_seg=256,
             max_resolution=192),
        # the smallest optimisation step: 320 triangles on a 32^3 grid, float32 vertices
        dict(name="fit_small_32", kind="fit", mesh="ico", a=2, b=0, resolution=30, pad=1,
             precision="fp64", dtype="float32"),
        # an optimisation step on a 65k-triangle surface at 128 cells, mixed precision
        dict(name="fit_surface_128", kind="fit", mesh="sh", a=256, b=128, resolution=126, pad=1,
             precision="mixed", dtype="float64"),
        # orient3d and insphere signs for a mesher: a tenth exactly degenerate, another
        # tenth within a few ulps of it
        dict(name="predicates_2m", kind="predicates", n=2_000_003, degenerate=0.1, near=0.1,
             exact_mode=False),
        # sizes for a mesher: 1M queries of a jittered 82,944-tetrahedron background
        dict(name="sizing_1m", kind="sizing", cells=24, jitter=0.3, n=1_000_003),
        # a 512k-triangle STL image in: vertices merged, checked, simplified
        dict(name="intake_512k", kind="intake", bodies=400, subdiv=3, grid=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, big):
    kind = rng.choice(["ico", "sh", "boxtorus", "field"])
    if kind == "ico":
        return dict(mesh=kind, a=rng.randint(1, 5 if big else 4), b=0)
    if kind == "sh":
        n = _log(rng, 12, 256 if big else 96)
        return dict(mesh=kind, a=n, b=max(6, n // 2 + rng.randint(-3, 3)))
    if kind == "boxtorus":
        return dict(mesh=kind, a=_log(rng, 16, 512 if big else 160), b=_log(rng, 16, 256 if big else 100))
    return dict(mesh=kind, a=_log(rng, 4, 160 if big else 60), b=rng.randint(1, 3))


def draw(rng):
    kind = rng.choice(["voxelize", "voxelize", "voxelize_ex", "voxelize_ex", "batch", "fit", "fit",
                       "predicates", "sizing", "intake"])
    if kind in ("voxelize", "voxelize_ex", "fit"):
        res = _log(rng, 14, 120 if kind == "fit" else 250)
        c = dict(kind=kind, **_draw_mesh(rng, res > 60), resolution=res, pad=rng.randint(0, 4))
        if kind == "voxelize":
            c["mode"] = rng.choice(["sdf", "sdf", "occupancy"])
        else:
            c["precision"] = rng.choice(["fp64", "mixed"])
        if kind == "voxelize_ex":
            c["near"] = rng.random() < 0.4
        if kind == "fit":
            c["dtype"] = rng.choice(["float32", "float64"])
        return c
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 24), max_subdiv=rng.randint(2, 5),
                    max_seg=_log(rng, 20, 256), max_resolution=_log(rng, 40, 180))
    if kind == "predicates":
        return dict(kind=kind, n=_log(rng, 1000, 2_000_000), degenerate=round(rng.uniform(0, 0.2), 3),
                    near=round(rng.uniform(0, 0.1), 3), exact_mode=rng.random() < 0.4)
    if kind == "sizing":
        return dict(kind=kind, cells=rng.randint(2, 24), jitter=round(rng.uniform(0, 0.3), 3),
                    n=_log(rng, 1000, 1_000_000))
    return dict(kind=kind, bodies=_log(rng, 3, 400), subdiv=rng.randint(1, 3), grid=_log(rng, 8, 256))


# --------------------------------------------------------------------------- inputs

#: every mesh of a case fills the same box, so that its grid has the same cells at any seed
_BOX = np.array([1.0, 0.9140625, 0.97265625])


def _boxed(p, axes=(0, 1, 2)):
    lo, hi = p.min(0), p.max(0)
    return (p - lo) / (hi - lo) * _BOX[list(axes)]


def _mesh(case, seed):
    """Points and triangles of a case: the repository's generators with the seed in their
    shape, turned (all but the axis-aligned box and the field of bodies) and fitted to
    the box."""
    rng = np.random.default_rng([17, seed])
    a, b = case["a"], case["b"]
    if case["mesh"] == "field":
        p, t = W.ellipsoid_field(a, seed=1000 + seed, subdiv=b, amin=0.02, amax=0.06)
        return _boxed(p), t
    if case["mesh"] == "boxtorus":
        p, t = W.merge(W.unit_box(float(rng.uniform(0.8, 1.2))),
                       W.torus(float(rng.uniform(0.3, 0.4)), float(rng.uniform(0.08, 0.14)),
                               (0.5, 0.5, 1.3), a, b))
        return _boxed(p, (1, 2, 0)), t
    if case["mesh"] == "ico":
        p, t = W.jittered_icosphere(a, 0.02, seed=1000 + seed)
    else:
        p, t = W.sh_sphere(a, b, seed=1000 + seed)
    return _boxed(p @ W._rotation(rng).T), t


def _precision(case):
    return cm.PREC_MIXED if case["precision"] == "mixed" else cm.PREC_FP64


def _outputs(case):
    if case["near"]:
        return cm.OUT_OCCUPANCY | cm.OUT_SDF_F64 | cm.OUT_NEAREST
    return cm.OUT_OCCUPANCY | cm.OUT_SDF_F32


def _batch_items(case, seed):
    """(points, triangles, resolution) of a batch: half icospheres, half tori of many
    sizes (the case says which), turned and proportioned by the seed."""
    which, rng = np.random.default_rng([case["count"], case["max_seg"]]), np.random.default_rng([4, seed])
    top, out = case["max_resolution"], []
    for _ in range(case["count"]):
        kind, sub = which.random() < 0.5, int(which.integers(1, case["max_subdiv"] + 1))
        nu, nv = (int(which.integers(16, case["max_seg"] + 1)) for _ in range(2))
        res = max(8, int(top * which.choice([1 / 6, 1 / 4, 1 / 3, 1 / 2, 2 / 3, 1])))
        p, t = W.jittered_icosphere(sub, 0.02, seed=int(rng.integers(1 << 30))) if kind else \
            W.torus(rng.uniform(0.3, 0.45), rng.uniform(0.05, 0.15), (0, 0, 0), nu, nv)
        out.append((_boxed(p @ W._rotation(rng).T), t, res))
    return out


def _fit_inputs(case, seed):
    """Mesh, grid, vertices and target of a fit: the target is the distance field of a
    sphere around the mesh's centre, as fitting a body to a simpler one has."""
    p, t = _mesh(case, seed)
    if case["dtype"] == "float32":
        p = p.astype(np.float32).astype(np.float64)
    corner, h, dims = cm.plc_grid(cm.PLC.from_arrays(p, t), case["resolution"], case["pad"])
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") for n in dims]
    x, y, z = (corner[i] + (ax[i] + 0.5) * h for i in range(3))
    c, r = p.mean(0), float(np.linalg.norm(p - p.mean(0), axis=1).mean())
    target = ((x[:, None, None] - c[0]) ** 2 + (y[None, :, None] - c[1]) ** 2 +
              (z[None, None, :] - c[2]) ** 2).sqrt() - 0.9 * r
    return p, t, (tuple(corner), h, dims), target


def _intake_mesh(case, seed):
    """Separate bodies, the last of them copied and shifted so that some triangles cross.
    The seed sets the bodies' order in the file, the axes' and the unit (a power of two,
    so that as many points, pairs and cells come of it)."""
    rng = np.random.default_rng([23, seed])
    n, nv, nt = case["bodies"], 10 * 4 ** case["subdiv"] + 2, 20 * 4 ** case["subdiv"]
    p, t = W.ellipsoid_field(n, seed=1000 + n, subdiv=case["subdiv"], amin=0.015, amax=0.045)
    p = np.concatenate([p, p[-nv:] + 0.011])[:, rng.permutation(3)] * 2.0 ** rng.integers(-4, 5)
    t = np.concatenate([t, t[-nt:] + nv])
    return p, t.reshape(n + 1, nt, 3)[rng.permutation(n + 1)].reshape(-1, 3).astype(np.int32)


def _sizing_inputs(case, seed):
    P, T = W.kuhn_tet_mesh(case["cells"], case["jitter"], seed=1000 + seed)
    S = np.random.default_rng([5, seed]).uniform(0.01, 0.2, len(P))
    return P, T, S, W.sizing_queries(P, T, case["n"], seed=2000 + seed)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind in ("voxelize", "voxelize_ex"):
        s["plc"] = cm.PLC.from_arrays(*_mesh(case, seed))
    elif kind == "batch":
        items = _batch_items(case, seed)
        s["batch"] = cm.Batch([cm.PLC.from_arrays(p, t) for p, t, _ in items],
                              [r for _, _, r in items], [1] * len(items),
                              outputs=cm.OUT_OCCUPANCY | cm.OUT_SDF_F32, precision=cm.PREC_MIXED)
    elif kind == "fit":
        p, t, grid, target = _fit_inputs(case, seed)
        dt = getattr(torch, case["dtype"])
        s["plan"] = torch_sdf.SDFPlan(p, t, grid, precision=_precision(case))
        s["v"] = torch.tensor(p, dtype=dt, device="cuda", requires_grad=True)
        s["target"] = target.to(dt)
    elif kind == "predicates":
        for name, k in (("o", "orient3d"), ("i", "insphere")):
            q = W.predicate_stream(case["n"], k, case["degenerate"], case["near"], seed=1000 + seed)
            s[name] = torch.from_numpy(q).cuda()
        s["mode"] = cm.PRED_EXACT if case["exact_mode"] else cm.PRED_COMPAT
    elif kind == "sizing":
        P, T, S, Q = _sizing_inputs(case, seed)
        s["field"] = cm.SizingField(P, T, S, 1.25)
        s["q"] = torch.from_numpy(Q).cuda()
    else:
        s["stl"] = W.stl_binary(*_intake_mesh(case, seed))
    return s


# --------------------------------------------------------------------------- passes

def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "voxelize":
        return cm.voxelize(s["plc"], case["resolution"], case["mode"], case["pad"]).grid
    if kind == "voxelize_ex":
        r = cm.voxelize_ex(s["plc"], resolution=case["resolution"], pad=case["pad"],
                           outputs=_outputs(case), precision=_precision(case))
        if case["near"]:
            return {"occupancy": r.occupancy, "sdf": r.sdf64, "triangle": r.nearest_triangle,
                    "region": r.nearest_region}
        return {"occupancy": r.occupancy, "sdf": r.sdf32}
    if kind == "batch":
        s["batch"].run()
        out = []
        for i in range(len(s["batch"])):
            r = s["batch"].result(i)
            out.append([r.occupancy, r.sdf32])
        return out
    if kind == "fit":
        d = torch_sdf.sdf(s["v"], s["plan"])
        loss = ((d - s["target"]) ** 2).mean()
        (grad,) = torch.autograd.grad(loss, s["v"])
        return {"sdf": d.detach(), "grad": grad}
    if kind == "predicates":
        st = torch.cuda.current_stream().cuda_stream
        out = {}
        for name, fn in (("o", cm.orient3d_stream), ("i", cm.insphere_stream)):
            q = s[name]
            signs = torch.empty(q.shape[1], dtype=torch.int8, device="cuda")
            fn(([q[k].data_ptr() for k in range(q.shape[0])], q.shape[1], signs.data_ptr()), s["mode"], st)
            out[name] = signs
        return out
    if kind == "sizing":
        return s["field"].eval(s["q"])
    plc = cm.plc_from_stl(s["stl"])
    pairs = cm.self_intersections(plc)
    small = cm.simplify(plc, case["grid"])
    return {"points": plc.points, "triangles": plc.triangles, "pairs": pairs,
            "simple_points": small.points, "simple_triangles": small.triangles}


# --------------------------------------------------------------------------- work

def _mesh_size(case):
    a, b = case["a"], case["b"]
    if case["mesh"] == "ico":
        return 10 * 4 ** a + 2, 20 * 4 ** a
    if case["mesh"] == "field":
        return a * (10 * 4 ** b + 2), a * 20 * 4 ** b
    if case["mesh"] == "boxtorus":
        return a * b + 8, 2 * a * b + 12
    return a * (b - 1) + 2, 2 * a * (b - 1)


def _cells(case):
    """Cells of a case's grid, to within a layer."""
    return math.prod(case["resolution"] * e + 2 * case["pad"] for e in _BOX)


def work(case):
    """Bytes: inputs read once, outputs written once. Flops: one point-triangle distance
    (79) per cell or cell adjoint, one containment test (96) per sizing query inside, one
    determinant per predicate (23 / 71)."""
    kind = case["kind"]
    if kind in ("voxelize", "voxelize_ex", "fit"):
        nv, nt = _mesh_size(case)
        cells = _cells(case)
        mesh = 24 * nv + 12 * nt
        if kind == "voxelize":
            sdf = case["mode"] == "sdf"
            return {"bytes": mesh + cells * (4 if sdf else 1), "flops": cells * 79 if sdf else 23 * nt}
        if kind == "voxelize_ex":
            return {"bytes": mesh + cells * (14 if case["near"] else 5), "flops": cells * 79}
        e = 4 if case["dtype"] == "float32" else 8
        # forward, target read, difference written and read by the adjoint, gradient
        return {"bytes": mesh + 24 * nv + 4 * e * cells, "flops": 2 * 79 * cells}
    if kind == "batch":
        n, top = case["count"], case["max_resolution"]
        cells = n * 0.25 * top ** 3
        tris = n * 0.5 * (20 * 4 ** case["max_subdiv"] * 0.27 + case["max_seg"] ** 2 * 0.5)
        return {"bytes": 24 * tris + 5 * cells, "flops": 79 * cells}
    if kind == "predicates":
        return {"bytes": case["n"] * (97 + 121), "flops": case["n"] * (23 + 71)}
    if kind == "sizing":
        return {"bytes": case["n"] * 32 + 6 * case["cells"] ** 3 * 16, "flops": case["n"] * 96}
    nt = (case["bodies"] + 1) * 20 * 4 ** case["subdiv"]
    return {"bytes": nt * (50 + 12 + 12) + 12 * nt, "flops": nt * 50}


# --------------------------------------------------------------------------- 64-bit values

def _closest(p, a, b, c):
    """Squared distance of points to triangles and the closest points' barycentric
    weights (broadcast over the leading axes), in 64 bits: the projection when it falls
    inside, else the nearest of the three edges."""
    def dot(u, v):
        return (u * v).sum(-1)

    def edge(u, v):
        d = v - u
        t = (dot(p - u, d) / dot(d, d).clamp_min(1e-300)).clamp(0, 1)
        r = p - (u + t[..., None] * d)
        return dot(r, r), t

    n = torch.linalg.cross(b - a, c - a)
    nn = dot(n, n).clamp_min(1e-300)
    wb = dot(torch.linalg.cross(p - a, (c - a).expand_as(p - a)), n) / nn
    wc = dot(torch.linalg.cross((b - a).expand_as(p - a), p - a), n) / nn
    h = dot(p - a, n)
    inside = (wb >= 0) & (wc >= 0) & (wb + wc <= 1)
    best = torch.where(inside, h * h / nn, torch.full_like(h, math.inf))
    w1, w2 = wb, wc
    zero = torch.zeros_like(h)
    for (u, v), f in (((a, b), lambda t: (t, zero)), ((b, c), lambda t: (1 - t, t)),
                      ((c, a), lambda t: (zero, 1 - t))):
        d, t = edge(u, v)
        less = d < best
        best = torch.where(less, d, best)
        x, y = f(t)
        w1, w2 = torch.where(less, x, w1), torch.where(less, y, w2)
    return best, torch.stack([1 - w1 - w2, w1, w2], -1)


def _nearest(p, t, corner, h, dims, block=16):
    """Squared distance and nearest triangle of every cell ((nz, ny, nx) order), by blocks
    of cells over the triangles whose bounding sphere can reach the block."""
    P = torch.as_tensor(p, device="cuda")
    V = P[torch.as_tensor(t, device="cuda").long()]
    cen = V.mean(1)
    rad = (V - cen[:, None]).norm(dim=-1).amax(1)
    nx, ny, nz = dims
    d2 = torch.empty((nz, ny, nx), dtype=torch.float64, device="cuda")
    tri = torch.empty((nz, ny, nx), dtype=torch.int64, device="cuda")
    ax = [corner[i] + (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * h for i, n in enumerate(dims)]
    for z in range(0, nz, block):
        for y in range(0, ny, block):
            for x in range(0, nx, block):
                X, Y, Z = ax[0][x:x + block], ax[1][y:y + block], ax[2][z:z + block]
                mid = torch.stack([(X[0] + X[-1]) / 2, (Y[0] + Y[-1]) / 2, (Z[0] + Z[-1]) / 2])
                rb = float((mid - torch.stack([X[0], Y[0], Z[0]])).norm())
                dc = (cen - mid).norm(dim=1)
                near = torch.nonzero(dc - rad <= float((dc + rad).min()) + 2 * rb + 1e-9)[:, 0]
                q = torch.stack(torch.meshgrid(Z, Y, X, indexing="ij")[::-1], -1).reshape(-1, 1, 3)
                best = torch.full((q.shape[0],), math.inf, dtype=torch.float64, device="cuda")
                which = torch.zeros(q.shape[0], dtype=torch.int64, device="cuda")
                step = max(1, 6_000_000 // q.shape[0])
                for k in range(0, len(near), step):
                    T = V[near[k:k + step]]
                    d, _ = _closest(q, T[None, :, 0], T[None, :, 1], T[None, :, 2])
                    m, j = d.min(1)
                    less = m < best
                    best, which = torch.where(less, m, best), torch.where(less, near[k + j], which)
                shape = (len(Z), len(Y), len(X))
                d2[z:z + block, y:y + block, x:x + block] = best.reshape(shape)
                tri[z:z + block, y:y + block, x:x + block] = which.reshape(shape)
    return d2, tri


def _inside(p, t, corner, h, dims):
    """Cells inside, by the parity of the surface's crossings above them ((nz, ny, nx))."""
    nx, ny, nz = dims
    V = p[np.asarray(t)]
    lo = np.ceil((V[:, :, :2].min(1) - corner[:2]) / h - 0.5).astype(np.int64)
    hi = np.floor((V[:, :, :2].max(1) - corner[:2]) / h - 0.5).astype(np.int64)
    lo, hi = np.maximum(lo, 0), np.minimum(hi, [nx - 1, ny - 1])
    w = np.maximum(hi - lo + 1, 0)
    count = w[:, 0] * w[:, 1]
    k = np.repeat(np.arange(len(V)), count)
    at = np.arange(len(k)) - np.repeat(np.cumsum(count) - count, count)
    i, j = lo[k, 0] + at % w[k, 0], lo[k, 1] + at // w[k, 0]
    x, y = corner[0] + (i + 0.5) * h, corner[1] + (j + 0.5) * h
    a, b, c = V[k, 0], V[k, 1], V[k, 2]

    def side(u, v):
        return (v[:, 0] - u[:, 0]) * (y - u[:, 1]) - (v[:, 1] - u[:, 1]) * (x - u[:, 0])

    wa, wb, wc = side(b, c), side(c, a), side(a, b)
    hit = ((wa > 0) & (wb > 0) & (wc > 0)) | ((wa < 0) & (wb < 0) & (wc < 0))
    i, j = i[hit], j[hit]
    height = ((wa * a[:, 2] + wb * b[:, 2] + wc * c[:, 2]) / np.where(hit, wa + wb + wc, 1.0))[hit]
    below = np.clip(np.ceil((height - corner[2]) / h - 0.5), 0, nz).astype(np.int64)
    flips = np.zeros((nz + 1, ny, nx), dtype=np.int64)
    np.add.at(flips, (below, j, i), 1)
    # a crossing flips the cells under it: layers 0 .. below-1
    return torch.as_tensor(np.cumsum(flips[::-1], 0)[::-1][1:] % 2 == 1, device="cuda")


def _exact_field(p, t, grid):
    corner, h, dims = np.asarray(grid[0]), grid[1], grid[2]
    d2, tri = _nearest(p, t, corner, h, dims)
    inside = _inside(p, t, corner, h, dims)
    return torch.where(inside, -d2.sqrt(), d2.sqrt()), tri, inside


def _affordable(cells, tris):
    # a block of 16^3 cells tests the triangles that can reach it: a tenth of a small
    # mesh, fewer of a large one
    return cells * (0.1 * min(tris, 20_000) + 0.03 * max(0, tris - 20_000)) < _EXACT_PAIRS


def _exact_fit(case, seed):
    p, t, grid, target = _fit_inputs(case, seed)
    d, tri, inside = _exact_field(p, t, grid)
    # the loss's derivative at the field in the fit's type, as a 64-bit loss has it
    target = target.to(getattr(torch, case["dtype"])).double()
    g = 2 * (d.permute(2, 1, 0) - target) / d.numel()
    corner, h, dims = grid
    ax = [corner[i] + (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * h for i, n in enumerate(dims)]
    q = torch.stack(torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")[::-1], -1).reshape(-1, 3)
    T = torch.as_tensor(t, device="cuda").long()[tri.reshape(-1)]
    V = torch.as_tensor(p, device="cuda")[T]
    _, w = _closest(q, V[:, 0], V[:, 1], V[:, 2])
    r = q - (w[..., None] * V).sum(1)
    n = r / r.norm(dim=1, keepdim=True).clamp_min(1e-300)
    sign = torch.where(inside.reshape(-1), -1.0, 1.0)
    push = -(g.permute(2, 1, 0).reshape(-1) * sign)[:, None] * n
    grad = torch.zeros(p.shape, dtype=torch.float64, device="cuda")
    for k in range(3):
        grad.index_add_(0, T[:, k], w[:, k, None] * push)
    return {"sdf": d.permute(2, 1, 0), "grad": grad}


def _exact_sizing(case, seed):
    P, T, S, Q = (torch.as_tensor(x, device="cuda") for x in _sizing_inputs(case, seed))
    n, best = case["cells"], torch.full((len(Q),), 1 << 30, dtype=torch.int64, device="cuda")
    val = torch.zeros(len(Q), dtype=torch.float64, device="cuda")
    base = (Q * n).floor().long()
    for o in range(27):
        cell = base + torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device="cuda")
        ok = ((cell >= 0) & (cell < n)).all(1)
        cid = (cell[:, 0] * n + cell[:, 1]) * n + cell[:, 2]
        for k in range(6):
            tet = torch.where(ok, cid * 6 + k, 0)
            V = P[T[tet].long()]
            M = (V[:, 1:] - V[:, :1]).transpose(1, 2)
            r = Q - V[:, 0]
            c = torch.linalg.cross(M[:, :, 1], M[:, :, 2])
            det = (M[:, :, 0] * c).sum(1)
            l1 = (r * c).sum(1) / det
            l2 = (M[:, :, 0] * torch.linalg.cross(r, M[:, :, 2])).sum(1) / det
            l3 = (M[:, :, 0] * torch.linalg.cross(M[:, :, 1], r)).sum(1) / det
            lam = torch.stack([1 - l1 - l2 - l3, l1, l2, l3], 1)
            hit = ok & (lam >= -1e-9).all(1) & (tet < best)
            best = torch.where(hit, tet, best)
            val = torch.where(hit, (lam * S[T[tet].long()]).sum(1), val)
    out = torch.nonzero(best == 1 << 30)[:, 0]
    for k in range(0, len(out), 4096):
        m = out[k:k + 4096]
        val[m] = S[((Q[m, None] - P[None]) ** 2).sum(-1).argmin(1)]
    return val * 1.25


def _exact_intake(case, seed):
    p, t = _intake_mesh(case, seed)
    v = p.astype(np.float32).astype(np.float64)[t].reshape(-1, 3)

    def first_seen(keys):
        _, first, inv = np.unique(keys, return_index=True, return_inverse=True)
        rank = np.empty(len(first), dtype=np.int64)
        rank[np.argsort(first)] = np.arange(len(first))
        return np.sort(first), rank[inv.ravel()]

    rows = np.ascontiguousarray(v + 0.0).view(np.dtype((np.void, 24))).ravel()
    at, _ = first_seen(rows)
    pts = v[at]
    ext = (pts.max(0) - pts.min(0)).max()
    cell = np.clip(((pts - pts.min(0)) * (case["grid"] / ext)).astype(np.int64), 0, case["grid"] - 1)
    _, rep = first_seen((cell[:, 0] * case["grid"] + cell[:, 1]) * case["grid"] + cell[:, 2])
    n = np.bincount(rep)
    centroid = np.stack([np.bincount(rep, pts[:, k]) / n for k in range(3)], 1)
    return {"points": pts, "triangles": None, "pairs": None, "simple_points": centroid,
            "simple_triangles": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("voxelize", "voxelize_ex", "fit"):
        if case.get("mode") == "occupancy" or not _affordable(_cells(case), _mesh_size(case)[1]):
            return None
        # the axis-aligned box puts edges on the columns of some grids, where the plain
        # parity has no answer
        if case["mesh"] == "boxtorus":
            return None
        if kind == "fit":
            return _exact_fit(case, seed)
        p, t = _mesh(case, seed)
        d, _, _ = _exact_field(p, t, cm.plc_grid(cm.PLC.from_arrays(p, t), case["resolution"], case["pad"]))
        if kind == "voxelize":
            return d.permute(2, 1, 0)
        if case["near"]:
            return {"occupancy": None, "sdf": d.reshape(-1), "triangle": None, "region": None}
        return {"occupancy": None, "sdf": d.reshape(-1)}
    if kind == "sizing":
        return _exact_sizing(case, seed)
    if kind == "intake":
        return _exact_intake(case, seed)
    return None
