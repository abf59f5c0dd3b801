"""Performance cases: what a program that uses this framework has it do, by public entry point.

A case is a dict of plain values; ``kind`` says which entry points it goes through:

* ``unfold``   -- one-call batched unfold of prepared charts (solve_batch): upload, assembly,
                  PCG, driver, UVs back to the host;
* ``pipeline`` -- a raw mesh to UVs: prepare_mesh on the context's device, then unfold_charts;
* ``cg``       -- the drop-in solver boundary (GpuSolver.cg_solve_precond) on a host CSR system;
* ``grad``     -- one step of an optimisation over vertex positions: lscm_forward,
                  distortion_loss, lscm_backward;
* ``keep``     -- the unfold that keeps each chart's area (UnfoldOptions.keep_metric);
* ``metrics``  -- what follows an unfold: chart_distortion and rectangularize of given UVs.

Meshes are the ones the benchmark and the tests use: welded boxes, polar disk patches, height
fields.  Topology depends on the case alone and is kept between preparations; positions, right-
hand sides and targets come from the seed.
"""
import math

import numpy as np
import torch

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

_PRECOND = {"none": R.Precond.NONE, "jacobi": R.Precond.JACOBI, "ic0": R.Precond.IC0,
            "ic0color": R.Precond.IC0_COLOR, "amg": R.Precond.AMG, "amgsa": R.Precond.AMG_SA}
_PRECISION = {"fp64": R.Precision.FP64, "mixed": R.Precision.MIXED}


def listed():
    return [
        # the first mesh anyone unfolds: a box of six charts, FP64 with the reference's IC(0)
        {"name": "box_ic0_fp64", "kind": "unfold", "mesh": "box", "n": 6, "precond": "ic0", "precision": "fp64",
         "pinned": False},
        # a prop: a few dozen small charts with the default options (Jacobi, mixed precision)
        {"name": "prop_default", "kind": "unfold", "mesh": "disks", "charts": 40, "t_min": 50, "t_max": 2500,
         "precond": "jacobi", "precision": "mixed", "pinned": False},
        # an ordinary asset: some hundred charts, the fast preconditioner, page-locked arrays
        {"name": "asset_amgsa", "kind": "unfold", "mesh": "disks", "charts": 300, "t_min": 50, "t_max": 20000,
         "precond": "amgsa", "precision": "mixed", "pinned": True},
        # the benchmark's batch: 4096 uneven charts, about 30 million triangles
        {"name": "disks4096_amgsa", "kind": "unfold", "mesh": "disks", "charts": 4096, "t_min": 50, "t_max": 50000,
         "precond": "amgsa", "precision": "mixed", "pinned": True},
        # one large chart, two million unknowns
        {"name": "field1024_amgsa", "kind": "unfold", "mesh": "field", "n": 1024, "sines": 8, "amp": 0.15,
         "precond": "amgsa", "precision": "mixed", "pinned": True},
        # one mid-size chart solved throughout in FP64 with the reference's default preconditioner
        {"name": "field301_jacobi_fp64", "kind": "unfold", "mesh": "field", "n": 301, "sines": 8, "amp": 0.15,
         "precond": "jacobi", "precision": "fp64", "pinned": False},
        # a hard-surface model: a raw mesh that the dihedral test cuts into hundreds of charts, to UVs
        {"name": "model_pipeline", "kind": "pipeline", "boxes": 100, "n": 12, "precond": "amgsa",
         "precision": "mixed"},
        # a host program's own systems through the solver boundary
        {"name": "cg_poisson400_jacobi", "kind": "cg", "system": "poisson", "n": 400, "precond": "jacobi"},
        {"name": "cg_poisson181_ic0color", "kind": "cg", "system": "poisson", "n": 181, "precond": "ic0color"},
        # a step of shape optimisation through the unfold (FP64: a smooth right-hand side asks
        # more of the solve than the mixed loop's 48 bits hold on charts of this size)
        {"name": "grad_disks64", "kind": "grad", "charts": 64, "t_min": 100, "t_max": 20000, "precond": "amgsa",
         "precision": "fp64"},
        # area-keeping unfold of a prop (FP64 for the same reason)
        {"name": "keep_disks32", "kind": "keep", "charts": 32, "t_min": 100, "t_max": 6000, "precond": "jacobi",
         "precision": "fp64"},
        # distortion report and rectangular layout of an asset's charts
        {"name": "metrics_disks256", "kind": "metrics", "charts": 256, "t_min": 50, "t_max": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["unfold", "unfold", "unfold", "unfold", "pipeline", "cg", "cg", "grad", "keep", "metrics"])
    pc = rng.choice(["jacobi", "amgsa", "amgsa", "amg"])
    prec = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    if kind == "unfold":
        mesh = rng.choice(["box", "disks", "disks", "disks", "field"])
        c = {"kind": kind, "mesh": mesh, "precond": pc, "precision": prec, "pinned": rng.random() < 0.5}
        if mesh == "box":
            c["n"] = _log(rng, 3, 48)
            c["precond"] = rng.choice(["ic0", "ic0color", "jacobi", "amgsa"])
        elif mesh == "disks":
            c["charts"] = _log(rng, 1, 2000)
            c["t_min"] = _log(rng, 50, 400)
            c["t_max"] = _log(rng, 2 * c["t_min"], 50000)
        else:
            c["n"] = _log(rng, 33, 1024 if pc == "amgsa" and prec == "mixed" else 400)
            c["sines"], c["amp"] = 8, 0.15
        return c
    if kind == "pipeline":
        return {"kind": kind, "boxes": _log(rng, 1, 300), "n": _log(rng, 3, 24), "precond": pc, "precision": "mixed"}
    if kind == "cg":
        system = rng.choice(["poisson", "poisson", "banded"])
        if system == "poisson":
            return {"kind": kind, "system": system, "n": _log(rng, 20, 400),
                    "precond": rng.choice(["none", "jacobi", "ic0color", "amg", "amgsa"])}
        return {"kind": kind, "system": system, "n": _log(rng, 300, 500000), "band": rng.randint(1, 6),
                "precond": rng.choice(["none", "jacobi", "ic0color"])}
    t_min = _log(rng, 50, 400)
    small = prec == "mixed"  # (smooth right-hand sides: see listed())
    return {"grad": {"kind": kind, "charts": _log(rng, 1, 200), "t_min": 60 if small else t_min,
                     "t_max": _log(rng, 120, 600) if small else _log(rng, 2 * t_min, 20000),
                     "precond": pc, "precision": prec},
            "keep": {"kind": kind, "charts": _log(rng, 1, 100), "t_min": 60 if small else t_min,
                     "t_max": _log(rng, 120, 600) if small else _log(rng, 2 * t_min, 8000),
                     "precond": pc, "precision": prec},
            "metrics": {"kind": kind, "charts": _log(rng, 1, 600), "t_min": t_min,
                        "t_max": _log(rng, 2 * t_min, 40000)}}[kind]


# ------------------------------------------------------------------ meshes
_TOPO: dict = {}   # the last few cases' topology (it does not depend on the seed)
_DISK: dict = {}


def _kept(key, make):
    if key not in _TOPO:
        while len(_TOPO) >= 2:
            _TOPO.pop(next(iter(_TOPO)))
        _TOPO[key] = make()
    return _TOPO[key]


def _disk(rings):
    """Polar disk: ring k has 6k vertices, alternate rings turned by half a step, rings joined
    by advancing whichever next vertex comes first in angle."""
    if rings in _DISK:
        return _DISK[rings]
    start = np.concatenate([[0, 1], 1 + np.cumsum(6 * np.arange(1, rings + 1))])
    nv = int(start[-1])
    rad, ang, faces = np.zeros(nv), np.zeros(nv), []
    for k in range(1, rings + 1):
        s, m = start[k], 6 * k
        rad[s:s + m] = k / rings
        ang[s:s + m] = 2 * np.pi * (np.arange(m) + 0.5 * (k % 2)) / m
    i = np.arange(6)
    faces.append(np.stack([np.zeros(6, np.int64), 1 + i, 1 + (i + 1) % 6], 1))
    for k in range(2, rings + 1):
        si, mi, so, mo = start[k - 1], 6 * (k - 1), start[k], 6 * k
        ni = ang[si:si + mi] + 2 * np.pi / mi
        no = ang[so:so + mo] + 2 * np.pi / mo
        i, j = np.arange(mi), np.arange(mo)
        at = np.searchsorted(no, ni + 1e-12)
        faces.append(np.stack([si + i, so + at % mo, si + (i + 1) % mi], 1))
        at = np.searchsorted(ni, no - 1e-12)
        faces.append(np.stack([si + at % mi, so + j, so + (j + 1) % mo], 1))
    f = np.concatenate(faces).astype(np.int32)
    nbr = np.tile(np.arange(nv, dtype=np.int64)[:, None], (1, 8))  # each vertex's neighbours, itself where fewer
    e = np.unique(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]], f[:, [1, 0]], f[:, [2, 1]], f[:, [0, 2]]]), axis=0)
    at = np.arange(len(e)) - np.searchsorted(e[:, 0], e[:, 0])
    keep = at < 8
    nbr[e[keep, 0], at[keep]] = e[keep, 1]
    _DISK[rings] = (rad, ang, f, nbr)
    return _DISK[rings]


def _disk_topology(charts, t_min, t_max):
    rng = np.random.Generator(np.random.PCG64([charts, t_min, t_max]))
    t = np.exp(rng.uniform(np.log(t_min), np.log(t_max), charts))
    rings = np.maximum(1, np.rint(np.sqrt(t / 6.0)).astype(np.int64))
    parts = [_disk(int(r)) for r in rings]
    vo = np.concatenate([[0], np.cumsum([len(p[0]) for p in parts])]).astype(np.int64)
    to = np.concatenate([[0], np.cumsum([len(p[2]) for p in parts])]).astype(np.int64)
    put = lambda xs, dt: torch.from_numpy(np.concatenate(xs)).to("cuda", dt)  # noqa: E731
    return {"vo": vo, "to": to, "tris": np.concatenate([p[2] for p in parts]),
            "rad": put([p[0] for p in parts], torch.float64), "ang": put([p[1] for p in parts], torch.float64),
            "h": put([np.full(len(p[0]), 1.0 / r) for p, r in zip(parts, rings)], torch.float64),
            "nbr": put([p[3].astype(np.int32) + np.int32(v) for p, v in zip(parts, vo)], torch.int32)}


def _disk_charts(case, seed):
    """Disk patches with smoothed radial and normal displacements of a tenth of a ring step,
    the border on the unit circle; one chart per patch."""
    key = (case["charts"], case["t_min"], case["t_max"])
    T = _kept(("disks",) + key, lambda: _disk_topology(*key))
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    noise = torch.randn(2, len(T["rad"]), generator=g, device="cuda", dtype=torch.float32).double()
    for _ in range(3):
        mean = torch.zeros_like(noise)
        for k in range(8):
            mean += noise[:, T["nbr"][:, k]]
        noise = 0.5 * noise + mean / 16
    noise *= torch.where(T["rad"] > 1.0 - 1e-9, 0.0, 0.1) * T["h"]
    r = T["rad"] + torch.where(T["rad"] > 0, noise[0], 0.0)
    p = torch.stack([r * torch.cos(T["ang"]), r * torch.sin(T["ang"]), noise[1]], 1).float().double().cpu().numpy()
    return R.prepare_patches(T["vo"], T["to"], p, T["tris"], ctx=_ctx())


def _field(case, seed):
    n = case["n"]
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    k = case["sines"]
    a, fr, ph = rng.uniform(0.2, 1.0, k), rng.integers(1, 7, size=(k, 2)), rng.uniform(0.0, 2.0 * np.pi, k)
    x = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda")
    z = sum(float(a[i]) * torch.sin(2.0 * math.pi * (float(fr[i, 0]) * x[None, :] + float(fr[i, 1]) * x[:, None])
                                    + float(ph[i])) for i in range(k)) * case["amp"]
    p = torch.stack([x[None, :].expand(n, n), x[:, None].expand(n, n), z], 2).reshape(-1, 3).float().double()
    return p.cpu().numpy(), _kept(("grid", n), lambda: W.grid_faces(n, n))


def _box(case, seed):
    """Boxes of six n x n faces, every face with its own vertices (welding joins them)."""
    n, boxes = case["n"], case.get("boxes", 1)
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    t = np.linspace(-0.5, 0.5, n + 1)
    v, u = np.meshgrid(t, t, indexing="ij")
    # inner vertices of a face move within it: a different triangulation of the same flat face
    inner = (np.abs(u) < 0.499) & (np.abs(v) < 0.499)
    pos, grid = np.zeros((boxes, 6, n + 1, n + 1, 3)), W.grid_faces(n + 1, n + 1)
    for f in range(6):
        axis, side = f // 2, (-0.5, 0.5)[f % 2]
        p = pos[:, f]
        b, c = ((axis + 1) % 3, (axis + 2) % 3) if side > 0 else ((axis + 2) % 3, (axis + 1) % 3)
        p[..., axis] = side
        p[..., b] = u + np.where(inner, rng.uniform(-0.2, 0.2, p.shape[:3]) / n, 0.0)
        p[..., c] = v + np.where(inner, rng.uniform(-0.2, 0.2, p.shape[:3]) / n, 0.0)
    pos *= rng.uniform(0.6, 1.6, (boxes, 1, 1, 1, 3))
    pos[..., 0] += 2.0 * np.arange(boxes)[:, None, None, None]
    first = np.arange(6 * boxes, dtype=np.int32) * np.int32((n + 1) ** 2)
    return pos.reshape(-1, 3), (grid[None] + first[:, None, None]).reshape(-1, 3).astype(np.int32)


def _charts(case, seed):
    if case.get("mesh", "disks") == "disks":
        return _disk_charts(case, seed)
    if case["mesh"] == "field":
        p, f = _field(case, seed)
        return R.prepare_patches([0, len(p)], [0, len(f)], p, f, ctx=_ctx())
    p, f = _box(case, seed)
    return R.prepare_mesh(p, f)


def _system(case, seed):
    """5-point Poisson or a banded diagonally dominant system with a seeded diagonal."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    n = case["n"]
    if case["system"] == "poisson":
        i = np.arange(n * n)
        x, y = i % n, i // n
        offs, ok, off = [-n, -1, 0, 1, n], [y > 0, x > 0, i >= 0, x < n - 1, y < n - 1], [-1.0, -1.0, 0.0, -1.0, -1.0]
        diag = 4.0 + rng.uniform(0.0, 0.01, n * n)
    else:
        i, b = np.arange(n), case["band"]
        offs = list(range(-b, b + 1))
        ok = [(i + d >= 0) & (i + d < n) for d in offs]
        off = [-0.25 / abs(d) if d else 0.0 for d in offs]
        diag = 4.0 + rng.uniform(0.0, 8.0, n)
    keep = np.stack(ok, 1)
    cols = (i[:, None] + np.array(offs)[None, :])[keep]
    vals = np.where(np.array(offs)[None, :] == 0, diag[:, None], np.array(off)[None, :])[keep]
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))])
    return R.CsrMatrix(vals, cols, rp), rng.uniform(0.0, 2.0, len(i))


# ------------------------------------------------------------------ preparation and one pass
_SHARED: dict = {}


def _ctx():
    """The program's one context, as GpuSolver.global_ keeps one."""
    if "ctx" not in _SHARED:
        _SHARED["ctx"] = R.Context(0)
    return _SHARED["ctx"]


def _opts(case, **kw):
    return R.UnfoldOptions(precond=_PRECOND[case["precond"]], precision=_PRECISION[case["precision"]], **kw)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ctx": _ctx()}
    if kind == "pipeline":
        s["pos"], s["faces"] = _box(case, seed)
        s["opts"] = _opts(case)
        return s
    if kind == "cg":
        s["solver"], s["pc"] = R.GpuSolver(_ctx()), _PRECOND[case["precond"]]
        s["a"], s["b"] = _system(case, seed)
        return s
    charts = s["charts"] = _charts(case, seed)
    vo = charts.i64("chart.vert_off")
    s["n"], s["nc"] = int(vo[-1]), len(vo) - 1
    if kind == "metrics":
        # UVs near the charts' frames, resident with their batch on a context of their own
        s["ctx"] = R.Context(0)
        rng = np.random.Generator(np.random.PCG64(int(seed)))
        p2 = charts.f64("chart.p2").reshape(-1, 2)
        s["uv"] = p2 @ np.array([[1.0, 0.13], [-0.07, 0.9]]) + 1e-4 * rng.standard_normal(p2.shape)
        s["border"] = R.border_flags(charts)
        R.solve_batch(s["ctx"], charts.batch(), R.UnfoldOptions(max_cg_iter=1), s["n"])
        return s
    s["opts"] = _opts(case, keep_metric=kind == "keep")
    s["area"] = charts.f64("chart.area3d")
    s["batch"] = charts.batch()
    if kind == "unfold" and case["pinned"]:
        s["batch"], s["arrays"] = R.pinned_batch(_ctx(), charts)
    if kind == "grad":
        rng = np.random.Generator(np.random.PCG64(int(seed)))
        p2 = charts.f64("chart.p2").reshape(-1, 2)
        s["target"] = p2 + 0.01 * rng.standard_normal(p2.shape)
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind in ("unfold", "keep"):
        uv, stats, _ = R.solve_batch(ctx, s["batch"], s["opts"], s["n"], area3d=s["area"])
        return {"uv": uv, "iters": np.array([t.driver_iters for t in stats], np.int32),
                "status": np.array([t.status for t in stats], np.int32)}
    if kind == "pipeline":
        charts = R.prepare_mesh(s["pos"], s["faces"], ctx=ctx)
        res = R.unfold_charts(ctx, charts, s["opts"])
        return {"uv": np.concatenate([r.uv for r in res]), "vertex": charts.i64("chart.vertex_ids"),
                "tris": charts.i64("chart.tris"), "status": np.array([int(r.status) for r in res], np.int32)}
    if kind == "cg":
        got = s["solver"].cg_solve_precond(s["a"], s["b"], 20000, 1e-12, s["pc"])
        if got is None:
            raise RuntimeError(s["solver"].last_error)
        return {"x": got[0]}
    if kind == "grad":
        uv, _ = R.lscm_forward(ctx, s["batch"], s["opts"], s["n"])
        loss, duv, dp = R.distortion_loss(ctx, uv, s["nc"])
        dps, _ = R.lscm_backward(ctx, duv + (uv - s["target"]), s["opts"], s["nc"])
        return {"uv": uv, "loss": loss, "grad": dp + dps}
    return {"distortion": R.chart_distortion(ctx, s["uv"], s["nc"]),
            "rect": list(R.rectangularize(ctx, s["uv"], s["border"], s["nc"]))}


def _sizes(case):
    """(vertices, triangles) of a case's mesh."""
    if case.get("mesh") == "field":
        return case["n"] ** 2, 2 * (case["n"] - 1) ** 2
    if case["kind"] == "pipeline" or case.get("mesh") == "box":
        return 6 * case.get("boxes", 1) * (case["n"] + 1) ** 2, 12 * case.get("boxes", 1) * case["n"] ** 2
    rng = np.random.Generator(np.random.PCG64([case["charts"], case["t_min"], case["t_max"]]))
    t = np.exp(rng.uniform(np.log(case["t_min"]), np.log(case["t_max"]), case["charts"]))
    r = np.maximum(1, np.rint(np.sqrt(t / 6.0)))
    return float((1 + 3 * r * (r + 1)).sum()), float((6 * r * r).sum())


def work(case):
    """Inputs once, outputs once; arithmetic: the cotangents of every triangle once and one
    application of the operator to its right-hand sides."""
    kind = case["kind"]
    if kind == "cg":
        n = case["n"] ** 2 if case["system"] == "poisson" else case["n"]
        nnz = n * (5 if case["system"] == "poisson" else 2 * case["band"] + 1)
        return {"bytes": 12.0 * nnz + 20.0 * n, "flops": 2.0 * nnz}
    v, t = _sizes(case)
    if kind == "metrics":
        return {"bytes": 24.0 * v + 12.0 * t + 16.0 * v + v + 16.0 * v, "flops": 150.0 * t + 72 * 8.0 * v}
    if kind == "pipeline":
        return {"bytes": 24.0 * v + 12.0 * t + 16.0 * v + 12.0 * t, "flops": 150.0 * t + 28.0 * v}
    both = 2 if kind in ("grad", "keep") else 1
    b = 24.0 * v + 12.0 * t + 33.0 * v + 16.0 * v + (40.0 * v if kind == "grad" else 0.0)
    return {"bytes": b, "flops": (100.0 * t + 28.0 * v) * both}


# ------------------------------------------------------------------ exact values
def _batch_arrays(charts):
    vo, to = charts.i64("chart.vert_off"), charts.i64("chart.tri_off")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    tri = charts.i64("chart.tris").reshape(-1, 3) + np.repeat(vo[:-1], np.diff(to))[:, None]
    chart = np.repeat(np.arange(len(vo) - 1), np.diff(vo))
    return {"p": dev(charts.f64("chart.p3").reshape(-1, 3)), "t": dev(tri),
            "pin": dev(charts.i64("chart.pinned").astype(bool)), "puv": dev(charts.f64("chart.pin_uv").reshape(-1, 2)),
            "p2": dev(charts.f64("chart.p2").reshape(-1, 2)), "chart": dev(chart), "nc": len(vo) - 1,
            "tchart": dev(np.repeat(np.arange(len(to) - 1), np.diff(to)))}


def _edges(p, t):
    """The half edges (i, j) of every triangle corner and their coefficients cot / |e|^2."""
    out_i, out_j, out_c = [], [], []
    for m in range(3):
        o, i, j = t[:, m], t[:, (m + 1) % 3], t[:, (m + 2) % 3]
        a, b, e = p[i] - p[o], p[j] - p[o], p[j] - p[i]
        cot = ((a * b).sum(1) / torch.linalg.cross(a, b).norm(dim=1)).clamp_min(0.0)
        out_i.append(i), out_j.append(j), out_c.append(cot / (e * e).sum(1))
    return torch.cat(out_i), torch.cat(out_j), torch.cat(out_c)


def _laplacian(A):
    """The free block of the weighted graph Laplacian (CSR) and the rows' vertices."""
    i, j, c = _edges(A["p"], A["t"])
    free = ~A["pin"]
    row = torch.cumsum(free, 0) - 1
    n = int(free.sum())
    ii, jj, cc = torch.cat([i, j]), torch.cat([j, i]), torch.cat([c, c])
    k = free[ii]
    ii, jj, cc = ii[k], jj[k], cc[k]
    inner = free[jj]
    r, q = row[ii], row[jj]
    L = torch.sparse_coo_tensor(torch.stack([torch.cat([r[inner], r]), torch.cat([q[inner], r])]),
                                torch.cat([-cc[inner], cc]), (n, n)).coalesce()
    rhs = torch.zeros(n, 2, dtype=torch.float64, device="cuda").index_add_(
        0, r[~inner], cc[~inner, None] * A["puv"][jj[~inner]])
    return L.to_sparse_csr(), rhs, free


def _cg(L, rhs, diag, limit=12000):
    """Conjugate gradients in 64 bits, restarted from the true residual until it stalls."""
    x, dinv = torch.zeros_like(rhs), 1.0 / diag[:, None]
    best, goal = math.inf, 4e-16 * float(rhs.norm())
    for _ in range(4):
        r = rhs - L @ x
        now = float(r.norm())
        if not now > goal or now > 0.5 * best:
            break
        best, z = now, dinv * r
        p, d, rz = z.clone(), torch.zeros_like(r), (r * z).sum(0)
        for k in range(limit):
            q = L @ p
            a = rz / (p * q).sum(0).clamp_min(1e-300)
            d += a * p
            r -= a * q
            z = dinv * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
            if k % 32 == 31 and float(r.norm()) < 1e-9 * now + 0.1 * goal:
                break
        x = x + d
    return x


def _diagonal(L):
    n = L.shape[0]
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), L.crow_indices().diff())
    on = L.col_indices() == rows
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows[on], L.values()[on])


def _unfolded(A):
    L, rhs, free = _laplacian(A)
    uv = A["puv"].clone()
    uv[free] = _cg(L, rhs, _diagonal(L))
    # a chart whose frame already is its solution stays as it is
    per = lambda d: torch.zeros(A["nc"], dtype=torch.float64, device="cuda").index_add_(0, A["chart"], (d * d).sum(1)).sqrt()  # noqa: E731
    still = per(uv - A["p2"]) < 1e-8 * per(A["p2"]).clamp_min(1e-30)
    return torch.where(still[A["chart"], None], A["p2"], uv), L, free


def _distortion_terms(p, uv, t):
    """area (s1 / s2 - 1)^2 of every triangle, s1 >= s2 the singular values of its map."""
    a, b = p[t[:, 1]] - p[t[:, 0]], p[t[:, 2]] - p[t[:, 0]]
    la = a.norm(dim=1)
    x = (a * b).sum(1) / la
    twice = torch.linalg.cross(a, b).norm(dim=1)
    y = twice / la
    d1, d2 = uv[t[:, 1]] - uv[t[:, 0]], uv[t[:, 2]] - uv[t[:, 0]]
    f0 = d1 / la[:, None]
    f1 = (d2 - f0 * x[:, None]) / y[:, None]
    s = torch.hypot(f0[:, 0] + f1[:, 1], f1[:, 0] - f0[:, 1])
    d = torch.hypot(f0[:, 0] - f1[:, 1], f1[:, 0] + f0[:, 1])
    s1 = 0.5 * (s + d)
    det = f0[:, 0] * f1[:, 1] - f0[:, 1] * f1[:, 0]
    return 0.5 * twice * (s1 * s1 / det.abs() - 1.0) ** 2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pipeline", "keep", "metrics"):
        return None  # (structure and per-chart decisions beside the numbers)
    if kind == "cg":
        a, b = _system(case, seed)
        L = torch.sparse_csr_tensor(torch.from_numpy(a.row_ptr).long().cuda(), torch.from_numpy(a.cols).long().cuda(),
                                    torch.from_numpy(a.vals).cuda(), (len(b), len(b)))
        return {"x": _cg(L, torch.from_numpy(b).cuda()[:, None], _diagonal(L))[:, 0].cpu().numpy()}
    v, _ = _sizes(case)
    if v > (1.5e6 if case["kind"] == "unfold" and case["mesh"] == "disks" else 3e5):
        return None
    A = _batch_arrays(_charts(case, seed))
    uv, L, free = _unfolded(A)
    if kind == "unfold":
        return {"uv": uv.cpu().numpy(), "iters": None, "status": None}
    p2 = A["p2"].cpu().numpy()
    target = p2 + 0.01 * np.random.Generator(np.random.PCG64(int(seed))).standard_normal(p2.shape)
    p, u = A["p"].clone().requires_grad_(), uv.clone().requires_grad_()
    live = ~A["pin"][A["t"]].all(1)  # (a triangle of three pins has no say in the loss)
    terms = _distortion_terms(p, u, A["t"][live])
    gp, gu = torch.autograd.grad(terms.sum(), [p, u])
    loss = torch.zeros(A["nc"], dtype=torch.float64, device="cuda").index_add_(0, A["tchart"][live], terms.detach())
    g = gu + (uv - torch.from_numpy(target).cuda())
    lam = torch.zeros_like(uv)
    lam[free] = _cg(L, g[free], _diagonal(L))
    q = A["p"].clone().requires_grad_()
    i, j, c = _edges(q, A["t"])
    energy = -(c * ((lam[i] - lam[j]) * (uv[i] - uv[j])).sum(1)).sum()
    return {"uv": uv.cpu().numpy(), "loss": loss.cpu().numpy(),
            "grad": (gp + torch.autograd.grad(energy, q)[0]).cpu().numpy()}
