"""AMG hierarchies from three million rows on (two matching rounds and a third smoothed level) and the
smoothers' weight.  The large form against the small one (RUV_AMG_ROUNDS, RUV_AMG_SA_LEVELS);
group matching on rows with more neighbour groups than the warp kernel holds in registers; and, on
charts of badly shaped triangles, that the weight 0.85 damps on every level: lambda_max(D^-1 A) < 2 / 0.85."""
import numpy as np
import pytest
import scipy.sparse as sp

import researchuv_gb300 as R
from oracle import oracle as O
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _field(monkeypatch, n, small):
    p, f = W.height_field(n, 8, 0.15, seed=2)
    C = R.prepare_patches(np.array([0, len(p)]), np.array([0, len(f)]), p, f)
    out = []
    for form in (None, small):
        for knob, v in (form or {}).items():
            monkeypatch.setenv(knob, v)
        out.append(R.unfold_charts(R.Context(0), C, R.UnfoldOptions(precond=R.Precond.AMG_SA))[0])
    assert [r.status for r in out] == [R.Status.OK] * 2
    return out


SMALL = {"RUV_AMG_ROUNDS": "3", "RUV_AMG_SA_LEVELS": "2"}


def test_a_million_rows_take_the_small_form(monkeypatch):
    a, b = _field(monkeypatch, 1024, SMALL)
    assert a.cg_iters == b.cg_iters and np.array_equal(a.uv, b.uv)


def test_large_form_solves_as_the_small_one(monkeypatch):
    a, b = _field(monkeypatch, 1740, SMALL)  # 3,020,644 free rows
    assert a.n_free >= 3000000
    assert not np.array_equal(a.uv, b.uv)  # (two hierarchies)
    assert O.uv_error(a.uv, b.uv) <= 1e-6


# `more`: neighbour aggregates that some row has; each holds a neighbour group of its own, so the row's group has
# at least as many keys (a lane's second key from 32 on, those past the lanes' two from 64)
@pytest.mark.parametrize("n,degree,more", [(900, 120, 32), (6000, 500, 66)])
def test_more_neighbour_groups_than_registers(monkeypatch, n, degree, more):
    rng = np.random.Generator(np.random.PCG64(n))
    i, j = rng.integers(0, n, n * degree // 2), rng.integers(0, n, n * degree // 2)
    g = sp.csr_matrix((rng.uniform(0.5, 1.0, len(i)), (i, j)), shape=(n, n))
    g = g + g.T
    g.setdiag(0.0)
    g.eliminate_zeros()
    m = (sp.diags(np.asarray(g.sum(1)).ravel() + 1.0) - g).tocsr()
    m.sort_indices()
    out = []
    for graph in ("0", "1"):
        monkeypatch.setenv("RUV_AMG_GROUP_GRAPH", graph)
        out.append(R.GpuSolver(R.Context(0)).amg_level(R.CsrMatrix(m.data, m.indices, m.indptr), 0, False))
    agg = out[0]["agg"]
    assert max(len(set(agg[m.indices[m.indptr[r]:m.indptr[r + 1]]])) for r in range(n)) > more
    assert np.array_equal(agg, out[1]["agg"]) and out[0]["next_rows"] == out[1]["next_rows"]


def _stretched(sx, jitter, n=90, graded=1.0):
    rng = np.random.Generator(np.random.PCG64(11))
    y, x = np.meshgrid(np.linspace(0, 1, n), np.linspace(0, 1, n) ** graded, indexing="ij")
    z = 0.05 * np.sin(5 * x) * np.cos(4 * y)
    x = x + jitter / n * rng.uniform(-0.5, 0.5, x.shape)
    return np.stack([sx * x.ravel(), y.ravel(), z.ravel()], 1), W.grid_faces(n, n)


@pytest.mark.parametrize("smoothed", [True, False])
@pytest.mark.parametrize("sx,jitter,graded", [(1, 0.0, 1.0), (30, 0.0, 1.0), (1000, 0.0, 1.0), (1, 1.5, 1.0), (100, 1.5, 1.0),
                                              (1, 0.5, 4.0)])
def test_the_weight_damps_on_every_level(monkeypatch, sx, jitter, graded, smoothed):
    p, f = _stretched(sx, jitter, graded=graded)
    C = R.prepare_patches(np.array([0, len(p)]), np.array([0, len(f)]), p, f)
    ctx = R.Context(0)
    R.solve_batch(ctx, C.batch(), R.UnfoldOptions(precond=R.Precond.NONE, precision=R.Precision.FP64), len(p), check=False)
    rp, cols, vals, _ = R.export_chart_system(ctx, 0)
    m = sp.csr_matrix((vals, cols, rp))[0::2][:, 0::2].tocsr()  # (one of the two equal columns)
    m.sort_indices()
    s = R.GpuSolver(R.Context(0))
    for sa in ("2", "3"):
        monkeypatch.setenv("RUV_AMG_SA_LEVELS", sa)
        k, levels = 0, 1
        while k < levels:
            lv = s.amg_level(R.CsrMatrix(m.data, m.indices, m.indptr), k, smoothed)
            levels = lv["levels"]
            a = sp.csr_matrix((lv["A"][2], lv["A"][1], lv["A"][0]), shape=(lv["rows"], lv["rows"]))
            d = sp.diags(a.diagonal() ** -0.5)
            x = np.random.Generator(np.random.PCG64(k)).standard_normal(lv["rows"])
            for _ in range(200):
                y = d @ (a @ (d @ (x / np.linalg.norm(x))))
                x = y
            assert np.linalg.norm(x) < 2.0 / 0.85, (sa, k)
            k += 1


@pytest.mark.parametrize("ns,large", [((1098,), True), ((1097,), False), ((1000, 600, 600), False)])
def test_large_form_by_the_largest_chart(monkeypatch, ns, large):
    vo, to, p3, tr = [0], [0], [], []
    for k, n in enumerate(ns):
        p, f = W.height_field(n, 8, 0.15, seed=5 + k)
        p3.append(p)
        tr.append(f)
        vo.append(vo[-1] + len(p))
        to.append(to[-1] + len(f))
    C = R.prepare_patches(np.array(vo), np.array(to), np.concatenate(p3), np.concatenate(tr))
    out = []
    for form in ({}, SMALL):
        for knob, v in form.items():
            monkeypatch.setenv(knob, v)
        out.append(R.unfold_charts(R.Context(0), C, R.UnfoldOptions(precond=R.Precond.AMG_SA)))
    assert (out[0][0].n_free >= 1200000) == large
    for a, b in zip(*out):
        assert a.status == R.Status.OK and b.status == R.Status.OK
        assert np.array_equal(a.uv, b.uv) != large
        assert O.uv_error(a.uv, b.uv) <= 1e-6
