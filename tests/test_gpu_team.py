"""Team solver (team.cu: a chart's whole CG loop in one kernel of a CTA or a cluster) against the
launch-per-step loop (RUV_TEAM=0): the same statuses, and UVs within the solves' own accuracy, at
the sizes where the team's layout changes (one row, one CTA's rows, 2 to 16 CTAs, the largest),
for every preconditioner, precision and column stream."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _grid(nx, ny, seed=3):
    """One bumpy nx x ny chart: (nx - 2)(ny - 2) free vertices."""
    rng = np.random.Generator(np.random.PCG64(seed))
    y, x = np.meshgrid(np.linspace(0, 1, ny), np.linspace(0, 1, nx), indexing="ij")
    z = 0.05 * np.sin(5 * x) * np.cos(4 * y) + 0.1 / max(nx, ny) * rng.uniform(-0.5, 0.5, x.shape)
    return np.stack([x.ravel(), y.ravel(), z.ravel()], 1), W.grid_faces(nx, ny)


def _both(monkeypatch, C, opts):
    out = []
    for team in ("0", None):
        if team is None:
            monkeypatch.delenv("RUV_TEAM", raising=False)
        else:
            monkeypatch.setenv("RUV_TEAM", team)
        out.append(R.unfold_charts(R.Context(0), C, opts))
    return out


def _agree(a, b, tol=1e-9):
    for c, (p, q) in enumerate(zip(a, b)):
        assert p.status == q.status == R.Status.OK, (c, p.status, q.status)
        assert p.iters == q.iters, c
        assert np.abs(p.uv - q.uv).max(initial=0.0) <= tol * max(np.abs(p.uv).max(initial=0.0), 1e-30), c


# free rows 1, 31 ... around one row per lane, one CTA's 512 threads and 1024 rows, the steps to
# 2, 4, 8 and 16 CTAs, and several rows per thread of a full team
SIZES = [(3, 3), (33, 3), (34, 3), (18, 34), (34, 34), (35, 34), (66, 34), (67, 66), (130, 66), (200, 170)]


@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
@pytest.mark.parametrize("precond", [R.Precond.NONE, R.Precond.JACOBI, R.Precond.AMG_SA, R.Precond.AMG, R.Precond.IC0,
                                     R.Precond.IC0_COLOR])
def test_team_matches_launch_loop(monkeypatch, precond, precision):
    vo, to, p3, tr = [0], [0], [], []
    for nx, ny in SIZES:
        p, f = _grid(nx, ny)
        p3.append(p)
        tr.append(f)
        vo.append(vo[-1] + len(p))
        to.append(to[-1] + len(f))
    C = R.prepare_patches(np.array(vo), np.array(to), np.concatenate(p3), np.concatenate(tr))
    _agree(*_both(monkeypatch, C, R.UnfoldOptions(precond=precond, precision=precision)))


@pytest.mark.parametrize("stream", ["wide", "row-relative"])
@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
def test_team_column_streams(monkeypatch, precision, stream):
    """A batch with a chart above 65536 rows: 32-bit or row-relative columns for every chart, the
    small ones by teams, the large one by the launch loop or (mixed) a full team."""
    p, f = _grid(300, 240)
    q, g = _grid(40, 30)
    C = R.prepare_patches(np.array([0, len(p), len(p) + len(q)]), np.array([0, len(f), len(f) + len(g)]),
                          np.concatenate([p, q]), np.concatenate([f, g]))
    if stream == "wide":
        monkeypatch.setenv("RUV_NARROW_COLS", "0")
    _agree(*_both(monkeypatch, C, R.UnfoldOptions(precond=R.Precond.JACOBI, precision=precision)))


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 4097])
@pytest.mark.parametrize("precond", [R.Precond.NONE, R.Precond.JACOBI, R.Precond.IC0, R.Precond.IC0_COLOR,
                                     R.Precond.AMG_SA])
def test_team_scalar_systems(monkeypatch, n, precond):
    """The one-column FP64 systems of the solver boundary: rows of up to 13 entries (beyond one
    sweep of eight), a start-up-scale right-hand side and a tiny one."""
    band = min(6, n - 1)
    i = np.arange(n)
    dense = np.zeros((n, 2 * band + 1))
    cols = i[:, None] + np.arange(-band, band + 1)[None, :]
    dense[:] = np.where(np.arange(-band, band + 1) == 0, 4.0 + (i % 11)[:, None] * 0.75,
                        -0.25 / np.maximum(np.abs(np.arange(-band, band + 1)), 1))
    ok = (cols >= 0) & (cols < n)
    a = R.CsrMatrix(dense[ok], cols[ok], np.concatenate([[0], np.cumsum(ok.sum(1))]))
    for scale in (1.0, 1e-150):
        b = scale * ((i % 97) * 0.01 + 1.0)
        got = []
        for team in ("0", "1"):
            monkeypatch.setenv("RUV_TEAM", team)
            got.append(R.GpuSolver.new().cg_solve_precond(a, b, 1000, 1e-12, precond))
        assert (got[0] is None) == (got[1] is None)
        if got[0] is not None:
            assert abs(got[0][1] - got[1][1]) <= 1
            assert np.abs(got[0][0] - got[1][0]).max() <= 1e-11 * np.abs(got[0][0]).max()
