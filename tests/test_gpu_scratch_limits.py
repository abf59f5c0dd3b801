"""Limits that no iteration meets, by teams and by the launch-per-step loop alike: the identity, whose first
iteration leaves a residual of exactly zero, and a batch with a chart that has no free vertex."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu

PRECONDS = [R.Precond.NONE, R.Precond.JACOBI, R.Precond.IC0, R.Precond.IC0_COLOR, R.Precond.AMG]


def _identity(n):
    i = np.arange(n)
    return R.CsrMatrix(np.ones(n), i, np.arange(n + 1)), 1.0 + i % 3


@pytest.mark.parametrize("team", ["0", "1"])
@pytest.mark.parametrize("precond", PRECONDS)
def test_no_iterations_under_a_negative_limit(monkeypatch, precond, team):
    monkeypatch.setenv("RUV_TEAM", team)
    s = R.GpuSolver(R.Context(0))
    a, b = _identity(40)
    assert s.cg_solve_precond(a, b, -100, 1e-12, precond) is None
    assert s.last_error.startswith("NOT_CONVERGED")
    x, iters = s.cg_solve_precond(a, b, 0, 1e-12, precond)  # (a limit of zero: one iteration, as ever)
    assert iters == 1 and np.array_equal(x, b)


@pytest.mark.parametrize("team", ["0", "1"])
@pytest.mark.parametrize("tol", [-1.0, float("nan")])
@pytest.mark.parametrize("precond", PRECONDS)
def test_zero_residual_does_not_meet_a_negative_tolerance(monkeypatch, precond, tol, team):
    monkeypatch.setenv("RUV_TEAM", team)
    s = R.GpuSolver(R.Context(0))
    a, b = _identity(40)
    assert s.cg_solve_precond(a, b, 50, tol, precond) is None
    assert s.last_error.startswith("BREAKDOWN")  # p.q = 0 in the second iteration


@pytest.mark.parametrize("knobs", [{"RUV_TEAM": "0", "RUV_TILE_STEPS": "0"}, {"RUV_TEAM": "0", "RUV_TILE_STEPS": "1"},
                                   {"RUV_TEAM": "1"}])
@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
@pytest.mark.parametrize("precond", [R.Precond.JACOBI, R.Precond.AMG_SA])
def test_chart_without_free_vertices_under_a_negative_tolerance(monkeypatch, precond, precision, knobs):
    vo, to, p3, tr = W.disks(1, t_min=500, t_max=501, seed=3)
    tri = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]])
    C = R.prepare_patches(np.array([0, 3, 3 + vo[-1]]), np.array([0, 1, 1 + to[-1]]), np.concatenate([tri, p3]),
                          np.concatenate([[[0, 1, 2]], tr]).astype(np.int32))
    for k, v in knobs.items():
        monkeypatch.setenv(k, v)
    opts = R.UnfoldOptions(precond=precond, precision=precision, tol=-1.0, max_cg_iter=3)
    _, stats, _ = R.solve_batch(R.Context(0), C.batch(), opts, 3 + int(vo[-1]), check=False)
    assert stats[0].n_free == 0
    assert [(s.status, s.cg_iters) for s in stats] == [(R.Status.BREAKDOWN, 0), (R.Status.NOT_CONVERGED, 3)]
