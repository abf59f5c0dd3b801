"""Limits that no iteration meets, by teams and by the launch-per-step loop alike: the identity, whose first
iteration leaves a residual of exactly zero, and a batch with a chart that has no free vertex."""
import numpy as np
import pytest

import researchuv_gb300 as R

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
