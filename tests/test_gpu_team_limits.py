"""Which systems of the solver boundary the team solver takes (team.cu team_solve): its limits fall with a row's
entries, since a team gives a row one thread.  A system left to the launch-per-step loop has that loop's
bits and launches (RUV_TEAM=0); one that a team takes has far fewer launches."""
import numpy as np
import pytest
import scipy.sparse as sp

import researchuv_gb300 as R

pytestmark = pytest.mark.gpu


def _system(n, per_row):
    """Diagonally dominant, about per_row entries in each row, near the diagonal."""
    half = per_row // 2
    rng = np.random.Generator(np.random.PCG64(per_row))
    off = rng.permutation(np.arange(1, 4 * half))[:half]
    w = rng.uniform(0.5, 1.0, half)
    g = sp.diags([np.full(n - o, v) for o, v in zip(off, w)], off, shape=(n, n), format="csr")
    g = g + g.T
    m = (sp.diags(np.asarray(g.sum(1)).ravel() * 1.001 + 1e-3) - g).tocsr()
    m.sort_indices()
    return R.CsrMatrix(m.data, m.indices, m.indptr)


@pytest.mark.parametrize("precond,n,per_row,team", [
    (R.Precond.JACOBI, 39000, 5, True), (R.Precond.JACOBI, 47000, 5, False),
    (R.Precond.JACOBI, 25000, 7, True), (R.Precond.JACOBI, 36000, 7, False),
    (R.Precond.JACOBI, 36000, 13, True), (R.Precond.JACOBI, 47000, 13, False),
    (R.Precond.JACOBI, 36000, 41, True),
    (R.Precond.JACOBI, 15000, 95, True), (R.Precond.JACOBI, 30000, 95, False),
    (R.Precond.AMG, 30000, 7, True), (R.Precond.AMG, 10000, 95, False),
    (R.Precond.IC0_COLOR, 20000, 13, True), (R.Precond.IC0_COLOR, 36000, 61, False),
])
def test_long_rows_lower_the_limit(monkeypatch, precond, n, per_row, team):
    a = _system(n, per_row)
    b = np.cos(np.arange(n))
    got, launches = [], []
    for form in ("0", None):
        if form:
            monkeypatch.setenv("RUV_TEAM", form)
        else:
            monkeypatch.delenv("RUV_TEAM", raising=False)
        s = R.GpuSolver(R.Context(0))
        n0 = R.lib().ruv_kernel_launches(s.ctx.h)
        got.append(s.cg_solve_precond(a, b, 3000, 1e-12, precond))
        assert got[-1] is not None, s.last_error
        launches.append(R.lib().ruv_kernel_launches(s.ctx.h) - n0)
    if team:
        assert launches[0] - launches[1] >= got[0][1]
        assert np.abs(got[0][0] - got[1][0]).max() <= 1e-9 * np.abs(got[0][0]).max()
    else:
        assert launches[0] == launches[1] and got[0][1] == got[1][1]
        assert np.array_equal(got[0][0], got[1][0])
