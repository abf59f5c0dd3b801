"""The team solver's bounded waits (team.cu team_reduce, team_leave).  With no try allowed
(RUV_SPIN_LIMIT=0) every wait of a team of several CTAs for its sums runs out at once; with one,
some CTAs of a team give up while others go on.  Either way the call ends, a loss is reported as
TIMEOUT, and the same context then solves the batch to the bits it gave before."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _charts():
    vo, to, p3, tr = W.disks(12, t_min=400, t_max=12000, seed=31)
    return R.prepare_patches(vo, to, p3, tr)


@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
@pytest.mark.parametrize("precond", [R.Precond.JACOBI, R.Precond.AMG_SA, R.Precond.IC0_COLOR])
def test_waits_that_run_out_end_the_call(monkeypatch, precond, precision):
    C = _charts()
    n = int(C.i64("chart.vert_off")[-1])
    opts = R.UnfoldOptions(precond=precond, precision=precision)
    monkeypatch.setenv("RUV_TEAM_PER", "64")  # teams of up to 16 CTAs
    ctx = R.Context(0)
    want, _, st = R.solve_batch(ctx, C.batch(), opts, n)
    assert st == R.Status.OK
    several = precond != R.Precond.IC0_COLOR  # (its teams go by the width of a colour: one CTA here)
    for limit in ("0", "1", "1", "2"):
        monkeypatch.setenv("RUV_SPIN_LIMIT", limit)
        _, _, st = R.solve_batch(ctx, C.batch(), opts, n, check=False)
        assert st in (R.Status.OK, R.Status.TIMEOUT), R.Status(st).name
        if limit == "0" and several:
            assert st == R.Status.TIMEOUT
        if st == R.Status.TIMEOUT:
            assert "RUV_SPIN_LIMIT" in ctx.last_error()
        monkeypatch.delenv("RUV_SPIN_LIMIT")
        uv, _, st = R.solve_batch(ctx, C.batch(), opts, n)
        assert st == R.Status.OK and np.array_equal(uv, want)
