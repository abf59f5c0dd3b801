"""IC(0) batches whose charts would wait for each other's SMs as teams stay with the launch-per-step loop (its bits
and launches, RUV_TEAM=0); the others are solved by teams, in far fewer launches."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond,precision,charts,t_min,t_max,team", [
    (R.Precond.IC0, R.Precision.MIXED, 150, 500, 600, True), (R.Precond.IC0, R.Precision.MIXED, 450, 500, 600, False),
    (R.Precond.IC0, R.Precision.FP64, 150, 500, 600, True), (R.Precond.IC0, R.Precision.FP64, 300, 500, 600, False),
    (R.Precond.IC0, R.Precision.MIXED, 2400, 20, 60, False), (R.Precond.IC0, R.Precision.FP64, 450, 100, 700, True),
    (R.Precond.IC0_COLOR, R.Precision.MIXED, 1200, 50, 300, True), (R.Precond.IC0_COLOR, R.Precision.MIXED, 10000, 20, 60, False),
    (R.Precond.IC0_COLOR, R.Precision.FP64, 600, 50, 300, True), (R.Precond.IC0_COLOR, R.Precision.FP64, 10000, 50, 90, False),
])
def test_waiting_teams_leave_the_batch_to_the_loop(monkeypatch, precond, precision, charts, t_min, t_max, team):
    vo, to, p3, tr = W.disks(charts, t_min=t_min, t_max=t_max, seed=8)
    C = R.prepare_patches(vo, to, p3, tr)
    out, launches = [], []
    for form in ("0", None):
        if form:
            monkeypatch.setenv("RUV_TEAM", form)
        else:
            monkeypatch.delenv("RUV_TEAM", raising=False)
        ctx = R.Context(0)
        n0 = R.lib().ruv_kernel_launches(ctx.h)
        uv, stats, st = R.solve_batch(ctx, C.batch(), R.UnfoldOptions(precond=precond, precision=precision), int(vo[-1]))
        assert st == R.Status.OK
        launches.append(R.lib().ruv_kernel_launches(ctx.h) - n0)
        out.append((uv, [s.cg_iters for s in stats]))
    if team:
        assert launches[0] - launches[1] >= 3 * max(out[0][1])
        assert np.abs(out[0][0] - out[1][0]).max() <= 1e-9 * np.abs(out[0][0]).max()
    else:
        assert launches[0] == launches[1]
        assert out[0][1] == out[1][1] and np.array_equal(out[0][0], out[1][0])
