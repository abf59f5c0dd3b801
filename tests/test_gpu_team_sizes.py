"""Teams of every size under every limit: RUV_TEAM_ROWS lifts the limits on a chart's rows, which lie below the
largest chart here for some solves, and RUV_TEAM_PER sets the rows of a CTA, so that the same charts run
on 1 to 16 CTAs, with the operator in shared memory and without.  Against the launch-per-step loop
(RUV_TEAM=0); the launch counts show that teams ran."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# 1, 1024, 2048, 8192 and 33,264 free rows
SIZES = [(3, 3), (34, 34), (66, 34), (130, 66), (200, 170)]


@pytest.fixture(scope="module")
def charts():
    vo, to, p3, tr = [0], [0], [], []
    for nx, ny in SIZES:
        y, x = np.meshgrid(np.linspace(0, 1, ny), np.linspace(0, 1, nx), indexing="ij")
        z = 0.05 * np.sin(5 * x) * np.cos(4 * y)
        p3.append(np.stack([x.ravel(), y.ravel(), z.ravel()], 1))
        tr.append(W.grid_faces(nx, ny))
        vo.append(vo[-1] + nx * ny)
        to.append(to[-1] + len(tr[-1]))
    return R.prepare_patches(np.array(vo), np.array(to), np.concatenate(p3), np.concatenate(tr))


@pytest.mark.parametrize("per", ["256", "1024", "4096"])
@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
@pytest.mark.parametrize("precond", [R.Precond.JACOBI, R.Precond.AMG_SA, R.Precond.AMG])
def test_every_team_size_matches_the_launch_loop(monkeypatch, charts, precond, precision, per):
    n = int(charts.i64("chart.vert_off")[-1])
    monkeypatch.setenv("RUV_TEAM_ROWS", "1000000")
    monkeypatch.setenv("RUV_TEAM_PER", per)
    out, launches = [], []
    for team in ("0", "1"):
        monkeypatch.setenv("RUV_TEAM", team)
        ctx = R.Context(0)
        n0 = R.lib().ruv_kernel_launches(ctx.h)
        uv, stats, st = R.solve_batch(ctx, charts.batch(), R.UnfoldOptions(precond=precond, precision=precision), n)
        assert st == R.Status.OK
        launches.append(R.lib().ruv_kernel_launches(ctx.h) - n0)
        out.append((uv, [s.cg_iters for s in stats]))
    # every chart by a team: no iteration of the launch loop, which is three launches and more for each
    assert launches[0] - launches[1] >= 3 * max(out[0][1])
    if precision == R.Precision.FP64:  # (the mixed loop's last refresh may come some iterations sooner or later)
        assert all(abs(a - b) <= 1 for a, b in zip(out[0][1], out[1][1]))
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-9 * np.abs(out[0][0]).max()
