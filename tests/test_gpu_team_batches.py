"""Which batches under a V-cycle the team solver takes whole (team.cu team_solve): by their rows, the largest
chart's, the precision and the hierarchy.  A batch left to the launch-per-step loop has that loop's bits and
launches (RUV_TEAM=0)."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _grids(count, nx, ny):
    """count bumpy charts of (nx - 2)(ny - 2) free vertices."""
    y, x = np.meshgrid(np.linspace(0, 1, ny), np.linspace(0, 1, nx), indexing="ij")
    f = W.grid_faces(nx, ny)
    p3 = [np.stack([x.ravel(), y.ravel(), (0.02 * (c % 7) * np.sin(5 * x) * np.cos(4 * y)).ravel()], 1) for c in range(count)]
    return R.prepare_patches(np.arange(count + 1) * len(p3[0]), np.arange(count + 1) * len(f), np.concatenate(p3),
                             np.concatenate([f] * count))


# 98 x 100 = 9,800 rows a chart, 60 x 65 = 3,900, 120 x 125 = 15,000
@pytest.mark.parametrize("count,nx,ny,precond,precision,team", [
    (20, 100, 102, R.Precond.AMG_SA, R.Precision.FP64, True),
    (31, 100, 102, R.Precond.AMG_SA, R.Precision.FP64, False),
    (31, 100, 102, R.Precond.AMG, R.Precision.FP64, True),
    (56, 100, 102, R.Precond.AMG, R.Precision.FP64, False),
    (56, 100, 102, R.Precond.AMG_SA, R.Precision.MIXED, True),
    (140, 62, 67, R.Precond.AMG_SA, R.Precision.FP64, True),
    (24, 122, 127, R.Precond.AMG_SA, R.Precision.MIXED, True),
    (30, 122, 127, R.Precond.AMG_SA, R.Precision.MIXED, False),
])
def test_batches_by_size(monkeypatch, count, nx, ny, precond, precision, team):
    C = _grids(count, nx, ny)
    n = int(C.i64("chart.vert_off")[-1])
    got, launches = [], []
    for form in ("0", None):
        if form:
            monkeypatch.setenv("RUV_TEAM", form)
        else:
            monkeypatch.delenv("RUV_TEAM", raising=False)
        ctx = R.Context(0)
        n0 = R.lib().ruv_kernel_launches(ctx.h)
        uv, stats, st = R.solve_batch(ctx, C.batch(), R.UnfoldOptions(precond=precond, precision=precision), n)
        assert st == R.Status.OK
        launches.append(R.lib().ruv_kernel_launches(ctx.h) - n0)
        got.append((uv, [s.cg_iters for s in stats]))
    if team:
        assert launches[0] - launches[1] >= max(got[0][1])
    else:
        assert launches[0] == launches[1]
        assert got[0][1] == got[1][1] and np.array_equal(got[0][0], got[1][0])
