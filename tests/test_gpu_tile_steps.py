"""The launch-per-step loop's chart steps at the end of the tile kernels (a chart's last tile to arrive) against
steps in kernels of their own: the partials are combined in the same order, so the same bits, from one
tile to a chart's many, for every loop (RUV_TILE_STEPS picks the form, RUV_TEAM=0 the loop)."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _launches(ctx):
    return R.lib().ruv_kernel_launches(ctx.h)


@pytest.mark.parametrize("precision", [R.Precision.MIXED, R.Precision.FP64])
@pytest.mark.parametrize("precond", [R.Precond.NONE, R.Precond.JACOBI, R.Precond.AMG_SA, R.Precond.IC0_COLOR])
def test_steps_in_tiles_same_bits(monkeypatch, precond, precision):
    vo, to, p3, tr = W.disks(9, t_min=60, t_max=9000, seed=61)
    p, f = W.height_field(190, 6, 0.1, seed=4)  # 35,000 rows: more tiles than a chart step has threads
    vo = np.concatenate([vo, [vo[-1] + len(p)]])
    to = np.concatenate([to, [to[-1] + len(f)]])
    C = R.prepare_patches(vo, to, np.concatenate([p3, p]), np.concatenate([tr, f]).astype(np.int32))
    monkeypatch.setenv("RUV_TEAM", "0")
    got, launches = [], []
    for form in ("0", "1"):
        monkeypatch.setenv("RUV_TILE_STEPS", form)
        ctx = R.Context(0)
        n0 = _launches(ctx)
        uv, stats, st = R.solve_batch(ctx, C.batch(), R.UnfoldOptions(precond=precond, precision=precision), int(vo[-1]))
        assert st == R.Status.OK
        launches.append(_launches(ctx) - n0)
        got.append((uv, [s.cg_iters for s in stats]))
    assert launches[1] < launches[0]
    assert got[0][1] == got[1][1] and np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("n", [1, 511, 513, 30000])
def test_steps_in_tiles_same_bits_one_column(monkeypatch, n):
    i = np.arange(n)
    keep = np.stack([i > 0, i >= 0, i < n - 1], 1)
    cols = (i[:, None] + np.array([-1, 0, 1])[None, :])[keep]
    vals = np.where(np.array([False, True, False])[None, :], 2.5 + (i % 7)[:, None], -1.0)[keep]
    a = R.CsrMatrix(vals, cols, np.concatenate([[0], np.cumsum(keep.sum(1))]))
    monkeypatch.setenv("RUV_TEAM", "0")
    got = []
    for form in ("0", "1"):
        monkeypatch.setenv("RUV_TILE_STEPS", form)
        got.append(R.GpuSolver(R.Context(0)).cg_solve_precond(a, np.cos(i), 1000, 1e-12, R.Precond.JACOBI))
    assert got[0][1] == got[1][1] and np.array_equal(got[0][0], got[1][0])
