"""The launch-per-step loop's kernels on batches whose charts teams would solve (RUV_TEAM=0 keeps them in the
loop): the autotuner's pick on the LU bar, the column streams, lane rules, shapes and tile rows of the
V-cycle.  Bit for bit where the sums have one order (one lane adds its row in entry order, a row does not
know its tile, a narrow column is the same column), within the mixed solve's bar else."""
import numpy as np
import pytest

import researchuv_gb300 as R
from oracle import oracle as O
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MIXED_TOL = 1e-6


@pytest.fixture(scope="module")
def disks():
    vo, to, p3, tr = W.disks(10, t_min=100, t_max=8000, seed=29)
    C = R.prepare_patches(vo, to, p3, tr)
    ref = []
    for c in range(len(vo) - 1):
        P = O.Pipeline(p3[vo[c]:vo[c + 1]], tr[to[c]:to[c + 1]], weld_tol=0.0, lu_limit=0)
        ref.append(P.superlu_uv(0))
    return C, ref


def _check(res, ref):
    for c, r in enumerate(res):
        assert r.status == R.Status.OK, (c, r.status)
        assert O.uv_error(r.uv, ref[c]) <= MIXED_TOL, c


def _same(a, b):
    assert [r.cg_iters for r in a] == [r.cg_iters for r in b]
    assert all(np.array_equal(x.uv, y.uv) for x, y in zip(a, b))


def test_autotuned_loop_meets_the_bar(monkeypatch, disks):
    C, ref = disks
    monkeypatch.setenv("RUV_TEAM", "0")
    ctx = R.Context(0)
    opts = R.UnfoldOptions(precond=R.Precond.AMG_SA)
    _check(R.unfold_charts(ctx, C, opts), ref)
    R.autotune(ctx, R.Precision.MIXED, reps=2)
    _check(R.unfold_charts(ctx, C, opts), ref)


@pytest.mark.parametrize("knobs", [{"RUV_AMG_L1SHAPE": "0"}, {"RUV_AMG_L2SHAPE": "1"}, {"RUV_AMG_TILE": "1024/256"},
                                   {"RUV_NARROW_COLS": "0"}])
def test_forms_with_the_same_bits(monkeypatch, disks, knobs):
    C, ref = disks
    monkeypatch.setenv("RUV_TEAM", "0")
    ctx = R.Context(0)
    opts = R.UnfoldOptions(precond=R.Precond.AMG_SA)
    base = R.unfold_charts(ctx, C, opts)
    _check(base, ref)
    for k, v in knobs.items():
        monkeypatch.setenv(k, v)
    _same(base, R.unfold_charts(ctx, C, opts))


@pytest.mark.parametrize("knobs", [{"RUV_AMG_SMOOTH_LANES": "0"}, {"RUV_AMG_LANES": "2/4/16/1"}, {"RUV_AMG_TLANES": "1,8"}])
def test_lane_rules_meet_the_bar(monkeypatch, disks, knobs):
    C, ref = disks
    monkeypatch.setenv("RUV_TEAM", "0")
    for k, v in knobs.items():
        monkeypatch.setenv(k, v)
    _check(R.unfold_charts(R.Context(0), C, R.UnfoldOptions(precond=R.Precond.AMG_SA)), ref)
