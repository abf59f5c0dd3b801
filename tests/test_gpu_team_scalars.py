"""The team solver's scalars (team.cu team_reduce) against the launch-per-step loop (RUV_TEAM=0) where
their range shows: sums over a chart are formed in FP64 from warps' sums, also under FP32 vectors."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FLT_MAX = float(np.finfo(np.float32).max)


def _chart(scale, n=100):
    y, x = np.meshgrid(np.linspace(0, 1, n), np.linspace(0, 1, n), indexing="ij")
    p = scale * np.stack([x.ravel(), y.ravel(), 0.05 * np.sin(5 * x).ravel()], 1)
    f = W.grid_faces(n, n)
    return R.prepare_patches(np.array([0, len(p)]), np.array([0, len(f)]), p, f), len(p)


def _solve(C, n, monkeypatch, team):
    monkeypatch.setenv("RUV_TEAM", team)
    ctx = R.Context(0)
    opts = R.UnfoldOptions(precond=R.Precond.NONE, precision=R.Precision.MIXED)
    uv, stats, st = R.solve_batch(ctx, C.batch(), opts, n, check=False)
    return ctx, uv, stats, st


def test_a_charts_sum_beyond_fp32(monkeypatch):
    """Without a preconditioner p.q of the first iteration (its largest) goes with the fourth power
    of a chart's size.  At 2.5 times FP32's largest number the sums of 128 rows, the smallest tile of
    the launch loop, and of a team's warps still fit in FP32: both loops solve the chart."""
    C, n = _chart(1.0)
    ctx, _, _, st = _solve(C, n, monkeypatch, "0")
    assert st == R.Status.OK
    rp, cols, vals, b = R.export_chart_system(ctx, 0)
    q = np.add.reduceat(vals * b[cols], rp[:-1])
    e = (b * q).reshape(-1, 2).sum(1)  # p.q of the first iteration, by rows (p = b)
    pad = np.concatenate([e, np.zeros(-len(e) % 128)]).reshape(-1, 128).sum(1)
    scale = (e.sum() / (2.5 * FLT_MAX)) ** 0.25
    assert pad.max() / scale**4 < 0.9 * FLT_MAX < FLT_MAX < 2.4 * FLT_MAX < e.sum() / scale**4
    C, n = _chart(scale)
    uv = []
    for team in ("0", "1"):
        _, u, stats, st = _solve(C, n, monkeypatch, team)
        assert st == R.Status.OK and stats[0].status == R.Status.OK, team
        uv.append(u)
    assert np.abs(uv[0] - uv[1]).max() <= 1e-6 * np.abs(uv[0]).max()
