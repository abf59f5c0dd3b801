"""chart_distortion of many short charts (a thread for each) has the bits of the same charts in batches so small that a
CTA takes each, charts without triangles' worth of area and folded ones among them."""
import numpy as np
import pytest

import researchuv_gb300 as R
from researchuv_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charts,t_min,t_max", [(2500, 20, 60), (6000, 50, 300), (3000, 6, 7)])
def test_thread_form_has_the_bits_of_the_cta_form(charts, t_min, t_max):
    vo, to, p3, tr = W.disks(charts, t_min=t_min, t_max=t_max, seed=17)
    assert to[-1] > 1400 * np.diff(to).max()
    rng = np.random.Generator(np.random.PCG64(1))
    uv = p3[:, :2] + 0.05 * rng.standard_normal((len(p3), 2))  # (some triangles flip)
    uv[vo[3]:vo[4]] = 0.5  # a chart without area
    uv[vo[5]:vo[6], 0] *= -1.0  # one turned over
    ctx = R.Context(0)

    def metrics(a, b):
        C = R.prepare_patches(vo[a:b + 1] - vo[a], to[a:b + 1] - to[a], p3[vo[a]:vo[b]], tr[to[a]:to[b]])
        R.solve_batch(ctx, C.batch(), R.UnfoldOptions(), int(vo[b] - vo[a]), check=False)  # (the batch becomes resident)
        return R.chart_distortion(ctx, uv[vo[a]:vo[b]], b - a)

    many = metrics(0, charts)
    for a in range(0, charts, 1000):
        b = min(a + 250, charts)  # (a quarter of them)
        assert to[b] - to[a] <= 1400 * np.diff(to[a:b + 1]).max()
        assert np.array_equal(many[a:b], metrics(a, b), equal_nan=True)
