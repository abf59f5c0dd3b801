"""The IC(0) sweeps' division by a row's pivot through its kept reciprocal (fp64rn.cuh div_by): the IEEE bits of
the division on 2^26 seeded inputs per class -- moderate exponents; arbitrary bit patterns, exponents at
the cut-offs of the short form, zeros over subnormals, infinities and NaNs; quotients near a midpoint."""
import pytest

import researchuv_gb300 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [6, 7, 8])
def test_div_by_bitwise(mode):
    ctx = R.Context(0)
    for seed in (1, 0x5EED0000 + mode):
        bad, first = R.selftest_fp64(ctx, mode, seed, 1 << 26)
        assert bad == 0, (mode, bad, [float.hex(v) for v in first])
