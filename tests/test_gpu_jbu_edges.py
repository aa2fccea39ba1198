"""The ways the joint bilateral upsampling takes its taps, against the oracle
at the tolerance of the other JBU tests: inner blocks (exact coordinates, only
the taps in reach), blocks at the borders and scales that are no power of two
(taps in reach with clamped coordinates), and blocks with a value that is not
finite in reach (every tap, so that a weight of zero still meets it)."""
import numpy as np
import pytest

import hpm_b200 as hb
import oracle as orc

pytestmark = pytest.mark.gpu


def _inputs(w, h, sw, sh, seed):
    r = np.random.default_rng(seed)
    n = r.normal(size=(sh, sw, 3)).astype(np.float32)
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    return (r.uniform(0, 255, (h, w)).round().astype(np.float32), r.uniform(2, 8, (sh, sw)).astype(np.float32), n)


@pytest.mark.parametrize("w,h,sw,sh", [(8, 8, 4, 4), (33, 9, 16, 4), (160, 120, 40, 30), (161, 119, 40, 29),
                                       (128, 96, 16, 12), (120, 90, 40, 30)])
def test_jbu_taps_match_the_oracle(w, h, sw, sh):
    guide, depth, normal = _inputs(w, h, sw, sh, w + h)
    od, on = orc.jbu(guide, depth, normal)
    with hb.Context() as ctx:
        gd, gn = ctx.jbu(guide, depth, normal)
    np.testing.assert_allclose(gd, od, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(gn, on, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_jbu_meets_values_that_are_not_finite(value):
    """One such depth spoils the depths of every pixel whose window holds it,
    at whatever weight, and no other."""
    guide, depth, normal = _inputs(320, 240, 80, 60, 3)
    depth[30, 40] = value
    od, on = orc.jbu(guide, np.where(np.isfinite(depth), depth, 0), normal)
    with hb.Context() as ctx:
        gd, gn = ctx.jbu(guide, depth, normal)
    y, x = np.mgrid[0:240, 0:320]
    window = (np.abs(30 - y // 4) <= 8) & (np.abs(40 - x // 4) <= 8)
    assert not np.isfinite(gd[window]).any()
    np.testing.assert_allclose(gd[~window], od[~window], rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(gn, on, rtol=1e-4, atol=1e-5)
