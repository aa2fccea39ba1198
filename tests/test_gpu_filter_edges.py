"""The median filter against the oracle where its two ways meet: images with no
pixel, one pixel and many pixels that have all 21 neighbours, equal depths,
and depths that are not a number."""
import numpy as np
import pytest

import hpm_b200 as hb
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(3, 2), (10, 10), (11, 11), (12, 33), (70, 41)])
@pytest.mark.parametrize("what", ["distinct", "ties", "nan"])
def test_median_filter_matches_the_oracle(w, h, what):
    r = np.random.default_rng(w * h)
    depth = r.permutation(w * h).reshape(h, w).astype(np.float32) / (w * h) + 1
    if what == "ties":
        depth = r.integers(1, 4, (h, w)).astype(np.float32)
    if what == "nan":
        depth[r.random((h, w)) < 0.02] = np.nan
    planes = np.zeros((h, w, 4), np.float32)
    planes[..., 2], planes[..., 3] = -1, depth  # fronto-parallel: the distance is the depth
    costs = r.random((h, w)).astype(np.float32)
    costs[r.random((h, w)) < 0.1] = 0.0005  # below 0.001: left as it is
    cams = np.zeros(2, hb.CAMERA_DTYPE)
    cams["K"], cams["R"] = [64, 0, w / 2, 0, 64, h / 2, 0, 0, 1], np.eye(3).reshape(-1)
    cams["t"][1] = [0.1, 0, 0]
    cams["width"], cams["height"], cams["depth_min"], cams["depth_max"] = w, h, 1, 5
    want = orc.depth_normal_filter(cams[0], planes, costs)
    with hb.Context() as ctx:
        ctx.set_views([np.zeros((h, w), np.float32)] * 2, cams)
        got = ctx.depth_normal_filter(planes, costs)
    # a median moves by no more than its values: the depth's division, 2 ulp
    np.testing.assert_allclose(got, want, rtol=4 * 2.0**-23, atol=0)
