"""Half-steps at the edges of their tiles, against the oracle.

A block of the half-step kernels updates a patch of 16x8 pixels (one colour:
two warps of 8x4 lanes) and its lanes score windows for one another, so the
sizes here leave lanes, rows of lanes, whole warps and most of a block without
a pixel, and the source counts lie on both sides of the widths the selection
is compiled for and of the 16 view weights per word.  Grids of up to 296 blocks
run eight warps per block, up to 592 (the last size) four."""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import hpm_b200 as hb
import oracle as orc
import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sources", [(7, 5, 1), (16, 8, 2), (17, 9, 3), (15, 41, 9), (33, 17, 13), (47, 12, 17),
                                         (272, 201, 5)])
@pytest.mark.parametrize("half_steps", [0, 2])
def test_half_steps_at_the_edges_of_the_tiles(w, h, sources, half_steps):
    sc = syn.make_scene(40 + w, w, h, sources + 1, n_planes=4, low_texture=0.0, arc_step_deg=min(8.0, 32.0 / sources))
    imgs, cams = syn.view_set(sc, sources // 2)
    dmin, dmax = sc.depth_min * 0.6, sc.depth_max * 1.2
    op, oc, _ = orc.run_patchmatch(imgs, cams, depth_min=dmin, depth_max=dmax, seed=11, salt=0,
                                   half_steps=half_steps, finalize=False)
    with hb.Context() as ctx:
        ctx.set_views(imgs, cams)
        ctx.run_partial(hb.default_params(dmin, dmax, seed=11), half_steps, False)
        gp, gc = ctx.get_result()
    # the shares of test_half_steps_agree_with_oracle (0.999 and 0.95 of the
    # planes, 0.99 of their costs), less three standard deviations of a share
    # of so few pixels
    def least(share):
        return share - 3.0 * math.sqrt(share * (1.0 - share) / (w * h))

    same = np.isclose(gp, op, rtol=1e-4, atol=1e-6).all(-1)
    close = np.isclose(gc[same], oc[same], rtol=1e-3, atol=1e-3, equal_nan=True)
    assert same.mean() >= least(0.999 if half_steps == 0 else 0.95), same.mean()
    assert close.mean() >= least(0.99), close.mean()


def test_two_threads_with_different_source_counts():
    """The refinement's shared memory follows the source count; contexts of two threads launch it side by side."""
    def problem(sources):
        sc = syn.make_scene(70, 48, 36, sources + 1, n_planes=4, low_texture=0.0, arc_step_deg=2.0)
        imgs, cams = syn.view_set(sc, 0)
        return imgs, cams, hb.default_params(sc.depth_min * 0.6, sc.depth_max * 1.2, seed=3)

    def passes(inputs):
        imgs, cams, p = inputs
        maps = []
        with hb.Context() as ctx:
            ctx.set_views(imgs, cams)
            for _ in range(60):  # each with its own random streams
                ctx.run_partial(p, 2, False)
                maps.append(ctx.get_result()[0])
        return maps

    inputs = [problem(2), problem(14)]
    alone = [passes(k) for k in inputs]
    with ThreadPoolExecutor(2) as pool:
        got = list(pool.map(passes, inputs))
    for one, other in zip(alone, got):
        assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(one, other))
