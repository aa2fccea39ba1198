"""Half-steps in the block form of ordinary image sizes (two warps a block, from
593 blocks of 64 pixels on) against the oracle, in every mode that has kernels
or branches of its own: the smaller images of the other half-step tests run four
or eight warps a block.  401x203 is 676 blocks, odd both ways, so the blocks at
both far edges own few pixels.  The prior-net form's proposal is compared with
the wide forms bit for bit in the batched tests."""
import numpy as np
import pytest

import hpm_b200 as hb
import oracle as orc
import synthetic as syn

pytestmark = pytest.mark.gpu

# the shares of equal planes, and of their equal costs, that the other tests ask
# for after two half-steps; a prior adds decisions between products of
# exponentials, in FP32 on the GPU and in the oracle's libm: 0.9 there
MIN_SAME = {"plain": 0.95, "geometric": 0.95, "prior": 0.9, "acmm geometric": 0.95, "acmm hierarchy": 0.95}
MIN_CLOSE = 0.99


@pytest.mark.parametrize("mode,sources", [(m, 4) for m in MIN_SAME] + [("geometric", 9), ("geometric", 17)])
def test_two_warps_a_block(mode, sources):
    w, h, nv = 401, 203, sources + 1
    sc = syn.make_scene(90, w, h, nv, n_planes=6, n_spheres=1, arc_step_deg=min(8.0, 32.0 / sources))
    ref = nv // 2
    imgs, cams = syn.view_set(sc, ref)
    dmin, dmax = sc.depth_min * 0.6, sc.depth_max * 1.2
    r = np.random.default_rng(4)
    gt = sc.gt_depth[ref]
    n = sc.gt_normal[ref] + r.normal(0, 0.1, gt.shape + (3,))
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    planes = np.concatenate([n, (gt * r.uniform(0.95, 1.05, gt.shape))[..., None]], -1).astype(np.float32)
    costs = r.uniform(0, 1, gt.shape).astype(np.float32)
    opts, start = {}, {}
    if mode != "plain":
        start = dict(planes=planes, costs=costs)
    if "geometric" in mode:
        opts["geom"] = True
        depths = [sc.gt_depth[i] * (r.random(gt.shape) > 0.05) for i in [ref] + list(sc.pairs[ref][1])]
        start["depth_maps"] = [d.astype(np.float32) for d in depths]
    if mode == "prior":
        opts["prior"] = True
        start["prior_planes"] = syn.gt_planes_ref_frame(sc, ref)
        start["masks"] = (r.random(gt.shape) < 0.7).astype(np.uint32)
    if "acmm" in mode:
        opts["variant"] = 1
    if "hierarchy" in mode:
        opts["hierarchy"] = 1
    with hb.Context() as ctx:
        ctx.set_views(imgs, cams)
        if "depth_maps" in start:
            ctx.set_geom_depths(start["depth_maps"])
        if "planes" in start:
            ctx.set_hypotheses(planes, costs)
        if "masks" in start:
            ctx.set_prior(start["prior_planes"], start["masks"])
        ctx.run_partial(hb.default_params(dmin, dmax, seed=21, **opts), 2, False)
        gp, gc = ctx.get_result()
    if "hierarchy" in mode:
        start["pre_costs"] = np.zeros(gt.shape, np.float32)
    op, oc, _ = orc.run_patchmatch(imgs, cams, depth_min=dmin, depth_max=dmax, seed=21, salt=0, half_steps=2,
                                   finalize=False, **opts, **start)
    same = np.isclose(gp, op, rtol=1e-4, atol=1e-6).all(-1)
    close = np.isclose(gc[same], oc[same], rtol=1e-3, atol=1e-3, equal_nan=True)
    print(f"{mode} S={sources}: planes {same.mean():.4f} costs {close.mean():.4f}")
    assert same.mean() >= MIN_SAME[mode], same.mean()
    assert close.mean() >= MIN_CLOSE, close.mean()
    # nor do they gather at the edges of the image, where blocks are part empty
    edge = np.ones_like(same)
    edge[8:-8, 16:-16] = False
    assert same[edge].mean() >= MIN_SAME[mode] - 0.05, same[edge].mean()
