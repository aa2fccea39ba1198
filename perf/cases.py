"""The work this library does for its users, as timed cases.

Each case is one call sequence through the public Python binding, over a seeded synthetic scene: textured planes
and spheres in front of a backdrop, rendered on the GPU, handed over as the host arrays that a program has after
decoding its images (the maps come back as host arrays too, as the .dmb writers take them).  Only the network and
the allocation-free JBU work on device buffers, as their callers hold them.

Kinds of case:
  pass     hpm_set_views, one plain PatchMatch pass, its planes, costs and selected views
  geom     one geometric-consistency pass from a previous pass's maps and the views' depth maps
  problem  one reference view through the planar-prior pyramid (hpm_process_problem)
  scene    every view of a scene, view after view: prior pyramid, then two geometric iterations (hpm_run_scene)
  net      every view of a scene of uneven sizes in the batched prior-net form (hpm_run_scene_batched_net)
  acmm     every view of a scene through the ACMM+NESP variant's image pyramid (hpm_run_scene_acmm)
  fuse     the final maps of a scene to a coloured point cloud (hpm_fuse)
  jbu      joint bilateral upsampling of a coarse depth and normal map, device buffers in and out
  train    loss and gradients of the proposal network on a batch of coarse views
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hpm-mvs_b200"))

import hpm_b200 as hb  # noqa: E402
import priornet  # noqa: E402

DEV = "cuda"
DEPTH_RANGE = (2.0, 8.0)
#: FLOP of one bilateral NCC window (36 taps of 34, and 80 for the homography and the last steps)
WINDOW = 36 * 34 + 80


def listed():
    return [
        # the smallest call: a thumbnail-sized problem, where launches and copies are all there is
        {"name": "pass_96x72", "kind": "pass", "w": 96, "h": 72, "sources": 4},
        # the ordinary single-scale problem: VGA, five views
        {"name": "pass_640x480", "kind": "pass", "w": 640, "h": 480, "sources": 4},
        # an odd size with many sources (the widest refinement kernel)
        {"name": "pass_801x601_s20", "kind": "pass", "w": 801, "h": 601, "sources": 20},
        # the largest view the path takes without rescaling, ten sources
        {"name": "pass_3200x2133", "kind": "pass", "w": 3200, "h": 2133, "sources": 10},
        # the second half of the work on every view: a pass with the geometric term
        {"name": "geom_1600x1200", "kind": "geom", "w": 1600, "h": 1200, "sources": 10},
        # one view of the usual dataset size from images to final pass-A maps
        {"name": "problem_1600x1200", "kind": "problem", "w": 1600, "h": 1200, "sources": 10, "levels": 2},
        # a whole small scene in the drop-in order
        {"name": "scene_6x480x360", "kind": "scene", "w": 480, "h": 360, "views": 6},
        # a scene of uneven sizes in the fast form
        {"name": "net_6x1600x1200", "kind": "net", "w": 1600, "h": 1200, "views": 6},
        # the variant that works coarse to fine over images
        {"name": "acmm_5x1200x900", "kind": "acmm", "w": 1200, "h": 900, "views": 5},
        # the last stage of a reconstruction
        {"name": "fuse_8x800x600", "kind": "fuse", "w": 800, "h": 600, "views": 8},
        # a prior at quarter scale brought to full scale, inside a caller's own loop
        {"name": "jbu_1600x1200_x4", "kind": "jbu", "w": 1600, "h": 1200, "scale": 4},
        # one gradient step of the proposal network at its training size
        {"name": "train_400x300_b8", "kind": "train", "w": 400, "h": 300, "batch": 8},
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["pass", "pass", "geom", "problem", "scene", "net", "acmm", "fuse", "jbu", "train"])
    aspect = rng.choice([3 / 4, 9 / 16, 2 / 3])
    if kind in ("pass", "geom"):
        w = between(64, 2400)
        return {"kind": kind, "w": w, "h": int(w * aspect) + rng.randrange(2), "sources": between(1, 20 if w < 1200 else 10)}
    if kind == "problem":
        w = between(200, 1600)
        return {"kind": kind, "w": w, "h": int(w * aspect) + rng.randrange(2), "sources": between(3, 10),
                "levels": rng.choice([-1, 0, 1, 2])}
    if kind in ("scene", "net"):
        w = between(160, 640 if kind == "scene" else 1400)
        return {"kind": kind, "w": w, "h": int(w * aspect) + rng.randrange(2), "views": rng.randint(3, 6)}
    if kind == "acmm":
        w = between(240, 1200)
        return {"kind": kind, "w": w, "h": int(w * aspect) + rng.randrange(2), "views": rng.randint(3, 5)}
    if kind == "fuse":
        w = between(120, 900)
        return {"kind": kind, "w": w, "h": int(w * aspect) + rng.randrange(2), "views": rng.randint(3, 8)}
    if kind == "jbu":
        s = rng.choice([2, 4])
        w, h = between(40, 1600) // s * s + s, between(40, 1200) // s * s + s
        return {"kind": kind, "w": w, "h": h, "scale": s}
    return {"kind": kind, "w": between(40, 400), "h": between(30, 300), "batch": rng.randint(1, 8)}


# ---------------------------------------------------------------------------
# Synthetic scenes, rendered on the GPU
# ---------------------------------------------------------------------------


def _textures(count, size, g, low_texture):
    """Periodic 1/f^2 noise (mean 128, std 40), with blobs of low texture (std 2) over `low_texture` of each."""
    fy = torch.fft.fftfreq(size, device=DEV)[:, None]
    fx = torch.fft.rfftfreq(size, device=DEV)[None]
    f = torch.sqrt(fx * fx + fy * fy)
    turn = torch.exp(2j * math.pi * torch.rand(2, count, *f.shape, generator=g, device=DEV))
    amp = torch.where((f > 0) & (f <= 0.25), 1 / f.clamp_min(1 / size), 0.0)
    tex = torch.fft.irfft2(amp * turn[0], s=(size, size))
    tex = 128 + 40 * (tex - tex.mean((1, 2), keepdim=True)) / tex.std((1, 2), keepdim=True)
    field = torch.fft.irfft2(((f > 0) & (f < 4 / size)) * turn[1], s=(size, size))
    cut = torch.quantile(field.flatten(1), 1 - low_texture, dim=1)[:, None, None]
    level = 70 + 120 * torch.rand(count, 1, 1, generator=g, device=DEV)
    return torch.where(field > cut, level + 2 * torch.randn(count, size, size, generator=g, device=DEV), tex)


def _cameras(sizes, w0):
    """Pinhole cameras 8 degrees apart on a 5 m arc around the scene's centre; the field of view is that of 640
    pixels at focal length 512."""
    cams = np.zeros(len(sizes), hb.CAMERA_DTYPE)
    centre = np.array([0.0, 0.0, sum(DEPTH_RANGE) / 2])
    step = math.radians(min(8.0, 80.0 / len(sizes)))
    for i, (w, h) in enumerate(sizes):
        a = (i - (len(sizes) - 1) / 2) * step
        pos = centre + 5 * np.array([math.sin(a), 0.0, -math.cos(a)])
        z = (centre - pos) / np.linalg.norm(centre - pos)
        x = np.cross([0.0, 1.0, 0.0], z)
        x /= np.linalg.norm(x)
        R = np.stack([x, np.cross(z, x), z])
        f = 512 * w / 640
        cams[i]["K"] = [f, 0, w / 2, 0, f, h / 2, 0, 0, 1]
        cams[i]["R"], cams[i]["t"] = R.reshape(-1), -R @ pos
        cams[i]["width"], cams[i]["height"] = w, h
        cams[i]["depth_min"], cams[i]["depth_max"] = DEPTH_RANGE
    return cams


def _scene(sizes, seed, planes=10, spheres=3, low_texture=0.4):
    """(images, depths, world normals) per view as float32 CUDA tensors, and the cameras."""
    g = torch.Generator(DEV).manual_seed(seed)
    r = np.random.RandomState(seed % (1 << 31))
    cams = _cameras(sizes, sizes[0][0])
    tex = _textures(planes + spheres, 512, g, low_texture)
    texel = 0.6 * 5.0 / (0.8 * max(w for w, _ in sizes))
    objs = []
    for k in range(planes):
        tilt, az = math.radians(r.uniform(0, 25 if k == 0 else 55)), r.uniform(0, 2 * math.pi)
        n = np.array([math.sin(tilt) * math.cos(az), math.sin(tilt) * math.sin(az), -math.cos(tilt)])
        z = r.uniform(2.3, 6.8)
        p = np.array([r.uniform(-0.36, 0.36) * z, r.uniform(-0.25, 0.25) * z, z]) if k else np.array([0, 0, 7.4])
        half = (r.uniform(0.3, 0.9) * z * 0.25, r.uniform(0.3, 0.9) * z * 0.25) if k else (1e3, 1e3)
        u = np.cross([1.0, 0, 0] if abs(n[1]) > 0.9 else [0, 1.0, 0], n)
        u /= np.linalg.norm(u)
        objs.append((n, p, half, u, np.cross(n, u)))
    balls = []
    for _ in range(spheres):
        z = r.uniform(2.8, 6.5)
        balls.append((np.array([r.uniform(-0.32, 0.32) * z, r.uniform(-0.22, 0.22) * z, z]), r.uniform(0.25, 0.7)))
    light = torch.tensor([0.3, -0.5, 0.8], device=DEV) / math.sqrt(0.98)

    def t3(v):
        return torch.tensor(np.asarray(v, np.float32), device=DEV)

    images, depths, normals = [], [], []
    for c in cams:
        w, h = int(c["width"]), int(c["height"])
        R, K = c["R"].reshape(3, 3).astype(np.float64), c["K"]
        C = -R.T @ c["t"].astype(np.float64)
        ys, xs = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                                torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
        d = torch.stack([(xs - float(K[2])) / float(K[0]), (ys - float(K[5])) / float(K[4]), torch.ones_like(xs)], -1) @ t3(R)
        best = torch.full((h, w), math.inf, device=DEV)
        grey, nrm = torch.zeros(h, w, device=DEV), torch.zeros(h, w, 3, device=DEV)
        for i in range(planes + spheres):
            if i < planes:
                n, p, half, u, v = objs[i]
                t = float((p - C) @ n) / (d @ t3(n))
                rel = t3(C - p) + t[..., None] * d
                su, sv = rel @ t3(u), rel @ t3(v)
                ok = (t > 0.05) & (su.abs() <= half[0]) & (sv.abs() <= half[1])
                nn = t3(n).expand(h, w, 3)
            else:
                o, rad = balls[i - planes]
                b, a = 2 * (d @ t3(C - o)), (d * d).sum(-1)
                disc = b * b - 4 * a * float((C - o) @ (C - o) - rad * rad)
                t = (-b - disc.clamp_min(0).sqrt()) / (2 * a)
                nn = (t3(C - o) + t[..., None] * d) / rad
                su = torch.atan2(nn[..., 0], -nn[..., 2]) * rad
                sv = torch.asin(nn[..., 1].clamp(-1, 1)) * rad
                ok = (disc > 0) & (t > 0.05)
            ok &= t < best
            uv = torch.stack([su / texel, sv / texel], -1)
            lo = uv.floor()
            fr, lo = uv - lo, lo.long() % 512
            hi = (lo + 1) % 512
            T, (x0, y0), (x1, y1) = tex[i], lo.unbind(-1), hi.unbind(-1)
            fx, fy = fr.unbind(-1)
            val = (1 - fy) * ((1 - fx) * T[y0, x0] + fx * T[y0, x1]) + fy * ((1 - fx) * T[y1, x0] + fx * T[y1, x1])
            nn = torch.where(((nn * d).sum(-1) > 0)[..., None], -nn, nn)
            shade = 0.45 + 0.55 * (-(nn @ light)).clamp(0, 1)
            grey = torch.where(ok, val * shade / 0.8, grey)
            nrm = torch.where(ok[..., None], nn, nrm)
            best = torch.where(ok, t, best)
        grey = grey + 2 * torch.randn(h, w, generator=g, device=DEV)
        images.append(grey.round().clamp(0, 255))
        depths.append(torch.where(best.isfinite(), best, 0.0))
        normals.append(nrm)
    return images, depths, normals, cams


def _nearest(ref, n, count):
    return sorted((j for j in range(n) if j != ref), key=lambda j: (abs(j - ref), j))[:count]


def _host(ts):
    return [np.ascontiguousarray(t.cpu().numpy()) for t in ts]


def _noisy(depths, normals, g):
    """Maps as a pass leaves them: 0.3 % depth noise, a tenth of the pixels off the surface, normals a few degrees off."""
    ds, ns = [], []
    for d, n in zip(depths, normals):
        e = 1 + 0.003 * torch.randn(d.shape, generator=g, device=DEV)
        off = torch.rand(d.shape, generator=g, device=DEV) < 0.1
        wild = DEPTH_RANGE[0] + 6 * torch.rand(d.shape, generator=g, device=DEV)
        ds.append(torch.where(off, wild, d * e))
        ns.append(torch.nn.functional.normalize(n + 0.05 * torch.randn(n.shape, generator=g, device=DEV), dim=-1))
    return ds, ns


def prepare(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    g = torch.Generator(DEV).manual_seed(seed + 1)
    s = {"kind": kind, "seed": seed, "case": case}
    if kind in ("pass", "geom", "problem"):
        n = case["sources"] + 1
        images, depths, normals, cams = _scene([(w, h)] * n, seed)
        order = [n // 2] + _nearest(n // 2, n, n - 1)
        s["images"] = _host([images[i] for i in order])
        s["cams"] = cams[order].copy()
        if kind == "geom":
            ds, ns = _noisy([depths[i] for i in order], [normals[i] for i in order], g)
            s["depths"] = _host(ds)
            s["planes"] = np.ascontiguousarray(torch.cat([ns[0], ds[0][..., None]], -1).cpu().numpy())
            s["costs"] = _host([0.3 * torch.rand(h, w, generator=g, device=DEV)])[0]
        s["ctx"] = hb.Context(0)
    elif kind in ("scene", "net", "acmm"):
        v = case["views"]
        sizes = [(w, h)] * v
        if kind == "net":  # thirds of full size, three quarters and a half
            sizes = [((w, h), (w * 3 // 4, h * 3 // 4), (w // 2, h // 2))[i * 3 // v] for i in range(v)]
        images, _, _, cams = _scene(sizes, seed)
        s["images"], s["cams"] = _host(images), cams
        s["pairs"] = [(i, _nearest(i, v, v - 1)) for i in range(v)]
        s["ctx"] = hb.Context(0)
        if kind == "net":
            s["net"] = priornet.Net.load()
    elif kind == "fuse":
        v = case["views"]
        images, depths, normals, cams = _scene([(w, h)] * v, seed)
        ds, ns = _noisy(depths, normals, g)
        s["depths"], s["normals"], s["cams"] = _host(ds), _host(ns), cams
        s["colors"] = [np.repeat(i.astype(np.uint8)[..., None], 3, -1) for i in _host(images)]
        s["pairs"] = [(i, _nearest(i, v, 6)) for i in range(v)]
        cap = v * w * h
        s["out"] = (np.zeros((cap, 3), np.float32), np.zeros((cap, 3), np.float32), np.zeros((cap, 3), np.uint8))
    elif kind == "jbu":
        k = case["scale"]
        images, depths, normals, _ = _scene([(w, h)], seed)
        ds, ns = _noisy(depths, normals, g)
        s["guide"] = images[0].contiguous()
        s["depth"] = ds[0][::k, ::k].contiguous()
        s["normal"] = ns[0][::k, ::k].contiguous()
        s["out"] = (torch.empty(h, w, device=DEV), torch.empty(h, w, 3, device=DEV))
    else:
        s["net"] = priornet.Net(0, seed=seed)
        s["trainer"] = priornet.Trainer(s["net"])
        s["views"] = _samples(case, seed)
    return s


def _samples(case, seed):
    """Coarse views as the training takes them: the 16 input channels, target depth and normal, and which count."""
    w, h = case["w"], case["h"]
    g = torch.Generator(DEV).manual_seed(seed)
    images, depths, normals, _ = _scene([(w, h)] * case["batch"], seed, planes=6, spheres=2)
    ds, ns = _noisy(depths, normals, g)
    views = []
    for img, d, n, td, tn in zip(images, ds, ns, depths, normals):
        conf = torch.rand(h, w, 1, generator=g, device=DEV)
        x = torch.cat([img[..., None] / 255, d[..., None] / 10, n, conf, d[..., None] / 10, (conf > 0.3).float(),
                       torch.zeros(h, w, 8, device=DEV)], -1).to(torch.bfloat16).contiguous()
        m = (torch.rand(h, w, generator=g, device=DEV) < 0.6) & (td > 0)
        views.append((x, td.contiguous(), tn.contiguous(), m.to(torch.uint8).contiguous()))
    return views


def run(s):
    kind = s["kind"]
    if kind in ("pass", "geom"):
        ctx = s["ctx"]
        ctx.set_views(s["images"], s["cams"])
        if kind == "geom":
            ctx.set_geom_depths(s["depths"])
            ctx.set_hypotheses(s["planes"], s["costs"])
        ctx.run_patchmatch(hb.default_params(DEPTH_RANGE[0] * 0.6, DEPTH_RANGE[1] * 1.2, seed=s["seed"], geom=kind == "geom"))
        planes, costs = ctx.get_result()
        return planes, costs, ctx.get_selected_views()
    if kind == "problem":
        s["ctx"].set_views(s["images"], s["cams"])
        return s["ctx"].process_problem(seed=s["seed"], pyramid_levels=s["case"]["levels"])
    if kind == "scene":
        return s["ctx"].run_scene(s["images"], s["cams"], s["pairs"], seed=s["seed"])
    if kind == "net":
        return s["ctx"].run_scene(s["images"], s["cams"], s["pairs"], seed=s["seed"], pyramid_levels=0,
                                  planar_prior=2, net=s["net"].weights(), batched=True)
    if kind == "acmm":
        return s["ctx"].run_scene_acmm(s["images"], s["cams"], s["pairs"], seed=s["seed"])
    if kind == "fuse":
        return _fuse(s)
    if kind == "jbu":
        (rows, cols), (s_rows, s_cols) = s["guide"].shape, s["depth"].shape
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in (s["guide"], s["depth"], s["normal"], *s["out"])]
        rc = hb.lib().hpm_jbu_noalloc(0, ptr[0], cols, rows, ptr[1], ptr[2], s_cols, s_rows, ptr[3], ptr[4], None)
        if rc != hb.HPM_OK:
            raise hb.HpmError(f"hpm_jbu_noalloc: {rc}")
        return s["out"]
    tr = s["trainer"]
    for t in tr.gw + tr.gb + [tr.loss]:
        t.zero_()
    for x, d, n, m in s["views"]:
        tr.accumulate(x, d, n, m, *DEPTH_RANGE, 1.0 / (x.shape[0] * x.shape[1]))
    return tr.gw, tr.gb, tr.loss


def _fuse(s):
    """hpm_fuse into the caller's point buffers, and the number of points."""
    v, cams, xyz = len(s["cams"]), s["cams"], s["out"][0]
    refs = np.array([r for r, _ in s["pairs"]], np.int32)
    counts = np.array([len(x) for _, x in s["pairs"]], np.int32)
    srcs = np.zeros((v, hb.MAX_IMAGES - 1), np.int32)
    for i, (_, x) in enumerate(s["pairs"]):
        srcs[i, : len(x)] = x
    maps = [(ctypes.c_void_p * v)(*[m.ctypes.data for m in s[k]]) for k in ("depths", "normals", "colors")]
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (cams, refs, counts, srcs, *s["out"])]
    points = ctypes.c_longlong()
    rc = hb.lib().hpm_fuse(0, v, ptr[0], *maps, v, *ptr[1:], ctypes.c_longlong(len(xyz)), ctypes.byref(points))
    if rc != hb.HPM_OK:
        raise hb.HpmError(f"hpm_fuse: {rc}")
    return (*s["out"], points.value)


def work(case):
    """Inputs in and outputs out, and for the passes the windows of every candidate in every source view: one at the
    start, then eight neighbours and five refinements in each of three iterations."""
    kind, w, h = case["kind"], case["w"], case["h"]
    px = w * h
    if kind in ("pass", "geom", "problem"):
        n = case["sources"]
        passes = 1 if kind != "problem" else 2 + (case["levels"] if case["levels"] >= 0 else sum(max(w, h) > 1000 * 2**k for k in range(3)))
        more = 4 * px * (n + 1) + 20 * px if kind == "geom" else 0
        return {"bytes": 4 * px * (n + 1) + more + 24 * px, "flops": passes * px * n * (1 + 39) * WINDOW}
    if kind in ("scene", "net", "acmm"):
        v = case["views"]
        if kind == "net":
            px *= (1 + 9 / 16 + 1 / 4) / 3
        passes = {"scene": 2 + 2, "net": 1 + 2 + 1 / 16, "acmm": 1 + 2 * 2 / 3}[kind]
        return {"bytes": v * px * (4 + 20), "flops": v * px * passes * (v - 1) * 40 * WINDOW}
    if kind == "fuse":
        v = case["views"]
        return {"bytes": v * px * (16 + 3 + 27), "flops": v * px * min(6, v - 1) * 150}
    if kind == "jbu":
        k = case["scale"]
        taps = {2: 25, 4: 289}[k]
        return {"bytes": px * (4 + 16) + px // (k * k) * 16, "flops": px * taps * 14}
    macs = 9 * (16 * 32 + 32 * 32 + 32 * 32 + 32 * 16)
    return {"bytes": case["batch"] * px * (32 + 17), "flops": case["batch"] * px * 2 * (3 * macs - 9 * 16 * 32)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "jbu":
        return _exact_jbu(prepare(case, seed))
    if kind == "train":
        return _exact_train(case, seed)
    # the passes choose among random candidates by comparing costs, and the fusion by tests and an order: what they
    # return are the choices, which have no value in more bits
    return None


def _exact_jbu(s):
    """Per pixel the weighted mean of the coarse depths and normals in the window around it: a Gaussian of the
    distance in coarse pixels (0.5), times one of the guide's difference (25.5), taken as many fine pixels away as
    the coarse sample is coarse ones."""
    guide, depth, normal = (s[k].double() for k in ("guide", "depth", "normal"))
    (rows, cols), (s_rows, s_cols) = guide.shape, depth.shape
    r = (s["case"]["scale"] ** 2 + 1) // 2
    y, x = torch.arange(rows, device=DEV), torch.arange(cols, device=DEV)
    oy, ox = y * (s_cols / cols), x * (s_cols / cols)
    maps = torch.cat([normal, depth[..., None], torch.ones_like(depth)[..., None]], -1)
    total = torch.zeros(rows, cols, 5, dtype=torch.float64, device=DEV)
    for j in range(-r, r + 1):
        cy = (oy + j).trunc().long().clamp(0, s_rows - 1)
        for i in range(-r, r + 1):
            cx = (ox + i).trunc().long().clamp(0, s_cols - 1)
            far = (oy - cy)[:, None] ** 2 + (ox - cx)[None] ** 2
            other = guide[(y + j).clamp(0, rows - 1)][:, (x + i).clamp(0, cols - 1)]
            wgt = torch.exp(-far / (2 * 0.5**2) - (guide - other) ** 2 / (2 * 25.5**2))
            total += wgt[..., None] * maps[cy][:, cx]
    return total[..., 3] / total[..., 4], torch.nn.functional.normalize(total[..., :3], dim=-1)


def _exact_train(case, seed):
    net = priornet.Net(0, seed=seed)
    ws = [w.to(torch.bfloat16).double().requires_grad_() for w in net.w]
    bs = [b.double().requires_grad_() for b in net.b]
    lo, hi = DEPTH_RANGE
    total = torch.zeros((), dtype=torch.float64, device=DEV)
    for x, d, n, m in _samples(case, seed):
        y = x.double().permute(2, 0, 1)[None]
        for i, (w, b) in enumerate(zip(ws, bs)):
            y = torch.nn.functional.conv2d(y, w, b, padding=1)
            if i < 3:
                y = y.relu()
        m = m.bool()
        o = y[0].permute(1, 2, 0)[m]
        depth = lo + (hi - lo) * torch.sigmoid(o[:, 0])
        cos = (torch.nn.functional.normalize(o[:, 1:4], dim=1) * n[m].double()).sum(1)
        t = d[m].double()
        total = total + ((depth - t).abs() / t + 0.5 * (1 - cos)).sum()
    inv = 1.0 / (case["w"] * case["h"])
    total.backward()
    return [w.grad * inv for w in ws], [b.grad * inv for b in bs], total.detach().reshape(1)
