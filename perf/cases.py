"""The work that a user of this framework has it do, as measurable cases.

Every case goes through a public entry point of the Python binding (dpe_b200, ncc_autograd): the
per-view PatchMatch call of each schedule stage, the batched call, the whole-scene schedule, the two
kinds of fusion, edge and label maps, and the NCC with its gradient.  Scenes are ray-cast by scene.py
on the GPU (planes and spheres textured with value noise, as the tests and the benchmark use).

Run from the repository's root.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "dpe-mvs-fast_b200"))

import dpe_b200 as D  # noqa: E402
import scene as S  # noqa: E402

_ctx = None


def _context():
    """The one context a program keeps per host thread."""
    global _ctx
    if _ctx is None:
        _ctx = D.Context(0)
    return _ctx


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest per-view call a test or a preview makes: launches and latency count
        dict(name="pm_init_small", kind="pm_init", width=160, height=120, images=4, level=False),
        # the plain workload: 5 views at 640x480, 3 red/black iterations
        dict(name="pm_init_vga", kind="pm_init", width=640, height=480, images=5, level=False),
        # one ordinary view of the batching workload: 1600x1200 with 10 sources (the most work)
        dict(name="pm_init_large", kind="pm_init", width=1600, height=1200, images=11, level=False),
        # the first call of a finer pyramid level: edge, label and weak-texture paths on an interpolated
        # level image (values that are no whole numbers), odd sizes
        dict(name="pm_refine_level", kind="pm_refine", width=801, height=603, images=10, level=True, geom=False),
        # the schedule's commonest call: a geometric-consistency pass at the finest level
        dict(name="pm_refine_geom", kind="pm_refine", width=1600, height=1200, images=10, level=False, geom=True),
        # many views of uneven size in one call on host arrays, FP16 staging and the Gauss-Newton
        # hypothesis (the batching, precision and differentiation forms together)
        dict(name="pm_batch_fp16_gn", kind="pm_batch", width=400, height=300, images=6, views=5, fp16_gn=True),
        # a whole scene through the pyramid schedule and fusion, host arrays in and out, edge and label
        # maps made on the device
        dict(name="scene_schedule", kind="scene", width=400, height=300, views=5, levels=2, refine_calls=1),
        # fusion of a scene's depth maps, the reference's rule with double arithmetic
        dict(name="fuse_scene", kind="fuse", width=1600, height=1200, views=10, rule="eth"),
        # the Tanks-and-Temples rule, float arithmetic, odd sizes
        dict(name="fuse_tat", kind="fuse", width=641, height=479, views=7, rule="tat_intermediate"),
        # the label and edge maps of one full-resolution image (every view, every level needs them)
        dict(name="edge_maps", kind="edges", width=1600, height=1200),
        # autograd through the NCC: forward and backward for planes and source images
        dict(name="ncc_autograd", kind="ncc_grad", width=640, height=480, images=5, queries=100000),
        # a small allocation-free batch of NCC queries on a program's own stream: latency counts
        dict(name="ncc_eval_small", kind="ncc_eval", width=320, height=240, images=3, queries=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pm_init", "pm_init", "pm_refine", "pm_refine", "pm_batch", "scene", "fuse", "edges", "ncc_grad",
                       "ncc_eval"])
    aspect = rng.uniform(0.55, 0.85)
    if kind == "pm_init":
        w = _log_int(rng, 96, 1600)
        return dict(kind=kind, width=w, height=max(64, int(w * min(aspect, 0.75))), images=rng.randint(3, 11),
                    level=rng.random() < 0.4)
    if kind == "pm_refine":
        w = _log_int(rng, 160, 1600)
        return dict(kind=kind, width=w, height=max(96, int(w * min(aspect, 0.75))), images=rng.randint(3, 10),
                    level=rng.random() < 0.5, geom=rng.random() < 0.6)
    if kind == "pm_batch":
        w = _log_int(rng, 128, 480)
        return dict(kind=kind, width=w, height=int(w * aspect), images=rng.randint(3, 7), views=rng.randint(2, 6),
                    fp16_gn=rng.random() < 0.5)
    if kind == "scene":
        w = _log_int(rng, 200, 480)
        return dict(kind=kind, width=w, height=int(w * aspect), views=rng.randint(3, 6), levels=rng.randint(1, 2),
                    refine_calls=rng.randint(1, 2))
    if kind == "fuse":
        w = _log_int(rng, 160, 1600)
        return dict(kind=kind, width=w, height=int(w * min(aspect, 0.75)), views=rng.randint(3, 10),
                    rule=rng.choice(["eth", "eth", "tat_intermediate", "tat_advanced"]))
    if kind == "edges":
        w = _log_int(rng, 320, 1600)
        return dict(kind=kind, width=w, height=int(w * min(aspect, 0.75)))
    w = _log_int(rng, 96, 640)
    if kind == "ncc_grad":
        return dict(kind=kind, width=w, height=int(w * min(aspect, 0.75)), images=rng.randint(2, 5),
                    queries=_log_int(rng, 1000, 100000))
    return dict(kind=kind, width=min(w, 400), height=int(min(w, 400) * min(aspect, 0.75)), images=rng.randint(2, 4),
                queries=_log_int(rng, 64, 65536))


# ------------------------------------------------------------------------------------------ inputs
def _scene(width, height, views, seed, weak):
    """A rendered scene at this size: the plain workload's strongly textured objects, or the full
    pipeline's, half of whose area has weak texture."""
    f = 0.8203125 * width
    spec = S.SceneSpec(width=width, height=height, n_views=views, fx=f, fy=f, cx=width / 2.0, cy=height / 2.0,
                       n_planes=6 if weak else 3, n_spheres=2 if weak else 1, weak_sigma=3.0 if weak else None,
                       tex_freq=0.0375 * width, supersample=1)
    return S.make_scene(spec, seed=seed, device="cuda")


def _params(sc, images, state, geom=False, weak_peak=6):
    """The per-call parameters of the schedule (first call of the coarsest level, later calls at the
    finest of three levels)."""
    p = D.default_params()
    p.num_images = images
    p.state = state
    refine = state != D.FIRST_INIT
    p.use_APD = p.use_edge = p.use_limit = p.use_label = 1 if refine else 0
    p.geom_consistency = 1 if geom else 0
    p.max_iterations = 3
    p.weak_peak_radius = weak_peak
    if refine:
        p.ransac_threshold = np.float32(0.01 - 2 * 0.00125)
        p.rotate_time = 4
    p.depth_min = np.float32(sc.spec.depth_min) * np.float32(0.6)
    p.depth_max = np.float32(sc.spec.depth_max) * np.float32(1.2)
    return p


def _images(sc, ids, level):
    """float32 images on the device: 8-bit values, or an interpolated level image's."""
    out = []
    for i in ids:
        g = torch.from_numpy(sc.gray[i]).cuda().to(torch.float32)
        if level:
            g = (g + g.roll(1, 0) + g.roll(1, 1) + g.roll((1, 1), (0, 1))) * 0.25
        out.append(g.contiguous())
    return out


def _edges_and_labels(gray):
    """Edges (the strongest gradients) and connected regions between them, as the edge and label maps
    of a level: 0 / 255; 0 on edges, -1 on small regions, else the region."""
    H, W = gray.shape
    g = F.avg_pool2d(gray[None, None], 5, 1, 2)[0, 0]
    mag = torch.zeros_like(g)
    mag[1:-1, 1:-1] = torch.hypot(g[1:-1, 2:] - g[1:-1, :-2], g[2:, 1:-1] - g[:-2, 1:-1])
    thr = torch.quantile(mag.reshape(-1)[:: max(1, mag.numel() // 100000)], 0.93)
    edge = (mag > thr).to(torch.uint8) * 255
    free = F.max_pool2d(edge[None, None].float(), 4, 4, ceil_mode=True)[0, 0] == 0
    lab = torch.where(free, torch.arange(1, free.numel() + 1, device=g.device).reshape(free.shape).double(), 0.0)
    for _ in range(96):  # spread the largest index through each region
        lab = torch.where(free, F.max_pool2d(lab[None, None], 3, 1, 1)[0, 0], 0.0)
    lab = lab.to(torch.int64)
    counts = torch.bincount(lab.reshape(-1))
    lab = torch.where((counts[lab] < 40) & (lab > 0), -1, lab).to(torch.int32)
    full = lab.repeat_interleave(4, 0).repeat_interleave(4, 1)[:H, :W].contiguous()
    full[edge > 0] = 0
    return edge.contiguous(), edge[::4, ::4].contiguous(), full.contiguous()


def _prior_state(sc, ref, gray, gen, n):
    """What an earlier call left: depths near the truth with some outliers, jittered normals, WEAK
    where the texture is weak, UNKNOWN at places, and each pixel's selected sources."""
    dev = gray.device
    H, W = gray.shape
    rnd = lambda *s: torch.rand(s, generator=gen, device=dev)
    gauss = lambda *s: torch.randn(s, generator=gen, device=dev)
    depth = torch.from_numpy(sc.depth[ref]).cuda()
    normal = torch.from_numpy(sc.normal[ref]).cuda()
    lo, hi = 0.65 * sc.spec.depth_min, 1.15 * sc.spec.depth_max
    depth = depth * (1.0 + 0.002 * gauss(H, W))
    depth = torch.where(rnd(H, W) < 0.08, lo + (hi - lo) * rnd(H, W), depth).clamp(lo, hi)
    normal = F.normalize(normal + 0.1 * gauss(H, W, 3), dim=2)
    plane = torch.cat([normal, depth[..., None]], 2).contiguous()
    m = F.avg_pool2d(gray[None, None], 9, 1, 4)[0, 0]
    std = (F.avg_pool2d((gray * gray)[None, None], 9, 1, 4)[0, 0] - m * m).clamp_min(0).sqrt()
    weak = torch.full((H, W), D.STRONG, dtype=torch.uint8, device=dev)
    cells = (rnd((H + 3) // 4, (W + 3) // 4) < 0.25).repeat_interleave(4, 0).repeat_interleave(4, 1)[:H, :W]
    weak[(std < 3.5) & cells & (rnd(H, W) < 0.95)] = D.WEAK  # about a fifth of the pixels
    weak[rnd(H, W) < 0.04] = D.UNKNOWN
    weak[:6], weak[-6:], weak[:, :6], weak[:, -6:] = (D.UNKNOWN,) * 4
    views = torch.zeros((H, W), dtype=torch.int32, device=dev)
    cells = ((H + 7) // 8, (W + 7) // 8)
    for j in range(n):  # nearer sources are selected more often
        on = (rnd(*cells) < (0.85 if j < 2 else 0.55 if j < 5 else 0.25)).to(torch.int32)
        views |= on.repeat_interleave(8, 0).repeat_interleave(8, 1)[:H, :W] << j
    return plane, weak.contiguous(), views.contiguous()


def _queries(sc, n, images, gen):
    """NCC queries: random pixels and sources, planes near the truth."""
    dev = "cuda"
    H, W = sc.gray.shape[1:]
    px = torch.randint(0, W, (n,), generator=gen, device=dev, dtype=torch.int32)
    py = torch.randint(0, H, (n,), generator=gen, device=dev, dtype=torch.int32)
    src = torch.randint(1, images, (n,), generator=gen, device=dev, dtype=torch.int32)
    cam = S.camera_struct(sc, 0)
    R = torch.from_numpy(np.asarray(cam["R"], np.float32).reshape(3, 3)).cuda()
    K = np.asarray(cam["K"], np.float32).reshape(3, 3)
    at = (py.long(), px.long())
    depth = torch.from_numpy(sc.depth[0]).cuda()[at] * (1.0 + 0.02 * torch.randn(n, generator=gen, device=dev))
    nw = torch.from_numpy(sc.normal[0]).cuda()[at]
    nr = F.normalize(nw @ R.T + 0.05 * torch.randn((n, 3), generator=gen, device=dev), dim=1)
    ray = torch.stack([(px - float(K[0, 2])) / float(K[0, 0]), (py - float(K[1, 2])) / float(K[1, 1]), torch.ones(n, device=dev)], 1)
    w = -depth * (nr * ray).sum(1)
    return px, py, src, torch.cat([nr, w[:, None]], 1).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    st = dict(kind=kind, case=case)
    W, H = case["width"], case["height"]
    if kind in ("pm_init", "pm_refine"):
        n_img = case["images"]
        sc = _scene(W, H, n_img, seed, weak=kind == "pm_refine")
        ref = n_img // 2
        ids = [ref] + sc.pairs[ref]
        st["images"] = _images(sc, ids, case["level"])
        st["cameras"] = [S.camera_struct(sc, i) for i in ids]
        st["out"] = dict(plane=torch.empty((H, W, 4), device="cuda"), weak=torch.empty((H, W), dtype=torch.uint8, device="cuda"),
                         views=torch.empty((H, W), dtype=torch.int32, device="cuda"), costs=torch.empty((H, W), device="cuda"))
        st["kw"] = dict(seed=1000 + seed, memory=D.MEM_DEVICE)
        if kind == "pm_init":
            st["params"] = _params(sc, n_img, D.FIRST_INIT)
        else:
            geom = case["geom"]
            st["params"] = _params(sc, n_img, D.REFINE_ITER if geom else D.REFINE_INIT, geom, 2 if geom else 6)
            plane, weak, views = _prior_state(sc, ref, st["images"][0], gen, n_img - 1)
            edge, low, label = _edges_and_labels(st["images"][0])
            st["kw"].update(plane_in=plane, weak_in=weak, views_in=views, edge=edge, edge_low=low, label=label)
            if geom:  # the sources' depth maps of the previous call
                st["kw"]["depths"] = [
                    (torch.from_numpy(sc.depth[i]).cuda() * (1.0 + 0.002 * torch.randn((H, W), generator=gen, device="cuda"))).contiguous()
                    for i in ids]
        torch.cuda.synchronize()  # the library works on its own stream
    elif kind == "pm_batch":
        st["calls"] = []
        for v in range(case["views"]):  # uneven sizes, 8-bit images in host memory
            w, h = W - 37 * v % (W // 3), H - 23 * v % (H // 3)
            sc = _scene(w, h, case["images"], seed * 16 + v, weak=False)
            st["calls"].append(dict(images=[np.ascontiguousarray(g.astype(np.float32)) for g in sc.gray],
                                    cameras=[S.camera_struct(sc, i) for i in range(sc.n)],
                                    params=_params(sc, sc.n, D.FIRST_INIT), seed=1000 + seed * 16 + v))
    elif kind == "scene":
        sc = _scene(W, H, case["views"], seed, weak=True)
        st["args"] = (list(sc.gray), list(sc.bgr), [S.camera_struct(sc, v) for v in range(sc.n)], sc.pairs)
        st["kw"] = dict(num_levels=case["levels"], refine_calls=case["refine_calls"], max_iterations=3, min_consistent=2,
                        seed=1000 + seed, device_edges=True, device_labels=True)
    elif kind == "fuse":
        sc = _scene(W, H, case["views"], seed, weak=True)
        st["views"] = []
        for v in range(sc.n):
            plane, weak, _ = _prior_state(sc, v, torch.from_numpy(sc.gray[v]).cuda().float(), gen, 1)
            good = torch.rand((H, W), generator=gen, device="cuda") < 0.9
            depth = torch.where(good, plane[..., 3], 0.0)
            st["views"].append(dict(depth=depth.contiguous(), normal=plane[..., :3].contiguous(), weak=weak,
                                    bgr=torch.from_numpy(sc.bgr[v]).cuda(), camera=S.camera_struct(sc, v), src=sc.pairs[v]))
        torch.cuda.synchronize()
    elif kind == "edges":
        sc = _scene(W, H, 1, seed, weak=True)
        st["gray"] = torch.from_numpy(sc.gray[0]).cuda()
        torch.cuda.synchronize()
    else:
        n_img = case["images"]
        sc = _scene(W, H, n_img, seed, weak=False)
        st["cameras"] = [S.camera_struct(sc, i) for i in range(n_img)]
        st["params"] = _params(sc, n_img, D.FIRST_INIT)
        st["q"] = _queries(sc, case["queries"], n_img, gen)
        st["images"] = _images(sc, range(n_img), False)
        if kind == "ncc_grad":
            st["stack"] = torch.stack(st["images"]).requires_grad_(True)
            st["planes"] = st["q"][3].clone().requires_grad_(True)
            st["gout"] = torch.randn(case["queries"], generator=gen, device="cuda")
        else:
            st["costs"] = torch.empty(case["queries"], device="cuda")
    return st


# ------------------------------------------------------------------------------------------ passes
def _whole(points):
    """The point buffer that the binding's slice of the produced points looks into (zeros follow them):
    the same shape whatever the number of points."""
    return points if points.base is None else points.base


def run(state):
    kind = state["kind"]
    if kind in ("pm_init", "pm_refine"):
        _context().pm_run(state["images"], state["cameras"], state["params"], out=state["out"], **state["kw"])
        return {k: state["out"][k] for k in ("plane", "weak", "views", "costs")}
    if kind == "pm_batch":
        ctx = _context()
        if state["case"]["fp16_gn"]:
            ctx.set_options(staging=D.STAGE_FP16, gn_refine=1)
        out = ctx.pm_run_batch(state["calls"])
        if state["case"]["fp16_gn"]:
            ctx.set_options()
        return [{k: o[k] for k in ("plane", "weak", "views", "costs")} for o in out]
    if kind == "scene":
        r = _context().scene_run(*state["args"], **state["kw"])
        out = {k: r[k] for k in ("depth", "normal", "weak", "views", "points")}
        return dict(out, xyz=_whole(r["xyz"]), bgr=_whole(r["bgr"]))
    if kind == "fuse":
        rule = state["case"]["rule"]
        if rule == "eth":
            r = _context().fuse(state["views"], D.FUSE_FP64, memory=D.MEM_DEVICE, min_consistent=2)
        else:
            variant = D.TAT_INTERMEDIATE if rule == "tat_intermediate" else D.TAT_ADVANCED
            r = _context().fuse_tat(state["views"], variant, D.FUSE_FLOAT, memory=D.MEM_DEVICE)
        return dict(count=r["count"], **{k: _whole(r[k]) for k in ("xyz", "bgr", "origin", "num_consistent")})
    if kind == "edges":
        ctx = _context()
        return {"edge": ctx.edge_map(state["gray"], memory=D.MEM_DEVICE),
                "labels": ctx.edge_labels(state["gray"], 0, memory=D.MEM_DEVICE),
                "labels_half": ctx.edge_labels(state["gray"], 1, memory=D.MEM_DEVICE)}
    px, py, src, planes = state["q"]
    if kind == "ncc_grad":
        import ncc_autograd

        cost = ncc_autograd.NCCCost.apply(state["planes"], state["stack"], state["cameras"], state["params"], px, py, src)
        gp, gi = torch.autograd.grad(cost, (state["planes"], state["stack"]), state["gout"])
        return {"cost": cost.detach(), "grad_planes": gp, "grad_images": gi}
    D.ncc_eval_noalloc(state["images"], state["cameras"], state["params"], px, py, src, planes, state["costs"])
    return {"cost": state["costs"]}


# ------------------------------------------------------------------------------------------ work
_STRONG = 1176  # FLOP of one strong NCC evaluation (36 taps)
_WEAK = 3672    # FLOP of one deformable evaluation (108 taps)


def _pm_work(px, images, host, refine=False, geom=False, iters=3):
    n = images - 1
    sel = min(n, 4)  # sources a pixel samples or has selected, about
    strong = n + iters * (8 * n + 6 * sel) + (61 + 12) * sel
    flops = px * strong * _STRONG
    size = 4 * images + 16 + 1 + 4 + 4
    if refine:  # about a fifth of the pixels are WEAK
        flops = px * (sel + 0.8 * iters * (8 * n + 6 * sel) + (61 + 12) * sel) * _STRONG
        flops += 0.2 * px * iters * (10 * n + 5 * sel) * _WEAK
        size += 16 + 4 + 1 + 1 + 4 + (4 * images if geom else 0)
    return px * size, flops


def work(case):
    kind = case["kind"]
    px = case["width"] * case["height"]
    if kind == "pm_init":
        b, f = _pm_work(px, case["images"], False)
    elif kind == "pm_refine":
        b, f = _pm_work(px, case["images"], False, True, case["geom"])
    elif kind == "pm_batch":
        b, f = 0, 0
        W, H = case["width"], case["height"]
        for v in range(case["views"]):
            x, y = _pm_work((W - 37 * v % (W // 3)) * (H - 23 * v % (H // 3)), case["images"], True)
            b, f = b + x, f + y
    elif kind == "scene":
        V, b, f = case["views"], px * case["views"] * (4 + 21), 0.0
        for lvl in range(case["levels"]):
            p = px / 4.0 ** (case["levels"] - 1 - lvl)
            for call in range(1 + case["refine_calls"]):
                f += V * _pm_work(p, V, True, lvl > 0 or call > 0, call > 0)[1]
        b = int(b)
    elif kind == "fuse":
        V = case["views"]
        b, f = px * V * (4 + 12 + 1 + 3) + px * V * 24, px * V * (V - 1) * 120
    elif kind == "edges":
        b, f = px * (1 + 1 + 4 + 1), px * 40
    elif kind == "ncc_grad":
        n, q = case["images"], case["queries"]
        b, f = px * n * 4 + px * n * 4 + q * (28 + 4 + 4 + 16), q * 36 * 150
    else:
        b, f = px * case["images"] * 4 + case["queries"] * (28 + 4), case["queries"] * _STRONG
    return {"bytes": int(b), "flops": int(f)}


# ------------------------------------------------------------------------------------------ 64 bits
def _ncc64(stack, planes, cameras, params, px, py, src):
    """The bilateral NCC cost (n,) in 64 bits: weights from the reference image, source samples
    bilinear with clamp-to-edge, 1 - covariance / sqrt(variances) clamped to [0, 2]; 2 where the
    centre projects outside the source or a window is flat."""
    dev, f64 = stack.device, torch.float64
    H, W = stack.shape[1:]
    K = torch.tensor(np.stack([np.asarray(c["K"], np.float64).reshape(3, 3) for c in cameras]), device=dev)
    R = torch.tensor(np.stack([np.asarray(c["R"], np.float64).reshape(3, 3) for c in cameras]), device=dev)
    t = torch.tensor(np.stack([np.asarray(c["t"], np.float64) for c in cameras]), device=dev)
    Rrel = R[src] @ R[0].T
    trel = t[src] - (Rrel @ t[0])
    n, w = planes[:, :3], planes[:, 3]
    # points X of the plane satisfy n . X = -w
    Hm = K[src] @ (Rrel - trel[:, :, None] * n[:, None, :] / w[:, None, None]) @ torch.linalg.inv(K[0])
    r, inc = int(params.strong_radius), int(params.strong_increment)
    off = torch.arange(-r, r + 1, inc, device=dev)
    ox, oy = (o.reshape(-1) for o in torch.meshgrid(off, off, indexing="ij"))
    x, y = px.long()[:, None] + ox, py.long()[:, None] + oy

    def project(xs, ys):
        p = Hm @ torch.stack([xs, ys, torch.ones_like(xs)], 1).to(f64)
        return p[:, 0] / p[:, 2], p[:, 1] / p[:, 2]

    cu, cv = project(px[:, None], py[:, None])
    inside = ((cu >= 0) & (cu < W) & (cv >= 0) & (cv < H))[:, 0]
    u, v = project(x, y)
    u, v = torch.nan_to_num(u).clamp(-1, W - 1), torch.nan_to_num(v).clamp(-1, H - 1)
    u0, v0 = u.detach().floor(), v.detach().floor()
    a, b = u - u0, v - v0
    u0, v0 = u0.long(), v0.long()
    base = (src.long() * (H * W))[:, None]
    flat = stack.reshape(-1)
    px_at = lambda xx, yy: flat[base + yy.clamp(0, H - 1) * W + xx.clamp(0, W - 1)]
    s = (1 - b) * ((1 - a) * px_at(u0, v0) + a * px_at(u0 + 1, v0)) + b * ((1 - a) * px_at(u0, v0 + 1) + a * px_at(u0 + 1, v0 + 1))
    ref = stack[0].detach()
    c = ref[py.long(), px.long()][:, None]
    rv = ref[y.clamp(0, H - 1), x.clamp(0, W - 1)]
    ss, sc = float(params.sigma_spatial), float(params.sigma_color)
    wt = torch.exp(-torch.sqrt((ox * ox + oy * oy).to(f64)) / (2 * ss * ss) - (rv - c).abs() / (2 * sc * sc))
    wt = wt / wt.sum(1, keepdim=True)
    mean = lambda q: (wt * q).sum(1, keepdim=True)
    rd, sd = rv - mean(rv), s - mean(s)
    var_r, var_s, cov = mean(rd * rd)[:, 0], mean(sd * sd)[:, 0], mean(rd * sd)[:, 0]
    ok = inside & (var_r >= 1e-5) & (var_s >= 1e-5)
    cost = 1 - cov / torch.sqrt(torch.where(ok, var_r * var_s, torch.ones_like(var_r)))
    return torch.where(ok, cost.clamp(0, 2), torch.full_like(cost, 2.0))


def exact(case, seed):
    """Costs and gradients have a 64-bit value.  A PatchMatch call, a schedule and a fusion are chains
    of decisions between hypotheses drawn at random, and maps are whole numbers: no such value."""
    if case["kind"] not in ("ncc_grad", "ncc_eval"):
        return None
    st = prepare(case, seed)
    px, py, src, planes = st["q"]
    src = src.long()
    n, step = int(px.numel()), 25000
    want = case["kind"] == "ncc_grad"
    stack = torch.stack(st["images"]).double().requires_grad_(want)
    planes = planes.double().requires_grad_(want)
    costs, gp, gi = [], torch.zeros_like(planes), torch.zeros_like(stack)
    for k in range(0, n, step):
        at = slice(k, k + step)
        c = _ncc64(stack, planes[at], st["cameras"], st["params"], px[at], py[at], src[at])
        costs.append(c.detach())
        if want:
            a, b = torch.autograd.grad(c, (planes, stack), st["gout"][at].double())
            gp += a
            gi += b
    if not want:
        return {"cost": torch.cat(costs)}
    return {"cost": torch.cat(costs), "grad_planes": gp, "grad_images": gi}
