"""The workloads this engine's speed is measured on.

Each case is one call (or one submit-and-drain) through the package's public
entry points on a rendered scene: textured spheres and tilted planes before a
background plane, seen by pinhole cameras on an arc around it, which is what
the engine's tests and benchmark solve.  Scenes, images and jobs follow from
the seed alone.

Kinds of case:
  stage  run_patchmatch_mvs on host images: upload, solve, geometric filter,
         maps back on the host (the drop-in call of the reconstruction pipeline)
  solve  Context.solve on resident images into device maps
  plan   Plan.run: a batch of views prepared once and solved repeatedly
  serve  Server: requests submitted, solved together and drained
  cost   Context.ncc_cost: the matching cost of given planes
  fuse   Context.fuse_views: solved maps into one point cloud
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

hp = importlib.import_module("hemiphoto3d-private_b200")

DEPTH_RANGE = (1.0, 6.0)
ARC_RADIUS = 3.0
BACKGROUND_Z = 4.5
MAX_EST_TAPS = 1.1e11  # algorithmic taps of the largest listed case: the bound on a drawn one


def listed():
    """The listed cases, smallest calls first."""
    return [
        # A preview at the reference's window (11 x 11, every pixel): one small view, few iterations.
        dict(name="solve_preview_f32", kind="solve", w=320, h=240, views=1, sources=2, spacing=10.0, radius=5,
             stride=1, iterations=4, precision="f32", dtype="u8"),
        # One request-sized view on the fast path, odd sides.
        dict(name="solve_vga_f16acc", kind="solve", w=641, h=479, views=1, sources=4, spacing=7.5, radius=7,
             stride=2, iterations=8, precision="f16acc", dtype="u8"),
        # The pipeline stage as the reference calls it: five host images, 11 x 11 window, filter on.
        dict(name="stage_vga_f32", kind="stage", w=640, h=480, views=5, sources=4, spacing=10.0, radius=5,
             stride=1, iterations=8, precision="f32", dtype="u8"),
        # The plain workload of the benchmark (15 x 15 window, stride 2, 6 sources, 12 iterations), two views.
        dict(name="solve_hd_f32", kind="solve", w=1920, h=1080, views=2, sources=6, spacing=3.2, radius=7,
             stride=2, iterations=12, precision="f32", dtype="u8"),
        # The same on the FP16-accumulate path, four views.
        dict(name="solve_hd_f16acc", kind="solve", w=1920, h=1080, views=4, sources=6, spacing=3.2, radius=7,
             stride=2, iterations=12, precision="f16acc", dtype="u8"),
        # The reference's window at full HD on the fast path, one view.
        dict(name="solve_hd_dense_f16acc", kind="solve", w=1920, h=1080, views=1, sources=6, spacing=3.2, radius=5,
             stride=1, iterations=12, precision="f16acc", dtype="u8"),
        # The precision form: FP16 images with sensor noise, 8 sources.
        dict(name="solve_6mp_f16acc", kind="solve", w=3000, h=2000, views=1, sources=8, spacing=2.0, radius=7,
             stride=2, iterations=12, precision="f16acc", dtype="f16"),
        # The largest view of the batched and serving mixes.
        dict(name="solve_12mp_f16acc", kind="solve", w=4000, h=3000, views=1, sources=5, spacing=7.5, radius=7,
             stride=2, iterations=6, precision="f16acc", dtype="u8"),
        # A batch of uneven views in one plan.
        dict(name="plan_uneven_f16acc", kind="plan", w=1280, h=720, views=5, sources=8, spacing=7.5, radius=7,
             stride=2, iterations=12, precision="f16acc", dtype="u8"),
        # Requests of uneven size and length served together.
        dict(name="serve_uneven_f16acc", kind="serve", w=1920, h=1080, views=6, sources=8, spacing=7.5, radius=7,
             stride=2, iterations=12, precision="f16acc", dtype="u8"),
        # The matching cost alone, at the reference's window.
        dict(name="cost_hd_f32", kind="cost", w=1920, h=1080, views=1, sources=6, spacing=3.2, radius=5, stride=1,
             iterations=0, precision="f32", dtype="u8"),
        # Fusing solved maps into a cloud.
        dict(name="fuse_hd", kind="fuse", w=1920, h=1080, views=8, sources=6, spacing=3.2, radius=7, stride=2,
             iterations=0, precision="f32", dtype="f32"),
    ]


def draw(rng):
    """One more case of the same ranges: every kind, size, window, source count and precision."""
    while True:
        kind = rng.choice(["solve", "solve", "solve", "stage", "plan", "serve", "cost", "fuse"])
        w = int(round(math.exp(rng.uniform(math.log(160), math.log(4000)))))
        h = max(120, min(3000, int(round(w * rng.uniform(0.55, 0.8)))))
        c = dict(kind=kind, w=w, h=h, views=rng.randint(1, 4), sources=rng.randint(2, 8),
                 spacing=round(rng.uniform(2.0, 8.0), 2), radius=rng.choice([3, 5, 5, 7, 7]), stride=rng.randint(1, 2),
                 iterations=rng.randint(4, 12), precision=rng.choice(["f32", "f16acc"]),
                 dtype=rng.choice(["u8", "u8", "f16", "f32"]))
        if kind == "stage":  # host images, at least two views (the filter needs another map)
            c.update(views=rng.randint(2, 5), dtype="u8", w=min(w, 1920), h=min(h, 1080))
        elif kind in ("plan", "serve"):
            c.update(views=rng.randint(3, 6), w=max(320, min(w, 1920)), h=max(240, min(h, 1080)))
        elif kind == "cost":
            c.update(views=1, iterations=0, w=min(w, 2560), h=min(h, 1440))
        elif kind == "fuse":
            c.update(views=rng.randint(3, 8), iterations=0, radius=7, stride=2, precision="f32", dtype="f32",
                     w=min(w, 2560), h=min(h, 1440))
        if sum(_taps(v) for v in _views(c)) <= MAX_EST_TAPS:
            return c


# --------------------------------------------------------------------------------------------
# The views of a case
# --------------------------------------------------------------------------------------------

def _side(case):
    return (2 * case["radius"]) // case["stride"] + 1


def _views(case):
    """Size, sources and iterations of each solved view.  Plans and request streams mix sizes (full, three
    quarters, half, odd sides), 2 to `sources` sources and half to all iterations, by position."""
    out = []
    for k in range(case["views"]):
        w, h, s, it = case["w"], case["h"], case["sources"], case["iterations"]
        if case["kind"] in ("plan", "serve"):
            num, den = ((1, 1), (1, 2), (3, 4), (1, 3))[k % 4]
            w, h = w * num // den - k % 2, h * num // den - (k // 2) % 2
            s = max(2, s - (3 * k) % 7)
            it = max(1, it - (it * k) // (2 * case["views"]))
        out.append(dict(w=w, h=h, s=s, it=it, taps=_side(case) ** 2))
    return out


def _taps(v):
    """Window samples of one view as the algorithm states it: the initial cost, then per iteration four
    neighbour planes and two perturbed ones on every pixel."""
    return float(v["w"]) * v["h"] * v["s"] * v["taps"] * (1 + 6 * v["it"])


def _cameras(n, spacing, w, h):
    """(K, R, t) of n cameras `spacing` degrees apart on the arc, aimed at its centre."""
    f = 0.78 * w
    K = np.array([[f, 0, w / 2.0], [0, f, h / 2.0], [0, 0, 1.0]])
    target = np.array([0.0, 0.0, ARC_RADIUS])
    cams = []
    for i in range(n):
        a = math.radians((i - (n - 1) / 2.0) * spacing)
        c = target + ARC_RADIUS * np.array([math.sin(a), 0.0, -math.cos(a)])
        z = (target - c) / np.linalg.norm(target - c)
        x = np.cross([0.0, 1.0, 0.0], z)
        x /= np.linalg.norm(x)
        R = np.stack([x, np.cross(z, x), z])
        cams.append((K, R, -R @ c))
    return cams


def _nearest(n, ref, k):
    """The k cameras nearest to `ref` on the arc (ties: lower index)."""
    return sorted((i for i in range(n) if i != ref), key=lambda i: (abs(i - ref), i))[:k]


def _albedo(gen, n=1024, sigma=1.5):
    """Uniform noise blurred by a periodic Gaussian, mean 0.5, standard deviation 0.15."""
    x = torch.rand(n, n, generator=gen, device="cuda")
    r = int(4 * sigma)
    g = torch.exp(-0.5 * (torch.arange(-r, r + 1, device="cuda") / sigma) ** 2)
    g = g / g.sum()
    x = sum(g[i + r] * torch.roll(x, i, 0) for i in range(-r, r + 1))
    x = sum(g[i + r] * torch.roll(x, i, 1) for i in range(-r, r + 1))
    return (0.5 + 0.15 * (x - x.mean()) / x.std()).clamp(0.0, 1.0)


def _layout(rng):
    """Three spheres and two tilted planes at seeded poses: (kind, point, size, normal, texture offset)."""
    objs = [("plane", np.array([0.0, 0.0, BACKGROUND_Z]), 1e9, np.array([0.0, 0.0, -1.0]), (0.0, 0.0))]
    for _ in range(3):
        objs.append(("sphere", np.array([rng.uniform(-1, 1), rng.uniform(-0.5, 0.5), rng.uniform(2.4, 4.0)]),
                     rng.uniform(0.3, 0.55), None, tuple(rng.uniform(0, 5, 2))))
    for _ in range(2):
        tilt, az = math.radians(rng.uniform(15, 45)), rng.uniform(0, 2 * math.pi)
        n = np.array([math.sin(az) * math.sin(tilt), math.cos(az) * math.sin(tilt), -math.cos(tilt)])
        objs.append(("plane", np.array([rng.uniform(-1.2, 1.2), rng.uniform(-0.5, 0.5), rng.uniform(2.0, 3.8)]),
                     rng.uniform(0.3, 0.6), n, tuple(rng.uniform(0, 5, 2))))
    return objs


def _render(objs, tex, cam, w, h):
    """(image in [0, 1], depth, camera-frame normal) of one view, float32 on the GPU."""
    K, R, t = cam
    dev = dict(device="cuda", dtype=torch.float32)
    x = (torch.arange(w, **dev) - K[0, 2]) / K[0, 0]
    y = (torch.arange(h, **dev) - K[1, 2]) / K[1, 1]
    ray = torch.stack([x.expand(h, w), y[:, None].expand(h, w), torch.ones(h, w, **dev)], -1)
    Rt = torch.tensor(R, **dev)
    d = ray @ Rt  # world direction with camera z = 1: the ray parameter is the depth
    c = torch.tensor(-R.T @ t, **dev)
    depth = torch.full((h, w), float("inf"), **dev)
    image = torch.full((h, w), 0.5, **dev)
    normal = torch.zeros(h, w, 3, **dev)
    tpm = 0.78 * w / 3.5  # about one texel per pixel at the scene's typical depth
    n = tex.shape[0]
    for kind, p, size, nv, off in objs:
        pt = torch.tensor(p, **dev)
        if kind == "plane":
            nt = torch.tensor(nv, **dev)
            s = ((pt - c) @ nt) / (d @ nt)
            X = c + s[..., None] * d
            q = X - pt
            hit = (s > 0) & (q[..., 0].abs() < size) & (q[..., 1].abs() < size)
            N = nt.expand(h, w, 3)
        else:
            oc = c - pt
            a, b, cc = (d * d).sum(-1), d @ oc, oc @ oc - size * size
            disc = b * b - a * cc
            s = (-b - disc.clamp(min=0).sqrt()) / a
            X = c + s[..., None] * d
            q = X - pt
            hit = (disc > 0) & (s > 0)
            N = q / size
        hit &= s < depth
        u, v = (q[..., 0] + off[0]) * tpm, (q[..., 1] + off[1]) * tpm
        u0, v0 = u.floor(), v.floor()
        fu, fv = u - u0, v - v0
        i, j = u0.long() % n, v0.long() % n
        i1, j1 = (i + 1) % n, (j + 1) % n
        val = (1 - fv) * ((1 - fu) * tex[j, i] + fu * tex[j, i1]) + fv * ((1 - fu) * tex[j1, i] + fu * tex[j1, i1])
        image = torch.where(hit, val, image)
        normal = torch.where(hit[..., None], N, normal)
        depth = torch.where(hit, s, depth)
    return image, depth, normal @ Rt.T


def _stored(image, dtype, gen):
    if dtype == "u8":
        return (image * 255.0).round().to(torch.uint8)
    if dtype == "f16":  # with sensor noise
        return (image + 0.01 * torch.randn(image.shape, generator=gen, device="cuda")).clamp(0, 1).half()
    return image.contiguous()


def _params(case):
    return hp.default_params(radius=case["radius"], stride=case["stride"],
                             precision=hp.PRECISION_F16ACC if case["precision"] == "f16acc" else hp.PRECISION_F32)


def _inputs(case, seed):
    """Rendered scene of a case: one group per image size, each with its cameras and views, and what to solve:
    (group, reference index, source indices, iterations) per solved view."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    tex, objs = _albedo(gen), _layout(rng)
    specs = _views(case)
    groups, jobs = {}, []
    for v in specs:
        g = groups.setdefault((v["w"], v["h"]), dict(w=v["w"], h=v["h"], refs=0, sources=0))
        g["refs"] += 1
        g["sources"] = max(g["sources"], v["s"])
    for g in groups.values():
        n = max(g["refs"], g["sources"] + 1)
        g["cams"] = _cameras(n, case["spacing"], g["w"], g["h"])
        g["views"] = [_render(objs, tex, cam, g["w"], g["h"]) for cam in g["cams"]]
        g["images"] = [_stored(v[0], case["dtype"], gen) for v in g["views"]]
        g["first"], g["next"] = (n - g["refs"]) // 2, 0  # the solved views lie around the arc's middle
    for v in specs:
        g = groups[(v["w"], v["h"])]
        ref = g["first"] + g["next"]
        g["next"] += 1
        jobs.append((g, ref, _nearest(len(g["cams"]), ref, v["s"]), v["it"]))
    return groups, jobs, gen


def prepare(case, seed):
    groups, specs, gen = _inputs(case, seed)
    kind = case["kind"]
    if kind == "stage":
        (g,) = groups.values()
        cams = [hp.make_camera(*c) for c in g["cams"]]
        images = [i.cpu().numpy() for i in g["images"]]
        views = [hp.ViewParams(ref, srcs, *DEPTH_RANGE) for _, ref, srcs, _ in specs]
        cfg = hp.MVSConfig(mvs_iterations=case["iterations"], mvs_patch_size=2 * case["radius"] + 1,
                           window_stride=case["stride"], precision=_params(case).precision)
        return dict(kind=kind, ctx=hp.Context(0), images=images, cams=cams, views=views, cfg=cfg)
    if kind == "fuse":
        (g,) = groups.values()
        depths, normals, conf, grays = [], [], [], []
        for img, d, n in g["views"]:
            noise = torch.randn(d.shape, generator=gen, device="cuda")
            drop = torch.rand(d.shape, generator=gen, device="cuda") < 0.05  # what the filter removed
            depths.append(torch.where(drop, 0.0, d * (1.0 + 0.002 * noise)).contiguous())
            normals.append(n.contiguous())
            conf.append((0.5 + 0.5 * torch.rand(d.shape, generator=gen, device="cuda")).contiguous())
            grays.append(img.contiguous())
        views, keep = [], [depths, normals, conf, grays]
        for k, cam in enumerate(g["cams"]):
            nb = np.array(_nearest(len(depths), k, min(case["sources"], len(depths) - 1)), np.int32)
            keep.append(nb)
            views.append(hp.FuseView(hp.make_camera(*cam), depths[k].data_ptr(), normals[k].data_ptr(),
                                     conf[k].data_ptr(), grays[k].data_ptr(),
                                     nb.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), len(nb), g["w"], g["h"]))
        # The caller's cloud buffers: room for half the pixels, what lies past the count stays zero.
        room = len(depths) * g["w"] * g["h"] // 2
        outs = [torch.zeros(room, 3, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        return dict(kind=kind, ctx=hp.Context(0), views=views, outs=outs, keep=keep,
                    params=hp.fuse_params(memory=hp.MEMORY_DEVICE))
    torch.cuda.synchronize()  # uploads and solves run on the context's own stream
    ctx = hp.Context(0)
    ids = {id(g): [ctx.upload(i) for i in g["images"]] for g in groups.values()}
    jobs, maps, outs = [], [], []
    for k, (g, ref, srcs, it) in enumerate(specs):
        im = ids[id(g)]
        jobs.append(hp.make_job(im[ref], [im[s] for s in srcs], hp.make_camera(*g["cams"][ref]),
                                [hp.make_camera(*g["cams"][s]) for s in srcs], *DEPTH_RANGE, seed=42 + seed,
                                view_id=k, iterations=it))
        shape = (g["h"], g["w"])
        arr = [torch.empty(shape, device="cuda"), torch.empty(shape + (3,), device="cuda"),
               torch.empty(shape, device="cuda")]
        if kind == "cost":  # planes near the surface, as a solve holds them half-way
            _, d, n = g["views"][ref]
            arr[0].copy_(d * (1.0 + 0.005 * torch.randn(shape, generator=gen, device="cuda")))
            tilted = n + 0.1 * torch.randn(shape + (3,), generator=gen, device="cuda")
            arr[1].copy_(tilted / tilted.norm(dim=-1, keepdim=True))
        outs.append(tuple(arr))
        maps.append(hp.maps_of(*arr))
    torch.cuda.synchronize()
    ctx.synchronize()
    state = dict(kind=kind, ctx=ctx, jobs=jobs, maps=maps, outs=outs, params=_params(case))
    if kind == "plan":
        state["plan"] = hp.Plan(ctx, jobs, state["params"], maps)
    elif kind == "serve":
        state["server"] = hp.Server(ctx, state["params"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "stage":
        res = hp.run_patchmatch_mvs(state["images"], state["cams"], state["views"], state["cfg"], ctx=state["ctx"])
        return [(m.depth, m.normal, m.confidence) for m in res]
    if kind == "fuse":
        out = hp.PointCloudC(hp.MEMORY_DEVICE, *(o.data_ptr() for o in state["outs"]), state["outs"][0].shape[0], 0)
        count = state["ctx"].fuse_views(state["views"], state["params"], out)
        return count, state["outs"]
    if kind == "solve":
        state["ctx"].solve(state["jobs"], state["params"], state["maps"])
    elif kind == "plan":
        state["plan"].run()
    elif kind == "serve":
        for job, maps in zip(state["jobs"], state["maps"]):
            state["server"].submit(job, maps)
        state["server"].drain()
        state["server"].poll()
    else:
        state["ctx"].ncc_cost(state["jobs"][0], state["params"], state["maps"][0])
        return state["outs"][0][2]
    return state["outs"]


def work(case):
    """Bytes: each image read once, each map written once.  Operations: 20 per window sample (warp, bilinear
    sample and the five window sums) of the samples the algorithm states; samples that provably cannot change
    a result need not be taken."""
    specs = _views(case)
    px = sum(float(v["w"]) * v["h"] for v in specs)
    if case["kind"] == "fuse":  # depth, normal, confidence and colour in, about a third of the pixels out as points
        nb = min(case["sources"], case["views"] - 1)
        return {"bytes": px * (24.0 + 36.0 / 3.0), "flops": px * nb * 60.0}
    size = {"u8": 1, "f16": 2, "f32": 4}[case["dtype"]]
    groups = {}
    for v in specs:
        n, s = groups.get((v["w"], v["h"]), (0, 0))
        groups[(v["w"], v["h"])] = (n + 1, max(s, v["s"]))
    read = sum(float(w) * h * size * max(n, s + 1) for (w, h), (n, s) in groups.items())
    if case["kind"] == "cost":  # planes in, cost out
        return {"bytes": read + px * 20.0, "flops": 20.0 * px * specs[0]["s"] * specs[0]["taps"]}
    return {"bytes": read + px * 20.0, "flops": 20.0 * sum(_taps(v) for v in specs)}


def exact(case, seed):
    """The matching cost in 64 bits (exact bilinear samples).  None for the others: a solve is a chain of
    discrete choices between hypotheses, and which pixels become points of a fused cloud depends on thresholds, so
    neither has a value that another precision reproduces element by element."""
    if case["kind"] != "cost":
        return None
    groups, specs, gen = _inputs(case, seed)
    g, ref, srcs, _ = specs[0]
    h, w = g["h"], g["w"]
    _, d, n = g["views"][ref]
    depth = (d * (1.0 + 0.005 * torch.randn((h, w), generator=gen, device="cuda"))).double()
    tilted = n + 0.1 * torch.randn((h, w, 3), generator=gen, device="cuda")
    normal = (tilted / tilted.norm(dim=-1, keepdim=True)).double()
    def gray(i):
        x = i.double()
        return (x / 255.0).float().double() if i.dtype == torch.uint8 else x
    img = [gray(g["images"][i]) for i in [ref, *srcs]]
    Kr, Rr, tr = g["cams"][ref]
    Kinv = torch.tensor(np.linalg.inv(Kr), device="cuda")
    ys, xs = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                            torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    ray = torch.stack([xs, ys, torch.ones_like(xs)], -1) @ Kinv.T
    npd = (normal * ray).sum(-1) * depth
    m = (normal @ Kinv) / npd[..., None]  # K^-T n / (n . P)
    r, st, side = case["radius"], case["stride"], _side(case)
    costs = []
    for k, s in enumerate(srcs):
        K, R, t = g["cams"][s]
        Rrel = R @ Rr.T
        A = torch.tensor(K @ Rrel @ np.linalg.inv(Kr), device="cuda")
        b = torch.tensor(K @ (t - Rrel @ tr), device="cuda")
        cnt, sr, ss, srr, sss, srs = (torch.zeros(h, w, device="cuda", dtype=torch.float64) for _ in range(6))
        for i in range(side):
            for j in range(side):
                dy, dx = i * st - r, j * st - r
                px, py = xs + dx, ys + dy
                f = m[..., 0] * px + m[..., 1] * py + m[..., 2]
                wx, wy, wz = (A[q, 0] * px + A[q, 1] * py + A[q, 2] + b[q] * f for q in range(3))
                u, v = wx / wz, wy / wz
                ok = (wz.abs() >= 1e-8) & (u >= 0) & (u < w - 1) & (v >= 0) & (v < h - 1)
                u0 = u.clamp(0, w - 2).floor()
                v0 = v.clamp(0, h - 2).floor()
                fu, fv = (u - u0).clamp(0, 1), (v - v0).clamp(0, 1)
                at = v0.long() * w + u0.long()
                q = img[k + 1].reshape(-1)
                sv = (1 - fv) * ((1 - fu) * q[at] + fu * q[at + 1]) + fv * ((1 - fu) * q[at + w] + fu * q[at + w + 1])
                rv = img[0].reshape(-1)[((ys + dy).clamp(0, h - 1).long() * w + (xs + dx).clamp(0, w - 1).long())]
                o = ok.double()
                rv, sv = rv * o, sv * o
                cnt += o
                sr += rv
                ss += sv
                srr += rv * rv
                sss += sv * sv
                srs += rv * sv
        dr, ds = cnt * srr - sr * sr, cnt * sss - ss * ss
        ncc = ((cnt * srs - sr * ss) / (dr.clamp(min=1e-300).sqrt() * ds.clamp(min=1e-300).sqrt())).clamp(-1, 1)
        bad = (cnt < (side * side) // 2) | (dr < 1e-6) | (ds < 1e-6) | (npd.abs() < 1e-8)
        costs.append(torch.where(bad, 2.0, 1.0 - ncc))
    top = torch.stack(costs).sort(0).values[: min(3, len(costs))]
    return top.mean(0)
