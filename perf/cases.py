"""Performance cases of the splatting framework: what is timed, on which inputs.

``listed()`` are the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes what a user's program has in hand before
the call (inputs, batch, optimizer), ``run(state)`` is one pass through public
entry points, ``work(case)`` the bytes and operations a pass cannot do without
and ``exact(case, seed)`` the same outputs in 64 bits, where they are cheap
enough to form.

The scenes are the repository's own (dsplat/scenes.py): Gaussians or points
uniform in [-1,1]^3, log-scales uniform in [-4.5,-2.5], unit quaternions,
opacity = sigmoid(N(0,1)) in [0.01,0.99], RGB uniform, SH coefficients with
DC ~ U[0,1] and N(0,0.1) above, cameras at distance 3 with 60 degrees of
vertical field of view, drawn here on the device.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "del-splat_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

RESOLUTIONS = [(320, 240), (640, 480), (1280, 720), (1920, 1080)]
PARAMS = ("means", "log_scales", "quats", "opacity", "colors")
LR, BETAS, EPS = 1e-3, (0.9, 0.999), 1e-8
ADAM_STEPS_BEFORE = 2  # optimizer steps taken by prepare(), so that the moments are those of a running training


def listed():
    return [
        # a del-splat-cudarc caller (project, tile lists with the pair count
        # read back, raster), one view per call: a preview of a tiny cloud,
        # where launches and the read-back count ...
        {"name": "chain_tiny", "kind": "chain", "n": 1000, "w": 96, "h": 64, "ts": 16},
        # ... the plain forward scene of the tests and the README ...
        {"name": "chain_16k_256", "kind": "chain", "n": 16384, "w": 256, "h": 256, "ts": 16},
        # ... and one full-HD view of the benchmark's scene
        {"name": "chain_1m_1080p", "kind": "chain", "n": 1048576, "w": 1920, "h": 1080, "ts": 16},
        # point cloud preview through the DLPack package, ragged sizes
        {"name": "points_200k", "kind": "points", "n": 200003, "w": 641, "h": 479},
        # the benchmark's circle frame: packed z-buffer, RGBA words
        {"name": "circle_zbuf_1m", "kind": "circle_zbuf", "n": 1048576, "w": 1024, "h": 1024, "ts": 16, "rgba": True},
        # the reference's circle path: sphere projection, tile lists, painter
        {"name": "circle_tiles_50k", "kind": "circle_tiles", "n": 50021, "w": 500, "h": 375, "ts": 16, "radius": 0.01},
        # a small differentiable render (torch.autograd, defaults of
        # make_batch): unit-test and few-Gaussian fitting size
        {"name": "autograd_3k", "kind": "autograd", "n": 3000, "sh": 1, "views": 1, "w": 96, "h": 80, "ts": 16},
        # one training view per call, eager, at the default tile size
        {"name": "train_262k_720p", "kind": "train", "n": 262144, "sh": 3, "views": 1, "w": 1280, "h": 720, "ts": 16,
         "graph": False},
        # the headline: 16 views of mixed sizes in one captured step (0x0: the
        # four resolutions in turn), at the tile size the autotuner picks
        {"name": "train_1m_16views", "kind": "train", "n": 1048576, "sh": 3, "views": 16, "w": 0, "h": 0, "ts": 8,
         "graph": True},
        # the large training batch, without its optimizer step (next case) so
        # that every pass does the same work
        {"name": "train_4m_8x1080p", "kind": "train", "n": 4194304, "sh": 3, "views": 8, "w": 1920, "h": 1080, "ts": 8,
         "graph": True},
        # the optimizer step of a 1M-Gaussian scene
        {"name": "adam_1m", "kind": "adam", "n": 1048576, "sh": 3},
        # inference: eight orbit views of a captured-scene size, no loss
        {"name": "orbit_100k_8x480p", "kind": "orbit", "n": 100003, "sh": 3, "views": 8, "w": 640, "h": 480, "ts": 8},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["chain", "points", "circle_zbuf", "circle_tiles", "autograd", "train", "train", "train", "adam",
                       "orbit"])
    w = logint(64, 1920)
    h = min(1080, int(round(w * rng.uniform(0.5, 1.4))))  # wide screens to portrait
    ts = rng.choice([8, 16, 32])
    sh = rng.choice([-1, 0, 1, 2, 3, 3])
    if kind == "chain":
        return {"kind": kind, "n": logint(500, 1048576), "w": w, "h": h, "ts": rng.choice([8, 16, 16, 32])}
    if kind == "points":
        return {"kind": kind, "n": logint(1000, 4194304), "w": w, "h": h}
    if kind == "circle_zbuf":
        return {"kind": kind, "n": logint(1000, 2097152), "w": w, "h": h, "ts": 16, "rgba": rng.random() < 0.5}
    if kind == "circle_tiles":
        return {"kind": kind, "n": logint(1000, 524288), "w": w, "h": h, "ts": ts, "radius": rng.uniform(0.005, 0.03)}
    if kind == "autograd":
        w = logint(48, 640)
        return {"kind": kind, "n": logint(500, 65536), "sh": sh, "views": rng.randint(1, 4), "w": w,
                "h": int(round(w * rng.uniform(0.5, 1.4))), "ts": ts}
    if kind == "adam":
        return {"kind": kind, "n": logint(1000, 2097152), "sh": sh}
    n, views = logint(1000, 2097152), rng.randint(1, 16)
    if n * views > 16 * 1048576:
        views = max(1, 16 * 1048576 // n)
    if kind == "orbit":
        return {"kind": kind, "n": n, "sh": sh, "views": views, "w": w, "h": h, "ts": ts}
    return {"kind": kind, "n": n, "sh": sh, "views": min(views, 8), "w": w, "h": h, "ts": ts,
            "graph": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo


def _coeffs(case):
    return 1 if case["sh"] < 0 else (case["sh"] + 1) ** 2


def _gaussians(g, n, sh):
    quats = torch.randn(n, 4, generator=g, device="cuda")
    p = {"means": _rand(g, n, 3, lo=-1.0), "log_scales": _rand(g, n, 3, lo=-4.5, hi=-2.5),
         "quats": quats / quats.norm(dim=1, keepdim=True),
         "opacity": torch.sigmoid(torch.randn(n, generator=g, device="cuda")).clamp(0.01, 0.99)}
    if sh < 0:
        p["colors"] = _rand(g, n, 3)
    else:
        c = 0.1 * torch.randn(n, (sh + 1) ** 2, 3, generator=g, device="cuda")
        c[:, 0] = _rand(g, n, 3)
        p["colors"] = c
    return {k: v.contiguous() for k, v in p.items()}


def _eyes(seed, count):
    d = np.random.default_rng(int(seed)).standard_normal((count, 3))
    return 3.0 * d / np.linalg.norm(d, axis=1, keepdims=True)


def _matrix(eye, w, h):
    """World -> NDC (4x4, float32 values): 60 degrees vertical field of view, near 0.1, far 10, larger z = nearer."""
    f = -eye / np.linalg.norm(eye)
    up = np.array([0.0, 1.0, 0.0]) if abs(f[1]) < 0.999 else np.array([1.0, 0.0, 0.0])
    r = np.cross(f, up)
    r /= np.linalg.norm(r)
    u = np.cross(r, f)
    view = np.eye(4)
    view[0, :3], view[1, :3], view[2, :3] = r, u, -f
    view[:3, 3] = -r @ eye, -u @ eye, f @ eye
    t = 1.0 / math.tan(math.radians(60.0) / 2.0)
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1], proj[2, 2], proj[2, 3], proj[3, 2] = t * h / w, t, 10.1 / 9.9, 2.0 / 9.9, -1.0
    return (proj @ view).astype(np.float32)


def _sizes(case):
    if case["w"]:
        return [(case["w"], case["h"])] * case.get("views", 1)
    return [RESOLUTIONS[v % len(RESOLUTIONS)] for v in range(case["views"])]


def _views(case, seed):
    """(eye, matrix, width, height) of every view, the eyes on the sphere of radius 3."""
    return [(e, _matrix(e, w, h), w, h) for e, (w, h) in zip(_eyes(seed, case.get("views", 1)), _sizes(case))]


def _cameras(case, seed):
    from dsplat.scenes import Camera
    return [Camera(w, h, np.ascontiguousarray(m.T.reshape(16)), e.astype(np.float32)) for e, m, w, h in _views(case, seed)]


def _project_points(m, xyz, w, h):
    """Pixel x, pixel y, ndc z of points, as a caller without spheres forms them."""
    m = torch.as_tensor(m, device=xyz.device)
    c = [xyz[:, 0] * m[i, 0] + xyz[:, 1] * m[i, 1] + xyz[:, 2] * m[i, 2] + m[i, 3] for i in range(4)]
    return torch.stack([(c[0] / c[3] + 1) * (0.5 * w), (1 - c[1] / c[3]) * (0.5 * h), c[2] / c[3]], dim=1).contiguous()


def _inputs(case, seed):
    """The seeded inputs that prepare() and exact() share."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "chain":
        s = _gaussians(g, case["n"], -1)
        s["scales"] = s["log_scales"].exp()
        return s
    if kind in ("points", "circle_zbuf", "circle_tiles"):
        n, w, h = case["n"], case["w"], case["h"]
        s = {"xyz": _rand(g, n, 3, lo=-1.0), "rgb": _rand(g, n, 3)}
        if kind != "circle_tiles":
            s["xyd"] = _project_points(_views(case, seed)[0][1], s["xyz"], w, h)
        if kind == "circle_zbuf":
            s["rad"] = torch.randint(1, 5, (n,), generator=g, device="cuda").float()
            s["rgba"] = torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g, device="cuda", dtype=torch.int32)
        return s
    s = _gaussians(g, case["n"], case["sh"])
    if kind == "adam":
        s["grads"] = [{k: 1e-3 * torch.randn(s[k].shape, generator=g, device="cuda") for k in PARAMS}
                      for _ in range(ADAM_STEPS_BEFORE + 1)]
    elif kind != "orbit":
        s["target"] = _rand(g, 3 * sum(w * h for w, h in _sizes(case)))
    return s


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case), **_inputs(case, seed)}
    if kind == "chain":
        s["mvp"] = torch.as_tensor(_views(case, seed)[0][1].T.reshape(16).copy(), device="cuda")
    elif kind == "circle_tiles":
        s["world2ndc"] = torch.as_tensor(_views(case, seed)[0][1], device="cuda")
    elif kind == "adam":
        from dsplat.gauss import Adam
        params = {k: s.pop(k) for k in PARAMS}
        s["adam"] = Adam(params, case["sh"], lr=LR, betas=BETAS, eps=EPS)
        for k in range(ADAM_STEPS_BEFORE):
            s["adam"].step(s["grads"][k])
        s["grads"] = s["grads"][ADAM_STEPS_BEFORE]
    elif kind in ("autograd", "train", "orbit"):
        from dsplat.gauss import CapturedStep, GaussBatch
        params = {k: s.pop(k) for k in PARAMS}
        s["params"] = params
        s["batch"] = GaussBatch(case["n"], _cameras(case, seed), case["ts"], case["sh"], pair_capacity=1 << 20)
        s["batch"].ensure_capacity(params)
        if kind == "autograd":
            for v in params.values():
                v.requires_grad_(True)
            s["targets"] = s["batch"].images(s.pop("target"))
        elif kind == "train":
            s["grads"] = {k: torch.zeros_like(v) for k, v in params.items()}
            if case["graph"]:
                s["step"] = CapturedStep(s["batch"], params, s["grads"], s["target"])
        else:
            s["alpha"] = torch.empty(sum(w * h for w, h in _sizes(case)), device="cuda")
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "chain":
        from del_splat_dlpack.SplatGauss import torch as G
        size = (case["w"], case["h"])
        xyd, conic, aabb = G.project(s["means"], s["scales"], s["quats"], s["mvp"], size)
        tile2idx, idx2pnt = G.tile2idx_idx2pnt(size, case["ts"], xyd, aabb)
        image = G.rasterize(size, xyd, conic, aabb, s["opacity"], s["colors"], case["ts"], tile2idx, idx2pnt)
        # idx2pnt is not among the outputs: its length goes with the inputs (the image shows its entries and their order)
        return {"xyd": xyd, "conic": conic, "aabb": aabb, "tile2idx": tile2idx, "image": image}
    if kind == "points":
        from del_splat_dlpack.SplatPoint import torch as P
        return {"image": P.rasterize_pix_zbuffer(s["xyd"], s["rgb"], (case["w"], case["h"]))}
    if kind == "circle_zbuf":
        from del_splat_dlpack.SplatCircle import torch as C
        colors = s["rgba"] if case["rgba"] else s["rgb"]
        return {"image": C.splat_zbuffer(s["xyd"], s["rad"], colors, (case["w"], case["h"]), case["ts"])}
    if kind == "circle_tiles":
        from del_splat_dlpack.SplatCircle import torch as C
        from dsplat import cudarc
        size, ts = (case["w"], case["h"]), case["ts"]
        xyd, rad = C.from_project_spheres(s["xyz"], case["radius"], s["world2ndc"], size)
        tile2idx, idx2pnt = cudarc.splat_circle_tile2idx_idx2pnt(None, cudarc.tile_shape(size, ts), xyd, rad, ts)
        image = torch.zeros((case["h"], case["w"], 3), device=xyd.device)
        cudarc.splat_circle_splat(None, size, image, xyd, rad, s["rgb"], ts, tile2idx, idx2pnt)
        return {"xyd": xyd, "rad": rad, "tile2idx": tile2idx, "image": image}
    if kind == "autograd":
        from del_splat_dlpack.SplatGauss import torch as G
        p = s["params"]
        for v in p.values():
            v.grad = None
        images = G.render(*(p[k] for k in PARAMS), s["batch"])
        loss = sum(((i - t) ** 2).sum() for i, t in zip(images, s["targets"]))
        loss.backward()
        return {"images": [i.detach() for i in images], "loss": loss.detach(), "grads": {k: p[k].grad for k in PARAMS}}
    if kind == "train":
        batch = s["batch"]
        if case["graph"]:
            s["step"].replay()
        else:
            for g in s["grads"].values():
                g.zero_()
            batch.forward(s["params"], target=s["target"])
            batch.backward(s["params"], s["grads"])
        return {"images": batch.images(), "loss": batch.slab_loss().sum(), "grads": s["grads"]}
    if kind == "adam":
        a = s["adam"]
        a.step(s["grads"])
        return {"params": a.params, "exp_avg": a.exp_avg, "exp_avg_sq": a.exp_avg_sq}
    batch = s["batch"]
    batch.forward(s["params"], out_alpha=s["alpha"])
    return {"images": batch.images(), "alpha": s["alpha"]}


# ---------------------------------------------------------------- work
def work(case):
    """Bytes: every input read once, every output written once.  Operations of
    the rasterisers: with the scenes above a Gaussian's 3-sigma box measures
    about 0.005 h^2 pixels and the scene covers about 0.4 h^2, so a covered
    pixel meets about 0.0125 n Gaussians, and its alpha sum passes 0.999
    after about 64 of them; 20 operations blend one (the exponential counted
    as one), 40 more carry its gradient back."""
    n, kind = case["n"], case["kind"]
    if kind == "adam":
        floats = n * (11 + 3 * _coeffs(case))
        return {"bytes": 28 * floats, "flops": 15 * floats}
    sizes = _sizes(case)
    pix = sum(w * h for w, h in sizes)
    views = len(sizes)
    covered = sum(min(w * h, 0.4 * h * h) for w, h in sizes)
    blends = covered * min(0.0125 * n, 64.0)
    if kind == "points":
        return {"bytes": 12 * n + 24 * pix, "flops": 4 * n}
    if kind == "circle_zbuf":  # mean of pi r^2 over r = 1..4 is 23.6 pixels
        return {"bytes": 16 * n + (8 if case["rgba"] else 24) * pix, "flops": 23.6 * 6 * n}
    if kind == "circle_tiles":
        cover = sum(math.pi * (case["radius"] * 0.289 * h) ** 2 for _, h in sizes) * n
        pairs = n * (1 + 2 * case["radius"] * 0.289 * case["h"] / case["ts"]) ** 2
        return {"bytes": 28 * n + 4 * pairs + 12 * pix, "flops": 6 * cover + 60 * n}
    if kind == "chain":
        side = 0.07 * case["h"]
        pairs = n * min((1 + side / case["ts"]) ** 2, float(pix) / case["ts"] ** 2)
        return {"bytes": 40 * n + 40 * n + 16 * n + 4 * pairs + 12 * pix, "flops": 250 * n + 20 * blends}
    row = 11 + 3 * _coeffs(case)
    if kind == "orbit":
        return {"bytes": 4 * row * n + 16 * pix, "flops": 400 * n * views + 20 * blends}
    return {"bytes": 8 * row * n + 36 * pix, "flops": 1000 * n * views + 60 * blends}


# ---------------------------------------------------------------- 64 bits
def _f64_project(means, scales, quats, m, w, h):
    """Pixel centre and ndc z, conic and 3-sigma half extents in float64 (the
    2x3 ndc -> pixel map is applied to the Jacobian with its translation
    column, as this framework defines it)."""
    m = torch.as_tensor(m, device=means.device).double()
    a = means @ m[:3, :3].T + m[:3, 3]
    wc = (means @ m[3, :3] + m[3, 3])[:, None]
    ndc = a / wc
    jac = m[None, :3, :3] / wc[:, :, None] - a[:, :, None] * m[3, :3] / (wc * wc)[:, :, None]
    px, py = 0.5 * w * ndc[:, 0] + 0.5 * w, -0.5 * h * ndc[:, 1] + 0.5 * h
    n2p = torch.tensor([[0.5 * w, 0, 0.5 * w], [0, -0.5 * h, 0.5 * h]], dtype=torch.float64, device=means.device)
    x, y, z, q = quats.unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * q), 2 * (x * z + y * q),
                       2 * (x * y + z * q), 1 - 2 * (x * x + z * z), 2 * (y * z - x * q),
                       2 * (x * z - y * q), 2 * (y * z + x * q), 1 - 2 * (x * x + y * y)], dim=1).view(-1, 3, 3)
    pr = n2p @ jac @ rot
    sig = (pr * (scales * scales)[:, None, :]) @ pr.transpose(1, 2)
    sa, sb, sc = sig[:, 0, 0], sig[:, 0, 1], sig[:, 1, 1]
    # inverse, the smaller eigenvalue held at 1e-5 at least
    hm, hd = 0.5 * (sa + sc), 0.5 * (sa - sc)
    r = torch.sqrt((hd * hd + sb * sb).clamp_min(1e-300))
    l1, l2 = (hm + r).clamp_min(1e-5), hm - r
    det = sa * sc - sb * sb
    pa, pb, pc = (sa - l2) / (2 * r), sb / (2 * r), (sc - l2) / (2 * r)
    plain = l2 >= 1e-5
    conic = torch.stack([torch.where(plain, sc / det, pa / l1 + (1 - pa) / 1e-5),
                         torch.where(plain, -sb / det, pb / l1 - pb / 1e-5),
                         torch.where(plain, sa / det, pc / l1 + (1 - pc) / 1e-5)], dim=1)
    kd = conic[:, 0] * conic[:, 2] - conic[:, 1] ** 2
    half = 3 * torch.stack([torch.sqrt(conic[:, 2] / kd), torch.sqrt(conic[:, 0] / kd)], dim=1)
    return px, py, ndc[:, 2], conic, half


def _f64_blend(px, py, z, conic, half, opacity, rgb, w, h, chunk):
    """Front-to-back blend of every Gaussian over every pixel; a pixel stops after the entry that lifts its alpha
    sum over 0.999.  Differentiable (boxes and stops held fixed)."""
    dev = px.device
    ys, xs = torch.meshgrid(torch.arange(h, device=dev) + 0.5, torch.arange(w, device=dev) + 0.5, indexing="ij")
    xs, ys = xs.reshape(-1, 1).double(), ys.reshape(-1, 1).double()
    order = torch.argsort(z.detach(), descending=True)
    trans = torch.ones_like(xs)
    total = torch.zeros_like(xs)
    image = torch.zeros(w * h, 3, dtype=torch.float64, device=dev)
    for i in range(0, order.numel(), chunk):
        o = order[i:i + chunk]
        dx, dy = xs - px[o], ys - py[o]
        inside = (dx.abs() <= half[o, 0]) & (dy.abs() <= half[o, 1])
        q = conic[o, 0] * dx * dx + 2 * conic[o, 1] * dx * dy + conic[o, 2] * dy * dy
        alpha = torch.where(inside, opacity[o] * torch.exp(-0.5 * torch.where(inside, q, torch.zeros_like(q))), 0.0)
        after = trans * torch.cumprod(1 - alpha, dim=1)
        front = torch.cat([trans, after[:, :-1]], dim=1)
        wgt = alpha * front
        sums = total + torch.cumsum(wgt.detach(), dim=1)
        live = (sums - wgt.detach()) <= 0.999
        image = image + torch.where(live, wgt, 0.0) @ rgb[o]
        trans, total = after[:, -1:], sums[:, -1:]
    return image.view(h, w, 3)


def _sh_rgb(colors, dirs, sh):
    """max(sum_k b_k(dir) coefficient_k + 1/2, 0) in float64, real SH basis up to degree 3."""
    x, y, z = dirs.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    pi = math.pi
    b = [torch.full_like(x, 0.5 * math.sqrt(1 / pi))]
    if sh >= 1:
        c = math.sqrt(3 / (4 * pi))
        b += [-c * y, c * z, -c * x]
    if sh >= 2:
        c = 0.5 * math.sqrt(15 / pi)
        b += [c * x * y, -c * y * z, 0.25 * math.sqrt(5 / pi) * (2 * zz - xx - yy), -c * x * z, 0.5 * c * (xx - yy)]
    if sh >= 3:
        c0, c1, c2 = 0.25 * math.sqrt(35 / (2 * pi)), 0.25 * math.sqrt(105 / pi), 0.25 * math.sqrt(21 / (2 * pi))
        b += [-c0 * y * (3 * xx - yy), 2 * c1 * x * y * z, -c2 * y * (4 * zz - xx - yy),
              0.25 * math.sqrt(7 / pi) * z * (2 * zz - 3 * xx - 3 * yy), -c2 * x * (4 * zz - xx - yy),
              c1 * z * (xx - yy), -c0 * x * (xx - 3 * yy)]
    return (torch.einsum("nk,nkc->nc", torch.stack(b, dim=1), colors) + 0.5).clamp_min(0.0)


def _f64_scene_images(p, case, seed, chunk):
    """Images of every view from raw parameters (quaternions normalised here)."""
    quats = p["quats"] / p["quats"].norm(dim=1, keepdim=True)
    images = []
    for eye, m, w, h in _views(case, seed):
        px, py, z, conic, half = _f64_project(p["means"], p["log_scales"].exp(), quats, m, w, h)
        if case["sh"] < 0:
            rgb = p["colors"]
        else:
            d = p["means"] - torch.as_tensor(eye.astype(np.float32), device="cuda").double()
            rgb = _sh_rgb(p["colors"], d / d.norm(dim=1, keepdim=True), case["sh"])
        images.append(_f64_blend(px, py, z, conic, half, p["opacity"], rgb, w, h, chunk))
    return images


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    s = _inputs(case, seed)
    if kind == "chain":
        w, h = case["w"], case["h"]
        px, py, z, conic, half = _f64_project(s["means"].double(), s["scales"].double(), s["quats"].double(),
                                              _views(case, seed)[0][1], w, h)
        centre = torch.stack([px, py], dim=1)
        image = None
        if n * w * h <= 2 ** 31:
            image = _f64_blend(px, py, z, conic, half, s["opacity"].double(), s["colors"].double(), w, h, 64)
        return {"xyd": torch.stack([px, py, z], dim=1), "conic": conic,
                "aabb": torch.cat([centre - half, centre + half], dim=1), "tile2idx": None, "image": image}
    if kind == "points":
        # nearest point per pixel, the larger index where depths are equal
        w, h = case["w"], case["h"]
        x, y, z = s["xyd"].unbind(1)
        ok = (z > -1) & (z < 1) & (x < w) & (y < h)
        cell = y.clamp_min(0).long() * w + x.clamp_min(0).long()
        bits = (z + 1.0).view(torch.int32).long()
        key = torch.where(ok, (bits << 32) | torch.arange(n, device="cuda"), -1)
        best = torch.full((w * h,), -1, dtype=torch.int64, device="cuda")
        best.scatter_reduce_(0, torch.where(ok, cell, 0), key, "amax")
        rgb = s["rgb"].double()[(best & 0xffffffff).clamp_max(n - 1)]
        return {"image": torch.where((best >= 0)[:, None], rgb, 0.0).view(h, w, 3)}
    if kind == "adam":
        out = {"params": {}, "exp_avg": {}, "exp_avg_sq": {}}
        for k in PARAMS:
            p, m, v = s[k].double(), 0.0, 0.0
            for t in range(ADAM_STEPS_BEFORE + 1):
                g = s["grads"][t][k].double()
                m = BETAS[0] * m + (1 - BETAS[0]) * g
                v = BETAS[1] * v + (1 - BETAS[1]) * g * g
                step = t + 1
                p = p - LR * (m / (1 - BETAS[0] ** step)) / ((v / (1 - BETAS[1] ** step)).sqrt() + EPS)
                if k == "opacity":
                    p = p.clamp(0.0, 0.999)
            out["params"][k], out["exp_avg"][k], out["exp_avg_sq"][k] = p, m, v
        return out
    if kind in ("autograd", "train") and n * sum(w * h for w, h in _sizes(case)) <= 2 ** 25:
        p = {k: s[k].double().requires_grad_(True) for k in PARAMS}
        images = _f64_scene_images(p, case, seed, 256)
        flat = torch.cat([i.reshape(-1) for i in images])
        loss = ((flat - s["target"].double()) ** 2).sum()
        loss.backward()
        return {"images": [i.detach() for i in images], "loss": loss.detach(), "grads": {k: p[k].grad for k in PARAMS}}
    if kind == "orbit" and n * sum(w * h for w, h in _sizes(case)) <= 2 ** 31:
        with torch.no_grad():
            p = {k: s[k].double() for k in PARAMS}
            return {"images": _f64_scene_images(p, case, seed, 64), "alpha": None}
    return None
