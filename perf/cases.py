"""Performance cases of the renderer's hot path.

Every case goes through ``Renderer`` (the Python front end of the C ABI) or
``autograd.RenderFunction`` on a seeded synthetic indoor cloud: an 8 x 6 x 3 m
room with boxes on its floor, points uniform by surface area (or with a
per-surface density drawn log-uniformly over a 100x range) and 3 mm jitter,
uint8 colours, cameras inside the room -- the clouds and views that the tests
and the benchmark use, made here on the GPU so that 10^8 points take a moment.

Kinds of a case:
  knn         exact k nearest neighbours of query points
  precompute  upload + index build + nearest-neighbour radii
  render      one view in one launch (the drop-in per-view form)
  batch       all views in one persistent launch
  backward    gradients of an image loss through stored hit indices
  train       one optimisation step: re-index the cloud, render, loss, backward
"""
import math

import numpy as np
import torch

from renderer_ray_marching_gb300 import _abi
from renderer_ray_marching_gb300.autograd import RenderFunction
from renderer_ray_marching_gb300.renderer import Renderer, View

ROOM = (8.0, 6.0, 3.0)
MIXED = "640x480,1067x690,1920x1080"


def listed():
    return [
        # A picking or query tool that asks for the nearest point of a few
        # hundred positions of a small scan: latency and launches only.
        {"name": "knn_1k_k1_100k", "kind": "knn", "n": 100_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "queries": 1000, "k": 1},
        # Registration or normal estimation: the 10 nearest of every point of
        # another (unsorted) scan of the same room.
        {"name": "knn_500k_k10_2m", "kind": "knn", "n": 2_000_003, "boxes": 12, "density": 1.0, "leaf": 16,
         "queries": 500_001, "k": 10},
        # A small scan made ready for rendering, from device memory.
        {"name": "precompute_100k", "kind": "precompute", "n": 100_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "host": False},
        # The same for an ordinary scan as the command line does it: the
        # cloud comes from host memory and the radii go back there.
        {"name": "precompute_2m_host", "kind": "precompute", "n": 1_999_993, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.05, "host": True},
        # The benchmark's 20M-point cloud with 40 boxes.
        {"name": "precompute_20m", "kind": "precompute", "n": 20_000_000, "boxes": 40, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "host": False},
        # The largest cloud, with uneven density.
        {"name": "precompute_100m_uneven", "kind": "precompute", "n": 100_000_000, "boxes": 12, "density": 100.0,
         "leaf": 16, "max_radius": 0.1, "host": False},
        # A thumbnail of a small scan: the smallest render call.
        {"name": "render_160x120_100k", "kind": "render", "n": 100_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "size": "160x120", "host": False},
        # The per-view form at the reference's image size, 2M points.
        {"name": "render_1067x690_2m", "kind": "render", "n": 2_000_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.05, "size": "1067x690", "host": False},
        # The benchmark's batched workload (20M points, three resolutions), fewer views.
        {"name": "batch_24v_20m", "kind": "batch", "n": 20_000_000, "boxes": 40, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "sizes": MIXED, "views": 24},
        # Many small ragged views of an uneven cloud (a data loader's crops).
        {"name": "batch_65v_ragged_1m", "kind": "batch", "n": 1_000_001, "boxes": 12, "density": 100.0, "leaf": 16,
         "max_radius": 0.1, "sizes": "97x61,200x133,255x193,321x240", "views": 65},
        # Gradients of all views of an optimisation step, hits stored before.
        {"name": "backward_16v_1m", "kind": "backward", "n": 1_000_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "sizes": "1067x690", "views": 16},
        # One step of fitting a cloud to target images, end to end.
        {"name": "train_2v_1m", "kind": "train", "n": 1_000_000, "boxes": 12, "density": 1.0, "leaf": 16,
         "max_radius": 0.1, "sizes": "1067x690", "views": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    w = _log(rng, lo, hi)
    return "%dx%d" % (w, max(8, int(w * rng.uniform(0.5, 1.0))))


def draw(rng):
    kind = rng.choice(["knn", "precompute", "render", "batch", "backward", "train"])
    c = {"kind": kind, "boxes": rng.choice([6, 12, 24, 40]), "density": rng.choice([1.0, 1.0, 10.0, 100.0]),
         "leaf": rng.choice([8, 16, 16, 16, 32])}
    if kind == "knn":
        c.update(n=_log(rng, 20_000, 5_000_000), queries=_log(rng, 300, 1_000_000),
                 k=rng.choice([1, 2, 3, 5, 8, 10, 16, 20, 32]))
    elif kind == "precompute":
        host = rng.random() < 0.3
        c.update(n=_log(rng, 20_000, 4_000_000 if host else 60_000_000), max_radius=rng.choice([0.02, 0.05, 0.1]),
                 host=host)
    elif kind == "render":
        c.update(n=_log(rng, 20_000, 10_000_000), max_radius=rng.choice([0.02, 0.05, 0.1]),
                 size=_size(rng, 64, 1920), host=rng.random() < 0.3)
    elif kind == "batch":
        small = rng.random() < 0.5
        c.update(n=_log(rng, 50_000, 20_000_000), max_radius=rng.choice([0.05, 0.1]),
                 views=rng.randint(17, 80) if small else rng.randint(2, 16),
                 sizes=",".join(_size(rng, 48, 400) if small else _size(rng, 400, 1600) for _ in range(3)))
    elif kind == "backward":
        c.update(n=_log(rng, 50_000, 4_000_000), max_radius=0.1, views=rng.randint(1, 16),
                 sizes=",".join(_size(rng, 64, 1280) for _ in range(2)))
    else:
        c.update(n=_log(rng, 50_000, 2_000_000), max_radius=0.1, views=rng.randint(1, 4),
                 sizes=",".join(_size(rng, 64, 1067) for _ in range(2)))
    return c


# ------------------------------------------------------------------ inputs
def _surfaces(boxes):
    X, Y, Z = ROOM
    r = [((0, 0, 0), (X, 0, 0), (0, Y, 0)), ((0, 0, Z), (X, 0, 0), (0, Y, 0)),
         ((0, 0, 0), (X, 0, 0), (0, 0, Z)), ((0, Y, 0), (X, 0, 0), (0, 0, Z)),
         ((0, 0, 0), (0, Y, 0), (0, 0, Z)), ((X, 0, 0), (0, Y, 0), (0, 0, Z))]
    for x, y, sx, sy, sz in boxes:
        r += [((x, y, sz), (sx, 0, 0), (0, sy, 0)), ((x, y, 0), (sx, 0, 0), (0, 0, sz)),
              ((x, y + sy, 0), (sx, 0, 0), (0, 0, sz)), ((x, y, 0), (0, sy, 0), (0, 0, sz)),
              ((x + sx, y, 0), (0, sy, 0), (0, 0, sz))]
    return np.array(r, np.float64)


def _scene(case, seed):
    """(xyz float32 [n, 3], rgb uint8 [n, 3]) on the GPU, the boxes and each point's surface density (points per m^2)."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    boxes = []
    for _ in range(case["boxes"]):
        sx, sy, sz = rng.uniform(0.3, 1.5, 3)
        boxes.append((rng.uniform(0, ROOM[0] - sx), rng.uniform(0, ROOM[1] - sy), sx, sy, sz))
    rects = _surfaces(boxes)
    area = np.linalg.norm(np.cross(rects[:, 1], rects[:, 2]), axis=1)
    weight = area.copy()
    if case["density"] > 1.0:
        weight *= np.exp(rng.uniform(0.0, math.log(case["density"]), len(area)))
    counts = rng.multinomial(n, weight / weight.sum())
    base = rng.integers(0, 256, (len(area), 3))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dev = dict(device="cuda")
    order = torch.randperm(n, generator=g, **dev)
    sid = torch.repeat_interleave(torch.arange(len(area), **dev), torch.tensor(counts, **dev))[order]
    del order
    xyz = torch.empty((n, 3), dtype=torch.float32, **dev)
    a = torch.rand(n, generator=g, **dev)
    b = torch.rand(n, generator=g, **dev)
    rt = torch.tensor(rects, dtype=torch.float32, **dev)
    for ax in range(3):
        xyz[:, ax] = (rt[sid, 0, ax] + a * rt[sid, 1, ax] + b * rt[sid, 2, ax]
                      + 0.003 * torch.randn(n, generator=g, **dev))
    bt = torch.tensor(base, dtype=torch.int16, **dev)
    rgb = torch.empty((n, 3), dtype=torch.uint8, **dev)
    for ax in range(3):
        noise = torch.randint(-20, 21, (n,), generator=g, dtype=torch.int16, **dev)
        rgb[:, ax] = (bt[sid, ax] + noise).clamp_(0, 255).to(torch.uint8)
    rho = torch.tensor(counts / area, dtype=torch.float32, **dev)[sid]
    return xyz, rgb, boxes, rho


def _sizes(text):
    return [tuple(int(v) for v in s.split("x")) for s in text.split(",")]


def _views(case, seed, boxes):
    """(camera-to-world column-major float32[16], W, H, fov float32) per view: cameras in the room, outside the boxes."""
    rng = np.random.default_rng(seed + 7919)
    sizes = _sizes(case.get("sizes") or case["size"])
    out = []
    while len(out) < case.get("views", 1):
        c = rng.uniform([0.5, 0.5, 0.5], np.array(ROOM) - 0.5)
        if any(x - 0.2 <= c[0] <= x + sx + 0.2 and y - 0.2 <= c[1] <= y + sy + 0.2 and c[2] <= sz + 0.2
               for x, y, sx, sy, sz in boxes):
            continue
        yaw, pitch = rng.uniform(0, 2 * math.pi), math.radians(rng.uniform(-20, 20))
        f = np.array([math.cos(pitch) * math.cos(yaw), math.cos(pitch) * math.sin(yaw), math.sin(pitch)])
        right = np.cross(f, [0.0, 0.0, 1.0])
        right /= np.linalg.norm(right)
        m = np.eye(4)
        m[:3, 0], m[:3, 1], m[:3, 2], m[:3, 3] = right, np.cross(right, f), -f, c
        # each size of the list in turn, so that every seed's call has the same number of rays
        w, h = sizes[len(out) % len(sizes)]
        fov = np.float32(2.0 * math.atan(w / (2.0 * 0.75 * w)))
        out.append((np.ascontiguousarray(m.T.astype(np.float32)).reshape(16), w, h, fov))
    return out


def _rays(view):
    """Origin [3] and unit directions [H*W, 3] in 64 bits."""
    m, w, h, fov = view
    m = torch.tensor(m, dtype=torch.float64, device="cuda").reshape(4, 4).t()
    pane = w / (2.0 * math.tan(0.5 * float(fov)))
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                          torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    d = torch.stack([x - w / 2.0, y - h / 2.0, torch.full_like(x, -pane)], -1).reshape(-1, 3) @ m[:3, :3].t()
    return m[:3, 3], d / d.norm(dim=1, keepdim=True)


def _cached_radii(case, seed, rho):
    """Radii as a cache file holds them: nearest-neighbour distances of points that lie at random on a
    surface of density rho are Rayleigh-distributed; the jitter widens them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 31)
    u = torch.rand(case["n"], generator=g, device="cuda").clamp_(min=1e-6)
    return (1.3 * torch.sqrt(-torch.log(u) / (math.pi * rho))).clamp_(min=5e-4, max=case["max_radius"]).float()


def _splat(view, xyz, rad):
    """Hit map of the spheres by splatting: the first sphere along each pixel's ray among those whose
    projected disc covers it (up to 4 pixels from the centre), -1 where there is none and at pixels near
    the first sphere's silhouette, which a user masks out (the depth's gradient grows without bound there)."""
    m, w, h, _ = view
    o, d = _rays(view)
    mt = torch.tensor(m, dtype=torch.float64, device="cuda").reshape(4, 4).t()
    best = torch.full((w * h,), torch.iinfo(torch.int64).max, dtype=torch.int64, device="cuda")
    pane = w / (2.0 * math.tan(0.5 * float(view[3])))
    for lo in range(0, xyz.shape[0], 1 << 20):
        p = xyz[lo:lo + (1 << 20)].double() - o
        cam = p @ mt[:3, :3]
        z = -cam[:, 2]
        px = cam[:, 0] / z * pane + w / 2.0
        py = cam[:, 1] / z * pane + h / 2.0
        r = rad[lo:lo + (1 << 20)].double()
        reach = r / z * pane
        near = (z > 0.1) & (px > -4) & (px < w + 4) & (py > -4) & (py < h + 4)
        idx = torch.nonzero(near).reshape(-1)
        for dy in range(-4, 5):
            for dx in range(-4, 5):
                k = idx[reach[idx] > max(abs(dx), abs(dy)) - 1.0]
                x, y = px[k].round().long() + dx, py[k].round().long() + dy
                ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
                k, pix = k[ok], (y * w + x)[ok]
                b = (p[k] * d[pix]).sum(1)
                disc = r[k] ** 2 - ((p[k] - b[:, None] * d[pix]) ** 2).sum(1)
                ok = disc > 0
                t = (b[ok] - disc[ok].sqrt()) * 1e6
                best.scatter_reduce_(0, pix[ok], (t.long() << 32) | (k[ok] + lo), "amin")
    hit = torch.where(best == torch.iinfo(torch.int64).max, -1, best & 0xffffffff)
    p = xyz[hit.clamp(min=0)].double() - o
    off = p - (p * d).sum(1, keepdim=True) * d
    return torch.where((off ** 2).sum(1) < (0.9 * rad[hit.clamp(min=0)].double()) ** 2, hit, -1).int()


def _queries(case, seed, xyz):
    """Points of another scan of the same surfaces, in no order."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 101)
    pick = torch.randint(0, case["n"], (case["queries"],), generator=g, device="cuda")
    return xyz[pick] + 0.005 * torch.randn((case["queries"], 3), generator=g, device="cuda")


def _image_grads(case, seed, pixels):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 211)
    drgb = 2e-3 * torch.randn((pixels, 3), generator=g, device="cuda")
    ddep = 1e-3 * torch.sign(torch.randn(pixels, generator=g, device="cuda"))
    return drgb, ddep


def _renderer(case, xyz, rgb, radii="compute"):
    r = Renderer(leaf_size=case["leaf"])
    r.set_cloud(xyz, rgb)
    r.build_index()
    if isinstance(radii, str):
        r.compute_radii(case["max_radius"], device=True)
    elif radii is not None:
        r.set_radii(radii, case["max_radius"])
    return r


def prepare(case, seed):
    kind = case["kind"]
    xyz, rgb, boxes, rho = _scene(case, seed)
    s = {"case": case}
    if kind == "knn":
        s["q"] = _queries(case, seed, xyz)
        s["r"] = _renderer(case, xyz, rgb, None)
    elif kind == "precompute":
        s["r"] = Renderer(leaf_size=case["leaf"])
        s["xyz"], s["rgb"] = (xyz.cpu().numpy(), rgb.cpu().numpy()) if case["host"] else (xyz, rgb)
    elif kind in ("render", "batch"):
        s["r"] = _renderer(case, xyz, rgb)
        s["views"] = [View(m, w, h, float(fov)) for m, w, h, fov in _views(case, seed, boxes)]
        if kind == "batch":
            # a render loop keeps its frames and its view table
            pixels = sum(v.pixels for v in s["views"])
            s["rgbd"] = torch.empty((pixels, 4), device="cuda")
            s["hit"] = torch.empty(pixels, dtype=torch.int32, device="cuda")
            s["frames"] = (_abi.RmFrame * len(s["views"]))()
            lo = 0
            for fr, v in zip(s["frames"], s["views"]):
                fr.rgbd, fr.hit = s["rgbd"][lo:].data_ptr(), s["hit"][lo:].data_ptr()
                lo += v.pixels
            s["cviews"] = (_abi.RmView * len(s["views"]))(*[v.to_c() for v in s["views"]])
    elif kind == "backward":
        rad = _cached_radii(case, seed, rho)
        views = _views(case, seed, boxes)
        s["r"] = _renderer(case, xyz, rgb, rad)
        s["views"] = [View(m, w, h, float(fov)) for m, w, h, fov in views]
        s["hit"] = torch.cat([_splat(v, xyz, rad) for v in views])
        s["drgb"], s["ddep"] = _image_grads(case, seed, s["hit"].shape[0])
    else:
        rad = _cached_radii(case, seed, rho)
        s["r"] = Renderer(leaf_size=case["leaf"])
        s["views"] = [View(m, w, h, float(fov)) for m, w, h, fov in _views(case, seed, boxes)]
        s["xyz"], s["rgb"], s["rad"] = xyz.requires_grad_(), rgb, rad.requires_grad_()
        s["col"] = (rgb.float() / 255.0).requires_grad_()
        pixels = sum(v.pixels for v in s["views"])
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 307)
        s["t_rgb"] = torch.rand((pixels, 3), generator=g, device="cuda")
        s["t_depth"] = 6.0 * torch.rand(pixels, generator=g, device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    case, r = s["case"], s["r"]
    kind = case["kind"]
    if kind == "knn":
        return r.knn(s["q"], case["k"])
    if kind == "precompute":
        r.set_cloud(s["xyz"], s["rgb"])
        r.build_index()
        return r.compute_radii(case["max_radius"], device=not case["host"])
    if kind == "render":
        return r.render(s["views"][0], device=not case["host"])
    if kind == "batch":
        r.render_batch_into(s["views"], s["frames"], device=True, cviews=s["cviews"])
        r.synchronize()
        return s["rgbd"], s["hit"]
    n = case["n"]
    if kind == "backward":
        g_rgb = torch.zeros((n, 3), device="cuda")
        g_xyz = torch.zeros((n, 3), device="cuda")
        g_rad = torch.zeros(n, device="cuda")
        torch.cuda.current_stream().synchronize()  # the renderer works on its own stream
        r.backward(s["views"], s["drgb"], s["ddep"], s["hit"], g_rgb, g_xyz, g_rad)
        return g_rgb, g_xyz, g_rad
    # train: the points moved in the last step, so the cloud is indexed anew
    r.set_cloud(s["xyz"].detach(), s["rgb"])
    r.build_index()
    r.set_radii(s["rad"].detach(), case["max_radius"])
    for p in (s["col"], s["xyz"], s["rad"]):
        p.grad = None
    rgb, depth, hit = RenderFunction.apply(r, s["views"], s["col"], s["xyz"], s["rad"])
    loss = ((rgb - s["t_rgb"]) ** 2).sum() + (depth - s["t_depth"]).abs().sum()
    loss.backward()
    return rgb.detach(), depth.detach(), hit, s["col"].grad, s["xyz"].grad, s["rad"].grad


def _pixels(case):
    sizes = _sizes(case.get("sizes") or case["size"])
    return sum(w * h for w, h in (sizes[i % len(sizes)] for i in range(case.get("views", 1))))


# A ray takes about 13 distance steps; each needs the 10 nearest points'
# records (9 flops for a distance, 2 for the step value).
STEPS = 13


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "knn":
        m, k = case["queries"], case["k"]
        # the queries, the answers, and the records that are answers (at most the cloud)
        return {"bytes": 12 * m + 8 * m * k + 16 * min(n, m * k), "flops": 8 * m * k}
    cloud = 15 * n  # xyz and rgb
    if kind == "precompute":
        return {"bytes": cloud + 8 * n, "flops": 9 * n}
    px = _pixels(case)
    march = {"bytes": 24 * px + 16 * min(n, px), "flops": STEPS * 10 * 11 * px}
    if kind in ("render", "batch"):
        return march
    # loss gradients and hit in, the hit points' records, the gradients of the whole cloud out
    back = {"bytes": 20 * px + 16 * min(n, px) + 28 * n, "flops": 60 * px}
    if kind == "backward":
        return back
    return {"bytes": cloud + 4 * n + march["bytes"] + back["bytes"], "flops": march["flops"] + back["flops"]}


# ------------------------------------------------------------- 64-bit values
def _nearest(q, xyz, k):
    """Squared distances to the k nearest points and their indices, in 64 bits, by brute force."""
    p = xyz.double()
    ds, js = [], []
    rows = max(1, (1 << 27) // p.shape[0])
    for lo in range(0, q.shape[0], rows):
        c = q[lo:lo + rows].double()
        d2 = (c[:, None, 0] - p[None, :, 0]) ** 2
        d2 += (c[:, None, 1] - p[None, :, 1]) ** 2
        d2 += (c[:, None, 2] - p[None, :, 2]) ** 2
        v, j = torch.topk(d2, min(k, p.shape[0]), dim=1, largest=False)
        ds.append(v)
        js.append(j)
    return torch.cat(ds), torch.cat(js)


def _exact_render(case, seed, xyz, rgb, boxes):
    """The march in 64 bits: steps of min(distance - radius) over the 10 nearest points."""
    d2, _ = _nearest(xyz, xyz, 2)
    rad = d2[:, 1].sqrt().clamp(max=float(np.float32(case["max_radius"])))
    view = _views(case, seed, boxes)[0]
    o, d = _rays(view)
    m = torch.tensor(view[0], dtype=torch.float64, device="cuda").reshape(4, 4).t()
    cos = -(d @ m[:3, 2])
    t, far = 0.1 / cos, 100.0 / cos
    depth = torch.zeros_like(t)
    col = torch.zeros((t.shape[0], 3), dtype=torch.float64, device="cuda")
    live = torch.arange(t.shape[0], device="cuda")
    for _ in range(128):
        if live.numel() == 0:
            break
        q2, j = _nearest(o + t[live, None] * d[live], xyz, 10)
        step, at = (q2.sqrt() - rad[j]).min(dim=1)
        t[live] += step
        hit = step < 0.001
        depth[live[hit]] = t[live[hit]]
        col[live[hit]] = rgb[j[hit, at[hit]]].double() / 255.0
        live = live[~hit & ~(t[live] > far[live])]
    shape = (view[2], view[1])
    return {"rgbd": torch.cat([col, depth[:, None]], 1).reshape(*shape, 4), "hit": None,
            "depth": depth.reshape(shape)}


def _exact_backward(case, seed, xyz, rho, boxes):
    rad = _cached_radii(case, seed, rho)
    views = _views(case, seed, boxes)
    hits = [_splat(v, xyz, rad).long() for v in views]
    drgb, ddep = _image_grads(case, seed, sum(h.shape[0] for h in hits))
    g_rgb = torch.zeros((case["n"], 3), dtype=torch.float64, device="cuda")
    g_xyz, g_rad = torch.zeros_like(g_rgb), torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    lo = 0
    for v, hit in zip(views, hits):
        o, d = _rays(v)
        on = hit >= 0
        h, d = hit[on], d[on]
        lc, ld = drgb[lo:lo + hit.shape[0]][on].double(), ddep[lo:lo + hit.shape[0]][on].double()
        lo += hit.shape[0]
        oc, r = xyz[h].double() - o, rad[h].double()
        b = (d * oc).sum(1)
        off = oc - b[:, None] * d                   # from the ray's closest point to the centre
        disc = r * r - (off * off).sum(1)
        s = torch.where(disc > 0, 1.0 / disc.clamp(min=1e-300).sqrt(), torch.zeros_like(disc))
        g_rgb.index_add_(0, h, lc)
        g_xyz.index_add_(0, h, ld[:, None] * (d + off * s[:, None]))
        g_rad.index_add_(0, h, -ld * r * s)
    return g_rgb, g_xyz, g_rad


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "knn" and case["queries"] * n <= 2e10:
        xyz = _scene(case, seed)[0]
        return None, _nearest(_queries(case, seed, xyz), xyz, case["k"])[0]
    if kind == "precompute" and n <= 150_000:
        xyz = _scene(case, seed)[0]
        out = _nearest(xyz, xyz, 2)[0][:, 1].sqrt()
        return (out.cpu().numpy() if case["host"] else out), None
    if kind == "render" and n * _pixels(case) <= 3e9:
        xyz, rgb, boxes, _ = _scene(case, seed)
        out = _exact_render(case, seed, xyz, rgb, boxes)
        return {k: (v.cpu().numpy() if case["host"] and v is not None else v) for k, v in out.items()}
    if kind == "backward":
        xyz, _, boxes, rho = _scene(case, seed)
        return _exact_backward(case, seed, xyz, rho, boxes)
    return None
