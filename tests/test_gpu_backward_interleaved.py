"""Gradient sums where neighbouring pixels hit few points in turn."""
import time

import numpy as np
import pytest
import torch

from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


def _hits(kind, p, n):
    at = torch.arange(p, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    if kind.startswith("two by "):
        return (at // int(kind.split()[-1]) % 2).int()
    if kind.startswith("random "):
        return torch.randint(0, int(kind.split()[-1]), (p,), device="cuda", dtype=torch.int32, generator=g)
    if kind == "gaps":  # misses between the points
        return torch.where(at % 3 == 1, -1, at % 7 // 3).int()
    return (at // 5 * 7919 % n).int()  # runs of five, no point twice in a warp


@pytest.fixture(scope="module")
def scene():
    sc = syn.make_scene(20_000, n_boxes=4, seed=2)
    views = views_from_specs(syn.make_views(2, seed=5, boxes=sc.boxes, resolutions=[(333, 201)]))
    r = Renderer()
    r.set_cloud(sc.xyz, sc.rgb)
    r.build_index()
    r.compute_radii(0.1)
    return r, views, len(sc.xyz)


def _grads(n):
    return [torch.zeros((n, 3), device="cuda"), torch.zeros((n, 3), device="cuda"), torch.zeros(n, device="cuda")]


@pytest.mark.parametrize("kind", ["two by 1", "two by 2", "two by 3", "two by 4", "random 2", "random 10", "random 40",
                                  "gaps", "runs"])
def test_sums(scene, kind):
    r, views, n = scene
    p = sum(v.pixels for v in views)
    g = torch.Generator(device="cuda").manual_seed(9)
    hit = _hits(kind, p, n)
    # whole numbers, so that colour sums are exact in any order (below 2^24)
    drgb = torch.randint(-8, 9, (p, 3), device="cuda", generator=g).float()
    ddep = 0.5 + torch.rand(p, device="cuda", generator=g)
    out = _grads(n)
    r.backward(views, drgb, ddep, hit, *out)
    on = hit >= 0
    want = torch.zeros((n, 3), dtype=torch.float64, device="cuda").index_add_(0, hit[on].long(), drgb[on].double())
    assert torch.equal(out[0].double(), want)
    # Depth gradients: against the same pixels in 37 calls of every 37th, added in 64 bits.  A float32 sum of m
    # terms is off by no more than m 2^-24 of the sum of their magnitudes; radius gradients of positive dL/ddepth
    # have one sign, and a pixel's position gradient is no larger than dL/ddepth and its radius gradient together.
    xyz = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    rad = torch.zeros(n, dtype=torch.float64, device="cuda")
    at = torch.arange(p, device="cuda")
    for k in range(37):
        part = _grads(n)
        r.backward(views, drgb, ddep, torch.where(at % 37 == k, hit, -1), *part)
        xyz += part[1].double()
        rad += part[2].double()
    h = hit[on].long()
    m = torch.bincount(h, minlength=n).double()
    size = rad.abs() + torch.zeros_like(rad).index_add_(0, h, ddep[on].double())
    assert ((out[2].double() - rad).abs() <= 2 * m * 2.0 ** -24 * rad.abs()).all()
    assert ((out[1].double() - xyz).abs() <= (2.001 * m * 2.0 ** -24 * size)[:, None]).all()


def test_interleaved_hits_cost_no_more_atomics(scene):
    """Two points pixel by pixel take the time of one point (14 times that when
    every run had its own atomics); 4 times is allowed."""
    r, views, n = scene
    big = views_from_specs(syn.make_views(4, seed=5, resolutions=[(1067, 690)]))
    p = sum(v.pixels for v in big)
    drgb, ddep = torch.ones((p, 3), device="cuda"), torch.ones(p, device="cuda")
    out = _grads(n)
    took = []
    for hit in (torch.zeros(p, dtype=torch.int32, device="cuda"), _hits("two by 1", p, n)):
        best = 1e9
        for _ in range(10):
            torch.cuda.synchronize()
            t = time.perf_counter()
            r.backward(big, drgb, ddep, hit, *out)
            best = min(best, time.perf_counter() - t)
        took.append(best)
    assert took[1] < 4.0 * took[0]
