"""k-NN of many queries with k of 1 and 2: queries in spatial order and in none,
on grids, with places that are not finite, over small and larger clouds, near
and exact ties among them, against the oracle."""
import time

import numpy as np
import pytest
import torch

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn

pytestmark = pytest.mark.gpu

MANY = 262_144  # from here on, with 4 queries for each point or more


def _spatial(x):
    """Points in Morton order."""
    c = ((x - x.min(0)) / 0.01).astype(np.int64)
    key = np.zeros(len(x), np.int64)
    for b in range(11):
        for a in range(3):
            key |= ((c[:, a] >> b) & 1) << (3 * b + a)
    return np.ascontiguousarray(x[np.argsort(key, kind="stable")])


def _points(kind, n):
    rng = np.random.default_rng(n)
    if kind == "lattice":
        g = np.stack(np.meshgrid(*[np.arange(32, dtype=np.float32)] * 3, indexing="ij"), -1).reshape(-1, 3)
        return (g * np.float32(0.07))[rng.permutation(len(g))[:n]]
    xyz = syn.make_scene(max(n, 64), n_boxes=4, seed=n).xyz[:n].copy()
    if kind == "twins":
        xyz[: n // 2] = xyz[n - n // 2:]
    return xyz


def _check(r, ix, q, k, stride=3):
    full = np.full((len(q), stride), 7.0, np.float32)
    full[:, :3] = q
    i, d = r.knn(torch.from_numpy(full).cuda(), k)
    i, d = i.cpu().numpy(), d.cpu().numpy()
    bad = ~np.isfinite(q).all(1)
    oi, od = ix.knn(np.where(bad[:, None], np.float32(0), q), k)
    oi[bad], od[bad] = -1, np.inf
    assert np.array_equal(d.view(np.int32), od.view(np.int32))
    assert np.array_equal(i, oi)


@pytest.mark.parametrize("kind,n", [("room", 50_000), ("room", 6_000), ("lattice", 20_000), ("twins", 20_000)])
def test_many_queries_per_point(kind, n):
    xyz = _points(kind, n)
    ix = oracle.Index(xyz)
    rng = np.random.default_rng(5)
    m = MANY + 13
    near = xyz[rng.integers(0, n, m)] + rng.normal(0.0, 0.01, (m, 3)).astype(np.float32)
    grid = np.stack(np.meshgrid(*[np.linspace(lo, hi, 64) for lo, hi in ((0, 8), (0, 6), (0, 3))], indexing="ij"),
                    -1).reshape(-1, 3).astype(np.float32)
    exact = np.repeat(xyz, m // n + 1, axis=0)[:m]  # every point several times in a row
    holes = _spatial(near)
    holes[rng.permutation(m)[:500], 1] = np.nan
    holes[rng.permutation(m)[:500], 0] = np.inf
    for leaf in (8, 16, 32):
        r = Renderer(leaf_size=leaf)
        r.set_cloud(xyz)
        r.build_index()
        for k in (1, 2):
            for q in (near, _spatial(near), grid, exact, holes):
                _check(r, ix, q, k)
        _check(r, ix, _spatial(near), 2, stride=5)
        r.close()


@pytest.mark.parametrize("n", [1, 2, 3, 9, 33, 130, 1250, 5000])
def test_small_clouds(n):
    xyz = _points("room", n)
    ix = oracle.Index(xyz)
    rng = np.random.default_rng(n)
    q = rng.uniform(-1.0, 9.0, (65_536 + 5, 3)).astype(np.float32)
    q[77] = np.nan
    q[99, 2] = -np.inf
    for leaf in (8, 16, 32):
        r = Renderer(leaf_size=leaf)
        r.set_cloud(xyz)
        r.build_index()
        for k in (1, 2, 3):
            _check(r, ix, q, k)
            _check(r, ix, _spatial(np.nan_to_num(q, nan=1.0, neginf=0.0)), k)
        r.close()


def test_queries_in_spatial_order_are_the_faster_ones():
    """7 times as fast as in no order (equally fast when every query had a warp
    of its own); 1.5 times is asked for."""
    xyz = _points("room", 20_000)
    rng = np.random.default_rng(6)
    q = xyz[rng.integers(0, len(xyz), 1_000_000)] + np.float32(0.003)
    r = Renderer(leaf_size=8)
    r.set_cloud(xyz)
    r.build_index()
    took = []
    for a in (q, _spatial(q)):
        a = torch.from_numpy(a).cuda()
        best = 1e9
        for _ in range(10):
            torch.cuda.synchronize()
            t = time.perf_counter()
            r.knn(a, 1)
            best = min(best, time.perf_counter() - t)
        took.append(best)
    r.close()
    assert 1.5 * took[1] < took[0]
