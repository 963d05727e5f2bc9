"""Clouds with a few points far from the rest: results, and that the searches
near the rest cost no more for them."""
import time

import numpy as np
import pytest
import torch

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


def _cloud(kind, n, seed=21):
    xyz = syn.make_scene(n, n_boxes=6, seed=seed).xyz
    rng = np.random.default_rng(seed)
    if kind == "above":
        xyz[n // 2] = [1.0, 1.0, 20000.0]
    elif kind == "around":
        far = rng.normal(size=(max(1, n // 300), 3))
        xyz[rng.permutation(n)[: len(far)]] = 5e4 * far / np.linalg.norm(far, axis=1)[:, None]
    elif kind == "float range":
        xyz[0], xyz[n - 1] = [3e38, 0, 0], [-3e38, -1e30, 2e20]
    elif kind == "noise":
        k = rng.permutation(n)[: max(1, n // 100)]
        xyz[k, 2] += rng.uniform(-3000.0, 3000.0, len(k)).astype(np.float32)
    elif kind == "one place":  # nearly everything there, the rest a room
        xyz[rng.permutation(n)[: n - n // 80]] = [4.0, 3.0, 1.0]
    return xyz


@pytest.mark.parametrize("kind", ["above", "around", "float range", "noise", "one place"])
@pytest.mark.parametrize("n", [33, 1025, 30_011])
def test_radii_knn_and_rays(kind, n):
    if kind == "one place":
        n = min(n, 4001)  # coincident points are all neighbours of each other
    xyz = _cloud(kind, n)
    rng = np.random.default_rng(n)
    q = np.concatenate([xyz[rng.integers(0, n, 60)], rng.uniform(0.0, 8.0, (60, 3)).astype(np.float32)])
    ix = oracle.Index(xyz)
    orad, onn = ix.radii(0.0)
    onn = np.where(np.isinf(orad), -1, onn)  # a distance beyond float32: no neighbour
    for leaf in (8, 16, 32):
        r = Renderer(leaf_size=leaf)
        r.set_cloud(xyz)
        r.build_index()
        rad, nn = r.compute_radii(0.1)
        assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
        assert np.array_equal(nn, onn)
        for k in (1, 10, 32):
            i, d = r.knn(q, k)
            oi, od = ix.knn(q, k)
            oi = np.where(np.isinf(od), -1, oi)
            assert np.array_equal(i, oi) and np.array_equal(d.view(np.int32), od.view(np.int32))
        view = views_from_specs(syn.make_views(1, seed=3, resolutions=[(64, 48)]))[0]
        packets = r.render(view, outputs=("hit", "depth", "steps"))
        r.set_launch(search=0, ctas_per_sm=4)
        alone = r.render(view, outputs=("hit", "depth", "steps"))
        for f in packets:
            assert np.array_equal(packets[f].view(np.int32), alone[f].view(np.int32)), f
        r.close()


@pytest.mark.parametrize("kind", ["above", "around", "noise"])
def test_time_does_not_grow_with_distant_points(kind):
    """1.0 to 1.1 times the time of a cloud without any (700 times for one
    point 20 km above, 40 times for the noise, when the curve's cells spanned
    the bounds); 4 is allowed."""
    took = []
    for k in (None, kind):
        r = Renderer()
        r.set_cloud(torch.from_numpy(_cloud(k, 1_000_000)).cuda())
        r.build_index()
        best = 1e9
        for _ in range(8):
            torch.cuda.synchronize()
            t = time.perf_counter()
            r.compute_radii(0.1, device=True)
            best = min(best, time.perf_counter() - t)
        took.append(best)
        r.close()
    assert took[1] < 4.0 * took[0]
