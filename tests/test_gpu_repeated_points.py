"""Radii of clouds in which many points repeat others, exactly or to the last
bits (merged scans): the remaining points are no strays because of it."""
import time

import numpy as np
import pytest
import torch

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn

pytestmark = pytest.mark.gpu


def _cloud(n, share, jitter, seed):
    xyz = syn.make_scene(n, n_boxes=12, seed=seed).xyz
    rng = np.random.default_rng(seed)
    m = int(n * share) // 2
    if m:
        xyz[n - m:] = xyz[:m] + (rng.random((m, 3)) - 0.5).astype(np.float32) * np.float32(jitter)
    return xyz[rng.permutation(n)]


@pytest.mark.parametrize("jitter", [0.0, 1e-6])
@pytest.mark.parametrize("share", [0.5, 0.6, 0.9, 1.0])
def test_radii(share, jitter):
    xyz = _cloud(50_001, share, jitter, 11)
    orad, onn = oracle.Index(xyz).radii(0.0)
    for leaf in (8, 16, 32):
        r = Renderer(leaf_size=leaf)
        r.set_cloud(xyz)
        r.build_index()
        rad, nn = r.compute_radii(0.1)
        assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
        assert np.array_equal(nn, onn)
        r.close()


def test_time_does_not_grow_with_repeated_points():
    """1.1 times the time of a cloud without any (5 times when every other
    point beside repeated ones was searched for alone); 2.5 is allowed."""
    took = []
    for share in (0.0, 0.6):
        r = Renderer()
        r.set_cloud(torch.from_numpy(_cloud(2_000_000, share, 0.0, 12)).cuda())
        r.build_index()
        best = 1e9
        for _ in range(12):
            torch.cuda.synchronize()
            t = time.perf_counter()
            r.compute_radii(0.1, device=True)
            best = min(best, time.perf_counter() - t)
        took.append(best)
        r.close()
    assert took[1] < 2.5 * took[0]
