"""Searches over clouds whose distances agree to a few ulps: lattices with
spacings that are no binary fractions, shifted off the origin, so that boxes
and points at nominally one distance differ in their last bits and the bound
of a search lies among them.  Queries at the points and at cell centres
against the oracle; lattices with strays, whose radii are searched one by
one; and rays between the lattice's points, in packets and alone."""
import numpy as np
import pytest

import oracle
from renderer_ray_marching_gb300 import Renderer, View, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


def _lattice(spacing, offset, m, seed):
    g = np.stack(np.meshgrid(*[np.arange(m, dtype=np.float32)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xyz = g * np.float32(spacing) + np.array(offset, np.float32)
    return xyz[np.random.default_rng(seed).permutation(len(xyz))]


SPACINGS = [(0.05, (0, 0, 0), 31), (0.1, (0, 0, 0), 36), (0.03, (1.7, -0.3, 0.9), 40), (0.07, (0, 0, 0), 36),
            (0.02, (-3.1, 2.2, 0.4), 46)]


@pytest.mark.parametrize("leaf", [8, 16, 32])
@pytest.mark.parametrize("spacing,offset,m", SPACINGS)
def test_knn_on_lattices(spacing, offset, m, leaf):
    xyz = _lattice(spacing, offset, m, m)
    centres = xyz[:6000] + np.float32(0.5 * spacing)
    q = np.concatenate([xyz[:24000], centres])
    ix = oracle.Index(xyz)
    r = Renderer(leaf_size=leaf)
    r.set_cloud(xyz)
    r.build_index()
    for k in (1, 2, 3, 4, 7, 10, 17, 32):
        i, d = r.knn(q, k)
        oi, od = ix.knn(q, k)
        assert np.array_equal(d.view(np.int32), od.view(np.int32)), k
        assert np.array_equal(i, oi), k
    r.close()


@pytest.mark.parametrize("leaf", [8, 16, 32])
@pytest.mark.parametrize("spacing,offset,m", SPACINGS)
def test_radii_of_lattices_with_strays(spacing, offset, m, leaf):
    """A stray is many spacings from everything: more than a region's search
    is meant for, so it gets one of its own."""
    xyz = _lattice(spacing, offset, m, m + 1)
    rng = np.random.default_rng(m)
    far = xyz[rng.integers(0, len(xyz), 3000)].copy()
    far[:, 2] = xyz[:, 2].max() + np.float32(spacing) * rng.integers(9, 30, 3000).astype(np.float32)
    xyz = np.concatenate([xyz, far])[rng.permutation(len(xyz) + 3000)]
    orad, onn = oracle.Index(xyz).radii(0.0)
    r = Renderer(leaf_size=leaf)
    r.set_cloud(xyz)
    r.build_index()
    rad, nn = r.compute_radii(0.1)
    assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
    assert np.array_equal(nn, onn)
    r.close()


@pytest.mark.parametrize("leaf", [8, 16, 32])
def test_radii_of_a_flat_cloud_under_a_distant_point(leaf):
    """One point 20 km above makes the curve's cells as wide as the cloud, so
    blocks overlap and nearly every point is searched for alone."""
    xyz = syn.make_scene(60_000, n_boxes=6, seed=8).xyz
    xyz[17] = [1.0, 1.0, 20000.0]
    orad, onn = oracle.Index(xyz).radii(0.0)
    r = Renderer(leaf_size=leaf)
    r.set_cloud(xyz)
    r.build_index()
    rad, nn = r.compute_radii(0.1)
    assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
    assert np.array_equal(nn, onn)
    r.close()


@pytest.mark.parametrize("spacing,offset,m", [(0.1, (1.0, 0.5, 0.1), 36), (0.07, (3.0, 2.0, 0.2), 40)])
def test_rays_between_the_points_of_a_lattice(spacing, offset, m):
    xyz = _lattice(spacing, offset, m, m + 2)
    views = views_from_specs(syn.make_views(3, seed=9, resolutions=[(96, 72)]))
    views.append(View(np.array([1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 3.3, 2.9, 4.7, 1], np.float32), 96, 72, 1.0))
    r = Renderer()
    r.set_cloud(xyz)
    r.build_index()
    r.set_radii(np.full(len(xyz), 0.3 * spacing, np.float32), 0.0)
    fields = ("hit", "depth", "steps")
    packets = [r.render(v, outputs=fields) for v in views]
    assert r.stats()["solo_steps"] > 0
    r.set_launch(search=0, ctas_per_sm=4)
    for v, p in zip(views, packets):
        alone = r.render(v, outputs=fields)
        for f in fields:
            assert np.array_equal(alone[f].view(np.int32), p[f].view(np.int32)), f
    r.close()
