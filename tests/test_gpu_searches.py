"""The index's searches against the oracle at the sizes where they change
form: blocks of 1024 points and their tails, chunks of 32 queries, one and
two chunks per warp, exact ties and coincident points, and clouds whose
sorted neighbours say little about the nearest ones (strays over a dense
surface, clusters far apart), for every leaf size."""
import numpy as np
import pytest

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    rng = np.random.default_rng(n)
    if kind == "room":
        return syn.make_scene(n, n_boxes=3, seed=n).xyz
    if kind == "grid":  # nearly every distance is shared
        return (rng.integers(0, 24, (n, 3)) * 0.125).astype(np.float32)
    if kind == "twins":  # half of the points coincide with others
        xyz = rng.random((n, 3)).astype(np.float32)
        xyz[rng.integers(0, n, n // 2)] = xyz[rng.integers(0, n, n // 2)]
        return xyz
    if kind == "zeros":  # a third of the points at one place, as missing returns are stored
        xyz = syn.make_scene(n, n_boxes=3, seed=n).xyz
        xyz[rng.permutation(n)[: n // 3]] = 0.0
        return xyz
    if kind == "strays":  # a dense slab and a thin layer of points above it
        xyz = rng.random((n, 3)) * [4.0, 4.0, 0.004]
        xyz[: n // 50, 2] += 0.01
        return xyz.astype(np.float32)
    centres = rng.uniform(-500.0, 500.0, (max(1, n // 20), 3))  # clusters
    return (centres[rng.integers(0, len(centres), n)] + rng.normal(0.0, 0.01, (n, 3))).astype(np.float32)


@pytest.mark.parametrize("kind", ["room", "grid", "twins", "zeros", "strays", "clusters"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 129, 1023, 1025, 4099, 70001])
def test_radii_and_knn(kind, n):
    xyz = _cloud(kind, n)
    rng = np.random.default_rng(n + 1)
    q = np.concatenate([xyz[rng.integers(0, n, 40)], rng.uniform(-2.0, 9.0, (40, 3)).astype(np.float32)])
    ix = oracle.Index(xyz)
    orad, onn = ix.radii(0.0)
    for leaf in (8, 16, 32):
        r = Renderer(leaf_size=leaf)
        r.set_cloud(xyz)
        r.build_index()
        rad, nn = r.compute_radii(0.1)
        assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
        assert np.array_equal(nn, onn)
        for k in (1, 2, 10, 17, 32):
            i, d = r.knn(q, k)
            oi, od = ix.knn(q, k)
            assert np.array_equal(i, oi)
            assert np.array_equal(d.view(np.int32), od.view(np.int32))
        r.close()


@pytest.mark.parametrize("kind", ["room", "strays", "twins"])
@pytest.mark.parametrize("n", [(12 << 20) - 1, (12 << 20) + 4097])
def test_radii_on_both_sides_of_the_size_switches(kind, n):
    """Regions of one and two chunks; results to cloud order directly and
    through buckets."""
    xyz = _cloud(kind, n)
    orad, onn = oracle.Index(xyz).radii(0.0)
    r = Renderer()
    r.set_cloud(xyz)
    r.build_index()
    rad, nn = r.compute_radii(0.1)
    assert np.array_equal(rad.view(np.int32), orad.view(np.int32))
    assert np.array_equal(nn, onn)
    r.close()


@pytest.mark.parametrize("n,size", [(7, (40, 24)), (3000, (8, 4)), (3000, (161, 119)), (60_000, (900, 610)),
                                    (20_000, (3600, 2400))])
def test_rays_that_leave_their_packets(n, size):
    """Packets hand rays to the tail kernel after a budget that grows with the
    launch (the largest view also overruns the list of such rays); the march
    of every ray alone (search 0) gives the same images."""
    sc = syn.make_scene(n, n_boxes=6, seed=n)
    views = views_from_specs(syn.make_views(2, seed=4, boxes=sc.boxes, resolutions=[size]))
    r = Renderer()
    r.set_cloud(sc.xyz, sc.rgb)
    r.build_index()
    r.compute_radii(0.3)
    fields = ("rgbd", "hit", "depth", "steps")
    plain = [r.render(v, outputs=fields) for v in views]
    if n >= 3000 and size != (8, 4):
        assert r.stats()["solo_steps"] > 0 and r.stats()["packet_steps"] > 0
    batch = r.render_batch(views, outputs=fields, device=False)
    r.set_launch(search=0, ctas_per_sm=4)
    for v, p, b in zip(views, plain, batch):
        alone = r.render(v, outputs=fields)
        for f in fields:
            assert np.array_equal(alone[f].view(np.int32), p[f].view(np.int32)), f
            assert np.array_equal(alone[f].view(np.int32), b[f].view(np.int32)), f
    r.close()
