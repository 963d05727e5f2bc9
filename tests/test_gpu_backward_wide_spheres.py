"""Depth gradients at the silhouettes of spheres as wide as their distance,
one pixel per point: no further from long-double values than FP64 arithmetic
is (2^-50 of b^2 in the discriminant), or than float32's own rounding."""
import numpy as np
import pytest

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,ratio", [(3.0, 0.7), (3.0, 0.1), (0.5, 3.0), (200.0, 0.02), (3.0, 0.006), (3.0, 0.001)])
def test_silhouettes(scale, ratio):
    view = views_from_specs(syn.make_views(1, seed=6, resolutions=[(320, 240)]))[0]
    n = view.pixels
    r = Renderer()
    pane = r.view_pane([view])[0]
    ov = oracle.make_view(view.cam2world, view.width, view.height, float(pane))
    rays = [oracle.ray(ov, p % view.width, p // view.width)[:2] for p in range(n)]
    o = np.array([a[0] for a in rays], np.float64)
    d = np.array([a[1] for a in rays], np.float64)
    rng = np.random.default_rng(7)
    side = np.cross(d, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1)[:, None]
    xyz = (o + scale * rng.uniform(0.5, 1.0, (n, 1)) * d + ratio * scale * side).astype(np.float32)
    L = np.longdouble
    o, d = o.astype(L), d.astype(L)
    oc = xyz.astype(L) - o
    q = np.cross(d, oc)
    aa = (d * d).sum(1)
    # the radius nearest to the ray's distance from the centre, and its neighbours
    rad = (np.sqrt((q * q).sum(1) / aa)).astype(np.float32)
    for _ in range(2):
        rad = np.where(rng.random(n) < 0.5, np.nextafter(rad, np.float32(np.inf)), rad)
    ld = rng.normal(size=n).astype(np.float32)
    r.set_cloud(xyz)
    r.build_index()
    r.set_radii(rad, 0.0)
    g = [np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32), np.zeros(n, np.float32)]
    r.backward([view], np.zeros((n, 3), np.float32), ld, np.arange(n, dtype=np.int32), *g)
    r.close()
    rr, ldl = rad.astype(L), ld.astype(L)
    disc = aa * rr * rr - (q * q).sum(1)
    inside = disc > 0
    s = np.where(inside, 1 / np.sqrt(np.where(inside, disc, 1)), 0)
    gx = ldl[:, None] * (d - np.cross(d, q) * s[:, None]) / aa[:, None]
    gr = -ldl * rr * s
    noise = (oc * oc).sum(1) * L(2) ** -50
    ok = np.abs(disc) > 16 * noise  # else FP64 does not know the sign either
    assert ok.mean() > 0.5 and (inside & ok).any()
    amp = np.where(inside, noise / np.abs(disc), 0)
    mag = np.abs(ldl) * (1 + np.sqrt((np.cross(d, q) ** 2).sum(1)) * s)
    tol = mag * (L(2) ** -22 + amp)
    assert (np.abs(g[1] - gx)[ok] <= tol[ok, None]).all()
    assert (np.abs(g[2] - gr)[ok] <= (np.abs(gr) * (L(2) ** -22 + amp))[ok]).all()
