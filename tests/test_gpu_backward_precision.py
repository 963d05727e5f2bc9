"""The backward kernel's two-float arithmetic against quadruple (or x87)
precision, one pixel per point so that no sum hides an error: rays that pass
their sphere's centre at fractions of the radius up to the silhouette and
outside it, for near and far, small and large spheres, and a size that falls
back to FP64."""
import numpy as np
import pytest

import oracle
from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,radius", [(0.3, 1e-3), (3.0, 1e-3), (3.0, 2e-2), (60.0, 0.1), (1500.0, 5.0),
                                          (4e6, 2e4)])
def test_entry_gradient(scale, radius):
    view = views_from_specs(syn.make_views(1, seed=6, resolutions=[(64, 48)]))[0]
    n = view.pixels
    r = Renderer()
    pane = r.view_pane([view])[0]
    ov = oracle.make_view(view.cam2world, view.width, view.height, float(pane))
    rays = [oracle.ray(ov, p % view.width, p // view.width)[:2] for p in range(n)]
    o = np.array([a[0] for a in rays], np.float64)
    d = np.array([a[1] for a in rays], np.float64)
    rng = np.random.default_rng(1)
    side = np.cross(d, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1)[:, None]
    off = radius * np.resize([0.0, 0.3, 0.9, 0.99, 0.9999, 1.01, 3.0], n)
    xyz = (o + scale * rng.uniform(0.5, 1.0, (n, 1)) * d + off[:, None] * side).astype(np.float32)
    rad = (radius * rng.uniform(0.7, 1.0, n) / 0.7).astype(np.float32)
    ld = rng.normal(size=n).astype(np.float32)
    r.set_cloud(xyz)
    r.build_index()
    r.set_radii(rad, 0.0)
    g = [np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32), np.zeros(n, np.float32)]
    r.backward([view], np.zeros((n, 3), np.float32), ld, np.arange(n, dtype=np.int32), *g)
    r.close()
    L = np.longdouble
    o, d, c, rr, ldl = o.astype(L), d.astype(L), xyz.astype(L), rad.astype(L), ld.astype(L)
    oc = c - o
    q = np.cross(d, oc)
    aa = (d * d).sum(1)
    disc = aa * rr * rr - (q * q).sum(1)
    inside = disc > 0
    s = np.where(inside, 1 / np.sqrt(np.where(inside, disc, 1)), 0)
    gx = ldl[:, None] * (d - np.cross(d, q) * s[:, None]) / aa[:, None]
    gr = -ldl * rr * s
    # The result is rounded to float32 (and its last products before that):
    # 2^-22 of it.  q carries 2^-45 |oc| (2^-50 of b^2 in the FP64 fallback's
    # disc), which the root amplifies by |q| / disc; pixels whose sign of disc
    # that could change are left out.
    size = np.sqrt((oc * oc).sum(1))
    noise = 2 * np.sqrt((q * q).sum(1)) * size * L(2) ** -45 + (size ** 2 * L(2) ** -50 if scale > 1e6 else 0)
    ok = np.abs(disc) > 16 * noise
    assert ok.mean() > 0.8 and (inside & ok).any() and (~inside & ok).any()
    amp = np.where(inside, noise / np.abs(disc), 0)
    mag = np.abs(ldl) * (1 + np.sqrt((np.cross(d, q) ** 2).sum(1)) * s)
    tol = mag * (L(2) ** -22 + amp)
    assert (np.abs(g[1] - gx)[ok] <= tol[ok, None]).all()
    assert (np.abs(g[2] - gr)[ok] <= (np.abs(gr) * (L(2) ** -22 + amp))[ok]).all()
