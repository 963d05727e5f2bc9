"""Incoming depth gradients at the ends of float32 and beyond: infinities,
NaN, overflow and the smallest numbers give what 64-bit arithmetic gives,
rounded to float32."""
import numpy as np
import pytest

import oracle
from renderer_ray_marching_gb300 import Renderer, View, synthetic as syn, views_from_specs

pytestmark = pytest.mark.gpu

INF = np.float32(np.inf)


def _gradients(view, xyz, rad, ld):
    n = view.pixels
    r = Renderer()
    pane = r.view_pane([view])[0]
    r.set_cloud(xyz)
    r.build_index()
    r.set_radii(rad, 0.0)
    g = [np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32), np.zeros(n, np.float32)]
    r.backward([view], np.zeros((n, 3), np.float32), ld, np.arange(n, dtype=np.int32), *g)
    r.close()
    return pane, g


def _rays(view, pane):
    ov = oracle.make_view(view.cam2world, view.width, view.height, float(pane))
    rays = [oracle.ray(ov, p % view.width, p // view.width)[:2] for p in range(view.pixels)]
    return np.array([a[0] for a in rays], np.float64), np.array([a[1] for a in rays], np.float64)


def _exact(o, d, xyz, rad, ld):
    """In long double: gradient by centre and radius, disc, q, and what the root makes of an error of q."""
    L = np.longdouble
    o, d, c, rr, ld = o.astype(L), d.astype(L), xyz.astype(L), rad.astype(L), ld.astype(L)
    oc = c - o
    q = np.cross(d, oc)
    aa = (d * d).sum(1)
    disc = aa * rr * rr - (q * q).sum(1)
    s = np.where(disc > 0, 1 / np.sqrt(np.where(disc > 0, disc, 1)), 0)
    with np.errstate(invalid="ignore"):
        gx = ld[:, None] * ((d - np.cross(d, q) * s[:, None]) / aa[:, None])
        gr = ld * (-rr * s)
    return gx, gr, disc, q, oc, s


@pytest.mark.parametrize("ld", [INF, -INF, np.float32("nan"), 3e38, -1e30, 1e26, 1e24, 1e-24, 1e-26, -1e-37, 1e-44, 0.0])
def test_extreme_incoming_gradients(ld):
    view = views_from_specs(syn.make_views(1, seed=6, resolutions=[(32, 24)]))[0]
    n = view.pixels
    r = Renderer()
    pane = r.view_pane([view])[0]
    r.close()
    o, d = _rays(view, pane)
    rng = np.random.default_rng(2)
    side = np.cross(d, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1)[:, None]
    off = 0.02 * np.resize([0.1, 0.5, 0.9, 1.5], n)
    xyz = (o + rng.uniform(1.0, 4.0, (n, 1)) * d + off[:, None] * side).astype(np.float32)
    rad = np.full(n, 0.02, np.float32)
    lds = np.full(n, ld, np.float32)
    _, g = _gradients(view, xyz, rad, lds)
    gx, gr, disc, q, oc, s = _exact(o, d, xyz, rad, lds)
    with np.errstate(over="ignore", invalid="ignore"):
        for got, want in ((g[1], gx), (g[2], gr)):
            if not np.isfinite(ld):
                w = want.astype(np.float32)
                assert np.array_equal(np.isnan(got), np.isnan(w))
                assert np.array_equal(got[~np.isnan(w)], w[~np.isnan(w)])
                continue
            # rounding to float32 (2^-24 of it, or half of the smallest number) after sums of terms up to
            # `mag`, each good to 2^-40 here (q's 2^-45 |oc|, amplified by |q| / disc < 2^5); the
            # accumulation (atom.add.f32) replaces numbers below 2^-126 by zero, as PTX defines it
            mag = np.abs(lds.astype(np.longdouble)) * (1 + np.sqrt((q * q).sum(1)) * s)
            tol = np.abs(want) * np.longdouble(2) ** -23 + (mag if want.ndim == 1 else mag[:, None]) * \
                np.longdouble(2) ** -36 + np.longdouble(2) ** -149
            tiny = np.abs(want) < np.longdouble(2) ** -126 * (1 + np.longdouble(2) ** -20)
            tol = np.where(tiny, np.maximum(tol, np.abs(want)), tol)
            top = np.longdouble(np.finfo(np.float32).max)
            over = np.abs(want) > top * (1 + np.longdouble(2) ** -20)
            fits = np.abs(want) < top * (1 - np.longdouble(2) ** -20)
            assert np.array_equal(got[over], np.sign(want[over]).astype(np.float32) * INF)
            assert (np.abs(got[fits].astype(np.longdouble) - want[fits]) <= tol[fits]).all()


def test_rays_of_a_matrix_with_a_fourth_row():
    """Such rays are shorter than unit length, down to 1e-12 here."""
    m = np.array([1, 0, 0, 4e12, 0, 1, 0, 3e12, 0, 0, 1, 1e12, 0.5, 0.25, 4.0, 1], np.float32)
    view = View(m, 32, 24, 1.0)
    n = view.pixels
    r = Renderer()
    pane = r.view_pane([view])[0]
    r.close()
    o, d = _rays(view, pane)
    u = d / np.linalg.norm(d, axis=1)[:, None]
    rng = np.random.default_rng(3)
    side = np.cross(u, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1)[:, None]
    xyz = (o + rng.uniform(1.0, 4.0, (n, 1)) * u + 0.01 * side).astype(np.float32)
    rad = np.full(n, 0.02, np.float32)
    ld = rng.normal(size=n).astype(np.float32) * np.float32(1e-3)
    _, g = _gradients(view, xyz, rad, ld)
    gx, gr, disc, q, oc, s = _exact(o, d, xyz, rad, ld)
    mag = np.abs(ld) * (1 + np.sqrt((q * q).sum(1)) * s) / (d * d).sum(1) ** 0.5
    assert (np.abs(g[1] - gx) <= np.abs(gx) * 2.0 ** -22 + mag[:, None] * 2.0 ** -22).all()
    assert (np.abs(g[2] - gr) <= np.abs(gr) * 2.0 ** -22).all()
