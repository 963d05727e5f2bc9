"""The renderer's stream is not torch's: calls wait for what torch still has
queued on their inputs, and on the freed blocks that their outputs get."""
import numpy as np
import pytest
import torch

from renderer_ray_marching_gb300 import Renderer, synthetic as syn, views_from_specs
from renderer_ray_marching_gb300.autograd import RenderFunction

pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # clock cycles of a spinning kernel, about 50 ms


@pytest.fixture(scope="module")
def scene():
    sc = syn.make_scene(30_000, n_boxes=4, seed=2)
    views = views_from_specs(syn.make_views(2, seed=5, boxes=sc.boxes, resolutions=[(200, 150)]))
    return torch.from_numpy(sc.xyz).cuda(), torch.from_numpy(sc.rgb).cuda(), views


def _ready(scene):
    xyz, rgb, views = scene
    torch.cuda.synchronize()
    r = Renderer()
    r.set_cloud(xyz, rgb)
    r.build_index()
    radii, nn = r.compute_radii(0.1, device=True)
    torch.cuda.synchronize()
    return r, radii, nn


def _late(t):
    """A copy of `t` that is written after a long-running kernel."""
    out = torch.zeros_like(t)
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    out.copy_(t)
    return out


def _stale(*shapes_dtypes):
    """Frees blocks of these sizes that a queued kernel will still write."""
    blocks = [torch.empty(s, dtype=d, device="cuda") for s, d in shapes_dtypes]
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY)
    for b in blocks:
        b.fill_(77)


def test_inputs_still_being_written(scene):
    xyz, rgb, views = scene
    r, radii, nn = _ready(scene)
    q = (xyz[:500] + 0.01).contiguous()
    want = r.knn(q, 4)
    frame = r.render(views[0], device=True)
    torch.cuda.synchronize()
    s = Renderer()
    s.set_cloud(_late(xyz), _late(rgb))
    s.build_index()
    s.set_radii(_late(radii), 0.1)
    got = s.knn(_late(q), 4)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    other = s.render(views[0], device=True)
    for f in ("rgbd", "hit", "depth"):
        assert torch.equal(frame[f], other[f])


def test_outputs_in_blocks_with_queued_work(scene):
    xyz, rgb, views = scene
    r, radii, nn = _ready(scene)
    n, m, px = xyz.shape[0], 3000, views[0].pixels
    q = (xyz[:m] + 0.01).contiguous()
    want = r.knn(q, 4)
    frame = r.render(views[0], outputs=("rgbd", "hit"), device=True)
    batch = r.render_batch(views, outputs=("rgbd", "hit"))
    torch.cuda.synchronize()
    _stale(((n,), torch.float32), ((n,), torch.int32))
    got = r.compute_radii(0.1, device=True)
    torch.cuda.synchronize()
    assert torch.equal(got[0], radii) and torch.equal(got[1], nn)
    _stale(((m, 4), torch.int32), ((m, 4), torch.float32))
    got = r.knn(q, 4)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    _stale(((px, 4), torch.float32), ((px,), torch.int32))
    got = r.render(views[0], outputs=("rgbd", "hit"), device=True)
    torch.cuda.synchronize()
    assert torch.equal(got["rgbd"], frame["rgbd"]) and torch.equal(got["hit"], frame["hit"])
    _stale(*[s for v in views for s in (((v.pixels, 4), torch.float32), ((v.pixels,), torch.int32))])
    got = r.render_batch(views, outputs=("rgbd", "hit"))
    torch.cuda.synchronize()
    for g, b in zip(got, batch):
        assert torch.equal(g["rgbd"], b["rgbd"]) and torch.equal(g["hit"], b["hit"])


def test_render_function(scene):
    xyz, rgb, views = scene
    r, radii, nn = _ready(scene)
    px = sum(v.pixels for v in views)
    args = [t.clone().requires_grad_() for t in (rgb.float() / 255.0, xyz, radii.clamp(max=0.1))]
    want = [t.detach().clone() for t in RenderFunction.apply(r, views, *args)]
    torch.cuda.synchronize()
    _stale(((px, 4), torch.float32), ((px,), torch.int32))
    got = RenderFunction.apply(r, views, *args)
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def test_context_on_torchs_stream(scene):
    """Such a context is ordered by the stream itself."""
    xyz, rgb, views = scene
    _, radii, nn = _ready(scene)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        s = Renderer(stream=st.cuda_stream)
        s.set_cloud(_late(xyz), _late(rgb))
        s.build_index()
        got = s.compute_radii(0.1, device=True)
        st.synchronize()
        assert torch.equal(got[0], radii) and torch.equal(got[1], nn)
        s.close()
