"""RenderFunction's handling of its views and outputs, with a stand-in for the
renderer that fills host buffers."""
import ctypes

import numpy as np
import pytest
import torch

from renderer_ray_marching_gb300 import View
from renderer_ray_marching_gb300.autograd import RenderFunction


class FakeRenderer:
    def wait_for_torch(self):
        pass

    def synchronize(self):
        pass

    def render_batch_into(self, views, frames, device=True):
        for k, (v, f) in enumerate(zip(views, frames)):
            rgbd = np.arange(4 * v.pixels, dtype=np.float32) + 1000 * k
            hit = np.arange(v.pixels, dtype=np.int32) % 3
            ctypes.memmove(f.rgbd, rgbd.ctypes.data, rgbd.nbytes)
            ctypes.memmove(f.hit, hit.ctypes.data, hit.nbytes)

    def backward(self, views, dl_drgb, dl_ddepth, hit, g_rgb, g_xyz, g_radius):
        assert sum(v.pixels for v in views) == hit.shape[0]
        g_rgb.index_add_(0, hit.long(), dl_drgb)
        g_radius.index_add_(0, hit.long(), dl_ddepth)


def _views(*sizes):
    return [View(np.eye(4, dtype=np.float32).reshape(16), w, h, 1.0) for w, h in sizes]


def _apply(views):
    n = 3
    colours, xyz, radii = (torch.zeros(s, requires_grad=True) for s in ((n, 3), (n, 3), (n,)))
    return RenderFunction.apply(FakeRenderer(), views, colours, xyz, radii) + (colours, radii)


@pytest.mark.parametrize("sizes", [[(1, 1)], [(2, 1)], [(5, 3)], [(4, 2), (1, 1), (3, 3)]])
def test_outputs_are_tensors_of_their_own(sizes):
    rgb, depth, hit, colours, radii = _apply(_views(*sizes))
    want = np.concatenate([(np.arange(4 * w * h, dtype=np.float32) + 1000 * k).reshape(-1, 4)
                           for k, (w, h) in enumerate(sizes)])
    assert np.array_equal(rgb.detach().numpy(), want[:, :3])
    assert np.array_equal(depth.detach().numpy(), want[:, 3])
    assert rgb.is_contiguous() and depth.is_contiguous()
    assert rgb.untyped_storage().data_ptr() != depth.untyped_storage().data_ptr()
    rgb.mul_(2.0)  # in place, as on any output of a function
    depth.add_(1.0)
    (rgb.sum() + depth.sum()).backward()
    assert colours.grad.sum() == 2 * 3 * len(want) and radii.grad.sum() == len(want)


def test_views_from_an_iterator():
    """They are read once in the forward and again in the backward."""
    sizes = [(4, 2), (3, 3)]
    rgb, depth, hit, colours, radii = _apply(v for v in _views(*sizes))
    assert rgb.shape == (17, 3)
    depth.sum().backward()
    assert radii.grad.sum() == 17


def test_no_views():
    with pytest.raises(RuntimeError):
        _apply([])
