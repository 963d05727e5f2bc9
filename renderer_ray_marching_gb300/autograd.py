"""Thin torch binding of the forward marcher and the backward kernel.

``RenderFunction.apply(renderer, views, colours, xyz, radii)`` renders the
views with the renderer's current cloud and returns (rgb [P, 3], depth [P],
hit [P]) for all pixels of all views concatenated (row 0 of each view is
its bottom row).  Backward calls ``rm_backward``: gradients w.r.t. float32
colours, positions and radii through each pixel's stored hit index (see
include/rm.h).  ``colours``/``xyz``/``radii`` are the leaf tensors the
gradients are reported for; they must describe the cloud the renderer
holds (the forward does not re-upload them).
"""
from __future__ import annotations

import torch

from . import _abi


class RenderFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, renderer, views, colours, xyz, radii):
        dev = colours.device
        views = list(views)  # read again in the backward
        if len(views) == 0:
            raise RuntimeError("no views to render")
        # all views in one launch, into one buffer (a view after the other)
        pixels = sum(v.pixels for v in views)
        rgbd = torch.empty((pixels, 4), dtype=torch.float32, device=dev)
        hit = torch.empty(pixels, dtype=torch.int32, device=dev)
        frames = (_abi.RmFrame * len(views))()
        lo = 0
        for frame, v in zip(frames, views):
            frame.rgbd = rgbd.data_ptr() + 16 * lo
            frame.hit = hit.data_ptr() + 4 * lo
            lo += v.pixels
        renderer.wait_for_torch()  # earlier users of these blocks are done
        renderer.render_batch_into(views, frames, device=True)
        renderer.synchronize()
        # copies: contiguous() of a single pixel is a view of the buffer
        rgb = rgbd[:, :3].clone(memory_format=torch.contiguous_format)
        depth = rgbd[:, 3].clone(memory_format=torch.contiguous_format)
        ctx.renderer = renderer
        ctx.views = views
        ctx.n = xyz.shape[0]
        ctx.save_for_backward(hit)
        ctx.mark_non_differentiable(hit)
        return rgb, depth, hit

    @staticmethod
    def backward(ctx, g_rgb, g_depth, g_hit):
        (hit,) = ctx.saved_tensors
        dev = hit.device
        if g_rgb is None:
            g_rgb = torch.zeros((hit.shape[0], 3), dtype=torch.float32, device=dev)
        if g_depth is None:
            g_depth = torch.zeros(hit.shape[0], dtype=torch.float32, device=dev)
        g_rgb = g_rgb.to(torch.float32).contiguous()
        g_depth = g_depth.to(torch.float32).contiguous()
        n = ctx.n
        gc = torch.zeros((n, 3), dtype=torch.float32, device=dev)
        gx = torch.zeros((n, 3), dtype=torch.float32, device=dev)
        gr = torch.zeros(n, dtype=torch.float32, device=dev)
        ctx.renderer.backward(ctx.views, g_rgb, g_depth, hit, gc, gx, gr)
        ctx.renderer.synchronize()
        return None, None, gc, gx, gr


def render(renderer, views, colours, xyz, radii):
    return RenderFunction.apply(renderer, views, colours, xyz, radii)
