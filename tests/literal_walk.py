"""The per-ray walk on purpose: the default render form (ids 0-3) goes block-major where that pays, but not for a view
whose rays may stop early -- and an opacity that hardly any ray reaches stops none."""
import numpy as np


def walked(view):
    """The same view for the walk alone: a ray stops once its opacity passes the last float below 1."""
    v = type(view).from_buffer_copy(view)
    v.alpha_stop = float(np.nextafter(np.float32(1), np.float32(0)))
    return v


def render(ctx, plan, view, tf):
    """(RGBA bits, ARGB32, samples, kernels launched) of the second of two frames: its view is staged, and it starts from
    what the first one left."""
    import torch
    n = view.W * view.H
    rgba = torch.full((4 * n,), -1.0, device="cuda")
    argb = torch.zeros(n, dtype=torch.int32, device="cuda")
    samples = torch.zeros(1, dtype=torch.int64, device="cuda")
    plan.render(view, tf, rgba, argb)
    rgba.fill_(-1.0)
    before = ctx.launches
    plan.render(view, tf, rgba, argb, samples)
    launched = ctx.launches - before
    torch.cuda.synchronize()
    assert float(rgba.min()) >= 0.0  # every pixel written
    return rgba.view(torch.int32), argb, int(samples.item()), launched


def differences(a, b):
    """Pixels of two results of render() that differ in a bit, and samples."""
    return int((a[0] != b[0]).view(-1, 4).any(1).sum()), int((a[1] != b[1]).sum()), a[2] - b[2]
