"""The block-major frame where blocks of different depths make it share rays among 2, 4 or 8 lanes, against the per-ray
walk (render tile 0): the same pixels bit for bit and the same sample counts."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["f32", "f16", "bf16", "texture", "stop", "opaque", "quality"])
@pytest.mark.parametrize("size", [(38, 23), (160, 120), (332, 251)])
def test_shared_rays_match_walk(ctx, case, size):
    """One deep block among shallow ones in small viewports: few, long chains of samples.  Masked nodes leave samples
    outside the domain; `opaque` ends blocks early; `quality` makes the sample counts odd.  (Even widths: an odd one
    has a pixel column in the plane between blocks, where the walk takes one of the two and the block-major form
    both.)"""
    import torch
    from revise_gb300.api import FramePlan
    W, H = size
    w = workloads.small(seed=11, level=1, depths=(2, 3, 5, 7), W=W, H=H)
    assert w.blocks[:, 3].max() == 7
    if case == "opaque":
        w.tf = w.tf.copy()
        w.tf[:, 3] = 1.0
        w.threshold_rel = 1.0
    if case == "quality":
        w.quality = 0.77
    fmt = {"f16": _lib.BRICK_F16, "bf16": _lib.BRICK_BF16}.get(case, _lib.BRICK_F32)
    view = host.view_for(w, alpha_stop=0.9 if case == "stop" else 2.0,
                         filter=_lib.FILTER_TEXTURE if case == "texture" else _lib.FILTER_EXACT)
    sp, tf = torch.from_numpy(w.sparse).cuda(), torch.from_numpy(np.ascontiguousarray(w.tf)).cuda()
    out = {}
    for rt in (0, *range(_lib.RENDER_TILES_WALK, _lib.RENDER_TILES)):
        plan = FramePlan(ctx, w, fmt, render_tile=rt)
        rgba = torch.full((W * H * 4,), -1.0, device="cuda")
        argb = torch.zeros(W * H, dtype=torch.int32, device="cuda")
        samples = torch.zeros(1, dtype=torch.int64, device="cuda")
        plan.interp(sp)
        plan.render(view, tf, rgba, argb, samples)
        torch.cuda.synchronize()
        out[rt] = (rgba, argb, int(samples.item()))
        plan.close()
    assert (out[0][0][3::4] > 0).float().mean() > 0.02
    for rt, (rgba, argb, samples) in out.items():
        assert torch.equal(rgba.view(torch.int32), out[0][0].view(torch.int32)), rt
        assert torch.equal(argb, out[0][1]), rt
        if case != "stop":
            assert samples == out[0][2], rt
