"""Infinite values in bricks; values whose relative value overflows -- infinite, or finite but far outside a narrow field range -- under the texture
unit's filtering rule: they take the transfer function's end entries, as any value beyond the range does."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu

FAR = 1e30  # outside the range, its relative value representable


def _scene():
    w = workloads.small(seed=3, level=1, depths=(3,), W=48, H=40)
    view = host.view_for(w, filter=_lib.FILTER_TEXTURE)
    view.field_min, view.field_max, view.threshold = 0.0, 0.5, 0.25
    return w, view


@pytest.mark.parametrize("tile", [0, 4, _lib.RENDER_TILES_WALK])
@pytest.mark.parametrize("value", [-3e38, 3e38])
def test_frames(ctx, tile, value):
    import torch
    from revise_gb300.api import FramePlan
    w, view = _scene()
    tf = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda()
    plan = FramePlan(ctx, w, render_tile=tile)
    got = []
    for v in (value, np.copysign(FAR, value)):
        plan.bricks()[0].fill_(float(v))
        img = [torch.zeros(w.W * w.H, dtype=torch.int32, device="cuda") for _ in range(3)]
        plan.render(view, tf, None, img[0])
        for k, mode in enumerate((_lib.MODE_ARGB, _lib.MODE_ARGB_LIGHT)):
            plan.render_mode(view, host.presentation(mode, view), tf, None, None, img[1 + k])
        torch.cuda.synchronize()
        got.append(img)
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert value < 0 or int((got[0][0] != 0).sum()) > 0  # (the table starts transparent)
    plan.close()


@pytest.mark.parametrize("mode", [_lib.MODE_ARGB, _lib.MODE_ARGB_LIGHT])
@pytest.mark.parametrize("value", [-float("inf"), float("inf"), -3e38, 3e38])
def test_blocks(ctx, mode, value):
    """One block, its values read by the texture unit and, finite ones, by its rule in software."""
    import torch
    w, view = _scene()
    tf = torch.from_numpy(np.ascontiguousarray(w.tf[::-1])).cuda()  # opaque at the low end
    if value > 0:
        tf = tf.flip(0).contiguous()
    pres = host.presentation(mode, view)
    idx = w.blocks[0, :3]
    rect = host.block_view_rect(view, idx)
    got = []
    for v in (value, np.copysign(FAR, value)):
        dense = torch.full((9 ** 3,), float(v), device="cuda")
        tex = ctx.texture(3)
        tex.fill(dense)
        img = [torch.zeros(w.W * w.H, dtype=torch.int32, device="cuda") for _ in range(2)]
        ctx.render_block_texture(view, pres, tex, idx, rect, ctx.tf_texture(tf), img[0])
        if np.isfinite(value):
            ctx.render_block(view, pres, dense, 3, idx, rect, tf, img[1])
        torch.cuda.synchronize()
        got.append(img)
    assert mode == _lib.MODE_ARGB_LIGHT or int((got[0][0] != 0).sum()) > 0
    for a, b in zip(*(g if np.isfinite(value) else g[:1] for g in got)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("via", ["block", "part"])
def test_infinite_texels_show_in_the_argb_call(ctx, via):
    """s3r_render_block_argb leaves a sample out where a texel is NaN; infinite texels, whose weighted sum is a NaN, make
    its pixel transparent (a NaN as a byte is 0).  The Argb field mode leaves out what filters to a NaN."""
    import torch
    from revise_gb300.api import FramePlan, RenderSharedState, VsWorker
    w, view = _scene()
    view.filter = _lib.FILTER_EXACT
    tf = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda()
    plan = FramePlan(ctx, w)
    signs = torch.ones_like(plan.bricks()[0])
    signs[::2] = -1.0
    plan.bricks()[0].copy_(signs * float("inf"))
    pres = host.presentation(_lib.MODE_ARGB, view)
    seen = []
    for p in (None, pres):
        if via == "part":
            st = RenderSharedState(w, filter=_lib.FILTER_EXACT)
            st.view = view
            wk = VsWorker(ctx)
            wk.set_render_shared_state(st)
            wk.render_scene_part_plan(plan, w.level, (0, 0, 0), (2, 2, 2), p)
            seen.append(wk.viewport.clone())
            continue
        vp = torch.full((w.W * w.H,), -1, dtype=torch.int32, device="cuda")  # opaque white
        dense = plan.block_dense(0).contiguous()
        idx = w.blocks[0, :3]
        rect = host.block_view_rect(view, idx)
        if p is None:
            ctx.render_block_argb(view, dense, 3, idx, rect, tf, vp)
        else:
            ctx.render_block(view, p, dense, 3, idx, rect, tf, vp)
        seen.append(vp)
    torch.cuda.synchronize()
    if via == "block":
        assert int((seen[0] == 0x00ffffff).sum()) > 100  # transparent, its colour kept
        assert int((seen[1] != -1).sum()) == 0
    else:
        assert int((seen[0] != 0).sum()) == 0 and int((seen[1] != 0).sum()) == 0
    plan.close()
