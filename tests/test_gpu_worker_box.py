"""VsWorker.render_scene_part_device: the native call that a render without a `cancelled` callback takes against the
block loop that one with it takes, the blocks it puts on the device, and its stream."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu

def _worker(ctx, filt, **kw):
    from revise_gb300.api import RenderSharedState, VsWorker
    w = workloads.small(seed=6, level=2, depths=(2, 3, 4), W=96, H=72, **kw)
    wk = VsWorker(ctx)
    wk.set_render_shared_state(RenderSharedState(w, filter=filt))
    return wk, w


def _image(part, w):
    (ox, oy), (cw, ch), px = part
    out = np.zeros((w.H, w.W), np.uint32)
    if cw:
        out[oy:oy + ch, ox:ox + cw] = px.cpu().numpy().view(np.uint32).reshape(ch, cw)
    return out


@pytest.mark.parametrize("via", ["device", "native", "plan"])
def test_parts_run_on_the_current_stream(ctx, via):
    """What the caller queued before on its stream -- here, after a while, another transfer function -- is there."""
    import torch
    from revise_gb300.api import FramePlan
    wk, w = _worker(ctx, _lib.FILTER_EXACT)
    box = ((0, 0, 0), (4, 4, 4))
    plan = FramePlan(ctx, w)
    plan.interp(torch.from_numpy(w.sparse).cuda())
    call = {"device": lambda: wk.render_scene_part_device(2, *box), "native": lambda: wk.render_scene_part_native(2, *box),
            "plan": lambda: wk.render_scene_part_plan(plan, 2, *box)}[via]
    call()
    table = wk.renderer._tf
    other = table.flip(0).contiguous()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(100_000_000)
        table.copy_(other)
        got = _image(call(), w)
    torch.cuda.synchronize()
    want = _image(call(), w)
    assert np.array_equal(got, want) and want.any()
    plan.close()
