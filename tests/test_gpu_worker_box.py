"""VsWorker.render_scene_part_device: the native call that a render without a `cancelled` callback takes against the
block loop that one with it takes, the blocks it puts on the device, and its stream."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu

BOXES = [((0, 0, 0), (4, 4, 4)), ((0, 0, 0), (2, 4, 4)), ((1, 2, 0), (4, 3, 4)), ((3, 3, 3), (4, 4, 4))]


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


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("filt", [_lib.FILTER_EXACT, _lib.FILTER_TEXTURE])
def test_native_call_is_the_block_loop(ctx, filt, box):
    wk, w = _worker(ctx, filt)
    asked = []
    loop = wk.render_scene_part_device(2, *box, cancelled=lambda: bool(asked.append(1)))
    native = wk.render_scene_part_device(2, *box)
    assert len(asked) >= 2 * int(np.prod(np.subtract(box[1], box[0])))  # before and inside every block's render
    assert loop[:2] == native[:2] and np.array_equal(_image(loop, w), _image(native, w))
    assert loop[1][0] > 0


def test_empty_box_is_refused(ctx):
    wk, _ = _worker(ctx, _lib.FILTER_EXACT)
    for kw in ({}, {"cancelled": lambda: False}):
        with pytest.raises(_lib.S3RError):
            wk.render_scene_part_device(2, (2, 2, 2), (2, 4, 4), **kw)


def test_cancelled_between_blocks(ctx):
    wk, w = _worker(ctx, _lib.FILTER_EXACT)
    asked = []
    assert wk.render_scene_part_device(2, (0, 0, 0), (4, 4, 4), lambda: bool(asked.append(1)) or len(asked) > 9) is None
    assert len(asked) in (10, 11)  # (a block's render that is cancelled returns to the loop, which asks again)


def test_only_the_boxes_blocks_go_to_the_device(ctx):
    """A worker of one box holds that box's nodes; boxes after another hold a level's worth at most."""
    wk, w = _worker(ctx, _lib.FILTER_EXACT)
    st = wk.state
    for box in BOXES[1:4] + [((x, y, z), (x + 2, y + 2, z + 2)) for x in (0, 1) for y in (0, 1) for z in (0, 1)]:
        wk.render_scene_part_device(2, *box)
        inside = [b for b in range(w.nblocks) if all(l <= i < h for l, i, h in zip(box[0], w.blocks[b, :3], box[1]))]
        blocks, off, n2i, values = st.device_box(*(list(map(int, c)) for c in box))
        assert np.array_equal(blocks, w.blocks[inside])
        assert int(off[-1]) == values.numel() == sum(w.block_nodes(b)[1].size for b in inside)
        assert "all" not in st._dev
        assert sum(v[3].numel() for v in st._boxes.values()) <= w.nodes


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


def test_another_camera_than_the_workloads(ctx):
    """A state whose view was replaced: blocks in the order of the workload's eye, as the block loop takes them."""
    wk, w = _worker(ctx, _lib.FILTER_EXACT)
    wk.state.view = host.view_for(w, filter=_lib.FILTER_EXACT, eye=(-9.0, 4.0, -8.0))
    box = ((0, 0, 0), (4, 4, 4))
    a, b = wk.render_scene_part_device(2, *box, cancelled=lambda: False), wk.render_scene_part_device(2, *box)
    assert a[:2] == b[:2] and np.array_equal(_image(a, w), _image(b, w))
