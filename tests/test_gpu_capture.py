"""Default-form renders inside a caller's CUDA graph, replayed after other views, and on two streams at once."""
import numpy as np
import pytest

from revise_gb300 import host, workloads

pytestmark = pytest.mark.gpu


def walked(view):
    """The same view for the per-ray walk alone: rays may stop, at an opacity that ends no ray early."""
    v = type(view).from_buffer_copy(view)
    v.alpha_stop = float(np.nextafter(np.float32(1), np.float32(0)))
    return v


def _image(plan, view, tf):
    import torch
    rgba = torch.full((view.W * view.H * 4,), -1.0, device="cuda")
    plan.render(view, tf, rgba)
    torch.cuda.synchronize()
    return rgba


@pytest.mark.parametrize("run", [False, True])
def test_captured_default_render_follows_the_view(ctx, run):
    """A default render of a level that goes block-major, captured and replayed: for its own view, after a closer one
    (which needs larger buffers), after the host pipeline was used -- the image of the view staged then."""
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.small(seed=41, level=2, depths=(4, 5), W=160, H=120)
    tf, sp = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda(), torch.from_numpy(w.sparse).cuda()
    plan = FramePlan(ctx, w)
    plan.interp(sp)
    far, near = host.view_for(w, eye=(6.0, 12.0, 40.0)), host.view_for(w, eye=(3.0, 6.0, 14.0))
    _image(plan, far, tf)
    before = ctx.launches
    _image(plan, far, tf)
    assert ctx.launches - before == 2  # block-major: march and composite
    rgba = torch.full((w.W * w.H * 4,), -1.0, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run(far, sp, tf, rgba) if run else plan.render(far, tf, rgba)
    out = torch.zeros(w.W * w.H, dtype=torch.int32).pin_memory()
    for view in (far, near, far):
        want = _image(plan, walked(view), tf)
        assert float(want.max()) > 0
        _image(plan, view, tf)
        rgba.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(rgba.view(torch.int32), want.view(torch.int32))
        plan.run_host(view, torch.from_numpy(w.sparse).pin_memory(), tf, out)
        plan.host_sync()
    del graph
    plan.close()


@pytest.mark.parametrize("tile", [0, 16])
def test_two_streams_of_one_plan(ctx, tile):
    """One staged view with two transfer functions, on two streams without order between them: both images, every time."""
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.small(seed=42, level=2, depths=(4, 5, 6), W=200, H=150)
    sp = torch.from_numpy(w.sparse).cuda()
    plan = FramePlan(ctx, w, render_tile=tile)
    plan.interp(sp)
    view = host.view_for(w)
    tfs = [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in (w.tf, w.tf[::-1])]
    want = [_image(plan, walked(view), tf) for tf in tfs]
    _image(plan, view, tfs[0])  # staged
    streams = [torch.cuda.Stream() for _ in tfs]
    got = [[torch.full_like(want[0], -1.0) for _ in range(16)] for _ in tfs]
    torch.cuda.synchronize()
    for k in range(16):
        for q, s in enumerate(streams):
            plan.render(view, tfs[q], got[q][k], stream=s)
    torch.cuda.synchronize()
    for q in range(2):
        for k in range(16):
            assert torch.equal(got[q][k].view(torch.int32), want[q].view(torch.int32)), (q, k)
    plan.close()
