"""A plan left to the default render form goes block-major where that is faster: its image against several lanes per
ray of the per-ray walk (render tile 4, which shares the walk's choice of blocks and merges in another order), rays in
the planes between blocks among them, and the same plan from view to view."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu


def _render(plan, view, tf):
    import torch
    rgba = torch.full((view.W * view.H * 4,), -1.0, device="cuda")
    samples = torch.zeros(1, dtype=torch.int64, device="cuda")
    plan.render(view, tf, rgba, None, samples)
    torch.cuda.synchronize()
    return rgba, int(samples.item())


@pytest.mark.parametrize("level", [1, 2, 3])
@pytest.mark.parametrize("filt", [_lib.FILTER_EXACT, _lib.FILTER_TEXTURE])
@pytest.mark.parametrize("eye", [(3.0, 6.0, 14.0), (0.0, 0.0, 14.0), (0.0, 6.25, 14.0), (0.7, -0.4, 1.1), (60.0, 9.0, 3.0)])
def test_default_form_is_the_walk(ctx, level, filt, eye):
    """Odd viewports (pixel columns and rows in the planes between blocks), from outside, along the planes, from
    inside the level and from far away; the two plans' sample counts are equal."""
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.small(seed=20 + level, level=level, depths=(2, 3, 5), W=201, H=151)
    view = host.view_for(w, filter=filt, eye=eye)
    tf, sp = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda(), torch.from_numpy(w.sparse).cuda()
    got = {}
    for rt in (0, 4):
        plan = FramePlan(ctx, w, render_tile=rt)
        plan.interp(sp)
        got[rt] = _render(plan, view, tf)
        assert plan.info.render_tile == rt
        plan.close()
    assert float(got[0][0].min()) >= 0.0  # every pixel written
    # 1e-5: the bound the several-lane forms are held to (partial composites merged in another order); a pixel's
    # colour is divided by its alpha, so faint pixels are compared premultiplied
    a, b = (g[0].view(-1, 4).double() for g in (got[0], got[4]))
    assert float((a[:, 3] - b[:, 3]).abs().max()) <= 1e-5
    assert float((a[:, :3] * a[:, 3:] - b[:, :3] * b[:, 3:]).abs().max()) <= 1e-5
    assert got[0][1] == got[4][1]


def test_default_form_from_view_to_view(ctx):
    """One plan through near, far, small, large and mode renders and run(), each against a fresh plan: buffers grow,
    the form changes with the view, captured frames follow."""
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.small(seed=31, level=2, depths=(2, 3, 4), W=160, H=120)
    tf, sp = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda(), torch.from_numpy(w.sparse).cuda()
    plan = FramePlan(ctx, w)
    plan.interp(sp)
    cases = [((3.0, 6.0, 40.0), 160, 120), ((3.0, 6.0, 9.0), 160, 120), ((1.0, 2.0, 8.0), 1500, 1100),
             ((0.5, 0.3, 3.0), 640, 480), ((3.0, 6.0, 40.0), 160, 120), ((30.0, 6.0, 2.0), 301, 99)]
    for k, (eye, W, H) in enumerate(cases):
        w.W, w.H = W, H
        view = host.view_for(w, eye=eye)
        fresh = FramePlan(ctx, w)
        fresh.interp(sp)
        want, n = _render(fresh, view, tf)
        fresh.close()
        if k % 2:
            pres = host.presentation(_lib.MODE_MAX_INTENSITY, view)
            plan.render_mode(view, pres, tf, None, torch.zeros(W * H * 4, device="cuda"))
        got, m = _render(plan, view, tf)
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)) and n == m, k
        rgba = torch.full((W * H * 4,), -1.0, device="cuda")
        for _ in range(2):
            plan.run(view, sp, tf, rgba)
        torch.cuda.synchronize()
        assert torch.equal(rgba.view(torch.int32), want.view(torch.int32)), k
    plan.close()
