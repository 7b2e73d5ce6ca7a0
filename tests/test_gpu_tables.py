"""Transfer functions up to the largest table that every render takes (3072 entries, 48 KB of shared memory)."""
import dataclasses

import numpy as np
import pytest

import oracle
from revise_gb300 import _lib, host, workloads

from test_gpu_adjoint import REL_TOL, _gpu_grad, _keep, _rects, _setup

pytestmark = pytest.mark.gpu


def _resampled(tf, n):
    x = np.linspace(0.0, 1.0, tf.shape[0])
    return np.stack([np.interp(np.linspace(0.0, 1.0, n), x, tf[:, c]) for c in range(4)], 1).astype(np.float32)


@pytest.mark.parametrize("level", [0, 1])
@pytest.mark.parametrize("n", [2, 1024, 1025, 3070, 3071, 3072])
def test_renders_take_the_table(ctx, n, level):
    """The walk (level 0: always) against block-major, which keeps differences up to 1024 entries: bit for bit; the Argb
    mode within 2e-3 of the oracle's composition, the bound of the mode images."""
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.small(seed=5, level=level, depths=(5,) if level == 0 else (3, 5), W=96, H=64)
    w = dataclasses.replace(w, tf=_resampled(w.tf, n))
    view = host.view_for(w)
    sp, tf = torch.from_numpy(w.sparse).cuda(), torch.from_numpy(w.tf).cuda()
    img = {}
    for rt in (0, 1, 4, _lib.RENDER_TILES_WALK):
        plan = FramePlan(ctx, w, render_tile=rt)
        plan.interp(sp)
        img[rt] = torch.full((w.W * w.H * 4,), -1.0, device="cuda")
        plan.render(view, tf, img[rt])
        if rt == 1:
            mode = torch.full((w.W * w.H * 4,), -1.0, device="cuda")
            pres = host.presentation(_lib.MODE_ARGB, view)
            plan.render_mode(view, pres, tf, None, mode, None)
        torch.cuda.synchronize()
        plan.close()
    assert torch.equal(img[0], img[_lib.RENDER_TILES_WALK])
    assert torch.equal(img[1], img[_lib.RENDER_TILES_WALK])
    # several lanes to a ray merge partial composites in another order; faint pixels are compared premultiplied
    a, b = (img[rt].view(-1, 4).double() for rt in (1, 4))
    assert float((a[:, 3] - b[:, 3]).abs().max()) <= 1e-5
    assert float((a[:, :3] * a[:, 3:] - b[:, :3] * b[:, 3:]).abs().max()) <= 1e-5
    dense = oracle.interp_workload(w)
    rects = _rects(w, view)
    want = oracle.render_frame_mode(oracle.view_from(view), oracle.presentation_from(pres), w, dense, rects, w.tf,
                                    view.alpha_stop, None)
    assert np.abs(mode.cpu().numpy().reshape(-1, 4) - np.asarray(want).reshape(-1, 4)).max() <= 2e-3


@pytest.mark.parametrize("n", [2, 2700, 3072])
def test_adjoint_takes_the_table(ctx, n):
    """Gradients against the FP64 oracle's, the shared memory beside the table included."""
    w = _setup(40, 40)
    target_tf = _resampled(w.meta["target_tf"], n)
    w = dataclasses.replace(w, tf=_resampled(w.tf, n))
    view = host.view_for(w)
    ov, dense, rects = oracle.view_from(view), oracle.interp_workload(w), _rects(w, view)
    target, _ = oracle.render_frame_f64(ov, w, dense, rects, target_tf)
    keep = _keep(ov, w, dense, rects)
    p = np.arange(w.W * w.H)[keep]
    pixels = np.stack([p % w.W, w.H - 1 - p // w.W], 1)
    _, dtf64, dd64 = oracle.render_frame_grad_f64(ov, w, dense, rects, w.tf, target[keep], pixels)
    _, _, dtf, dd = _gpu_grad(ctx, w, target, keep)
    assert np.linalg.norm(dtf - dtf64) <= REL_TOL * np.linalg.norm(dtf64)
    m = ~np.isnan(dense)
    assert np.linalg.norm(dd[m] - dd64[m]) <= REL_TOL * np.linalg.norm(dd64[m])
