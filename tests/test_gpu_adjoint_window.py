"""The adjoint's transfer-function gradient with a field window much narrower than the data: nearly every sample lies far
beyond the table, at one of its end entries, and the gradient has to be as good there as inside (against the FP64 oracle,
to the adjoint's bound)."""
import numpy as np
import pytest

import oracle
from revise_gb300 import host, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1e-2, 1e-5])
def test_narrow_window(ctx, width):
    import torch
    from revise_gb300.api import FramePlan
    w = workloads.cfg5(W=96, H=96)
    w.tf = np.clip(w.tf, 0.0, 1.0).astype(np.float32)
    lo, hi = w.field_min, w.field_max
    w.field_min = float(np.median(w.sparse))
    w.field_max = w.field_min + width * (hi - lo)
    view = host.view_for(w)
    ov = oracle.view_from(view)
    dense = oracle.interp_workload(w)
    rects = np.array([host.block_view_rect(view, w.blocks[b, :3]) for b in range(w.nblocks)], np.int32)
    target, _ = oracle.render_frame_f64(ov, w, dense, rects, w.meta["target_tf"])
    keep = oracle.render_frame_f64(ov, w, dense, rects, w.tf)[1] == 0
    assert keep.mean() > 0.97
    p = np.arange(w.W * w.H)[keep]
    want = oracle.render_frame_grad_f64(ov, w, dense, rects, w.tf, target[keep],
                                        np.stack([p % w.W, w.H - 1 - p // w.W], 1))[1]
    plan = FramePlan(ctx, w)
    plan.interp(torch.from_numpy(w.sparse).cuda())
    tf = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda()
    rgba = torch.zeros(w.W * w.H * 4, device="cuda")
    plan.render(view, tf, rgba)
    dl = (rgba - torch.from_numpy(np.ascontiguousarray(target, np.float32).ravel()).cuda())
    dl = dl * torch.from_numpy(np.repeat(keep.astype(np.float32), 4)).cuda()
    dtf, dd = torch.zeros(w.tf.size, device="cuda"), torch.zeros_like(plan.bricks()[0])
    plan.backward(view, tf, rgba, dl, dtf, dd)
    torch.cuda.synchronize()
    plan.close()
    ends = [0, -1]  # the entries that the samples beyond the window take
    got = dtf.cpu().numpy().reshape(-1, 4).astype(np.float64)
    err = np.linalg.norm(got[ends] - want[ends]) / np.linalg.norm(want[ends])
    print(f"window {width:g}: {err:.2e}")
    assert err < 1e-3, err
