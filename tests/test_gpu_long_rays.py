"""Rays of more samples in a block than a float can count (2^24), through every march that the counts go into."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu

MORE = 128  # samples beyond 2^24


def _four_rays():
    """One block of 8 equal values, 2 x 2 pixels (of the 3 x 3, its view rectangle) looking straight through it: 2 quality
    samples of nothing each."""
    w = workloads.small(seed=1, level=0, depths=(1,), W=3, H=3)
    w.blocks = np.array([[0, 0, 0, 0]], np.uint32)
    w.node_off = np.array([0, 8], np.uint64)
    w.n2i = np.array([[q & 1, q >> 1 & 1, q >> 2] for q in range(8)], np.uint16)
    w.sparse = np.full(8, 0.5, np.float32)
    w.field_min, w.field_max = 0.0, 1.0
    w.ortho, w.ortho_height, w.eye = True, 10.0, (0.0, 0.0, -20.0)
    w.quality = float(2 ** 23 + MORE // 2)
    w.tf = np.zeros((4, 4), np.float32)
    return w


@pytest.mark.parametrize("tile", [0, _lib.RENDER_TILES_WALK])
def test_every_sample_is_taken(ctx, tile):
    """The walk and the block-major march (which shares so long a ray among lanes) end, having taken every sample."""
    import torch
    from revise_gb300.api import FramePlan
    w = _four_rays()
    view = host.view_for(w)
    tf, sp = torch.from_numpy(w.tf).cuda(), torch.from_numpy(w.sparse).cuda()
    plan = FramePlan(ctx, w, render_tile=tile)
    plan.interp(sp)
    rgba = torch.full((36,), -1.0, device="cuda")
    samples = torch.zeros(1, dtype=torch.int64, device="cuda")
    plan.render(view, tf, rgba, None, samples)
    torch.cuda.synchronize()
    assert int(samples.item()) == 4 * (2 ** 24 + MORE - 1)
    assert int((rgba != 0).sum()) == 0
    plan.close()


def test_adjoint_ends(ctx):
    import torch
    from revise_gb300.api import FramePlan
    w = _four_rays()
    view = host.view_for(w)
    tf, sp = torch.from_numpy(w.tf).cuda(), torch.from_numpy(w.sparse).cuda()
    plan = FramePlan(ctx, w)
    plan.interp(sp)
    rgba, dl = torch.zeros(36, device="cuda"), torch.tensor([0.0, 0.0, 0.0, 1.0] * 9, device="cuda")
    dtf, dense = torch.zeros(16, device="cuda"), torch.zeros_like(plan.bricks()[0])
    plan.backward(view, tf, rgba, dl, dtf, dense)
    torch.cuda.synchronize()
    # dA/d(alpha): the exponent of a sample's opacity times the threshold, of every sample, within a factor of 2 (an FP32
    # sum of 2^24 equal terms, each of them below the sum's last bit in the end)
    want = 4 * 100.0 / w.quality * (2 ** 24 + MORE - 1) * view.threshold
    assert 0.5 < float(dtf.view(4, 4)[:, 3].sum()) / want < 2.0
    plan.close()
