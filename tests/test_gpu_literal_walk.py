"""Every render form against the per-ray walk itself (tests/literal_walk.py), bit for bit with the same samples; the
kernels launched say which form ran: one for the walk, two for block-major."""
import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads
from literal_walk import differences, render, walked

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _plan(ctx, w, fmt=_lib.BRICK_F32, tile=0):
    from revise_gb300.api import FramePlan
    plan = FramePlan(ctx, w, fmt, render_tile=tile)
    plan.interp(_dev(w.sparse))
    return plan


def _thin(w):
    """A transfer function so transparent that no ray becomes opaque: the samples agree too."""
    w.tf = w.tf * np.array([1, 1, 1, 0.02], np.float32)
    return w


@pytest.mark.parametrize("distance,quality,half,eyes", [(300.0, 1.5, 0.05, 8), (10000.0, 150.0, 0.006, 12)])
def test_default_form_from_far_away(ctx, distance, quality, half, eyes):
    """A distant eye, where the walk's crossing times are large and rounded accordingly, looking through a narrow field of
    view at points where blocks meet, so that every ray grazes some of them, with samples close enough (5e-4) to show
    which."""
    w = _thin(workloads.small(seed=54, level=4, depths=(3,), W=48, H=36))
    w.fovy, w.quality = float(np.degrees(2 * np.arctan(half / distance))), quality
    plan, tf = _plan(ctx, w), _dev(w.tf)
    rng = np.random.default_rng(4)
    total = np.zeros(3, np.int64)
    for _ in range(eyes):
        d = rng.normal(size=3)
        w.center = tuple(float(x) for x in rng.integers(1, 16, 3) * 0.625 - 5.0)
        view = host.view_for(w, eye=tuple(float(x) for x in d / np.linalg.norm(d) * distance))
        want, got = render(ctx, plan, walked(view), tf), render(ctx, plan, view, tf)
        assert want[3] == 1 and got[3] == 2
        total += np.abs(differences(got, want))
    assert total.tolist() == [0, 0, 0]
    plan.close()
