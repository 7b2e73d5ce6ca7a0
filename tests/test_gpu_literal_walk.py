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


@pytest.mark.parametrize("eye", [(3.0, 6.0, 14.0), (0.0, 0.0, 14.0), (0.0, 6.25, 14.0), (2.5, 2.5, 9.0), (60.0, 9.0, 3.0)])
@pytest.mark.parametrize("level,depths,fmt,filt", [(2, (4, 5, 6), 0, 0), (2, (5, 6), 1, 0), (2, (4, 5), 2, 0),
                                                   (2, (4, 5), 0, 1), (3, (3, 4, 5), 0, 0), (4, (2, 3, 4), 0, 0)])
def test_default_form_is_the_walk_bit_for_bit(ctx, level, depths, fmt, filt, eye):
    """Odd viewports, eyes on the planes between blocks among them; brick formats and filters."""
    w = _thin(workloads.small(seed=60 + level, level=level, depths=depths, W=243, H=181))
    plan, tf = _plan(ctx, w, fmt), _dev(w.tf)
    view = host.view_for(w, filter=filt, eye=eye)
    want, got = render(ctx, plan, walked(view), tf), render(ctx, plan, view, tf)
    assert want[3] == 1 and got[3] == 2
    assert differences(got, want) == (0, 0, 0)
    plan.close()


def test_default_form_of_few_blocks(ctx):
    """8 blocks, deep ones, in a small view: block-major with several lanes to a ray."""
    w = workloads.small(seed=70, level=1, depths=(6, 7), W=121, H=83)
    plan, tf = _plan(ctx, w), _dev(w.tf)
    for eye in ((3.0, 6.0, 14.0), (0.0, 0.0, 14.0)):
        view = host.view_for(w, eye=eye)
        want, got = render(ctx, plan, walked(view), tf), render(ctx, plan, view, tf)
        assert want[3] == 1 and got[3] == 2
        assert differences(got, want) == (0, 0, 0)
    plan.close()


def test_walk_shapes_agree(ctx):
    """The four CTA shapes of the walk itself, on the 64-block benchmark frame, against the block-major forms."""
    w = workloads.cfg2()
    view, tf = host.view_for(w), _dev(w.tf)
    want = None
    for tile in (*range(4), *range(_lib.RENDER_TILES_WALK, _lib.RENDER_TILES)):
        plan = _plan(ctx, w, tile=tile)
        got = render(ctx, plan, walked(view) if tile < 4 else view, tf)
        plan.close()
        assert got[3] == (1 if tile < 4 else 2)
        want = want or got
        # (opaque pixels: the walk stops at an opacity of 1, with nothing behind it that would show)
        assert differences(got, want)[:2] == (0, 0), tile


@pytest.mark.parametrize("case", ["f16", "bf16", "texture", "inside", "opaque"])
def test_block_major_ids_match_the_walk(ctx, case):
    """An even width: a pixel column in the plane between blocks is marched in both of them by the ids 16-18."""
    w = workloads.small(seed=4, level=2, depths=(2, 3, 4), W=128, H=96)
    if case == "opaque":
        w.tf = w.tf.copy()
        w.tf[:, 3] = 0.9
    view = host.view_for(w, filter=_lib.FILTER_TEXTURE if case == "texture" else _lib.FILTER_EXACT,
                         eye=(0.7, -0.4, 1.1) if case == "inside" else None)
    fmt, tf = {"f16": _lib.BRICK_F16, "bf16": _lib.BRICK_BF16}.get(case, _lib.BRICK_F32), _dev(w.tf)
    plan = _plan(ctx, w, fmt)
    want = render(ctx, plan, walked(view), tf)
    plan.close()
    assert want[3] == 1
    for tile in range(_lib.RENDER_TILES_WALK, _lib.RENDER_TILES):
        plan = _plan(ctx, w, fmt, tile)
        got = render(ctx, plan, view, tf)
        plan.close()
        assert got[3] == 2
        # (opaque pixels: the walk stops at an opacity of 1, with nothing behind it that would show)
        assert differences(got, want)[:2] == (0, 0) and (case == "opaque" or got[2] == want[2]), tile


@pytest.mark.parametrize("case", ["f32", "f16", "bf16", "texture", "quality"])
@pytest.mark.parametrize("size", [(38, 23), (160, 120)])
def test_shared_rays_match_the_walk(ctx, case, size):
    """Several lanes to a ray against one."""
    w = workloads.small(seed=11, level=1, depths=(2, 3, 5, 7), W=size[0], H=size[1])
    if case == "quality":
        w.quality = 0.77
    view = host.view_for(w, filter=_lib.FILTER_TEXTURE if case == "texture" else _lib.FILTER_EXACT)
    fmt, tf = {"f16": _lib.BRICK_F16, "bf16": _lib.BRICK_BF16}.get(case, _lib.BRICK_F32), _dev(w.tf)
    plan = _plan(ctx, w, fmt)
    want = render(ctx, plan, walked(view), tf)
    plan.close()
    assert want[3] == 1
    for tile in range(_lib.RENDER_TILES_WALK, _lib.RENDER_TILES):
        plan = _plan(ctx, w, fmt, tile)
        got = render(ctx, plan, view, tf)
        plan.close()
        assert got[3] == 2 and differences(got, want) == (0, 0, 0), tile


@pytest.mark.parametrize("n", [2, 1024, 1025, 3072])
def test_tables_of_every_size(ctx, n):
    """The walk's table against the block-major form's, which keeps differences up to 1024 entries."""
    w = workloads.small(seed=5, level=1, depths=(3, 5), W=96, H=64)
    x = np.linspace(0.0, 1.0, w.tf.shape[0])
    w.tf = np.stack([np.interp(np.linspace(0.0, 1.0, n), x, w.tf[:, c]) for c in range(4)], 1).astype(np.float32)
    view, tf = host.view_for(w), _dev(w.tf)
    plan, other = _plan(ctx, w), _plan(ctx, w, tile=_lib.RENDER_TILES_WALK)
    want, got = render(ctx, plan, walked(view), tf), render(ctx, other, view, tf)
    assert want[3] == 1 and got[3] == 2
    assert differences(got, want) == (0, 0, 0)
    plan.close()
    other.close()


@pytest.mark.parametrize("stop", [False, True])
def test_host_pipeline_of_a_default_plan(ctx, stop):
    """s3r_frame_run_host in the default form, block-major and walking, over changing values and two views: the images of
    the walk, frame by frame."""
    import torch
    w = workloads.small(seed=23, level=2, depths=(4, 5), W=160, H=120)
    plan, tf = _plan(ctx, w), _dev(w.tf)
    views = [host.view_for(w), host.view_for(w, eye=(3.0, 12.0, 30.0))]
    rng = np.random.default_rng(5)
    frames = [np.where(w.sparse == 1e30, w.sparse, w.sparse * (1 + 0.1 * k) + rng.normal()).astype(np.float32)
              for k in range(6)]
    want = []
    for k, f in enumerate(frames):
        plan.interp(_dev(f))
        want.append(render(ctx, plan, walked(views[k // 3]), tf)[1].cpu().numpy())
    images = [torch.zeros(w.W * w.H, dtype=torch.int32).pin_memory() for _ in frames]
    for k, f in enumerate(frames):
        plan.run_host(walked(views[k // 3]) if stop else views[k // 3], torch.from_numpy(f).pin_memory(), tf, images[k])
    plan.host_sync()
    for k in range(len(frames)):
        assert np.array_equal(images[k].numpy(), want[k]), k
    assert len({x.tobytes() for x in want}) == len(want)
    plan.close()
