"""What the host side queues for frames -- streams, events, captured graphs, buffers -- on a stand-in for the CUDA
runtime: nothing races, outlives its memory or runs over it."""
import ctypes as C

import numpy as np
import pytest

from revise_gb300 import _lib
from tests import host_fake as hf

NEAR, FAR = (3.0, 6.0, 14.0), (6.0, 12.0, 40.0)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return hf.build(tmp_path_factory.mktemp("fake") / "libs3r_fake.so")


@pytest.fixture
def m(fake):
    x = hf.Machine(fake)
    yield x
    x.close()


def _level2(**kw):
    return hf.coarse_set(2, depth=5, **kw)


def _block_major(m, view, plan):
    n = m.calls("segments")
    m.render(plan, view)
    return m.calls("segments") > n


@pytest.mark.parametrize("tile", [0, 16])
def test_host_pipeline_orders_the_items(m, tile):
    """s3r_frame_run_host over views that change on either slot: a slot's block-major march comes after the expansion
    of the work items, on whichever slot's stream that was queued."""
    w = _level2()
    plan = m.plan(w, tile)
    sparse, tf = m.buffer(w.nodes), m.buffer(4 * 256)
    out = [m.buffer(w.W * w.H, np.uint32) for _ in range(2)]
    k = 0
    for eye in (NEAR, FAR, NEAR):
        view = hf.view_of(w, eye=eye)
        for _ in range(3):
            m.ok(m.lib.s3r_frame_run_host(m.h, plan, C.byref(view), sparse, tf, out[k & 1], None))
            k += 1
    m.ok(m.lib.s3r_frame_host_sync(m.h, plan))
    assert m.calls("segments") == k
    assert m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


def _captured(m, plan, view, tf, image, run):
    """A caller's graph of one frame of the staged view; run: (sparse values) interpolation and render."""
    s = m.stream()
    args = (C.byref(view), *([run] if run else []), tf, None, image, None, s)
    f = m.lib.s3r_frame_run if run else m.lib.s3r_frame_render
    return m.capture(s, lambda: m.ok(f(m.h, plan, *args))), s


@pytest.mark.parametrize("run", [False, True])
def test_captured_default_render_outlives_every_view(m, run):
    """A default render captured by the caller is replayed after closer views, views that walk, larger and smaller
    images, a field mode's view and the host pipeline: only memory that lives as long as the plan is in it, and each
    replay shows the view that is staged then."""
    w = _level2()
    plan = m.plan(w)
    sparse, tf, image = m.buffer(w.nodes), m.buffer(4 * 256), m.buffer(1500 * 1100, np.uint32)
    view = hf.view_of(w, eye=FAR)
    assert _block_major(m, view, plan)
    graph, s = _captured(m, plan, view, tf, image, sparse if run else None)
    w.W, w.H = 1500, 1100
    large = hf.view_of(w, eye=NEAR)
    w.W, w.H = 160, 120
    stop = hf.view_of(w, eye=NEAR)
    stop.alpha_stop = 0.9
    for other in (hf.view_of(w, eye=NEAR), large, stop, view):
        m.render(plan, other)
        m.lib.cudaDeviceSynchronize()
        m.launch(graph, s)
        m.lib.cudaDeviceSynchronize()
    near = hf.view_of(w, eye=NEAR)
    pres = hf.host.presentation(_lib.MODE_MAX_INTENSITY, near)
    m.ok(m.lib.s3r_frame_render_mode(m.h, plan, C.byref(near), C.byref(pres), tf, None, None, image, None))
    m.lib.cudaDeviceSynchronize()
    m.launch(graph, s)
    m.lib.cudaDeviceSynchronize()  # (views are staged in the caller's order)
    for _ in range(2):
        m.ok(m.lib.s3r_frame_run_host(m.h, plan, C.byref(view), sparse, tf, m.buffer(w.W * w.H, np.uint32), None))
    m.ok(m.lib.s3r_frame_host_sync(m.h, plan))
    m.launch(graph, s)
    m.lib.cudaDeviceSynchronize()
    assert m.trouble() == []
    assert m.calls("walk") >= 5  # the replays among them
    m.ok(m.lib.s3r_plan_destroy(plan))


def test_captured_block_major_render_keeps_its_buffers(m):
    """A render in a block-major form by its id, captured: replays follow the views of the same image size and at most
    as many work items, a field mode's view and the first use of the host pipeline."""
    w = _level2()
    plan = m.plan(w, 16)
    sparse, tf, image = m.buffer(w.nodes), m.buffer(4 * 256), m.buffer(w.W * w.H, np.uint32)
    near = hf.view_of(w, eye=NEAR)
    m.render(plan, near)
    graph, s = _captured(m, plan, near, tf, image, None)
    far = hf.view_of(w, eye=FAR)
    m.render(plan, far)
    m.lib.cudaDeviceSynchronize()
    m.launch(graph, s)
    m.lib.cudaDeviceSynchronize()
    pres = hf.host.presentation(_lib.MODE_MAX_INTENSITY, near)
    m.ok(m.lib.s3r_frame_render_mode(m.h, plan, C.byref(near), C.byref(pres), tf, None, None, image, None))
    m.lib.cudaDeviceSynchronize()
    m.launch(graph, s)
    m.lib.cudaDeviceSynchronize()  # (as above)
    m.ok(m.lib.s3r_frame_run_host(m.h, plan, C.byref(far), sparse, tf, m.buffer(w.W * w.H, np.uint32), None))
    m.ok(m.lib.s3r_frame_host_sync(m.h, plan))
    m.launch(graph, s)
    assert m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


@pytest.mark.parametrize("tile", [0, 16])
def test_two_streams_take_turns(m, tile):
    """Frames of one staged view on two streams, and of s3r_frame_run's graph beside them: the block-major form's
    results, masks and work queue serve one at a time."""
    w = _level2()
    plan = m.plan(w, tile)
    view = hf.view_of(w, eye=NEAR)
    sparse, tf = m.buffer(w.nodes), m.buffer(4 * 256)
    assert _block_major(m, view, plan)
    m.lib.cudaDeviceSynchronize()
    streams = [m.stream() for _ in range(3)]
    for k in range(6):
        m.render(plan, view, streams[k % 3])
    m.lib.cudaDeviceSynchronize()
    m.ok(m.lib.s3r_frame_run(m.h, plan, C.byref(view), sparse, tf, None, m.buffer(w.W * w.H, np.uint32), None, streams[0]))
    m.render(plan, view, streams[1])
    assert m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


def test_growing_views(m):
    """Default renders whose views cover more and more, on alternating streams with frames in flight: a plan's first
    frame waits for nothing, later ones give memory back only when the frames that use it are over."""
    w = _level2()
    plan = m.plan(w)
    streams = [m.stream(), m.stream()]
    waits = ("cudaFree", "cudaDeviceSynchronize", "cudaStreamSynchronize")
    for k, (W, H, eye) in enumerate([(100, 80, FAR), (160, 120, FAR), (160, 120, NEAR), (400, 300, NEAR)]):
        w.W, w.H = W, H
        view = hf.view_of(w, eye=eye)
        before = [m.calls(n) for n in waits]
        m.render(plan, view, streams[k % 2])
        assert k > 0 or [m.calls(n) for n in waits] == before
        m.lib.cudaStreamSynchronize(streams[k % 2])  # the caller's own order between views
        m.render(plan, view, streams[1 - k % 2])
    assert m.calls("segments") == 8
    assert m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


@pytest.mark.parametrize("tile", [0, 16])
def test_a_little_more_fits(m, tile):
    """Views that cover up to half as many pixels again as a plan's first one reuse its buffers."""
    w = _level2()
    plan = m.plan(w, tile)
    m.render(plan, hf.view_of(w, eye=FAR))
    before = m.calls("cudaMalloc")
    for z in (39.0, 38.0, 40.0):
        m.render(plan, hf.view_of(w, eye=(6.0, 12.0, z)))
    assert m.calls("cudaMalloc") == before and m.calls("segments") == 4
    m.ok(m.lib.s3r_plan_destroy(plan))


def test_no_room_for_results_walks(m):
    """Without memory for the block results the default form walks, and what other calls then queue is clean."""
    w = _level2(W=640, H=480)
    plan = m.plan(w)
    view = hf.view_of(w, eye=NEAR)
    m.lib.fake_limit(1 << 20)
    assert not _block_major(m, view, plan) and m.calls("walk") == 1
    m.lib.fake_limit(2 ** 64 - 1)
    assert not _block_major(m, view, plan)  # as staged
    assert _block_major(m, hf.view_of(w, eye=FAR), plan)
    assert m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


@pytest.mark.parametrize("level,eye", [(3, (0.1, 0.2, 0.3)), (4, (0.3, 0.2, 1.0)), (4, (0.0, 0.0, -6.0))])
def test_default_form_inside_the_level_walks(m, level, eye):
    """A camera inside the level or facing away from it: blocks with a corner behind the eye have the whole viewport for
    their rectangle, hundreds of times the rays that meet a block.  The default form walks and allocates nothing; seen
    from outside the same plan goes block-major."""
    w = hf.coarse_set(level, depth=1, W=300, H=200, quality=16.0)
    plan = m.plan(w)
    outside = hf.view_of(w, eye=NEAR)
    assert _block_major(m, outside, plan)
    inside = hf.view_of(w, eye=eye)
    if eye[2] < -5:  # the level behind the camera
        w.center = (0.0, 0.0, -9.0)
        inside = hf.view_of(w, eye=eye)
    before = m.lib.fake_used()
    assert not _block_major(m, inside, plan) and m.calls("walk") == 1
    assert m.lib.fake_used() == before and m.trouble() == []
    m.ok(m.lib.s3r_plan_destroy(plan))


@pytest.mark.parametrize("filt", [_lib.FILTER_EXACT, _lib.FILTER_TEXTURE])
@pytest.mark.parametrize("secondary", [False, True])
@pytest.mark.parametrize("room", [3 << 20, 12 << 20, 60 << 20])
def test_part_without_room_goes_block_by_block(m, filt, secondary, room):
    """A part whose textures, dense fields or pixel lists do not fit is rendered block by block, in one block's memory; a
    later part with room is not."""
    w = _level2(W=640, H=480)
    w.blocks[:, 3] = 5
    view = hf.view_of(w, eye=NEAR, filter=filt)
    pres = hf.host.presentation(_lib.MODE_VALUE_ON_ISOSURFACE, view, secondary_range=(0.0, 1.0)) if secondary else None
    m.lib.fake_limit(room)
    assert m.part(w, view, pres) == [0, 0, 640, 480]
    assert m.calls("render_block") == 64 and m.trouble() == []
    m.lib.fake_limit(2 ** 64 - 1)
    assert m.part(w, view, pres) == [0, 0, 640, 480]
    assert m.calls("render_block") == 64 and m.calls("part") == 1 and m.trouble() == []


@pytest.mark.parametrize("room", [1 << 20, 2 ** 64 - 1])
def test_part_of_bricks_without_room(m, room):
    w = _level2(W=640, H=480)
    plan = m.plan(w)
    view = hf.view_of(w, eye=NEAR)
    m.lib.fake_limit(room)
    lo, hi, rect = (C.c_uint32 * 3)(0, 0, 0), (C.c_uint32 * 3)(4, 4, 4), (C.c_int32 * 4)()
    m.ok(m.lib.s3r_render_scene_part_bricks(m.h, plan, C.byref(view), None, None, lo, hi, m.buffer(4 * 256),
                                            m.buffer(w.W * w.H, np.uint32), rect, None))
    assert rect[:] == [0, 0, 640, 480]
    assert m.calls("render_block") == (64 if room < 2 ** 63 else 0) and m.trouble() == []
    m.lib.fake_limit(2 ** 64 - 1)
    m.ok(m.lib.s3r_plan_destroy(plan))


def test_few_shallow_blocks_walk(m):
    """8 blocks of depths 2 to 4 go block-major for no view: their rays have too few samples to share, whatever deeper
    blocks would do."""
    w = hf.coarse_set(1, depth=4, W=407, H=407)
    w.blocks[:, 3] = [2, 3, 4, 2, 3, 4, 2, 3]
    w.n2i = np.concatenate([np.array([[q & 1, q >> 1 & 1, q >> 2] for q in range(8)], np.uint16) << d for d in w.blocks[:, 3]])
    plan = m.plan(w)
    for distance in (9.0, 14.0, 30.0, 60.0):
        assert not _block_major(m, hf.view_of(w, eye=(0.3 * distance, 0.2 * distance, distance)), plan)
    m.ok(m.lib.s3r_plan_destroy(plan))


def test_small_views_inside_the_level_go_block_major(m):
    """A camera inside the level, but so few pixels that empty rays cost nothing beside the chains of samples."""
    w = hf.coarse_set(2, depth=6, W=50, H=50)
    plan = m.plan(w)
    assert _block_major(m, hf.view_of(w, eye=(0.1, 0.2, 0.3)), plan)
    w.W, w.H = 500, 400
    assert not _block_major(m, hf.view_of(w, eye=(0.1, 0.2, 0.3)), plan)
    m.ok(m.lib.s3r_plan_destroy(plan))
