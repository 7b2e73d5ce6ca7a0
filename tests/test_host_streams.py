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
