"""A worker's part rendered in a few launches (s3r_render_scene_part, s3r_render_scene_part_bricks) against the same
blocks rendered one by one through the per-block calls, back to front: the same viewport, byte for byte."""
import dataclasses

import numpy as np
import pytest

from revise_gb300 import _lib, host, workloads

pytestmark = pytest.mark.gpu

MODES = [_lib.MODE_ISOSURFACE, _lib.MODE_ISOSURFACES, _lib.MODE_MAX_INTENSITY, _lib.MODE_ARGB, _lib.MODE_ARGB_LIGHT,
         _lib.MODE_DOMAIN_VOXELS, _lib.MODE_VALUE_ON_ISOSURFACE, _lib.MODE_VALUE_ON_ISOSURFACES]


def _presentation(mode, w, view):
    span = w.field_max - w.field_min
    return host.presentation(mode, view, isosurface_opacity=0.6, levels=[w.field_min + span * t for t in (0.3, 0.5, 0.7)],
                             secondary_range=(w.field_min, w.field_max))


def _second(w):
    return np.where(w.sparse == workloads.NO_FIELD, w.sparse, np.float32(0.3) - w.sparse).astype(np.float32)


def _block_by_block(ctx, w, view, pres, box, second, viewport, bricks):
    """Every block of the box, back to front, through the per-block calls; the texture filter through the texture
    unit, but on bricks, which are sampled in memory, by its rule in software."""
    import torch
    from revise_gb300.api import to_device_n2i
    tf = torch.from_numpy(np.ascontiguousarray(w.tf)).cuda()
    tex = view.filter == _lib.FILTER_TEXTURE and not bricks
    tf_tex = ctx.tf_texture(tf) if tex else None
    secondary = pres is not None and pres.mode in (_lib.MODE_VALUE_ON_ISOSURFACE, _lib.MODE_VALUE_ON_ISOSURFACES)
    clear = 0x7fc00000 if pres is not None and pres.mode == _lib.MODE_MAX_INTENSITY else 0
    ctx.clear_viewport(viewport, w.W, w.H, clear)
    where = {tuple(int(x) for x in b[:3]): i for i, b in enumerate(w.blocks)}
    cmin, cmax = host.index_box_world(w.level, *box)
    for idx in host.b2f_order(*box, cmin, cmax, view.cam.eye[:]):
        b = where.get(tuple(int(x) for x in idx))
        if b is None:
            continue
        depth = int(w.blocks[b, 3])
        n2i, vals = w.block_nodes(b)
        n2i_dev = to_device_n2i(n2i)
        fields = [vals] + ([second[int(w.node_off[b]):int(w.node_off[b + 1])]] if secondary else [])
        rect = host.block_view_rect(view, idx)
        if rect[2] == 0 or rect[3] == 0:
            continue
        if tex:
            texs = []
            for f in fields:
                t = ctx.texture(depth)
                ctx.interp_dense_texture(n2i_dev, torch.from_numpy(np.ascontiguousarray(f)).cuda(), t)
                texs.append(t)
            ctx.render_block_texture(view, pres, texs[0], idx, rect, tf_tex, viewport,
                                     texs[1] if secondary else None)
            torch.cuda.synchronize()  # the textures go with this iteration
        else:
            dense = [ctx.interp_dense(n2i_dev, torch.from_numpy(np.ascontiguousarray(f)).cuda(), depth) for f in fields]
            if pres is None:
                ctx.render_block_argb(view, dense[0], depth, idx, rect, tf, viewport)
            else:
                ctx.render_block(view, pres, dense[0], depth, idx, rect, tf, viewport,
                                 dense[1] if secondary else None)


def _check(ctx, w, filt, mode, box=None, bricks=False, eye=None):
    import torch
    from revise_gb300.api import FramePlan, RenderSharedState, VsWorker
    m = 1 << w.level
    box = box or ((0, 0, 0), (m, m, m))
    if eye is not None:
        w = dataclasses.replace(w, eye=eye)
    st = RenderSharedState(w, filter=filt)
    pres = None if mode is None else _presentation(mode, w, st.view)
    second = _second(w)
    wk = VsWorker(ctx)
    wk.set_render_shared_state(st)
    if bricks:
        plan, plan2 = FramePlan(ctx, w), FramePlan(ctx, w)
        plan.interp(torch.from_numpy(w.sparse).cuda())
        plan2.interp(torch.from_numpy(second).cuda())
        wk.render_scene_part_plan(plan, w.level, *box, pres, plan2.bricks()[0])
    else:
        wk.render_scene_part_native(w.level, *box, pres, torch.from_numpy(second).cuda())
    got = wk.viewport.clone()
    want = torch.empty_like(got)
    _block_by_block(ctx, w, st.view, pres, box, second, want, bricks)
    torch.cuda.synchronize()
    assert torch.equal(got, want), int((got != want).sum())
    assert int((want != want[0]).sum()) > 0


@pytest.mark.parametrize("mode", [None, *MODES])
@pytest.mark.parametrize("source", ["texture", "dense", "bricks", "bricks_texture_rule"])
def test_part_equals_block_by_block(ctx, mode, source):
    """Every field mode from every source; an odd viewport, a box that is not the whole level."""
    w = workloads.small(seed=5, level=2, depths=(2, 3, 4, 5), W=131, H=97)
    filt = _lib.FILTER_TEXTURE if source in ("texture", "bricks_texture_rule") else _lib.FILTER_EXACT
    _check(ctx, w, filt, mode, box=((1, 0, 0), (4, 4, 3)), bricks=source.startswith("bricks"))


@pytest.mark.parametrize("source", ["texture", "bricks"])
@pytest.mark.parametrize("scene", ["inside", "on_faces", "missing", "chunks", "strips", "two"])
def test_part_shapes(ctx, scene, source):
    """An eye inside the level and one on the planes between blocks with a pixel column and row along them (rays that
    pass two blocks' faces at once: more results a pixel than blocks on a path); missing blocks; more blocks than one
    chunk; lists larger than their memory, so several strips; a box of two blocks."""
    box, eye = None, None
    if scene == "chunks":
        w = workloads.small(seed=7, level=3, depths=(1, 2), W=160, H=120)
    elif scene == "strips":
        w = workloads.small(seed=8, level=2, depths=(1, 2), W=1920, H=1080, eye=(2.0, 3.0, 9.0))
    else:
        w = workloads.small(seed=6, level=2, depths=(2, 3, 4), W=129, H=95)
    if scene == "inside":
        eye = (0.7, -0.4, 1.1)
    elif scene == "on_faces":
        eye = (0.0, 0.0, 14.0)
    elif scene == "missing":
        keep = [b for b in range(w.nblocks) if b % 3]
        parts = [w.block_nodes(b) for b in keep]
        w = dataclasses.replace(w, blocks=w.blocks[keep], n2i=np.concatenate([p[0] for p in parts]),
                                sparse=np.concatenate([p[1] for p in parts]),
                                node_off=np.concatenate([[0], np.cumsum([len(p[1]) for p in parts])]).astype(np.uint64))
    elif scene == "two":
        box = ((1, 2, 1), (2, 3, 3))
    _check(ctx, w, _lib.FILTER_TEXTURE if source == "texture" else _lib.FILTER_EXACT, None, box=box,
           bricks=source == "bricks", eye=eye)
