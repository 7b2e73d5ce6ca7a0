"""The work a user of revise_gb300 has it do, as cases that can be timed and compared.

Every case is a block set of one block-tree level (octree node lists, one float per node) and a camera, taken
through the public entry points:

  block   one subtree's sparse nodes -> its dense grid (Context.interp_dense)
  frame   a whole level: interpolation and ray cast, FP32 / FP16 / BF16 bricks (FramePlan.run)
  orbit   several camera positions over a level that is already interpolated (FramePlan.render)
  mode    a level in one of the field modes, as the viewer's ARGB frame (FramePlan.render_mode)
  part    a worker's image part of an index box (VsWorker.render_scene_part_*), composed onto the frame
  adjoint the image and its gradients with respect to transfer function and bricks (autograd.render_frame)
  stream  a time series from pinned host buffers to host images (FramePlan.run_host)

exact() restates the interpolation and the ray cast in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

from revise_gb300 import _lib, host, schedule, workloads
from revise_gb300.api import Context, FramePlan, RenderSharedState, VsWorker, to_device_n2i
from revise_gb300.autograd import render_frame

NO_FIELD = 1e30
FORMATS = {"f32": _lib.BRICK_F32, "f16": _lib.BRICK_F16, "bf16": _lib.BRICK_BF16}
MODES = {"isosurface": _lib.MODE_ISOSURFACE, "isosurfaces": _lib.MODE_ISOSURFACES, "mip": _lib.MODE_MAX_INTENSITY,
         "argb": _lib.MODE_ARGB, "argb_light": _lib.MODE_ARGB_LIGHT, "domain": _lib.MODE_DOMAIN_VOXELS,
         "value_on_isosurface": _lib.MODE_VALUE_ON_ISOSURFACE, "value_on_isosurfaces": _lib.MODE_VALUE_ON_ISOSURFACES}
SCENE = {"level": 2, "depth": 6, "nodes": 0, "mask": "none", "W": 1920, "H": 1080, "dist": 18.0, "fovy": 60.0,
         "quality": 1.0, "tf": 256, "stop": 2.0}


def _scene(**over):
    return {**SCENE, **over}


def listed():
    return [
        # the per-block drop-in of a worker loop: most subtrees are small, so a call is launches and latency
        {"name": "block_small", "kind": "block", "depth": 4, "nodes": 700, "mask": "random"},
        # a deep subtree of a few thousand nodes, the deepest class of the mixed-depth benchmark level
        {"name": "block_deep", "kind": "block", "depth": 7, "nodes": 20000, "mask": "random"},
        # the largest subtree the kernels take: 513^3 vertices
        {"name": "block_largest", "kind": "block", "depth": 9, "nodes": 2000000, "mask": "sphere"},
        # the benchmark's level: 4096 blocks of depth 3 to 7, 20 % of the nodes masked, as the README runs it
        {"name": "frame_full_level", "kind": "frame", "fmt": "f32", "form": 0,
         **_scene(level=4, depth=0, nodes=2000, mask="random", dist=36.4)},
        # a uniform level close up, 16-bit bricks (half the memory for twice the data)
        {"name": "frame_uniform_f16", "kind": "frame", "fmt": "f16", "form": 0, **_scene()},
        # turning the camera around a loaded data set, in the render form the autotuner picks for such a level
        {"name": "orbit_mixed", "kind": "orbit", "fmt": "f32", "form": 16, "views": 4,
         **_scene(level=3, depth=0, nodes=2000, mask="random")},
        # lit isosurfaces of a loaded data set in a viewer window
        {"name": "mode_isosurfaces", "kind": "mode", "mode": "isosurfaces", **_scene(mask="sphere", W=1280, H=720)},
        # a worker thread's part of a level as the reference renders it, texture-unit sampling, volume rendering
        {"name": "part_texture", "kind": "part", "via": "native", "mode": "argb", **_scene()},
        # the smallest worker call: one split box of a coarse level in a small window, through the block loop
        {"name": "part_small", "kind": "part", "via": "device", "mode": "argb",
         **_scene(level=1, depth=3, mask="random", W=333, H=251)},
        # a worker's part of a mixed level whose bricks stay resident
        {"name": "part_bricks", "kind": "part", "via": "bricks", "mode": "argb",
         **_scene(level=3, depth=0, nodes=2000, mask="random")},
        # fitting a transfer function and a field to an image
        {"name": "adjoint", "kind": "adjoint", **_scene(level=1, W=512, H=512, dist=22.4, fovy=40.0)},
        # playing a time series: every frame's values come from host memory, every image goes back there
        {"name": "stream", "kind": "stream", "fmt": "f32", "form": 16, "frames": 4,
         **_scene(level=3, depth=0, nodes=2000, mask="random")},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "frame", "orbit", "mode", "part", "part", "adjoint", "stream"])
    if kind == "block":
        depth = rng.randint(2, 9)
        top = min(2000000, (2 ** depth + 1) ** 3)
        return {"kind": "block", "depth": depth, "nodes": _log_int(rng, min(64, top), top),
                "mask": rng.choice(["none", "random", "sphere"])}
    W = _log_int(rng, 200, 1920)
    c = _scene(W=W, H=max(96, min(1080, int(W * rng.choice([0.5625, 0.75, 1.0])) + rng.randint(0, 7))),
               dist=round(rng.uniform(11.0, 37.0), 2), fovy=rng.choice([40.0, 60.0]),
               quality=rng.choice([0.5, 1.0, 1.0, 1.5]), tf=rng.choice([64, 256, 256, 1000]),
               mask=rng.choice(["none", "random", "sphere"]), stop=rng.choice([2.0, 2.0, 0.99]))
    if rng.random() < 0.5:  # blocks of one depth
        c.update(level=rng.randint(0, 2), depth=rng.randint(2, 6))
    else:  # depths 3 to 7
        c.update(level=rng.randint(1, 3), depth=0, nodes=_log_int(rng, 500, 4000))
    c["kind"] = kind
    if kind in ("frame", "orbit", "stream"):
        c["fmt"] = rng.choice(["f32", "f32", "f16", "bf16"])
        c["form"] = rng.choice([0, 0, 1, 16, 17])
    if kind == "orbit":
        c["views"] = rng.randint(1, 6)
    if kind == "stream":
        c["frames"] = rng.randint(1, 6)
    if kind == "mode":
        c["mode"] = rng.choice(sorted(MODES))
    if kind == "part":
        c["via"] = rng.choice(["native", "native", "device", "bricks"])
        c["mode"] = "argb" if c["via"] == "device" else rng.choice(sorted(set(MODES) - {"mip"}))
        c["stop"] = 2.0
    if kind == "adjoint":
        c.update(level=min(c["level"], 1), W=min(c["W"], 512), H=min(c["H"], 512), dist=max(c["dist"], 20.0))
    return c


# ------------------------------------------------------------------------------------------------ inputs

def _depths(case):
    """Depth of every block: one depth, or the benchmark's mix in fixed shares (which block is which is drawn)."""
    nb = 8 ** case["level"]
    if case["depth"]:
        return np.full(nb, case["depth"])
    share = {7: 0.05, 6: 0.15, 5: 0.2, 4: 0.3}
    d = np.full(nb, 3)
    at = 0
    for depth, p in share.items():
        n = max(1, round(nb * p))
        d[at:at + n] = depth
        at += n
    return d


def _octrees(depth, target, gen):
    """Node sets of octrees grown level by level, all blocks at once: (block, x, y, z) of every node, blocks in
    order, each block's nodes in a random order.  target 0: 30 to 70 % of a level's cells are refined; else
    about so many nodes in all."""
    dev = "cuda"
    nb = depth.numel()
    cb = torch.arange(nb, device=dev)
    cells = torch.zeros(nb, 3, dtype=torch.int64, device=dev)
    corner = torch.tensor([[i & 1, (i >> 1) & 1, (i >> 2) & 1] for i in range(8)], device=dev)
    keys = torch.zeros(0, dtype=torch.int64, device=dev)
    for level in range(10):
        p = (cells[:, None, :] + corner) << (depth[cb] - level)[:, None, None]
        k = (cb[:, None] << 30) | (p[..., 2] << 20) | (p[..., 1] << 10) | p[..., 0]
        keys = torch.unique(torch.cat([keys, k.reshape(-1)]))
        live = depth[cb] > level
        cb, cells = cb[live], cells[live]
        if cb.numel() == 0:
            break
        count = torch.bincount(cb, minlength=nb)
        have = torch.bincount(keys >> 30, minlength=nb)
        left = (depth - level).clamp(min=1)
        grown = (target - have).clamp(min=0).double() / (10.0 * left)
        part = (0.3 + 0.4 * torch.rand(nb, device=dev, generator=gen, dtype=torch.float64)) * count
        want = torch.minimum(torch.where(target > 0, grown, part).round().long().clamp(min=1), count)
        order = torch.argsort(torch.rand(cb.numel(), device=dev, generator=gen, dtype=torch.float64) + cb)
        first = torch.cumsum(count, 0) - count
        rank = torch.arange(cb.numel(), device=dev) - first[cb[order]]
        take = order[rank < want[cb[order]]].sort().values
        cb = cb[take].repeat_interleave(8)
        cells = (cells[take][:, None, :] * 2 + corner).reshape(-1, 3)
    b = keys >> 30
    keys = keys[torch.argsort(torch.rand(keys.numel(), device=dev, generator=gen, dtype=torch.float64) + b)]
    return keys >> 30, keys & 1023, (keys >> 10) & 1023, (keys >> 20) & 1023


def _values(u, mask, gen):
    """Eight Gaussian blobs at unit-cube points u; masked nodes: a fifth at random, or those far from the centre."""
    dev = u.device
    c = torch.rand(8, 3, device=dev, generator=gen, dtype=torch.float64)
    s = 0.05 + 0.15 * torch.rand(8, device=dev, generator=gen, dtype=torch.float64)
    a = 2 * torch.rand(8, device=dev, generator=gen, dtype=torch.float64) - 1
    v = torch.zeros(u.shape[0], device=dev, dtype=torch.float64)
    for i in range(8):
        v += a[i] * torch.exp(-((u - c[i]) ** 2).sum(1) / (2 * s[i] ** 2))
    v = v.float()
    if mask == "random":
        v = torch.where(torch.rand(v.numel(), device=dev, generator=gen) < 0.2, NO_FIELD, v)
    elif mask == "sphere":
        v = torch.where(((u - 0.5) ** 2).sum(1) > 0.48 ** 2, NO_FIELD, v)
    return v


def _inputs(case, seed):
    """Blocks, nodes and values of a case, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    if case["kind"] == "block":
        depth = torch.tensor([case["depth"]], device="cuda")
        level, idx = 0, torch.zeros(1, 3, dtype=torch.int64, device="cuda")
        target = torch.full((1,), case["nodes"], device="cuda")
    else:
        level, m = case["level"], 1 << case["level"]
        depth = torch.from_numpy(_depths(case)).cuda()[torch.randperm(m ** 3, device="cuda", generator=gen)]
        i = torch.arange(m ** 3, device="cuda")
        idx = torch.stack([i % m, (i // m) % m, i // (m * m)], 1)
        target = torch.zeros(m ** 3, device="cuda", dtype=torch.int64)
        if case["nodes"]:
            spread = torch.randn(m ** 3, device="cuda", generator=gen).exp()
            target = (case["nodes"] * spread).long().clamp(8)
            target = torch.minimum(target, ((1 << depth) + 1) ** 3)
    b, x, y, z = _octrees(depth, target, gen)
    xyz = torch.stack([x, y, z], 1)
    u = (idx[b] + xyz / (1 << depth[b])[:, None]) / (1 << level)
    vals = _values(u, case["mask"], gen)
    turn = float(torch.rand(1, device="cuda", generator=gen)) * 2 * math.pi
    return {"depth": depth, "idx": idx, "b": b, "xyz": xyz, "vals": vals, "u": u, "turn": turn, "gen": gen}


def _eye(case, turn, k=0):
    r, a = case["dist"], turn + 0.15 * k
    return (r * 0.96 * math.sin(a), r * 0.28, r * 0.96 * math.cos(a))


def _range(vals):
    ok = vals[vals != NO_FIELD]
    lo, hi = (float(ok.min()), float(ok.max())) if ok.numel() else (0.0, 1.0)
    return (lo, hi) if hi > lo else (lo, lo + 1.0)


def _table(n, seed=None):
    if seed is not None:
        return np.random.default_rng(seed).uniform(0.0, 1.0, (n, 4)).astype(np.float32)
    return host.make_color_transfer(*workloads.colormap_points(), n)


def _workload(case, inp):
    counts = torch.bincount(inp["b"], minlength=inp["depth"].numel()).cpu().numpy()
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    blocks = torch.cat([inp["idx"], inp["depth"][:, None]], 1).cpu().numpy().astype(np.uint32)
    n2i = inp["xyz"].to(torch.int16).cpu().numpy().view(np.uint16)
    lo, hi = _range(inp["vals"])
    return workloads.Workload(case["kind"], case["level"], blocks, off, n2i, inp["vals"].cpu().numpy(), lo, hi,
                              case["W"], case["H"], _eye(case, inp["turn"]), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0),
                              case["fovy"], False, 0.0, case["quality"], 0.5, _table(case["tf"]))


_CTX = []


def _context():
    """A program keeps one context per host thread."""
    if not _CTX:
        _CTX.append(Context(0))
    return _CTX[0]


def _presentation(case, w, view):
    span = w.field_max - w.field_min
    levels = [w.field_min + span * t for t in (0.3, 0.45, 0.6, 0.75)]
    return host.presentation(MODES[case["mode"]], view, isosurface_opacity=0.7, levels=levels,
                             secondary_range=(w.field_min, w.field_max))


def _plan(ctx, w, case):
    plan = FramePlan(ctx, w, FORMATS[case.get("fmt", "f32")], render_tile=case.get("form", 0))
    bricks = plan.bricks()[0]  # the rows' padding is never read: the same values in every run
    if plan.fmt == _lib.BRICK_BF16:
        bricks = bricks.view(torch.bfloat16)
    bricks.fill_(float("nan"))
    return plan


def prepare(case, seed):
    inp = _inputs(case, seed)
    ctx = _context()
    kind = case["kind"]
    if kind == "block":
        n2i = to_device_n2i(inp["xyz"].to(torch.int16).cpu().numpy().view(np.uint16))
        return {"kind": kind, "ctx": ctx, "n2i": n2i, "sparse": inp["vals"], "depth": case["depth"]}
    w = _workload(case, inp)
    s = {"kind": kind, "ctx": ctx, "w": w, "sparse": inp["vals"], "fmt": case.get("fmt", "f32")}
    s["tf"] = torch.from_numpy(w.tf).cuda()
    npix = case["W"] * case["H"]
    if kind == "part":
        st = RenderSharedState(w, case["stop"], _lib.FILTER_EXACT if case["via"] == "bricks" else _lib.FILTER_TEXTURE)
        s["worker"] = VsWorker(ctx)
        s["worker"].set_render_shared_state(st)
        s["pres"] = None if case["mode"] == "argb" else _presentation(case, w, st.view)
        m = 1 << case["level"]
        s.update(via=case["via"], level=case["level"], box=((0, 0, 0), (m, m, m)))
        second = "value_on" in case["mode"]
        values2 = _values(inp["u"], case["mask"], inp["gen"])
        if case["via"] == "bricks":
            s["plan"] = _plan(ctx, w, case)
            s["plan"].interp(inp["vals"])
            s["plan2"] = _plan(ctx, w, case) if second else None
            if second:
                s["plan2"].interp(values2)
        elif case["via"] == "device":
            for b in range(w.nblocks):  # node lists and values are resident
                st.device_nodes(b)
        else:
            st.device_all()
            s["sparse2"] = values2 if second else None
        return s
    s["plan"] = _plan(ctx, w, case)
    s["view"] = host.view_for(w, case["stop"])
    if kind == "frame":
        s["rgba"] = torch.zeros(npix * 4, device="cuda")
        s["argb"] = torch.zeros(npix, dtype=torch.int32, device="cuda")
    elif kind == "orbit":
        s["plan"].interp(inp["vals"])
        s["views"] = [host.view_for(w, case["stop"], eye=_eye(case, inp["turn"], k)) for k in range(case["views"])]
        s["rgbas"] = [torch.zeros(npix * 4, device="cuda") for _ in s["views"]]
    elif kind == "mode":
        s["plan"].interp(inp["vals"])
        s["pres"] = _presentation(case, w, s["view"])
        s["plan2"] = None
        if "value_on" in case["mode"]:
            s["plan2"] = _plan(ctx, w, case)
            s["plan2"].interp(_values(inp["u"], case["mask"], inp["gen"]))
        s["argb"] = torch.zeros(npix, dtype=torch.int32, device="cuda")
    elif kind == "adjoint":
        s["plan"].interp(inp["vals"])
        target_tf = torch.from_numpy(_table(case["tf"], seed + 1)).cuda()
        s["target"] = torch.zeros(npix * 4, device="cuda")
        s["plan"].render(s["view"], target_tf, s["target"])
        s["target"] = s["target"].view(case["H"], case["W"], 4)
        s["tf"].requires_grad_()
        s["bricks"] = s["plan"].bricks()[0].requires_grad_()
    elif kind == "stream":
        s["in"], s["out"] = [], []
        for k in range(case["frames"]):
            v = inp["vals"] if k == 0 else _values(inp["u"], case["mask"], inp["gen"])
            s["in"].append(torch.empty(v.shape, pin_memory=True).copy_(v))
            s["out"].append(torch.zeros(npix, dtype=torch.int32, pin_memory=True))
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "block":
        return s["ctx"].interp_dense(s["n2i"], s["sparse"], s["depth"])
    if kind == "frame":
        s["plan"].run(s["view"], s["sparse"], s["tf"], s["rgba"], s["argb"])
        bricks = s["plan"].bricks()[0]
        return {"rgba": s["rgba"], "argb": s["argb"],
                "bricks": bricks.view(torch.bfloat16) if s["fmt"] == "bf16" else bricks}
    if kind == "orbit":
        for view, rgba in zip(s["views"], s["rgbas"]):
            s["plan"].render(view, s["tf"], rgba)
        return s["rgbas"]
    if kind == "mode":
        second = s["plan2"].bricks()[0] if s["plan2"] else None
        s["plan"].render_mode(s["view"], s["pres"], s["tf"], second, None, s["argb"])
        return s["argb"]
    if kind == "part":
        wk, (lo, hi) = s["worker"], s["box"]
        if s["via"] == "native":
            part = wk.render_scene_part_native(s["level"], lo, hi, s["pres"], s["sparse2"])
        elif s["via"] == "device":
            part = wk.render_scene_part_device(s["level"], lo, hi)
        else:
            second = s["plan2"].bricks()[0] if s["plan2"] else None
            part = wk.render_scene_part_plan(s["plan"], s["level"], lo, hi, s["pres"], second)
        w = s["w"]
        return [*part[:2], schedule.final_compose_device(s["ctx"], schedule.DevicePart(*part), w.W, w.H)]
    if kind == "adjoint":
        image = render_frame(s["plan"], s["view"], s["tf"], s["bricks"])
        dtf, dbricks = torch.autograd.grad(image, [s["tf"], s["bricks"]], image.detach() - s["target"])
        return {"rgba": image.detach(), "dtf": dtf, "dbricks": dbricks}
    for v, img in zip(s["in"], s["out"]):
        s["plan"].run_host(s["view"], v, s["tf"], img)
    s["plan"].host_sync()
    return s["out"]


def _brick_elems(case, itemsize):
    e = (1 << _depths(case).astype(np.int64)) + 1
    per = 32 // itemsize
    return int((e * e * ((e + per - 1) // per * per)).sum())


def work(case):
    """Every node (three 16-bit indices and a value) and every brick once, every pixel once.  Operations: for an
    image, eight-corner filtering, table lookup and blend of the samples of a ray through the whole level."""
    if case["kind"] == "block":
        e = 2 ** case["depth"] + 1
        return {"bytes": 10 * min(case["nodes"], e ** 3) + 4 * e ** 3, "flops": 2 * e ** 3}
    depths = _depths(case)
    e = 2.0 ** depths + 1
    nodes = float(np.minimum(1.5 * case["nodes"], e ** 3).sum()) if case["nodes"] else float((0.1 * e ** 3).sum())
    item = 2 if case.get("fmt", "f32") != "f32" else 4
    bricks = item * float((e ** 3).sum())
    npix = case["W"] * case["H"]
    seen = min(1.0, (11.0 / (2 * case["dist"] * math.tan(math.radians(case["fovy"] / 2)))) ** 2 * case["H"] / case["W"])
    image_flops = 60.0 * npix * seen * float(e.mean()) * (1 << case["level"]) * case["quality"]
    kind = case["kind"]
    if kind == "frame":
        return {"bytes": 10 * nodes + bricks + 20 * npix, "flops": 2 * bricks / item + image_flops}
    if kind == "orbit":
        return {"bytes": bricks + 16 * npix * case["views"], "flops": image_flops * case["views"]}
    if kind == "mode":
        return {"bytes": bricks + 4 * npix, "flops": image_flops}
    if kind == "part":
        return {"bytes": (bricks if case["via"] == "bricks" else 10 * nodes) + 4 * npix, "flops": image_flops}
    if kind == "adjoint":
        return {"bytes": 2 * bricks + 48 * npix, "flops": 4 * image_flops}
    return {"bytes": (10 * nodes + 4 * npix) * case["frames"],
            "flops": (2 * bricks / item + image_flops) * case["frames"]}


# ------------------------------------------------------------------------------------------------ 64 bits

def _fill(depth, b, xyz, vals, nb):
    """The dense grids (nb, e, e, e), z slowest, of nb subtrees of one depth: every level's edge, face and cell
    midpoints are the means of two, four and six neighbours where no node defines them."""
    e = (1 << depth) + 1
    g = torch.full((nb, e, e, e), float("nan"), dtype=torch.float64, device="cuda")
    v = vals.double()
    g[b, xyz[:, 2], xyz[:, 1], xyz[:, 0]] = torch.where(vals == NO_FIELD, float("inf"), v)
    for level in range(depth):
        h = 1 << (depth - level - 1)
        for odd in ((1,), (2,), (3,), (1, 2), (1, 3), (2, 3), (1, 2, 3)):
            at = [slice(None)] + [slice(h, None, 2 * h) if a in odd else slice(0, None, 2 * h) for a in (1, 2, 3)]
            total = 0.0
            for a in odd:
                for start in (0, 2 * h):
                    near = list(at)
                    near[a] = slice(start, e - h if start == 0 else None, 2 * h)
                    total = total + g[tuple(near)]
            old = g[tuple(at)]
            g[tuple(at)] = torch.where(torch.isnan(old), total / (2 * len(odd)), old)
    return torch.where(torch.isinf(g), float("nan"), g)


def _bricks64(case, inp, item):
    """Every block's grid, rows padded to whole 32-byte sectors, and per block {first element, pitch}."""
    depth = inp["depth"].cpu().numpy()
    e = (1 << depth.astype(np.int64)) + 1
    per = 32 // item
    pitch = (e + per - 1) // per * per
    off = np.concatenate([[0], np.cumsum(e * e * pitch)])
    out = torch.full((int(off[-1]),), float("nan"), dtype=torch.float64, device="cuda")
    for d in sorted(set(depth.tolist())):
        n, p = (1 << d) + 1, int(pitch[depth == d][0])
        which = np.flatnonzero(depth == d)
        step = max(1, (1 << 31) // (n ** 3 * 64))
        for k in range(0, len(which), step):
            blocks = torch.from_numpy(which[k:k + step]).cuda()
            local = torch.full((depth.size,), -1, dtype=torch.int64, device="cuda")
            local[blocks] = torch.arange(blocks.numel(), device="cuda")
            pick = local[inp["b"]] >= 0
            g = _fill(d, local[inp["b"][pick]], inp["xyz"][pick], inp["vals"][pick], blocks.numel())
            rows = torch.full((blocks.numel(), n, n, p), float("nan"), dtype=torch.float64, device="cuda")
            rows[..., :n] = g
            first = torch.from_numpy(off[which[k:k + step]]).cuda()
            out[first[:, None] + torch.arange(n * n * p, device="cuda")] = rows.reshape(blocks.numel(), -1)
            del g, rows
    return out, torch.from_numpy(off[:-1]).cuda(), torch.from_numpy(pitch).cuda()


def _camera64(case, eye):
    z = np.array(eye) / np.linalg.norm(eye)
    x = np.cross((0.0, 1.0, 0.0), z)
    x /= np.linalg.norm(x)
    y = np.cross(z, x)
    h = 0.2 * math.tan(math.radians(case["fovy"] / 2))
    return np.array(eye), x, y, z, h


def _cast64(case, inp, store, off, pitch, tf, eye, lo, hi):
    """The (H, W, 4) image of a level, rows top to bottom: every pixel's ray through every block whose view
    rectangle holds the pixel, the blocks' samples front to back, the blocks composited front to back."""
    dev, f8 = "cuda", torch.float64
    eye, ex, ey, ez, vh = _camera64(case, eye)
    W, H, m = case["W"], case["H"], 1 << case["level"]
    pix = vh / H
    half = 5.0 / m
    centre = -5.0 + half * (1 + 2 * inp["idx"].double())
    T = lambda a: torch.tensor(a, dtype=f8, device=dev)  # noqa: E731
    rot = torch.stack([T(ex), T(ey), T(ez)])
    corner = T([[i & 1, (i >> 1) & 1, i >> 2] for i in range(8)]) * 2 - 1
    q = ((centre[:, None, :] + half * corner) - T(eye)) @ rot.T
    full = (q[..., 2] >= 0).any(1)
    s = (-q[..., :2] / q[..., 2:] * 0.1 / pix).trunc() + T([W >> 1, H >> 1])
    s = torch.stack([s[..., 0].clamp(0, W - 1), s[..., 1].clamp(0, H - 1)], -1)
    r0, r1 = s.amin(1).long(), s.amax(1).long()
    r0[full] = 0
    r1[full] = torch.tensor([W, H], device=dev)
    size = (r1 - r0).clamp(min=0)
    area = size[:, 0] * size[:, 1]
    blk = torch.repeat_interleave(torch.arange(area.numel(), device=dev), area)
    j = torch.arange(blk.numel(), device=dev) - (torch.cumsum(area, 0) - area)[blk]
    px, py = r0[blk, 0] + j % size[blk, 0].clamp(min=1), r0[blk, 1] + j // size[blk, 0].clamp(min=1)
    u = ((px + 0.5) / W - 0.5) * (pix * W)
    v = ((py + 0.5) / H - 0.5) * vh
    d = -0.1 * T(ez) + u[:, None] * T(ex) + v[:, None] * T(ey)
    c = centre[blk]
    t0, t1 = (c - half - T(eye)) / d, (c + half - T(eye)) / d
    enter = torch.minimum(t0, t1).amax(1).clamp(min=1.0)
    leave = torch.maximum(t0, t1).amin(1)
    keep = leave > enter
    blk, px, py, d, c, enter, leave = (t[keep] for t in (blk, px, py, d, c, enter, leave))
    depth = inp["depth"][blk]
    n = (1 << depth) + 1
    texel = 2 * half / n
    count = (case["quality"] * (leave - enter) * (d * d).sum(1) / (texel * d.abs().sum(1))).trunc()
    step = d * ((leave - enter) / count)[:, None]
    p0 = T(eye) + d * enter[:, None]
    origin = c - (half + 0.5 * texel)[:, None]
    factor = n / (2 * (half + 0.5 * texel))
    expo = 100.0 / ((1 << (depth + case["level"])) * case["quality"])
    base, row = off[blk], pitch[blk]
    gain = 0.5
    acc = torch.zeros(blk.numel(), 4, dtype=f8, device=dev)
    live = torch.arange(blk.numel(), device=dev)
    for k in range(int(count.max()) - 1 if blk.numel() else 0):
        live = live[(count[live] > k + 1) & (acc.detach()[live, 3] <= 0.996)]
        if live.numel() == 0:
            break
        xb = (p0[live] + k * step[live] - origin[live]) * factor[live, None] - 0.5
        fl = xb.floor()
        f = xb - fl
        top = (n[live] - 1)[:, None]
        i0, i1 = torch.minimum(fl.long().clamp(min=0), top), torch.minimum((fl.long() + 1).clamp(min=0), top)
        val, ok = 0.0, torch.ones(live.numel(), dtype=torch.bool, device=dev)
        for o in range(8):
            i = [(i1 if (o >> a) & 1 else i0)[:, a] for a in range(3)]
            t = store[base[live] + (i[2] * n[live] + i[1]) * row[live] + i[0]]
            ok &= ~torch.isnan(t)
            w = math.prod([(f if (o >> a) & 1 else 1 - f)[:, a] for a in range(3)])
            val = val + w * torch.where(torch.isnan(t), 0.0, t)
        g = (val - lo) / (hi - lo) * tf.shape[0] - 0.5
        gl = g.detach().floor()
        a0, a1 = gl.long().clamp(0, tf.shape[0] - 1), (gl.long() + 1).clamp(0, tf.shape[0] - 1)
        col = tf[a0] + (g - gl)[:, None] * (tf[a1] - tf[a0])
        alpha = 1 - (1 - col[:, 3] * gain) ** expo[live]
        wgt = torch.where(ok, (1 - acc[live, 3]) * alpha, 0.0)
        add = torch.cat([wgt[:, None] * col[:, :3], wgt[:, None]], 1)
        acc = acc.index_add(0, live, add) if acc.requires_grad or add.requires_grad else acc.index_add_(0, live, add)
    order = torch.where(d < 0, m - 1 - inp["idx"][blk], inp["idx"][blk]).sum(1)
    out = torch.zeros(H * W, 4, dtype=f8, device=dev)
    at = (H - 1 - py) * W + px
    for k in range(3 * m - 2):
        pick = order == k
        a = at[pick]
        go = out.detach()[a, 3] <= case["stop"]
        a, part = a[go], acc[pick][go]
        add = (1 - out[a, 3:]) * part
        out = out.index_add(0, a, add)
    alpha = out[:, 3:]
    colour = torch.where(alpha > 0, out[:, :3] / torch.where(alpha > 0, alpha, 1.0), 0.0)
    return torch.cat([colour, alpha], 1).view(H, W, 4)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mode", "part", "stream"):
        return None  # whole-number pixels
    inp = _inputs(case, seed)
    if kind == "block":
        z = torch.zeros_like(inp["b"])
        return _fill(case["depth"], z, inp["xyz"], inp["vals"], 1).reshape(-1)
    lo, hi = _range(inp["vals"])
    item = 4 if case.get("fmt", "f32") == "f32" else 2
    store, off, pitch = _bricks64(case, inp, item)
    tf = torch.from_numpy(_table(case["tf"])).cuda().double()
    eye = _eye(case, inp["turn"])
    if kind == "adjoint":
        target = _cast64(case, inp, store, off, pitch, torch.from_numpy(_table(case["tf"], seed + 1)).cuda().double(),
                         eye, lo, hi)
        tf, store = tf.requires_grad_(), store.requires_grad_()
        image = _cast64(case, inp, store, off, pitch, tf, eye, lo, hi)
        dtf, dstore = torch.autograd.grad(image, [tf, store], image.detach() - target)
        return {"rgba": image.detach(), "dtf": dtf, "dbricks": dstore}
    if kind == "orbit":
        return [_cast64(case, inp, store, off, pitch, tf, _eye(case, inp["turn"], k), lo, hi).reshape(-1)
                for k in range(case["views"])]
    rgba = _cast64(case, inp, store, off, pitch, tf, eye, lo, hi).reshape(-1)
    if item == 2:  # stored as (value - minimum) / range of each block's nodes
        nb = off.numel()
        ok = inp["vals"] != NO_FIELD
        b, v = inp["b"][ok], inp["vals"][ok].double()
        least = torch.full((nb,), float("inf"), dtype=torch.float64, device="cuda").scatter_reduce(0, b, v, "amin")
        most = torch.full((nb,), float("-inf"), dtype=torch.float64, device="cuda").scatter_reduce(0, b, v, "amax")
        least, span = torch.where(torch.isinf(least), 0.0, least), most - least
        span = torch.where((span > 0) & torch.isfinite(span), span, 1.0)
        size = torch.diff(torch.cat([off, torch.tensor([store.numel()], device="cuda")]))
        owner = torch.repeat_interleave(torch.arange(nb, device="cuda"), size)
        store = (store - least[owner]) / span[owner]
    return {"rgba": rgba, "argb": None, "bricks": store}
