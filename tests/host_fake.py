"""The library's host side on a stand-in for the CUDA runtime (tests/host/fake_cuda.cpp): plans, contexts and calls as
on a GPU, with every kernel's accesses checked for order, lifetime and extent instead of carried out."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np

from revise_gb300 import _lib, host, workloads
from revise_gb300.build import cuda_home

ROOT = Path(__file__).resolve().parents[1]
vp = C.c_void_p


def build(out: Path) -> C.CDLL:
    csrc = ROOT / "revise_gb300" / "csrc"
    # -Bsymbolic: the stand-in's own functions, whatever runtime the process has loaded besides
    cmd = ["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wl,-Bsymbolic",
           "-I", str(ROOT / "include"), "-I", str(csrc), "-I", str(cuda_home() / "include"),
           str(ROOT / "tests" / "host" / "fake_cuda.cpp"), str(csrc / "host.cpp"), "-o", str(out)]
    subprocess.run(cmd, check=True)
    lib = _lib.load(out)
    lib.fake_trouble.restype = C.c_char_p
    lib.fake_calls.argtypes = [C.c_char_p]
    for f in (lib.fake_used, lib.fake_peak):
        f.restype = C.c_uint64
    lib.fake_limit.argtypes = [C.c_uint64]
    return lib


class Machine:
    """A context on the stand-in."""

    def __init__(self, lib):
        self.lib = lib
        h = vp()
        assert lib.s3r_ctx_create(0, C.byref(h)) == 0
        self.h = h
        lib.fake_reset()
        self._keep = []

    def close(self):
        self.lib.s3r_ctx_destroy(self.h)
        self.lib.fake_reset()

    def ok(self, rc):
        assert rc == 0, self.lib.s3r_last_error(self.h).decode()

    def trouble(self):
        return self.lib.fake_trouble().decode().split("\n")[:-1]

    def calls(self, name):
        return self.lib.fake_calls(name.encode())

    def buffer(self, n, dtype=np.float32):
        a = np.zeros(n, dtype)
        self._keep.append(a)
        return vp(a.ctypes.data)

    def stream(self):
        s = vp()
        assert self.lib.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        return s

    def capture(self, stream, body):
        """The graph, ready to launch, of what body() queues on `stream`."""
        g, x = vp(), vp()
        assert self.lib.cudaStreamBeginCapture(stream, 0) == 0
        body()
        assert self.lib.cudaStreamEndCapture(stream, C.byref(g)) == 0
        assert self.lib.cudaGraphInstantiate(C.byref(x), g, C.c_ulonglong(0)) == 0
        return x

    def launch(self, graph, stream):
        assert self.lib.cudaGraphLaunch(graph, stream) == 0

    def plan(self, w, render_tile=0, fmt=_lib.BRICK_F32):
        d = _lib.FrameDesc()
        blocks, off, n2i = (np.ascontiguousarray(a, t) for a, t in ((w.blocks, np.uint32), (w.node_off, np.uint64),
                                                                     (w.n2i, np.uint16)))
        d.level, d.nblocks, d.brick_format, d.tile_cells, d.render_tile = w.level, blocks.shape[0], fmt, 16, render_tile
        d.blocks, d.node_off, d.n2i = _lib.arr(blocks, C.c_uint32), _lib.arr(off, C.c_uint64), _lib.arr(n2i, C.c_uint16)
        h = vp()
        self.ok(self.lib.s3r_frame_plan(self.h, C.byref(d), C.byref(h)))
        return h

    def part(self, w, view, pres=None, stream=None):
        """s3r_render_scene_part of the whole level; returns the rectangle."""
        wb = _lib.WorkerBlocks()
        blocks, off = np.ascontiguousarray(w.blocks, np.uint32), np.ascontiguousarray(w.node_off, np.uint64)
        self._keep += [blocks, off]
        wb.nblocks, wb.blocks, wb.node_off = blocks.shape[0], _lib.arr(blocks, C.c_uint32), _lib.arr(off, C.c_uint64)
        wb.n2i, wb.sparse, wb.sparse2 = self.buffer(3 * w.nodes, np.uint16), self.buffer(w.nodes), self.buffer(w.nodes)
        lo, hi, rect = (C.c_uint32 * 3)(0, 0, 0), (C.c_uint32 * 3)(*[1 << w.level] * 3), (C.c_int32 * 4)()
        self.ok(self.lib.s3r_render_scene_part(self.h, C.byref(view), C.byref(pres) if pres is not None else None,
                                               C.byref(wb), lo, hi, self.buffer(4 * view.tf_n),
                                               self.buffer(view.W * view.H, np.uint32), rect, stream))
        return rect[:]

    def render(self, plan, view, stream=None, image=None):
        self.ok(self.lib.s3r_frame_render(self.h, plan, C.byref(view), self.buffer(4 * view.tf_n),
                                          None, image or self.buffer(view.W * view.H, np.uint32), None, stream))


def coarse_set(level, depth=0, W=160, H=120, quality=1.0):
    """Every block of a level, each of one depth with its 8 corners as nodes."""
    m, e = 1 << level, 1 << depth
    i = np.arange(m ** 3)
    blocks = np.stack([i % m, i // m % m, i // (m * m), np.full_like(i, depth)], 1).astype(np.uint32)
    corners = np.array([[q & 1, q >> 1 & 1, q >> 2] for q in range(8)], np.uint16) * e
    w = workloads.small(seed=1, level=0, depths=(1,), W=W, H=H)
    w.level, w.blocks, w.quality = level, blocks, quality
    w.node_off = (8 * np.arange(m ** 3 + 1)).astype(np.uint64)
    w.n2i = np.tile(corners, (m ** 3, 1))
    w.sparse = np.zeros(8 * m ** 3, np.float32)
    return w


def view_of(w, **kw):
    return host.view_for(w, **kw)
