"""Drop-in for the reference's erosion module, variant 3 (the one nixis.py
calls, nixis.py:410), plus the steepest-descent rule of find_lowest.

State on the GPU is binary32 pairs (hi + lo) with a per-planet power-of-two
scale (exact, see csrc/nx_erosion.cu); results are returned in the reference's float64
arrays, updated in place like the reference.
"""
import contextlib
import ctypes
import math

import numpy as np
import torch

from . import _dev
from . import autotune as _autotune
from . import mesh as _mesh
from ._lib import ErosionPlanet, NxError, call, lib

RAIN = 0.3 / 320            # erosion.py:182
EVAPORATION = 0.1 / 320     # erosion.py:205
SOLUBILITY = 0.01 / 320     # erosion.py:206
CAPACITY = 0.2 / 320        # erosion.py:207

# A run over an icosphere's own neighbour table takes the temporally blocked
# passes from this many vertex-iterations on, and from BLOCKED_ITERS
# iterations (ErosionRun.blocked).  They cost the tiling and ~300 us of host
# work, and save 16 us per million vertex-iterations where the state and the
# tables are larger than L2 (from ~800,000 vertices on), 2-6 below.  The line
# is where they pay at every size.  Measured (GB300, erode_terrain3 one
# iteration at a time against blocked, us), at it: 36,002 vertices x 1,000
# 6,420 / 4,733; 100,002 x 336 2,840 / 2,490; 225,002 x 150 1,787 / 1,480;
# 256,002 x 132 1,667 / 1,644; 400,002 x 84 1,466 / 1,417; 625,002 x 54 1,391 /
# 1,330; 1,024,002 x 33 1,613 / 1,308; 6,400,002 x 6 2,101 / 1,840; 10,000,002 x
# 5 2,940 / 2,444; below it: 256,002 x 50 765 / 983, 400,002 x 50 973 / 1,058,
# 1,024,002 x 16 924 / 941, 2,500,002 x 5 939 / 1,006 (from 1,000,000 vertices on
# they would pay from 2e7 on: 1,600,002 x 12 1,049 / 1,023, 2,500,002 x 8 1,152 /
# 1,102, 6,400,002 x 3 1,581 / 1,547).
# A pass rescales its planet before its iterations, not between them, for a
# growth below 16 per iteration: water grows by up to 2 + 6 d, so edges
# longer than BLOCKED_EDGE (a sphere in metres) go one iteration at a time.
BLOCKED_WORK = 1 << 25
BLOCKED_ITERS = 5
BLOCKED_EDGE = 2.0


class ErosionRun:
    """Resident erosion state of one planet (binary32 pairs).

    verts float64 (N,3) and neighbors int32 (N,6) as CUDA tensors (or
    numpy); fields are loaded from float64 heights / water / sediment.
    `iters`, if given, is the length of the run to come: where blocked passes
    pay for it, the table is compared with the icosphere's own."""

    def __init__(self, verts, neighbors, edge=None, stream=None, iters=0):
        self.stream = stream
        self.xyz = _dev.to_device(verts, np.float64, name="verts")
        _dev.check_vertices(self.xyz)
        self.n = self.xyz.shape[0]
        self.nbr = _dev.to_device(neighbors, np.int32, (self.n, 6), "neighbors")
        n = self.n
        with self._on_stream():
            # None: not the icosphere's own table, edges too long, or not worth finding out
            self.k = (self._icosphere_divisions()
                      if edge is None and iters >= BLOCKED_ITERS and iters * n >= BLOCKED_WORK else None)
            if edge is None and self.k is None:
                edge, err = _mesh.edge_lengths(self.xyz, self.nbr, stream=stream)
                bad = err.item()
            elif edge is None:
                edge = torch.empty((n, 6, 2), dtype=torch.float32, device="cuda")
                info = torch.zeros(2, dtype=torch.int32, device="cuda")
                call("nx_icosphere_edges", self.k, _dev.ptr(self.xyz), _dev.ptr(self.nbr), _dev.ptr(edge), _dev.ptr(info),
                     _dev.stream_handle(stream))
                info = info.cpu()
                bad = int(info[0])
                if not float(info.view(torch.float32)[1]) <= BLOCKED_EDGE:
                    self.k = None
            else:
                bad = 0
            if bad:
                raise IndexError("neighbors holds an id outside [-1, N)")
        self.edge = edge
        self.st = torch.empty((n, 8), dtype=torch.float32, device="cuda")    # (h, w, s as hi/lo pairs, 0, 0)
        self.st_tmp = torch.empty_like(self.st)
        self.ws = torch.zeros(int(lib().nx_erosion_workspace_size(n, 1)), dtype=torch.uint8, device="cuda")
        self.planet = torch.zeros(ctypes.sizeof(ErosionPlanet), dtype=torch.uint8, device="cuda")  # one descriptor
        self.iters_done = 0

    def _on_stream(self):
        """The run's stream as the current one, so that what the host reads
        back is ordered behind the run's kernels."""
        return torch.cuda.stream(self.stream) if self.stream is not None else contextlib.nullcontext()

    def _icosphere_divisions(self):
        """k if the neighbour table's face-interior rows are those of this
        library's icosphere of k divisions (the vertices may be any)."""
        k = math.isqrt(max(0, (self.n - 2) // 10))
        if k < 2 or 10 * k * k + 2 != self.n or self.nbr.data_ptr() % 8:
            return None
        _mesh._ensure_tables()
        differ = torch.zeros(1, dtype=torch.int32, device="cuda")
        call("nx_icosphere_like", k, _dev.ptr(self.nbr), _dev.ptr(differ), _dev.stream_handle(self.stream))
        return None if int(differ.item()) else k

    def load(self, heights, water=None, sediment=None):
        h = _dev.to_device(heights, np.float64, (self.n,), "heights")
        w = None if water is None else _dev.to_device(water, np.float64, (self.n,), "water")
        s = None if sediment is None else _dev.to_device(sediment, np.float64, (self.n,), "sediment")
        call("nx_erosion_load", _dev.ptr(h), _dev.ptr(w), _dev.ptr(s), self.n, _dev.ptr(self.st),
             _dev.ptr(self.ws), self.ws.numel(), _dev.stream_handle(self.stream))
        self.iters_done = 0
        return self

    def steps(self, iters, rain=0.0, mass=False, flow=False):
        """Run `iters` iterations; returns (mass float64 (iters,3) or None,
        flow uint16 (N,) of the last iteration or None)."""
        iters = int(iters)
        m = torch.empty((max(iters, 1), 3), dtype=torch.float64, device="cuda") if mass else None
        f = torch.zeros(self.n, dtype=torch.int16, device="cuda") if flow else None
        call("nx_erosion_steps", _dev.ptr(self.nbr), _dev.ptr(self.edge), self.n, _dev.ptr(self.st),
             _dev.ptr(self.st_tmp), iters, float(rain), _dev.ptr(self.planet), _dev.ptr(m), _dev.ptr(f),
             _dev.ptr(self.ws), self.ws.numel(), _dev.stream_handle(self.stream))
        self.iters_done += iters
        return (m[:iters] if mass else None), f

    def blocked(self, iters, rain=0.0):
        """Run `iters` iterations as temporally blocked passes (the same bits
        as steps, which read the state and the tables once per iteration
        instead of once per pass); False, and nothing done, where the table
        is not known to be an icosphere's (see __init__) or the tiling does
        not fit."""
        iters = int(iters)
        if self.k is None or iters < 1:
            return False
        tb = _autotune.current()
        if tb.variant not in (0, 1, 4, 5):
            return False
        with self._on_stream():
            try:
                tl = _mesh.MeshTiling(self, tb.tile_side, tb.rings, self.stream)
                d = ErosionPlanet(0, self.n, self.nbr.data_ptr(), self.edge.data_ptr(), iters, float(rain), 0, 0,
                                  tl.dev.data_ptr(), tl.ntiles, tl.maxnl, tl.maxc)
                ws = torch.empty(int(lib().nx_erosion_workspace_size(max(self.n, 256 * tl.ntiles), 1)), dtype=torch.uint8,
                                 device="cuda")
            except RuntimeError:                     # too large a tile, or out of memory
                return False
            ws[:32].copy_(self.ws[:32])
            self.planet.copy_(torch.frombuffer(bytearray(bytes(d)), dtype=torch.uint8))
            # the state enters in the buffer that the number of passes asks for and ends in buffer 0
            st = (self.st, self.st_tmp) if -(-iters // tb.rings) % 2 == 0 else (self.st_tmp, self.st)
            try:
                call("nx_erosion_run_as", _dev.ptr(self.planet), ctypes.byref(d), 1, tb.rings, tb.threads, tb.variant,
                     _dev.ptr(st[0]), _dev.ptr(st[1]), _dev.ptr(ws), ws.numel(), _dev.stream_handle(self.stream))
            except NxError as e:
                if e.code != 1:                      # NX_EINVAL: refused before any launch (the tiles do not fit)
                    raise
                return False
            self.st, self.st_tmp = st
            self.ws, self.tiling = ws, tl            # (in use until the run's stream has passed them)
        self.iters_done += iters
        return True

    def store(self, heights, water=None, sediment=None):
        """Write the state as float64 true values into the given CUDA tensors."""
        call("nx_erosion_store", _dev.ptr(self.st), self.n, _dev.ptr(self.ws),
             _dev.ptr(heights), _dev.ptr(water), _dev.ptr(sediment), _dev.stream_handle(self.stream))

    def scale_exponent(self):
        return int(self.ws[:32].view(torch.int32)[3].item())

    def check(self):
        if self.error():
            raise IndexError("neighbors holds an id outside [-1, N)")

    def error(self):
        """The run's flag: 1 an id out of range, 2 or 3 a tiling that does
        not suit the passes."""
        with self._on_stream():
            return int(self.ws[:32].view(torch.int32)[6].item())


def erosion_iteration3(verts, neighbors, r_buff, wat, sed):
    """erosion.erosion_iteration3 (erosion.py:197-279): one Jacobi step;
    r_buff (heights), wat and sed are updated in place."""
    _run_inplace(verts, neighbors, r_buff, wat, sed, 1, 0.0, with_fields=True)


def erode_terrain3(nodes, neighbors, heights, num_iter=1, snapshot=False):
    """erosion.erode_terrain3 (erosion.py:172-192): num_iter <= 0 runs once;
    water and sediment start at zero and 0.3/320 of rain is added before
    each iteration; heights are updated in place.  Per-iteration PNG
    snapshots (image export) are not part of this library."""
    if snapshot:
        raise NotImplementedError("erosion snapshots (PNG export) are not provided by nixis_gb300")
    if num_iter <= 0:
        num_iter = 1
    _run_inplace(nodes, neighbors, heights, None, None, int(num_iter), RAIN, with_fields=False)


def _run_inplace(verts, neighbors, h, w, s, iters, rain, with_fields):
    host = _dev.is_host(h)
    for a in (h, w, s):
        if a is None:
            continue
        if host and (not isinstance(a, np.ndarray) or a.dtype != np.float64 or not a.flags.c_contiguous):
            raise ValueError("fields must be C-contiguous float64 arrays")
    if len(verts) == 0:
        # the reference's loop over vertices runs zero times
        for a, name in ((h, "heights"), (w, "water"), (s, "sediment")):
            if a is not None and tuple(a.shape) != (0,):
                raise ValueError(f"{name}: expected shape (0,), got {tuple(a.shape)}")
        return
    # (host fields before the run zeroes its workspace: a busy stream has them staged)
    hd, wd, sd = (_dev.to_device(a, np.float64) if host and a is not None else a for a in (h, w, s))
    run = ErosionRun(verts, neighbors, iters=iters)
    hd = _dev.to_device(hd, np.float64, (run.n,), "heights")
    wd = _dev.to_device(wd, np.float64, (run.n,), "water") if w is not None else None
    sd = _dev.to_device(sd, np.float64, (run.n,), "sediment") if s is not None else None
    run.load(hd, wd, sd)
    done = run.blocked(iters, rain)
    if done and run.error() > 1:
        run.load(hd, wd, sd)
        done = False
    if not done:
        run.steps(iters, rain=rain)
    run.check()
    if with_fields:
        run.store(hd, wd, sd)
    else:
        run.store(hd)
    if host:
        _dev.to_host(h, hd)
        if w is not None:
            _dev.to_host(w, wd)
            _dev.to_host(s, sd)
    else:
        for dst, src in ((h, hd), (w, wd), (s, sd)):
            if dst is not None and dst.data_ptr() != src.data_ptr():
                dst.copy_(src)


def find_lowest(vert, nbr, height):
    """erosion.find_lowest (erosion.py:398-406) for one vertex (host rule)."""
    alts = [height[i] for i in nbr if i != -1]
    lowest = min(alts)
    if lowest < height[vert]:
        return alts.index(lowest)
    return None


def steepest_descent(neighbors, heights, stream=None):
    """find_lowest for every vertex on the GPU: (pos int32 (N,), vid int32
    (N,)); pos is the reference's return value (-1 for None), vid the
    neighbour id it designates."""
    nb = _dev.to_device(neighbors, np.int32, name="neighbors")
    h = _dev.to_device(heights, np.float64, name="heights")
    n = nb.shape[0]
    pos = torch.empty(n, dtype=torch.int32, device="cuda")
    vid = torch.empty(n, dtype=torch.int32, device="cuda")
    call("nx_steepest_descent", _dev.ptr(nb), _dev.ptr(h), n, _dev.ptr(pos), _dev.ptr(vid), _dev.stream_handle(stream))
    return pos, vid


__all__ = ["erosion_iteration3", "erode_terrain3", "find_lowest", "steepest_descent", "ErosionRun",
           "ErosionPlanet", "RAIN", "EVAPORATION", "SOLUBILITY", "CAPACITY"]
