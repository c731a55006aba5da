"""The work whose speed is measured: what a program that uses this framework has it do.

A case is one call (or one short sequence of calls) of a program's, through the public entry points, over the sizes
of this repository's configurations, tests and benchmark: spheres of a few thousand to tens of millions of vertices, 4-12
octaves, up to 100 erosion iterations.  ``exact`` gives what the outputs would be in binary64, in plain torch.
"""
import math

import numpy as np
import torch

from nixis_gb300 import climate, erosion, mesh, opensimplex, planets, serve, terrain, util

EARTH = 6378100.0            # the driver program's world radius (m)
TILT = 23.44


def listed():
    return [
        # the smallest noise call (a preview sphere of 1,442 vertices): its latency
        dict(name="noise_preview", op="noise", k=12, octaves=4, radius=1.0, out="f64"),
        # the driver program's noise: its octaves, lacunarity 2.5 and radius (scales that are no powers of two)
        dict(name="noise_driver", op="noise", k=250, octaves=7, radius=EARTH, out="f64"),
        # a full-size planet's 12 octaves in binary32
        dict(name="noise_large_f32", op="noise", k=1000, octaves=12, radius=1.0, out="f32"),
        # the drop-in erosion loop on a full-size planet that is resident on the GPU
        dict(name="erode_large", op="erode", k=1000, iters=50),
        # the driver program from mesh to map on ordinary host arrays: mesh, noise, shaping, adjacency, erosion, insolation, map
        dict(name="driver_host", op="driver", k=160, iters=11, width=1024),
        # a batch of planets of uneven size, half of them with insolation: the headline's path, replayed as one graph
        dict(name="batch_mixed", op="batch", count=16, k_lo=100, k_hi=800, iters_hi=100, pick=7),
        # one very large planet with a year of insolation through the same path
        dict(name="planet_large", op="batch", count=1, k_lo=2000, k_hi=2000, iters_hi=60, pick=0),
        # a server with requests of log-uniform size that arrive together, results in host arrays
        dict(name="serve_burst", op="serve", count=16, k_lo=50, k_hi=1000, iters_hi=100, pick=11),
        # a year of hourly sun positions
        dict(name="insolation_year", op="year", k=1000, days=365),
        # a day of one-degree rotations on an ordinary sphere
        dict(name="insolation_day", op="day", k=500),
        # the first planet of a subdivision that is not resident: mesh, adjacency, edge lengths, tiling, then a short planet
        dict(name="new_size", op="new_size", k=700, octaves=4, iters=4),
        # the post-noise shaping of a large planet's heights
        dict(name="shape_heights", op="shape", k=800),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["noise", "noise", "erode", "erode", "driver", "batch", "batch", "planet", "serve", "year", "day", "new_size", "shape"])
    if op == "noise":
        return dict(op=op, k=size(12, 1000), octaves=rng.randint(4, 12), radius=rng.choice([1.0, EARTH]),
                    out=rng.choice(["f64", "f64", "f32"]))
    if op == "erode":
        return dict(op=op, k=size(30, 1000), iters=rng.randint(1, 50))
    if op == "driver":
        return dict(op=op, k=size(40, 160), iters=rng.randint(5, 15), width=2 * rng.randint(128, 512))
    if op == "batch":
        return dict(op=op, count=rng.randint(2, 8), k_lo=100, k_hi=rng.randint(300, 700), iters_hi=rng.randint(20, 80), pick=rng.randint(0, 999))
    if op == "planet":
        k = size(100, 1600)
        return dict(op="batch", count=1, k_lo=k, k_hi=k, iters_hi=60, pick=rng.randint(0, 999))
    if op == "serve":
        return dict(op=op, count=rng.randint(4, 14), k_lo=50, k_hi=800, iters_hi=100, pick=rng.randint(0, 999))
    if op == "year":
        return dict(op=op, k=size(50, 1000), days=rng.choice([365, 365, rng.randint(100, 500)]))
    if op == "day":
        return dict(op=op, k=size(50, 700))
    if op == "new_size":
        return dict(op=op, k=size(50, 900), octaves=rng.randint(4, 6), iters=rng.randint(1, 8))
    return dict(op=op, k=size(50, 900))


# What a program has before the call ------------------------------------------------------------------------------

def _requests(case, seed):
    """Planets of the case: sizes from its own draw (`pick`), noise seeds from `seed`; every second with insolation."""
    r = np.random.default_rng(case["pick"])
    n, lo, hi = case["count"], case["k_lo"], case["k_hi"]
    if case["op"] == "serve":
        ks = np.round(np.exp(r.uniform(np.log(lo), np.log(hi), n))).astype(int)
    else:
        ks = r.integers(lo, hi + 1, n)
    octaves = r.integers(4, 13, n) if n > 1 else [12]
    iters = r.integers(0, case["iters_hi"] + 1, n) if n > 1 else [case["iters_hi"]]
    return [planets.PlanetRequest(seed=seed + i, divisions=int(ks[i]), octaves=int(octaves[i]), erosion_iters=int(iters[i]),
                                  insolation=i % 2 == 0) for i in range(n)]


def _noise_args(case):
    """sample_octaves' octaves, first frequency and strength, lacunarity, persistence, radius."""
    if case["radius"] == 1.0:
        return case["octaves"], 1.0, 1.0, 2.0, 0.5, 1.0
    return case["octaves"], 1.5, 0.4, 2.5, 0.5, case["radius"]


def _day_tilt(seed):
    return TILT - 0.37 * (seed % 61)


def _terrain(xyz, seed):
    """Heights as the pipeline has them after the noise: 8 octaves on the sphere (an input, not the timed work)."""
    perm, pgi = opensimplex.init(seed)
    return terrain.sample_octaves(xyz, None, perm, pgi, 8, 1.0, 1.0, 2.0, 0.5, 1.0)


def prepare(case, seed):
    op, s = case["op"], {"case": case, "seed": seed}
    if op in ("noise", "year", "day"):
        xyz, _ = mesh.icosphere(case["k"], with_tris=False)
        if op == "noise":
            perm, pgi = opensimplex.init(seed)
            s.update(xyz=xyz * case["radius"], perm=torch.from_numpy(perm).cuda(), pgi=torch.from_numpy(pgi).cuda())
        else:
            s["radius"] = 1.0 + 0.25 * (seed % 7)
            s["xyz"] = xyz * s["radius"]
            s["tilt"] = _day_tilt(seed)
    elif op == "erode":
        m = mesh.PlanetMesh(case["k"])
        s.update(xyz=m.xyz, nbr=m.nbr, height=util.rescale(_terrain(m.xyz, seed), -4000.0, 8850.0))
    elif op == "batch":
        s["batch"] = planets.PlanetBatch(_requests(case, seed))
        s["batch"].capture()
    elif op == "serve":
        s["engine"] = serve.ServeEngine(hbm_budget=16 * 2**30, slots=256, host_bytes=2**29).warmup()
        s["stream"] = [(0.0, r) for r in _requests(case, seed)]
    elif op == "new_size":
        s["request"] = planets.PlanetRequest(seed=seed, divisions=case["k"], octaves=case["octaves"], erosion_iters=case["iters"])
    elif op == "shape":
        xyz, _ = mesh.icosphere(case["k"], with_tris=False)
        s["height"] = _terrain(xyz, seed)
    elif op != "driver":
        raise ValueError(op)
    return s


# The calls -------------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    op = case["op"]
    if op == "noise":
        if case["out"] == "f64":
            return terrain.sample_octaves(s["xyz"], None, s["perm"], s["pgi"], *_noise_args(case))
        n, f, a, lac, pers, radius = _noise_args(case)
        scale, strength = [f * lac**o / radius for o in range(n)], [a * pers**o / radius for o in range(n)]
        return terrain.fbm(s["xyz"], s["perm"], s["pgi"], scale, strength, radius, out_dtype=torch.float32)[0]
    if op == "erode":
        height = s["height"].clone()            # erosion works in place; the program keeps the uneroded heights
        erosion.erode_terrain3(s["xyz"], s["nbr"], height, num_iter=case["iters"])
        return height
    if op == "driver":
        return _driver(case["k"], s["seed"], case["iters"], case["width"])
    if op == "batch":
        s["batch"].run()
        got = s["batch"].results()
        return {"heights": [r.heights for r in got], "insolation": [r.insolation for r in got]}
    if op == "serve":
        got = s["engine"].run(s["stream"], realtime=False)
        s["engine"].done = []
        return {"heights": [t.heights for t in got], "insolation": [t.insolation for t in got]}
    if op == "year":
        return climate.annual_insolation(s["xyz"], s["radius"], s["tilt"], 365, case["days"], 24, mean_wm2=True)
    if op == "day":
        return climate.brute_daily_insolation(s["xyz"], None, s["radius"], s["tilt"])
    if op == "new_size":
        held = mesh.MeshCache()
        got = planets.generate_plain(s["request"], held, sync=False, blocked=True)
        m = held.get(case["k"])
        return {"heights": got.heights, "xyz": m.xyz, "nbr": m.nbr, "edge": m.edge}
    height, ocean, level = util.shape_heights(s["height"], -4000.0, 8850.0, 55.0)
    return {"height": height, "ocean": ocean, "level": level}


def _driver(k, seed, iters, width):
    """The driver program's steps with its defaults, numpy arrays throughout."""
    points, cells = util.create_mesh(k)
    points *= EARTH
    perm, pgi = opensimplex.init(seed)
    height = terrain.sample_octaves(points, None, perm, pgi, 7, 1.5, 0.4, 2.5, 0.5, EARTH)
    height, ocean, _ = util.shape_heights(height, -4000.0, 8850.0, 55.0)
    neighbors = util.build_adjacency(cells)
    util.sort_adjacency(neighbors)
    erosion.erode_terrain3(points, neighbors, height, num_iter=iters)
    insolation = climate.calc_instant_insolation(points, height, EARTH, 0.0, TILT)
    gray = util.equirect_map(points, neighbors, k, util.rescale(height, 0.0, 65535.0), width, width // 2, EARTH)
    return {"height": height, "insolation": insolation, "neighbors": neighbors, "ocean": ocean, "points": points,
            "map": gray}


# Bytes (each input read once, each output written once) and operations of a pass --------------------------------

NOISE_FLOPS = 160            # per vertex and octave: a binary64 noise3d's executed path
ERODE_FLOPS = 60             # per vertex and iteration: six neighbours' sums, the capacity test


def _planet_work(r):
    n = r.n_vertices
    mesh_bytes = 24 * n + ((24 + 48) * n if r.erosion_iters else 0)
    return (mesh_bytes + 8 * n + (4 * n if r.insolation else 0),
            n * (NOISE_FLOPS * r.octaves + ERODE_FLOPS * r.erosion_iters + (150 if r.insolation else 0)))


def work(case):
    op = case["op"]
    if op in ("batch", "serve"):
        w = [_planet_work(r) for r in _requests(case, 0)]
        return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}
    n = 10 * case["k"] ** 2 + 2
    if op == "noise":
        return {"bytes": n * (24 + (8 if case["out"] == "f64" else 4)), "flops": n * NOISE_FLOPS * case["octaves"]}
    if op == "erode":
        return {"bytes": n * (24 + 24 + 8 + 8), "flops": n * ERODE_FLOPS * case["iters"]}
    if op == "driver":
        pixels = case["width"] * (case["width"] // 2)
        return {"bytes": n * (24 + 8 + 1 + 24 + 4) + 4 * pixels, "flops": n * (7 * NOISE_FLOPS + ERODE_FLOPS * case["iters"] + 100) + 300 * pixels}
    if op == "year":
        return {"bytes": 28 * n, "flops": 150 * n}
    if op == "day":
        return {"bytes": 28 * n, "flops": 60 * n}
    if op == "new_size":  # vertices, neighbours and edge pairs, the tiling's copy of the last two, heights
        return {"bytes": n * (24 + 24 + 48 + 4 + 12 + 48 + 8), "flops": n * (120 + NOISE_FLOPS * case["octaves"] + ERODE_FLOPS * case["iters"])}
    return {"bytes": n * (8 + 8 + 1), "flops": 30 * n}


# The outputs in binary64, in plain torch -------------------------------------------------------------------------

def exact(case, seed):
    op = case["op"]
    if op == "noise":
        xyz = _sphere(case["k"])[0] * case["radius"]
        return _fbm(xyz, _tables(seed), *_noise_args(case))
    if op == "erode":
        xyz, nbr = _sphere(case["k"])
        h = _rescale(_fbm(xyz, _tables(seed), 8, 1.0, 1.0, 2.0, 0.5, 1.0), -4000.0, 8850.0)
        return _erode(xyz, nbr, h, case["iters"], 0.0, 0.3 / 320)
    if op == "driver":
        xyz, nbr = _sphere(case["k"])
        xyz = xyz * EARTH
        h, _, _ = _shape(_fbm(xyz, _tables(seed), 7, 1.5, 0.4, 2.5, 0.5, EARTH))
        h = _erode(xyz, nbr, h, case["iters"], 0.0, 0.3 / 320)
        return {"height": h, "insolation": _insolation(xyz, EARTH, [0.0], [TILT]), "neighbors": None, "ocean": None, "points": xyz, "map": None}
    if op in ("batch", "serve"):
        heights, inso = [], []
        for r in _requests(case, seed):
            xyz, nbr = _sphere(r.divisions)
            h = _rescale(_fbm(xyz, _tables(r.seed), r.octaves, 1.0, 1.0, 2.0, 0.5, 1.0), -8000.0, 8000.0)
            heights.append(_erode(xyz, nbr, h, r.erosion_iters, 1e-3, 0.0))
            inso.append(_year(xyz, 1.0, TILT, 365) if r.insolation else None)
            del xyz, nbr, h
        if op == "serve":
            heights, inso = [h.cpu().numpy() for h in heights], [None if i is None else i.cpu().numpy() for i in inso]
        return {"heights": heights, "insolation": inso}
    if op in ("year", "day"):
        radius, tilt = 1.0 + 0.25 * (seed % 7), _day_tilt(seed)
        xyz = _sphere(case["k"])[0] * radius
        if op == "year":
            return _year(xyz, radius, tilt, case["days"])
        return _insolation(xyz, radius, [-180.0 + i for i in range(360)], [tilt])
    if op == "new_size":
        xyz, nbr = _sphere(case["k"])
        h = _rescale(_fbm(xyz, _tables(seed), case["octaves"], 1.0, 1.0, 2.0, 0.5, 1.0), -8000.0, 8000.0)
        d = _lengths(xyz, nbr)
        hi = d.float().double()
        return {"heights": _erode(xyz, nbr, h, case["iters"], 1e-3, 0.0), "xyz": xyz, "nbr": None, "edge": torch.stack([hi, d - hi], 2)}
    h, _, level = _shape(_fbm(_sphere(case["k"])[0], _tables(seed), 8, 1.0, 1.0, 2.0, 0.5, 1.0))
    return {"height": h, "ocean": None, "level": level.reshape(1)}


DEVICE = "cuda"
CHUNK = 1 << 21
_PHI = (1.0 + 5.0**0.5) / 2.0
_CORNERS = [(-1, _PHI, 0), (1, _PHI, 0), (-1, -_PHI, 0), (1, -_PHI, 0), (0, -1, _PHI), (0, 1, _PHI), (0, -1, -_PHI), (0, 1, -_PHI),
            (_PHI, 0, -1), (_PHI, 0, 1), (-_PHI, 0, -1), (-_PHI, 0, 1)]
_FACES = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6), (7, 1, 8),
          (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10), (8, 6, 7), (9, 8, 1)]


def _unit(p):
    return p / torch.sqrt((p[:, 0] * p[:, 0] + p[:, 1] * p[:, 1]) + p[:, 2] * p[:, 2]).unsqueeze(1)


def _sphere(k):
    """The icosphere of k divisions: vertices (corners, edges, face interiors) and neighbour rings."""
    corner = _unit(torch.tensor(_CORNERS, dtype=torch.float64, device=DEVICE))
    edges = sorted({(min(f[a], f[b]), max(f[a], f[b])) for f in _FACES for a, b in ((0, 1), (1, 2), (2, 0))})
    number = {e: i for i, e in enumerate(edges)}
    t = torch.arange(1, k, dtype=torch.float64, device=DEVICE).unsqueeze(1)
    parts = [corner] + [_unit((k - t) * corner[a] + t * corner[b]) for a, b in edges]
    g = torch.arange(k + 1, device=DEVICE)
    i, j = g.unsqueeze(1), g.unsqueeze(0)
    inside = (i >= 1) & (j >= 1) & (i + j <= k - 1)
    fi, fj = (x.double().unsqueeze(1) for x in torch.nonzero(inside, as_tuple=True))
    up = torch.nonzero((i + j <= k - 1)[:k, :k])                          # grid triangles of a face, row by row
    key = torch.cat([2 * (up[:, 0] * (k + 1) + up[:, 1]), 2 * (up[:, 0] * (k + 1) + up[:, 1]) + 1])
    kind_down = torch.arange(key.numel(), device=DEVICE) >= up.shape[0]
    ui, uj = up[:, 0].repeat(2), up[:, 1].repeat(2)
    keep = ~kind_down | (ui + uj < k - 1)
    order = torch.argsort(key[keep])
    ui, uj, down = ui[keep][order], uj[keep][order], kind_down[keep][order].long()
    base, per, tris = 12 + 30 * (k - 1), (k - 1) * (k - 2) // 2, []
    for f, (a, b, c) in enumerate(_FACES):
        if per:
            parts.append(_unit(((k - fi - fj) * corner[a] + fi * corner[b]) + fj * corner[c]))
        v = torch.zeros((k + 1, k + 1), dtype=torch.int64, device=DEVICE)
        v[inside] = base + f * per + torch.arange(per, device=DEVICE)
        s = torch.arange(1, k, device=DEVICE)
        for (p, q), at in (((a, b), (s, 0 * s)), ((a, c), (0 * s, s)), ((b, c), (k - s, s))):
            e = number[(min(p, q), max(p, q))]
            v[at] = 12 + e * (k - 1) + (s if p < q else k - s) - 1
        v[0, 0], v[k, 0], v[0, k] = a, b, c
        tris.append(torch.stack([v[ui + down, uj], v[ui + 1, uj + down], v[ui, uj + 1]], 1))
    xyz, tri = torch.cat(parts), torch.cat(tris)
    n = xyz.shape[0]
    src, at = torch.sort(tri.reshape(-1), stable=True)
    dst = tri.roll(-1, 1).reshape(-1)[at]
    row = torch.full((n, 6), -1, dtype=torch.int64, device=DEVICE)
    row[:12, :5], row[12:] = dst[:60].view(12, 5), dst[60:].view(-1, 6)
    del src, at, dst, tri, tris
    ring = torch.full_like(row, -1)
    for b in range(0, n, CHUNK):
        r = row[b:b + CHUNK]
        cur, last = r[:, 0], torch.arange(b, b + r.shape[0], device=DEVICE)
        ring[b:b + CHUNK, 0] = cur
        for q in range(1, 6):
            o = row[cur.clamp(min=0)]
            hit = (r.unsqueeze(2) == o.unsqueeze(1)).any(2) & (r != last.unsqueeze(1)) & (r >= 0)
            last, cur = cur, torch.gather(r, 1, hit.int().argmax(1, keepdim=True)).squeeze(1)
            ring[b:b + CHUNK, q] = cur
    ring[:12, 5] = -1
    return xyz, ring


def _lengths(xyz, nbr):
    d = torch.empty(nbr.shape, dtype=torch.float64, device=DEVICE)
    for q in range(6):
        e = xyz - xyz[nbr[:, q].clamp(min=0)]
        d[:, q] = torch.sqrt(e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1] + e[:, 2] * e[:, 2]) * (nbr[:, q] >= 0)
    return d


def _tables(seed):
    """OpenSimplex permutation and gradient tables (each state of the generator cut to its low 32 bits, signed)."""
    def step(v):
        v = (v * 6364136223846793005 + 1442695040888963407) & 0xFFFFFFFF
        return v - (1 << 32) if v >> 31 else v

    pool, perm, st = list(range(256)), [0] * 256, step(step(step(seed)))
    for i in range(255, -1, -1):
        st = step(st)
        r = (st + 31) % (i + 1)
        perm[i], pool[r] = pool[r], pool[i]
    return torch.tensor(perm, device=DEVICE), torch.tensor([p % 24 for p in perm], device=DEVICE)


_G = [(-11, 4, 4), (-4, 11, 4), (-4, 4, 11), (11, 4, 4), (4, 11, 4), (4, 4, 11), (-11, -4, 4), (-4, -11, 4), (-4, -4, 11),
      (11, -4, 4), (4, -11, 4), (4, -4, 11)]
_GRAD = [(x, y, s * z) for s in (1, -1) for x, y, z in _G]


def _noise3(p, perm, pgi):
    """103 times OpenSimplex 3-D noise at the rows of p: skewed cell, region, its fixed corners and two extra points."""
    grad = torch.tensor(_GRAD, dtype=torch.float64, device=DEVICE)
    skew = ((p[:, 0] + p[:, 1]) + p[:, 2]) * (-1.0 / 6)
    ps = p + skew.unsqueeze(1)
    cell = torch.floor(ps)
    ins = ps - cell
    x, y, z = ins.unbind(1)
    total = (x + y) + z
    d0 = p - (cell + ((cell[:, 0] + cell[:, 1] + cell[:, 2]) * (1.0 / 3)).unsqueeze(1))
    cell = cell.long()
    low = total <= 1.0
    high = ~low & (total >= 2.0)
    mid = ~low & ~high
    # tetrahedra; the one at (1,1,1) is the other's mirror image
    s = torch.where(high, -1.0, 1.0).double()
    xy, zb, za = s * x >= s * y, s * z > s * y, s * z > s * x
    rb, ra = xy & zb, ~xy & za
    va, vb, ca, cb = torch.where(ra, z, x), torch.where(rb, z, y), torch.where(ra, 4, 1), torch.where(rb, 4, 2)
    w = torch.where(high, 3.0, 1.0) - total
    near = (s * w > s * va) | (s * w > s * vb)
    c = torch.where(near, torch.where(s * vb > s * va, cb, ca), ca | cb)
    b1, b2, b4 = (c & 1) != 0, (c & 2) != 0, (c & 4) != 0

    def pick(cond, a, b):
        return torch.where(cond, a, b).long() if not isinstance(a, int) or not isinstance(b, int) else torch.where(cond, torch.full_like(c, a), torch.full_like(c, b))

    e0 = [pick(near, pick(b1, 1, -1), pick(b1, 1, 0)), pick(near, pick(b2, pick(b2, 1, 1), pick(b1, -1, 0)), pick(b2, 1, 0)), pick(b4, 1, 0)]
    e1 = [pick(near, pick(b1, 1, 0), pick(b1, 1, -1)), pick(near, pick(b2, pick(b2, 1, 1), pick(b1, 0, -1)), pick(b2, 1, -1)), pick(b4, 1, -1)]
    e0, e1 = ([pick(high, 1 - e, e) for e in q] for q in (e0, e1))
    # octahedron between them
    p1, p2, p3 = x + y, x + z, y + z
    f1, f2, f3 = p1 > 1.0, p2 > 1.0, p3 > 1.0
    sa, sb, sc = (torch.where(f, v - 1.0, 1.0 - v) for f, v in ((f1, p1), (f2, p2), (f3, p3)))
    swa, swb = (sa <= sb) & (sa < sc), ~(sa <= sb) & (sb < sc)
    third = pick(f3, 6, 1)
    oa, ob = torch.where(swa, third, pick(f1, 3, 4)), torch.where(swb, third, pick(f2, 5, 2))
    fa, fb = torch.where(swa, f3, f1), torch.where(swb, f3, f2)
    same = fa == fb
    cs = torch.where(fa, oa & ob, oa | ob)
    s1, s2 = (cs & 1) != 0, (cs & 2) != 0
    ax, ay = torch.where(fa, s1, ~s1), torch.where(fa, ~s1 & s2, s1 & ~s2)
    q1, q2 = torch.where(fa, oa, ob), torch.where(fa, ob, oa)
    bx, by = (q1 & 1) == 0, ((q1 & 1) != 0) & ((q1 & 2) == 0)
    gx, gy = (q2 & 1) != 0, ((q2 & 1) == 0) & ((q2 & 2) != 0)
    one, hit, miss = pick(fa, 1, 0), pick(fa, 2, -1), pick(fa, 0, 1)
    o0 = [pick(same, one, pick(b, -1, 1)) for b in (bx, by, ~bx & ~by)]
    o1 = [pick(same, pick(a, hit, miss), pick(g, 2, 0)) for a, g in ((ax, gx), (ay, gy), (~ax & ~ay, ~gx & ~gy))]
    e0, e1 = [pick(mid, o, e) for o, e in zip(o0, e0)], [pick(mid, o, e) for o, e in zip(o1, e1)]

    def point(o, on):
        step = (d0.new_zeros(1) + o[0] + o[1] + o[2]) * (1.0 / 3)
        d = [d0[:, a] - o[a] - step for a in range(3)]
        attn = 2.0 - d[0] * d[0] - d[1] * d[1] - d[2] * d[2]
        h = perm[(cell[:, 0] + o[0]) & 255]
        h = perm[(h + cell[:, 1] + o[1]) & 255]
        g = grad[pgi[(h + cell[:, 2] + o[2]) & 255]]
        attn = torch.where(on, attn.clamp(min=0.0), 0.0)
        return (attn * attn) * (attn * attn) * (g[:, 0] * d[0] + g[:, 1] * d[1] + g[:, 2] * d[2])

    v = point((0, 0, 0), low) + point((1, 1, 1), high)
    for o in ((1, 0, 0), (0, 1, 0), (0, 0, 1)):
        v = v + point(o, ~high)
    for o in ((1, 1, 0), (1, 0, 1), (0, 1, 1)):
        v = v + point(o, ~low)
    every = torch.ones_like(low)
    return v + point(e0, every) + point(e1, every)


def _fbm(xyz, tables, octaves, f, a, lac, pers, radius):
    out = torch.zeros(xyz.shape[0], dtype=torch.float64, device=DEVICE)
    for _ in range(octaves):
        for b in range(0, xyz.shape[0], CHUNK):
            v = _noise3(xyz[b:b + CHUNK] * (f / radius), *tables) / 103.0
            out[b:b + CHUNK] += (v + 1.0) * 0.5 * (a / radius) * radius
        f, a = f * lac, a * pers
    return out


def _rescale(x, lo, hi):
    return (x - x.min()) / (x.max() - x.min()) * (hi - lo) + lo


def _shape(x, lo=-4000.0, hi=8850.0, percent=55.0):
    h = _rescale(x, lo, hi)
    level = h.min() + (h.max() - h.min()) * percent / 100.0
    ocean = h <= level
    for mask, power in ((ocean, 0.5), (~ocean, 2.0)):
        first, last = h.max(), h.min()
        v = h[mask]
        before = torch.cat([first.reshape(1), torch.cummin(v, 0).values[:-1]]).minimum(first)
        small, cand = torch.minimum(first, v.min()), v[v >= before]      # a new running minimum is no candidate for the maximum
        span = torch.maximum(last, cand.max()) - small if cand.numel() else last - small
        h[mask] = ((v - small) / span) ** power * span + small
    h = h - level
    return torch.where(h <= 0.0, (h - h.min()) / (0.0 - h.min()) * (0.0 - lo) + lo, h / h.max() * hi), ocean, level


def _erode(xyz, nbr, h, iters, water, rain):
    d, w, s = _lengths(xyz, nbr), torch.full_like(h, water), torch.zeros_like(h)
    at, sol, evap, cap = nbr.clamp(min=0), 0.01 / 320, 0.1 / 320, 0.2 / 320
    there = nbr >= 0
    for _ in range(iters):
        w = w + rain
        sed, wat = s.clone(), w.clone()
        for q in range(6):
            g = torch.sign(h[at[:, q]] - h) * there[:, q] * w[at[:, q]]
            sed += sol * g
            wat += g * d[:, q]
        h, s, w = h - sed, s + sed, w + (wat - wat * evap)
        over = (s - cap * w).clamp(min=0.0)
        h, s = h + over, s - over
    return h


def _insolation(xyz, radius, rotations, tilts):
    """The terms max(cos|lat|, 0) max(cos lon, 0) of vertices on the sphere, summed over rotations and tilts."""
    out = torch.zeros(xyz.shape[0], dtype=torch.float64, device=DEVICE)
    for b in range(0, xyz.shape[0], CHUNK // 4):
        x, y, z = xyz[b:b + CHUNK // 4].unbind(1)
        for t in tilts:
            ct, st = math.cos(math.radians(t)), math.sin(math.radians(t))
            zt = z * st
            for r in rotations:
                u = x * (math.cos(math.radians(r)) * ct) - y * (math.sin(math.radians(r)) * ct)
                out[b:b + CHUNK // 4] += (u + zt).clamp(min=0.0)
    return out / radius


def _year(xyz, radius, tilt, days):
    """Mean flux over days of 24 hourly positions; a rotation and its opposite add up to C + max(|C|, |u|)."""
    out = torch.zeros(xyz.shape[0], dtype=torch.float64, device=DEVICE)
    turn = torch.deg2rad(-180.0 + 15.0 * torch.arange(12, dtype=torch.float64, device=DEVICE))
    tilts = [math.radians(math.sin(math.radians(day / 365 * 360.0)) * tilt) for day in range(days)]
    for b in range(0, xyz.shape[0], CHUNK // 8):
        x, y, z = xyz[b:b + CHUNK // 8].unbind(1)
        u = (x.unsqueeze(0) * turn.cos().unsqueeze(1) - y.unsqueeze(0) * turn.sin().unsqueeze(1)).abs()
        for t in tilts:
            c = z * math.sin(t)
            out[b:b + CHUNK // 8] += 12 * c + torch.maximum(u * math.cos(t), c.abs().unsqueeze(0)).sum(0)
    return out / radius * (1361.0 / (days * 24))
