"""Insolation schedules summed by arcs and by breakpoints, against the terms summed one by one in binary64.

Tolerance (stated): 2e-6 of the largest sum.  By arcs a tilt's sum over n rotations is a difference of prefix sums of up
to n/pi, each rounded once (4 roundings of 2^-25), three products (2^-24 each) and at most one rotation misplaced at
either end of the arc, whose term is then within 1e-6 of 0; by breakpoints the lines' sums are rounded once and 12 values
of a few roundings each are added.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROTATIONS = {
    "degrees": [-180.0 + i for i in range(360)],                            # pairs, ascending
    "shuffled": list(np.random.default_rng(1).permutation(360) - 180.0),
    "uneven": list(np.random.default_rng(2).uniform(-400.0, 400.0, 129)),   # no pairs, beyond one turn
    "most": [-90.0 + 0.3515625 * i for i in range(1024)],
    "hourly": [-180.0 + 15.0 * i for i in range(24)],                       # by breakpoints
}


@pytest.mark.parametrize("tilts", [[0.0], [23.44, -7.5, 90.0, 135.0, 10.0]])
@pytest.mark.parametrize("name", list(ROTATIONS))
@pytest.mark.parametrize("radius", [1.0, 6378100.0])
def test_sums_equal_the_terms_in_binary64(name, tilts, radius):
    import torch
    from nixis_gb300 import climate, mesh
    xyz = mesh.icosphere(17, with_tris=False)[0]
    poles = torch.tensor([[0, 0, 1], [0, 0, -1], [1, 0, 0], [0, -1, 0], [1e-13, 0, 1]], dtype=torch.float64, device="cuda")
    xyz = torch.cat([xyz, poles / poles.norm(dim=1, keepdim=True)]) * radius
    if name == "uneven" and len(tilts) == 1:
        tilts = tilts * 3
    got = climate.insolation_sum(xyz, radius, ROTATIONS[name], tilts).double()
    rot, tilt = (torch.deg2rad(torch.tensor(v, dtype=torch.float64, device="cuda")) for v in (ROTATIONS[name], tilts))
    want = torch.zeros_like(got)
    x, y, z = (xyz / radius).unbind(1)
    for t in tilt:
        u = x[:, None] * torch.cos(rot) - y[:, None] * torch.sin(rot)
        want += (u * torch.cos(t) + (z * torch.sin(t))[:, None]).clamp(min=0.0).sum(1)
    assert (got - want).abs().max() <= 2e-6 * want.max()


def test_large_sphere_and_batch_rows_take_the_same_values():
    import torch
    from nixis_gb300 import climate, mesh
    from nixis_gb300.planets import PlanetBatch, PlanetRequest
    m = mesh.PlanetMesh(170)                                                # over 2^18 vertices: one tilt by arcs
    rot = [-180.0 + 2.0 * i for i in range(180)]
    one = climate.insolation_sum(m.xyz, 1.0, rot, [12.0])
    part = climate.insolation_sum(m.xyz[:5000], 1.0, rot, [12.0])           # rotation by rotation
    assert (one[:5000] - part).abs().max() <= 2e-6 * one.max()
    reqs = [PlanetRequest(seed=1, divisions=k, octaves=2, insolation=True, days=3, hours=h) for k, h in ((9, 360), (14, 360), (11, 24))]
    b = PlanetBatch(reqs)
    b.run()
    for r, got in zip(reqs, b.results()):
        rot, tilts = climate.annual_schedule(r.axial_tilt, r.days, r.days, r.hours)
        want = climate.insolation_sum(mesh.PlanetMesh(r.divisions).xyz, 1.0, rot, tilts) * (climate.SOLAR_CONSTANT / (r.days * r.hours))
        assert torch.equal(got.insolation, want)


@pytest.mark.parametrize("days", [1, 2, 7, 30, 127, 128, 255, 256, 300, 366, 400, 495, 511, 512, 513])
def test_bucket_tables_of_any_length(days):
    """Hourly positions over `days` days, days past the first year repeating (equal and nearly equal breakpoints), as
    the sum of its terms one by one."""
    import torch
    from nixis_gb300 import climate, mesh
    m = mesh.PlanetMesh(23)
    rot, tilts = climate.annual_schedule(23.44, 365, days, 24)
    got = climate.insolation_sum(m.xyz, 1.0, rot, tilts).double()
    r, t = (torch.tensor(v, dtype=torch.float64, device="cuda") * (math.pi / 180) for v in (rot, tilts))
    x, y, z = m.xyz.T
    want = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    for tau in t:
        u = (x[:, None] * r.cos() - y[:, None] * r.sin()) * tau.cos() + (z * tau.sin())[:, None]
        want += u.clamp(min=0).sum(1)
    assert (got - want).abs().max() <= 2e-6 * want.max()


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("where", [0, 77, 359])
def test_a_rotation_that_is_no_number_lights_nothing(where, bad):
    """It has no place among the sorted angles; the others' terms stay as they are rotation by rotation (120 at a time
    is below the arcs' range).  2e-6 of the largest sum: two orders of summation in binary32."""
    from nixis_gb300 import climate, mesh
    m = mesh.PlanetMesh(17)
    rot, tilts = [-180.0 + i for i in range(360)], [23.44, -7.5]
    rot[where] = bad
    got = climate.insolation_sum(m.xyz, 1.0, rot, tilts)
    want = sum(climate.insolation_sum(m.xyz, 1.0, rot[q:q + 120], tilts) for q in (0, 120, 240))
    assert (got - want).abs().max() <= 2e-6 * want.max()


@pytest.mark.parametrize("rotations", [24, 7, 360])
def test_vertices_at_the_bound_of_the_sphere_test(rotations):
    """| |v|^2 - r^2 | within 8e-14 r^2 of its bound of 1e-12 r^2: the formula is the one that binary64 picks, so a sum has
    the bits of a vertex well inside the bound (the same binary32 coordinates) or of a radius well off (the same binary32
    reciprocal)."""
    import torch
    from nixis_gb300 import climate
    gen = torch.Generator(device="cuda").manual_seed(8)
    n, r = 200_000, 1.25
    v = torch.randn(n, 3, dtype=torch.float64, device="cuda", generator=gen)
    v = v / v.norm(dim=1, keepdim=True) * r
    sign = torch.where(torch.arange(n, device="cuda") % 2 == 0, 1.0, -1.0).double()
    off = sign * (1e-12 + (torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 0.5) * 1.6e-13)
    at, inside = v * (1 + off / 2)[:, None], v * (1 + 0.2 * off)[:, None]
    # |at|^2 / r^2 - 1 as the kernel's binary64 forms it, but for two roundings (2e-16, left out below)
    over = ((at[:, 0] * at[:, 0] + at[:, 1] * at[:, 1] + at[:, 2] * at[:, 2]) / (r * r) - 1).abs() - 1e-12
    clear = (over.abs() > 2e-15) & (at.float() == inside.float()).all(1)
    assert clear.float().mean() > 0.9
    rot, tilts = [-180.0 + 360.0 / rotations * i for i in range(rotations)], [23.44, -11.0, 3.0]
    got = climate.insolation_sum(at, r, rot, tilts)
    on = climate.insolation_sum(inside, r, rot, tilts)
    far = climate.insolation_sum(at, r * (1 + 1e-9), rot, tilts)
    assert (on != far).float().mean() > 0.2
    want = torch.where(over < 0, on, far)
    assert torch.equal(got[clear], want[clear])


@pytest.mark.parametrize("axial", [23.44, 1e-3, 1e-6, 1e-8, 1e-20])
def test_years_of_small_tilts_at_the_poles(axial):
    """Where only the tilts light a vertex its sum is as exact as any other: within 5e-7 of itself (eight roundings of
    2^-24: the lines' sums, a product and the additions of 12 values and of the days' C terms)."""
    import torch
    from nixis_gb300 import climate
    gen = torch.Generator(device="cuda").manual_seed(3)
    lon = torch.rand(2000, dtype=torch.float64, device="cuda", generator=gen) * 2 * math.pi
    e = 1e-3 * axial * math.pi / 180 * torch.rand(2000, dtype=torch.float64, device="cuda", generator=gen)
    xyz = torch.stack([e * lon.cos(), e * lon.sin(), torch.sqrt(1 - e * e)], 1)
    xyz[::2, 2] *= -1
    rot, tilts = climate.annual_schedule(axial, 365, 365, 24)
    got = climate.insolation_sum(xyz, 1.0, rot, tilts).double()
    r, t = (torch.tensor(v, dtype=torch.float64, device="cuda") * (math.pi / 180) for v in (rot, tilts))
    x, y, z = xyz.T
    want = torch.zeros_like(got)
    for tau in t:
        want += ((x[:, None] * r.cos() - y[:, None] * r.sin()) * tau.cos() + (z * tau.sin())[:, None]).clamp(min=0).sum(1)
    assert ((got - want).abs() <= 5e-7 * want).all()


@pytest.mark.parametrize("axial, allowed", [(23.44, 5.27e-8), (1.0, 5.67e-8), (0.01, 4.94e-8)])
def test_a_years_error_is_no_larger_than_of_sums_in_binary64(axial, allowed):
    """Root mean square error over a sphere, against the one measured where the days' sums were kept in binary64 and
    looked up by their counts (the form that the tables of lines replaced)."""
    import torch
    from nixis_gb300 import climate, mesh
    xyz = mesh.icosphere(60, with_tris=False)[0]
    rot, tilts = climate.annual_schedule(axial, 365, 365, 24)
    got = climate.insolation_sum(xyz, 1.0, rot, tilts).double()
    r, t = (torch.tensor(v, dtype=torch.float64, device="cuda") * (math.pi / 180) for v in (rot, tilts))
    x, y, z = xyz.T
    u = x[:, None] * r.cos() - y[:, None] * r.sin()
    want = torch.zeros_like(got)
    for tau in t:
        want += (u * tau.cos() + (z * tau.sin())[:, None]).clamp(min=0).sum(1)
    assert (got - want).norm() <= allowed * want.norm()


@pytest.mark.parametrize("rotations, days", [(24, 2048), (24, 2049), (7, 700), (100, 90)])
def test_long_schedules_day_by_day(rotations, days):
    """Past the breakpoints' 512 days, past the 2,048 staged ones, and by single rotations, vertices on the sphere and off."""
    import torch
    from nixis_gb300 import climate, mesh
    xyz = mesh.icosphere(9, with_tris=False)[0]
    rot, tilts = climate.annual_schedule(23.44, days, days, rotations)
    r, t = (torch.tensor(v, dtype=torch.float64, device="cuda") * (math.pi / 180) for v in (rot, tilts))
    x, y, z = xyz.T
    want = torch.zeros(xyz.shape[0], dtype=torch.float64, device="cuda")
    for tau in t:
        want += ((x[:, None] * r.cos() - y[:, None] * r.sin()) * tau.cos() + (z * tau.sin())[:, None]).clamp(min=0).sum(1)
    assert (climate.insolation_sum(xyz, 1.0, rot, tilts).double() - want).abs().max() <= 2e-6 * want.max()
    off = climate.insolation_sum(xyz, 1.0 + 1e-9, rot, tilts).double()
    assert (off - want).abs().max() <= 1e-5 * want.max()


@pytest.mark.parametrize("radius", [1e-30, 1e-19, 1e19, 1e25])
def test_spheres_whose_squares_are_no_binary32_numbers(radius):
    """A one-degree day as the sum of three parts of 120 rotations (below the arcs' range), alone and in a batch; 2e-6 of
    the largest sum (two orders of summation in binary32)."""
    import ctypes
    import torch
    from nixis_gb300 import _dev, _lib, climate, mesh
    xyz = mesh.icosphere(20, with_tris=False)[0] * radius
    rot, tilts = [-180.0 + i for i in range(360)], [11.0]
    want = sum(climate.insolation_sum(xyz, radius, rot[q:q + 120], tilts) for q in (0, 120, 240))
    assert (climate.insolation_sum(xyz, radius, rot, tilts) - want).abs().max() <= 2e-6 * want.max()
    tab, nre, pairs = climate._plan(rot, tilts)
    table, out = torch.from_numpy(tab).cuda(), torch.empty(xyz.shape[0], dtype=torch.float32, device="cuda")
    d = (_lib.InsoPlanet * 1)()
    d[0].xyz, d[0].n, d[0].vbeg, d[0].radius = xyz.data_ptr(), xyz.shape[0], 0, radius
    dev = torch.frombuffer(bytearray(bytes(d)), dtype=torch.uint8).cuda()
    _lib.call("nx_insolation_batch", _dev.ptr(dev), ctypes.cast(d, ctypes.c_void_p), 1, _dev.ptr(table), nre, pairs, 1, _dev.ptr(out),
              _dev.stream_handle())
    assert (out - want).abs().max() <= 2e-6 * want.max()


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("rotations", [128, 129])
def test_a_tilt_that_is_no_number_gives_what_the_rotations_one_by_one_give(rotations, bad):
    """Three tilts by arcs (their 384 positions reach the rule's 360), each alone by maxima: no number in pairs, where both
    sides of a maximum are none, 0 otherwise.  2e-6 of the largest sum."""
    import torch
    from nixis_gb300 import climate, mesh
    xyz = mesh.icosphere(9, with_tris=False)[0]
    rot, tilts = [-180.0 + 360.0 / rotations * i for i in range(rotations)], [20.0, bad, -7.0]
    got = climate.insolation_sum(xyz, 1.0, rot, tilts)
    want = sum(climate.insolation_sum(xyz, 1.0, rot, [t]) for t in tilts)
    assert torch.equal(got.isnan(), want.isnan()) and bool(want.isnan().all()) == (rotations == 128)
    assert rotations == 128 or (got - want).abs().max() <= 2e-6 * want.max()


@pytest.mark.parametrize("rotations", [361, 511, 1023])
@pytest.mark.parametrize("tilt", [23.44, 75.0])
def test_vertices_lit_in_few_rotations_without_pairs(rotations, tilt):
    """Near where night lasts all day, by arcs.  Tolerance (stated): binary32 terms of three products of two or three
    rounded factors are within 6 2^-24 of themselves each, and a rotation misplaced at an end of the arc (an angle's
    cosine is off by 2^-23, twice) adds at most 4 2^-24: (6 m + 8) 2^-24 for a vertex lit in m rotations."""
    import torch
    from nixis_gb300 import climate
    rng = np.random.default_rng(7)
    t = math.radians(tilt)
    z = -math.cos(t) * (1.0 + rng.uniform(-1e-3, 1e-3, 6000))
    at = rng.uniform(-math.pi, math.pi, len(z))
    v = np.stack([np.sqrt(1.0 - z * z) * np.cos(at), np.sqrt(1.0 - z * z) * np.sin(at), z], axis=1)
    rot = [-180.0 + 360.0 / rotations * i for i in range(rotations)]
    got = climate.insolation_sum(torch.from_numpy(v).cuda(), 1.0, rot, [tilt]).double().cpu().numpy()
    r = np.radians(rot)
    u = (v[:, :1] * np.cos(r) - v[:, 1:2] * np.sin(r)) * math.cos(t) + v[:, 2:] * math.sin(t)
    lit = (u > 0.0).sum(1)
    assert ((lit >= 1) & (lit <= 8)).sum() > 100
    assert (np.abs(got - np.maximum(u, 0.0).sum(1)) <= (6 * lit + 8) * 2.0 ** -24)[lit <= 60].all()
