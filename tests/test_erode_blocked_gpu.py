"""erode_terrain3 by blocked passes against one iteration at a time: bit for bit the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K, ITERS = 150, 150          # 225,002 vertices: past the rule's 2^25 vertex-iterations, and through the rescale


def field(m, seed):
    from nixis_gb300 import opensimplex, terrain, util
    perm, pgi = opensimplex.init(seed)
    return util.rescale(terrain.sample_octaves(m.xyz, None, perm, pgi, 6, 1.0, 1.0, 2.0, 0.5, 1.0), -4000.0, 8850.0)


def one_at_a_time(xyz, nbr, h, iters):
    import torch
    from nixis_gb300 import erosion
    run = erosion.ErosionRun(xyz, nbr).load(h)
    run.steps(iters, rain=erosion.RAIN)
    run.check()
    out = torch.empty_like(h)
    run.store(out)
    return out


@pytest.mark.parametrize("iters", [ITERS, ITERS + 1])
@pytest.mark.parametrize("case", ["plain", "earth_radius", "host", "huge_heights"])
def test_blocked_runs_equal_iteration_at_a_time(case, iters):
    import torch
    from nixis_gb300 import erosion, mesh
    m = mesh.PlanetMesh(K)
    h = field(m, 5) * (2.0 ** 90 if case == "huge_heights" else 1.0)
    xyz = m.xyz * (6378100.0 if case == "earth_radius" else 1.0)
    # (edges of tens of kilometres: the water's growth within a pass would pass the state's range)
    expect = None if case == "earth_radius" else K
    assert iters * m.n >= erosion.BLOCKED_WORK and erosion.ErosionRun(xyz, m.nbr, iters=iters).k == expect
    want = one_at_a_time(xyz, m.nbr, h, iters)
    if case == "host":
        got = h.cpu().numpy()
        erosion.erode_terrain3(xyz.cpu().numpy(), m.nbr.cpu().numpy(), got, iters)
        assert np.array_equal(got, want.cpu().numpy())
    else:
        got = h.clone()
        erosion.erode_terrain3(xyz, m.nbr, got, iters)
        assert torch.equal(got, want)


@pytest.mark.parametrize("change", ["order", "row", "border"])
def test_other_tables_still_run(change):
    """Another vertex order, a turned ring inside a face, a changed row of an edge vertex."""
    import torch
    from nixis_gb300 import erosion, mesh
    m = mesh.PlanetMesh(K)
    xyz, nbr, h = m.xyz, m.nbr.clone(), field(m, 6)
    if change == "order":
        perm = torch.from_numpy(np.random.default_rng(1).permutation(m.n)).cuda()
        inv = torch.empty_like(perm)
        inv[perm] = torch.arange(m.n, device="cuda")
        xyz, h = xyz[perm], h[perm]
        nbr = torch.where(nbr[perm] >= 0, inv[nbr[perm].clamp(min=0).long()].int(), nbr[perm]).int()
    elif change == "row":
        nbr[m.n - 1000] = nbr[m.n - 1000].roll(2)
    else:
        nbr[40] = nbr[40].roll(1)
        nbr[41, 3] = -1
    want = one_at_a_time(xyz, nbr, h, ITERS)
    got = h.clone()
    erosion.erode_terrain3(xyz, nbr, got, ITERS)
    assert torch.equal(got, want)
    bad = nbr.clone()
    bad[50, 2] = m.n
    with pytest.raises(IndexError):
        erosion.erode_terrain3(xyz, bad, got, ITERS)
    assert torch.equal(got, want)


def test_load_and_store_keep_every_value():
    """Heights, water and sediment of every size and sign through the state: to 48 bits, and the scale's exponent."""
    import torch
    from nixis_gb300 import erosion, mesh
    m = mesh.PlanetMesh(10)
    rng = np.random.default_rng(3)
    for top in (1.0, 1e18, 1e25, 1e300):
        v = [torch.from_numpy(rng.normal(0.0, 1.0, m.n) * 10.0 ** rng.integers(-12, 1, m.n) * top).cuda() for _ in range(3)]
        v[0][:4] = torch.tensor([0.0, -0.0, top, -top], dtype=torch.float64)
        run = erosion.ErosionRun(m.xyz, m.nbr).load(*v)
        out = [torch.empty_like(x) for x in v]
        run.store(*out)
        for a, b in zip(v, out):
            assert ((a - b).abs() <= a.abs() * 2.0 ** -48).all()


def test_short_runs_do_no_work_for_blocked_passes(monkeypatch):
    """One iteration at a time, without asking for the setting of passes that are not made."""
    import torch
    from nixis_gb300 import autotune, erosion, mesh

    def unwanted():
        raise AssertionError("asked for")
    monkeypatch.setattr(autotune, "current", unwanted)
    m = mesh.PlanetMesh(20)
    h = field(m, 2)
    want = one_at_a_time(m.xyz, m.nbr, h, 3)
    erosion.erode_terrain3(m.xyz, m.nbr, h, 3)
    assert torch.equal(h, want)
