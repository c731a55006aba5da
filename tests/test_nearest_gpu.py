"""The three nearest vertices against brute force: bits, order and ties, for queries where the located triangle or the
ranking is in doubt (vertices, edges' middles, face borders, poles) and spheres of any radius."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 7, 40])
@pytest.mark.parametrize("radius", [1.0, 6378100.0, 1e-7, 3e20])
def test_equals_brute_force(k, radius):
    import torch
    from nixis_gb300 import mesh, util
    m = mesh.PlanetMesh(k)
    xyz = m.xyz * radius
    a = m.nbr[:, :5].long()
    gen = torch.Generator(device="cuda").manual_seed(3)
    pts = [m.xyz, (m.xyz + m.xyz[a[:, 0]]) / 2, (m.xyz + m.xyz[a[:, 0]] + m.xyz[a[:, 1]]) / 3,
           m.xyz * (1 + 1e-9), torch.randn(4000, 3, dtype=torch.float64, device="cuda", generator=gen),
           torch.tensor([[0, 0, 1], [0, 0, -1], [1, 0, 0], [0, 1, 0], [1e-30, 0, 1]], dtype=torch.float64, device="cuda")]
    q = torch.cat([p / p.norm(dim=1, keepdim=True) for p in pts]) * radius
    d, i = util.query_nearest3(xyz, m.nbr, k, q)
    for b in range(0, q.shape[0], 2000):
        e = q[b:b + 2000, None, :] - xyz[None]
        full = torch.sqrt((e[..., 0] * e[..., 0] + e[..., 1] * e[..., 1]) + e[..., 2] * e[..., 2])
        want, at = full.sort(dim=1, stable=True)
        assert torch.equal(d[b:b + 2000], want[:, :3]) and torch.equal(i[b:b + 2000], at[:, :3])


@pytest.mark.parametrize("size", [(3, 2), (64, 32), (257, 33), (1000, 65)])
def test_pixel_positions_are_the_scalar_formula(size):
    import math
    from nixis_gb300 import util
    w, h = size
    ll = util.make_ll_arr(w, h, 2.5)
    assert ll.shape == (h, w, 3)
    for r in sorted({0, 1, h // 2, h - 1}):
        for c in sorted({0, w // 3, w - 1}):
            x, y, z = util.latlon2xyz(max(90.0 - r * (180.0 / (h - 1)), -90.0), max(-180.0 + c * (360.0 / w), -180.0), 2.5)
            assert all(abs(u - v) <= 2 * math.ulp(2.5) for u, v in zip(ll[r, c], (x, y, z)))


@pytest.mark.parametrize("ratio", [1 / 1e3, 1 / 7.0, 16.0, 100.0, 1e3, 6.4e6])
def test_spheres_of_another_radius_than_the_queries(ratio):
    """Vertices `ratio` times as far out as the queries: the ranking's error is of the larger of the two."""
    import torch
    from nixis_gb300 import mesh, util
    k = 40
    m = mesh.PlanetMesh(k)
    xyz = m.xyz * ratio
    gen = torch.Generator(device="cuda").manual_seed(5)
    a = m.nbr[:, :5].long()
    q = torch.cat([torch.randn(6000, 3, dtype=torch.float64, device="cuda", generator=gen), m.xyz + 0.4999 * (m.xyz[a[:, 0]] - m.xyz)])
    q = q / q.norm(dim=1, keepdim=True)
    d, i = util.query_nearest3(xyz, m.nbr, k, q)
    for b in range(0, q.shape[0], 2000):
        e = q[b:b + 2000, None, :] - xyz[None]
        full = torch.sqrt((e[..., 0] * e[..., 0] + e[..., 1] * e[..., 1]) + e[..., 2] * e[..., 2])
        want, at = full.sort(dim=1, stable=True)
        assert torch.equal(d[b:b + 2000], want[:, :3]) and torch.equal(i[b:b + 2000], at[:, :3])


def test_queries_of_no_length_and_no_number():
    """The centre goes to the first face's first corner, as its coordinates there (0 / 0, taken as 0) always had it;
    queries below the smallest normal number by their direction; a component that is no number finds nothing."""
    import torch
    from nixis_gb300 import mesh, util
    k = 40
    m = mesh.PlanetMesh(k)
    u = m.xyz[200:260]
    q = torch.cat([torch.zeros(1, 3, dtype=torch.float64, device="cuda"), u * 1e-309])
    _, i = util.query_nearest3(m.xyz, m.nbr, k, q)
    toward = torch.cat([m.xyz[:1], u])
    far = (m.xyz[i] - toward[:, None]).norm(dim=2)          # the candidates: a triangle there and its rings
    assert far.max() <= 3 * 1.2 / k
    for bad in (float("nan"), float("inf")):
        d, i = util.query_nearest3(m.xyz, m.nbr, k, torch.tensor([[0.3, bad, 0.1]], dtype=torch.float64, device="cuda"))
        assert (i == -1).all() and torch.isinf(d).all()


@pytest.mark.parametrize("size", [(1, 65535 * 32 + 1), (2, 65535 * 32 + 70)])
def test_pixel_positions_of_maps_taller_than_a_grid(size):
    import math
    from nixis_gb300 import util
    w, h = size
    ll = util.make_ll_arr(w, h, 2.5, device=True)
    for r in (0, 31, 32, h // 2, 65535 * 32 - 1, 65535 * 32, h - 1):
        x, y, z = util.latlon2xyz(max(90.0 - r * (180.0 / (h - 1)), -90.0), -180.0, 2.5)
        assert all(abs(u - v) <= 2 * math.ulp(2.5) for u, v in zip(ll[r, 0].tolist(), (x, y, z)))
