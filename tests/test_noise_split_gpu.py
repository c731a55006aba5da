"""The noise of small spheres and remainders, whose octaves are dealt out to groups of warps: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("octaves", [0, 1, 2, 5, 12, 32])
def test_a_vertex_has_the_same_sum_in_every_launch(octaves):
    import torch
    from nixis_gb300 import mesh, opensimplex, terrain
    perm, pgi = opensimplex.init(7)
    xyz = mesh.icosphere(100, with_tris=False)[0]                    # 100,002 vertices: one round and a remainder
    scale, strength = [1.7 * 1.9 ** o for o in range(octaves)], [0.8 ** o for o in range(octaves)]
    whole = terrain.fbm(xyz, perm, pgi, scale, strength, 1.0)[0]
    for n in (1, 31, 32, 33, 511, 512, 513, 1442, 4864, 4865, 20000, 38913, 77823, 77824, 77825, 77857):
        part, fallbacks = terrain.fbm(xyz[:n].contiguous(), perm, pgi, scale, strength, 1.0, count_fallbacks=True)
        assert torch.equal(part, whole[:n]), n
        if n == 33:                                                  # (padding lanes are not counted)
            one = [terrain.fbm(xyz[i:i + 1].contiguous(), perm, pgi, scale, strength, 1.0, count_fallbacks=True)[1] for i in range(n)]
            assert fallbacks == sum(one)
    base = torch.linspace(-1.0, 1.0, 1442, dtype=torch.float64, device="cuda")
    out = base.clone()
    terrain.fbm(xyz[:1442].contiguous(), perm, pgi, scale, strength, 1.0, out=out, accumulate=True)
    assert torch.equal(out, base + whole[:1442])


@pytest.mark.parametrize("divisions", [[2], [2, 3, 5], [12, 40], [60, 61], [12, 100, 150]])
def test_small_batches_equal_planets_alone(divisions):
    import torch
    from nixis_gb300 import planets
    reqs = [planets.PlanetRequest(seed=i, divisions=k, octaves=1 + 5 * i, erosion_iters=0) for i, k in enumerate(divisions)]
    b = planets.PlanetBatch(reqs)
    b.run()
    for r, got in zip(reqs, b.results()):
        assert torch.equal(got.heights, planets.generate_plain(r).heights)
