"""The case tables of the binary32 decision: every order of the coordinates in every region, at and around its ties.

Decisions are binary64's (a lane whose margin is below TAU = 4e-6 is decided there), so they are equal, not close."""
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _near_ties(rng, reach):
    """Points whose position in the skewed cell is on, or `eps` off, one or two of the decision surfaces."""
    base = rng.random((60_000, 3))
    rows = [base]
    x, y, z = base.T
    one = np.ones_like(x)
    planes = [lambda: (x, x, z), lambda: (x, y, y), lambda: (x, y, x),                      # equal coordinates
              lambda: (x, y, one - x - y), lambda: (x, y, 2 - x - y),                       # the regions' borders
              lambda: (x, one - x, z), lambda: (x, y, one - x), lambda: (x, y, one - y),    # sums of two are 1
              lambda: (x, y, 2 - 2 * x - y), lambda: (x, 2 - 2 * y, y),                     # equal scores of the octahedron
              lambda: (x, (one - x) / 2, (one - x) / 4), lambda: (x, (one - x - y) / 1, y)]  # wins equal to a score
    for f in planes:
        p = np.stack([np.broadcast_to(c, x.shape) for c in f()], 1)
        p = p[((p >= 0) & (p <= 1)).all(1)][:4000]
        for eps in (0.0, 1e-9, 1e-7, 3e-6, 5e-6, 1e-5, 1e-3):
            rows.append(p + eps * rng.choice([-1.0, 0.0, 1.0], p.shape))
    ins = np.concatenate(rows)
    s = ins + rng.integers(-reach, reach + 1, ins.shape)
    return s + s.sum(1, keepdims=True) / 3           # unskewed


@pytest.mark.parametrize("reach", [0, 3, 40, 9000])
def test_decisions_around_ties(reach):
    from nixis_gb300 import opensimplex as osx
    pts = _near_ties(np.random.default_rng(reach), reach)
    perm, pgi = O.init(reach)
    val, tr, sl, nfb = osx.noise3d_trace(pts, perm, pgi)
    want, want_tr, _ = O.noise3d_batch(pts, perm, pgi, trace=True)
    assert np.array_equal(tr.cpu().numpy(), want_tr)
    np.testing.assert_allclose(val.cpu().numpy(), want, rtol=0, atol=2e-6)
    if reach <= 40:          # both kinds of lanes (at large coordinates the offsets drown)
        assert 0 < nfb < len(pts)
    # all the orders of every region were among them
    ins = np.mod(pts - pts.sum(1, keepdims=True) / 6, 1.0)
    seen = {(int(r), tuple(np.argsort(i))) for r, i in zip(want_tr[:, 3], ins)}
    assert seen == set(itertools.product((0, 1, 2), itertools.permutations(range(3))))


@pytest.mark.parametrize("reach", [0, 40])
def test_pair_values_around_ties(reach):
    """0.5 (noise + 1) in pairs, as one octave (renormalised) and as one of small amplitude, to the path's 2e-13 of the
    summed amplitudes."""
    from nixis_gb300 import terrain
    pts = _near_ties(np.random.default_rng(reach + 1), reach)
    perm, pgi = O.init(5)
    for strength in ([1.0], [1.0, 1.0 / 16]):
        got, _ = terrain.fbm(torch.from_numpy(pts).cuda(), perm, pgi, [1.0] * len(strength), strength, 1.0)
        want = (O.noise3d_batch(pts, perm, pgi) + 1.0) * 0.5 * sum(strength)
        assert np.abs(got.cpu().numpy() - want).max() <= 2e-13 * sum(strength)


def test_gradients_that_start_anywhere():
    """Tables whose entries are no multiples of 3: components index, index + 1 and index + 2 of the reference's table, in
    binary32.  The path's 2e-6 times 16.1 / 12.3, the longest such gradient against the longest of init()'s."""
    from nixis_gb300 import opensimplex as osx, terrain
    rng = np.random.default_rng(2)
    pts = rng.uniform(-30.0, 30.0, (50_000, 3))
    perm, _ = O.init(3)
    pgi = rng.integers(0, 70, 256).astype(np.int32)
    want = O.noise3d_batch(pts, perm, pgi)
    val = osx.noise3d_trace(pts, perm, pgi)[0].cpu().numpy()
    np.testing.assert_allclose(val, want, rtol=0, atol=2.7e-6)
    got = terrain.fbm(torch.from_numpy(pts).cuda(), perm, pgi, [1.0], [2.0], 1.0, out_dtype=torch.float32)[0]
    np.testing.assert_allclose(got.cpu().numpy(), want + 1.0, rtol=0, atol=2.7e-6)


@pytest.mark.parametrize("octaves, x", [(1, 1e17), (4, 1e16), (4, 1e17), (12, 1e15), (12, 1e16)])
def test_coordinates_past_the_integers(octaves, x):
    """No lattice point is near there, so an octave adds half its strength and no more."""
    from nixis_gb300 import opensimplex, terrain
    perm, pgi = opensimplex.init(5)
    strength = [0.5 ** o for o in range(octaves)]
    got = terrain.fbm(np.full((3, 3), x), perm, pgi, [2.0 ** o for o in range(octaves)], strength, 1.0)[0]
    assert torch.equal(got, torch.full_like(got, 0.5 * sum(strength)))
    for x in (np.inf, -np.inf, np.nan):
        assert terrain.fbm(np.full((3, 3), x), perm, pgi, [1.0, 2.0], [1.0, 0.5], 1.0)[0].isnan().all()
