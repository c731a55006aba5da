"""Height shaping at the edges of its chunks and of its number ranges, against the oracle.

rescale and the range, mask and level decisions are exact; the power step is held to 4 units in the last place of the
largest result, as elsewhere (the reference's libm pow is not correctly rounded).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def field(kind, n):
    rng = np.random.default_rng(n)
    return {
        "normal": lambda: rng.normal(0.0, 1.0, n),
        "descending": lambda: np.linspace(5.0, -5.0, n),          # every value a new running minimum
        "ascending": lambda: np.linspace(-5.0, 5.0, n),
        "constant": lambda: np.full(n, 3.25),                     # 0 / 0 everywhere
        "ties": lambda: np.round(rng.normal(0.0, 3.0, n)),
        "zeros": lambda: np.where(rng.random(n) < 0.5, 0.0, -0.0),
        "tiny": lambda: rng.normal(0.0, 1e-9, n),                 # a range below 2^-28
        "huge": lambda: rng.normal(0.0, 1e12, n),                 # a range above 2^28
        "spread": lambda: rng.normal(0.0, 1.0, n) * 10.0 ** rng.integers(-18, 12, n),
    }[kind]()


def ulps(got, want):
    if np.array_equal(got, want, equal_nan=True):
        return 0.0
    assert np.array_equal(np.isnan(got), np.isnan(want))
    return float(np.nanmax(np.abs(got - want)) / np.spacing(np.nanmax(np.abs(want))))


@pytest.mark.parametrize("kind", ["normal", "descending", "ascending", "constant", "ties", "zeros", "tiny", "huge", "spread"])
@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 100002])
def test_shaping_equals_the_oracle(kind, n):
    from nixis_gb300 import util
    x = field(kind, n)
    with np.errstate(all="ignore"):
        want, mask, level = O.shape_heights(x)
    got, gmask, glevel = util.shape_heights(x)
    assert np.array_equal(gmask, mask.astype(bool)) and (glevel == level or (np.isnan(glevel) and np.isnan(level)))
    # where the ocean or the land has one value, its curve is 0 / 0 and np.max's treatment of it decides the rest
    h1 = O.rescale_full(x, -4000.0, 8850.0)
    if not np.isnan(want).any() and min(len(np.unique(h1[gmask])), len(np.unique(h1[~gmask]))) > 1:
        assert ulps(got, want) <= 4
    for args in ({}, {"mid": 0.25}, {"mid": 0.0}, {"mid": 0.25, "mode": "lower"}, {"mid": -0.25, "mode": "upper"}):
        assert np.array_equal(util.rescale(x, -4000.0, 8850.0, **args), O.rescale_full(x, -4000.0, 8850.0, **args), equal_nan=True)
    m = np.random.default_rng(7).random(n) < 0.5
    for mode in (0, 1):
        for power in (0.5, 1.0, 2.0):
            with np.errstate(all="ignore"):
                want = O.power_rescale(x, m.astype(np.uint8), mode, power)
            assert ulps(util.power_rescale(x, m, mode, power), want) <= 4, (mode, power)


@pytest.mark.parametrize("field", [[5.0, 7.0, 6.0], [-5.0, -7.0, -6.0], [-1.0, 2.0, 0.5]])
@pytest.mark.parametrize("at", [0, 2, 3])
def test_nans_by_their_sign(field, at):
    """A negative NaN is the smallest key, so the minimum is NaN; a positive one counts as a number right below 0."""
    from nixis_gb300 import util
    x = np.insert(field, at, np.nan)
    y = x.copy()
    y.view(np.uint64)[at] ^= np.uint64(1 << 63)
    number = ~np.isnan(x)
    lo, hi = min(min(field), 0.0), max(max(field), 0.0)
    assert np.allclose(util.rescale(x, 0.0, 1.0), (x - lo) / (hi - lo), rtol=1e-15, equal_nan=True)
    assert np.isnan(util.rescale(y, 0.0, 1.0)).all()
    above = number & (x > 0.6)
    for v in (x, y):
        assert np.array_equal(util.rescale(v, 0.0, 1.0, mid=0.6)[above], ((x - 0.6) / (max(hi, 0.0) - 0.6) * 0.4 + 0.6)[above])
    assert np.array_equal(np.isnan(util.rescale(y, 0.0, 1.0, mid=0.6)), ~above)
    everywhere = np.ones(4, bool)
    assert np.array_equal(np.isnan(util.power_rescale(x, everywhere, 1, 2.0)), ~number)
    assert np.isnan(util.power_rescale(y, everywhere, 1, 2.0)).all()
    assert np.array_equal(np.isnan(util.shape_heights(x)[0]), ~number) and np.isnan(util.shape_heights(y)[0]).all()


@pytest.mark.parametrize("field, nans", [([0.0, 1.0, 0.99, 0.98], [0]), ([1.0, 0.0, 0.01, 0.02], [0, 1, 2, 3]), ([0.0, 1.0], [0, 1]),
                                         ([0.0, 0.8, 0.9, 1.0], [0])])
def test_a_single_vertex_of_ocean_or_land(field, nans):
    """Its curve is 0 / 0, the minimum of the last rescale: no number there and in the ocean, the land is mapped."""
    from nixis_gb300 import util
    h, _, level = util.shape_heights(np.array(field))
    assert np.flatnonzero(np.isnan(h)).tolist() == nans and level == 3067.5
