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


def test_the_sign_of_a_nan_does_not_matter():
    """A NaN of either sign is np.max's result and not np.min's, so what lies below `mid` keeps its values."""
    from nixis_gb300 import util
    x = np.random.default_rng(4).normal(size=5000)
    x[17] = np.nan
    y = x.copy()
    y.view(np.uint64)[17] ^= np.uint64(1 << 63)
    for args, nans in (({}, 5000), ({"mid": 0.25}, 1 + (x > 0.25).sum()), ({"mid": 0.25, "mode": "lower"}, 1),
                       ({"mid": -0.25, "mode": "upper"}, 1 + (x > -0.25).sum())):
        a, b = util.rescale(x, -1.0, 2.0, **args), util.rescale(y, -1.0, 2.0, **args)
        assert np.array_equal(a, b, equal_nan=True) and np.isnan(a).sum() == nans
    m = np.random.default_rng(5).random(5000) < 0.5
    for mode in (0, 1):
        assert np.array_equal(util.power_rescale(x, m, mode, 2.0), util.power_rescale(y, m, mode, 2.0), equal_nan=True)
    assert np.array_equal(util.make_bool_elevation_mask(x, 0.1), util.make_bool_elevation_mask(y, 0.1))
