"""Rescaling by every size of width: the product by the width is put together from integers, in binary64 outside its
range and where it ends in a half.  The reference's operations, in order, are binary64's, so results are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lower, upper", [(0.0, 65535.0), (-4000.0, 8850.0), (8850.0, -4000.0), (0.0, 1.0), (0.0, 3e-160), (1.0, 1.0),
                                          (-1e150, 1e160), (0.0, 5e-324), (-1e308, 1e307), (0.0, 2.0 ** 500), (0.0, 2.0 ** -501)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 3e5])
def test_rescale_is_the_reference_arithmetic(lower, upper, scale):
    from nixis_gb300 import util
    rng = np.random.default_rng(4)
    x = np.concatenate([rng.normal(size=20_000), np.round(rng.normal(0, 40, 4_000)) / 64, [0.0, -0.0, 1.0, 1.5]]) * scale
    with np.errstate(all="ignore"):
        want = (x - x.min()) / (x.max() - x.min()) * (upper - lower) + lower
        assert np.array_equal(util.rescale(x, lower, upper), want)


def test_products_that_end_in_a_half():
    """Significands of 27 and 27 bits, whose product has 53 bits and a half."""
    from nixis_gb300 import util
    rng = np.random.default_rng(5)
    a = (rng.integers(2 ** 26, 2 ** 27, 100_000) | 1) / 2.0 ** 27
    x = np.concatenate([[0.0, 1.0], a])                    # the span is 1, the quotients are x
    for w in (2.0 ** 26 + 1, 2.0 ** 27 - 1, 94_906_267.0):
        assert np.array_equal(util.rescale(x, 0.0, w), x / 1.0 * w + 0.0)
