"""Exact ties in the matrix profile: windows of a series that repeats itself
bitwise have many partners at distance zero, and the lowest one is reported,
also where the lists of near-minimal pairs overflow (short periods)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lowest_partner(s, m, period):
    """Lowest window at a multiple of the period with the window length between."""
    i = np.arange(s)
    first = i % period
    up = i + -(-m // period) * period  # the nearest later one
    return np.where(i - first >= m, first, np.where(up < s, up, -1))


# rows on one to several tiles of 4,032 rows and 896 lags, whole and cut tiles;
# 9,001 samples at period 97 and 2,000 at 24 overflow the lists
@pytest.mark.parametrize("n,m,period", [(3001, 16, 97), (2000, 8, 24), (5003, 64, 449),
                                        (9001, 128, 700), (9001, 128, 97), (13000, 300, 2999)])
def test_lowest_partner_of_a_periodic_series(gpu_dtwj, n, m, period):
    x = np.resize(np.random.default_rng(n + period).standard_normal(period), n)
    mp, mpi = gpu_dtwj.matrix_profile(x, m)
    ref = _lowest_partner(n - m + 1, m, period)
    has = ref >= 0
    np.testing.assert_array_equal(mpi[has], ref[has])
    # bitwise equal windows: their statistics are equal too, the distance is zero up to
    # the rounding of the two means (2 ulp of a mean per sample)
    assert mp[has].max() <= 1e-12
