"""VIEWSHED launch forms at the edges of their ranges, word for word against the oracle.

Whole windows up to roi 74, halves from 75, quarters from 119, halves again from
209, quarters from 216 and L1 beyond; steps up to 16 mark bytes and later ones bits;
a ray's steps come in groups of four.  Observers at corners, edges and one cell
inside make the mirrored rays of a pair end at different steps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _observers(n, roi, count, seed):
    rng = np.random.default_rng(seed)
    e = [0, n - 1, n * (n - 1), n * n - 1, 1, n + 1, n * (n // 2), n * (n // 2) + n - 1, n // 2,
         n * (n - 1) + n // 2, (n // 2) * n + 3, 2 * n + n // 2, (n - 2) * n + n - 5]
    e += [min(roi, n - 1) * n + min(roi, n - 1), (n // 2) * n + n // 2]
    return np.unique(np.r_[e, rng.integers(0, n * n, count)]).astype(np.int32)


@pytest.mark.parametrize("roi", [1, 2, 4, 5, 15, 16, 17, 20, 21, 31, 32, 33, 63, 65, 74, 75, 111, 112,
                                 118, 119, 128, 159, 160, 208, 209, 215, 216, 310, 330])
def test_viewshed_forms_match_oracle(native, oracle, roi):
    n = max(61, 2 * roi + 35) | 1
    dem = native.fbm_dem(n, seed=roi, octaves=7, range_max=40000)
    d2 = dem.reshape(n, n)
    d2[n // 3:n // 2, n // 4:n // 2] = 20000  # a plateau: equal elevations along rays
    obs = _observers(n, roi, 12, roi)
    for oht, tht in ((0, 0), (150, 20)):
        want = oracle.sheds(dem, n, roi, oht, tht, obs)
        with native.Context(0) as ctx:
            for plan in (-1, 1, 2, 0):
                ctx.autotune_clear()
                if plan >= 0:
                    ctx.autotune_set(roi, 1, native.Plan(0, -1, plan, 0))
                got = ctx.calc_sheds(n, dem, roi, oht, tht, obs)
                bad = int(np.count_nonzero(got != want))
                assert bad == 0, f"plan {plan}, heights {oht}, {tht}: {bad} words differ"


@pytest.mark.parametrize("oht,tht", [(-3, 5), (1500000, 0), (0, -40), (1000000, 1000000)])
def test_heights_beyond_the_reciprocal_table(native, oracle, oht, tht):
    """Observer heights outside 0..10^6 divide instead of using the table."""
    n, roi = 150, 40
    dem = native.fbm_dem(n, seed=9, octaves=7, range_max=60000)
    obs = _observers(n, roi, 12, 1)
    want = oracle.sheds(dem, n, roi, oht, tht, obs)
    with native.Context(0) as ctx:
        got = ctx.calc_sheds(n, dem, roi, oht, tht, obs)
    assert int(np.count_nonzero(got != want)) == 0


def test_many_observers_random_sizes(native, oracle):
    rng = np.random.default_rng(5)
    for roi in (23, 90, 140, 200):
        n = int(rng.integers(300, 420))
        dem = native.fbm_dem(n, seed=roi, octaves=8, range_max=15000)
        obs = _observers(n, roi, 150, roi)
        with native.Context(0) as ctx:
            got = ctx.calc_sheds(n, dem, roi, 7, 3, obs)
        assert np.array_equal(got, oracle.sheds(dem, n, roi, 7, 3, obs))


def test_a_cluster_takes_several_quarters(native, oracle):
    # one CTA an SM from radius 216 on; 1300 observers give each cluster four halves
    n, roi = 470, 216
    dem = native.fbm_dem(n, seed=3, octaves=7, range_max=40000)
    obs = _observers(n, roi, 1300, 3)
    want = oracle.sheds(dem, n, roi, 60, 5, obs)
    with native.Context(0) as ctx:
        assert np.array_equal(ctx.calc_sheds(n, dem, roi, 60, 5, obs), want)
        bad = obs.copy()
        bad[[0, 5, 6, 641]] = n * n, -1, n * n + 7, -5  # first, inside and last of a cluster's
        with pytest.raises(native.SitingError):
            ctx.calc_sheds(n, dem, roi, 60, 5, bad)
        assert np.array_equal(ctx.calc_sheds(n, dem, roi, 60, 5, obs), want)
