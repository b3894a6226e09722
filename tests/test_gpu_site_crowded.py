"""SITE on observers that lie close together.

The order of a selection is chosen for the mean number of candidates in a circle; where
they are crowded, the count taken with the gains leaves the job to the global order.
The picks are the same whichever it is.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _observers(n, count, spread, seed):
    """Observers about the middle of the raster; spread 0: all on one cell, inf: anywhere."""
    rng = np.random.default_rng(seed)
    if np.isinf(spread):
        return rng.integers(0, n * n, count).astype(np.int32)
    xy = np.clip((rng.normal(size=(count, 2)) * spread + n / 2).astype(int), 0, n - 1)
    return (xy[:, 0] * n + xy[:, 1]).astype(np.int32)


@pytest.mark.parametrize("n, roi, count, intervis, spread, crowded", [
    (400, 6, 1500, 0, np.inf, False), (400, 6, 1500, 0, 4, True), (400, 6, 1500, 0, 0, True),
    (500, 5, 5000, 1, np.inf, False), (500, 5, 5000, 1, 12, True), (600, 8, 17000, 1, np.inf, False),
    (600, 8, 17000, 1, 15, True), (90, 1, 400, 0, 0, True), (300, 70, 1200, 0, 3, None),
])
def test_crowded_observers(native, oracle, n, roi, count, intervis, spread, crowded):
    dem = native.fbm_dem(n, seed=n + roi, octaves=7, range_max=6000)
    obs = _observers(n, count, spread, count)
    sheds = oracle.sheds(dem, n, roi, 20, 20, obs)
    want, used, area, order = oracle.site(n, roi, intervis, obs, sheds, want_order=True)
    for how in (0, 1, 2):
        with native.Context(0) as ctx:
            ctx.set_site_order(how)
            sel, res = ctx.site_it(n, roi, intervis, obs, sheds)
            assert np.array_equal(ctx.last_pick_order(count), order), f"order {how}"
            # the clock of the cut runs in the global order alone
            in_global_order = ctx.last_site_phase_cycles()[12] > 0
        assert np.array_equal(sel, want)
        assert (res.nusedsheds, res.cumarea) == (used, area)
        if how:
            assert in_global_order == (how == 1)
        elif crowded is not None:
            assert in_global_order == crowded
