"""SITE in the global key order and by local dominance: the same picks in the same order.

Few, dense, sparse and equal candidates, with and without intervis, on both sides of the
lines by which the order is chosen; each pinned and chosen.  Every result is a whole
number, so all are compared exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, roi, count", [
    (40, 5, 1), (60, 9, 31), (200, 4, 127), (200, 4, 128), (300, 3, 129), (97, 40, 60),
    (33, 16, 500), (64, 3, 300), (50, 1, 2500), (300, 31, 1023), (300, 31, 1024), (300, 63, 700),
    (300, 64, 700), (260, 46, 1100), (260, 48, 1100), (900, 7, 160), (130, 130, 200),
])
@pytest.mark.parametrize("intervis", [0, 1])
def test_both_orders_match_the_sequential_greedy(native, oracle, n, roi, count, intervis):
    rng = np.random.default_rng(n + roi + count)
    dem = native.fbm_dem(n, seed=n + roi, octaves=7, range_max=6000)
    obs = rng.integers(0, n * n, count).astype(np.int32)  # any order, some cells twice
    sheds = oracle.sheds(dem, n, roi, 20, 20, obs)
    want, used, area, order = oracle.site(n, roi, intervis, obs, sheds, want_order=True)
    for ctas in (0, 1, 7):
        for how in (0, 1, 2):
            with native.Context(0) as ctx:
                ctx.set_site_ctas(ctas)
                ctx.set_site_order(how)
                sel, res = ctx.site_it(n, roi, intervis, obs, sheds)
                got = ctx.last_pick_order(count)
            assert np.array_equal(got, order), f"{ctas} CTAs, order {how}"
            assert np.array_equal(sel, want)
            assert (res.nusedsheds, res.cumarea) == (used, area)


@pytest.mark.parametrize("n, roi, bw, count, intervis", [
    (287, 20, 12, 648, 0), (287, 90, 12, 648, 0), (512, 60, 25, 400, 0), (400, 9, 20, 1600, 1)])
def test_jobs_in_both_orders(native, oracle, n, roi, bw, count, intervis):
    dem = native.fbm_dem(n, seed=n, octaves=7, range_max=6000)
    ref = oracle.run(dem, n, roi, 20, 16, bw, count, intervis)
    p = native.Params(nrows=n, roi=roi, height=20, ntests=16, bw=bw, nwanted0=count, intervis=intervis)
    for how in (0, 1, 2):
        with native.Context(0) as ctx:
            ctx.set_site_order(how)
            obs, sel, res = ctx.run(p, dem)
        assert np.array_equal(obs, ref["obs"])
        assert np.array_equal(sel, ref["selected"]), f"order {how}"
        assert (res.nusedsheds, res.cumarea) == (ref["nused"], ref["cumarea"])


def test_an_unknown_order_is_refused(native):
    with native.Context(0) as ctx:
        for how in (-1, 3):
            with pytest.raises(native.SitingError):
                ctx.set_site_order(how)


@pytest.mark.parametrize("n, roi, count, local", [
    (460, 19, 4096, True), (460, 19, 4095, False), (450, 19, 4096, False), (454, 28, 4096, True),
    (454, 29, 4096, False), (452, 12, 10000, True),
    (440, 12, 10000, False), (200, 3, 5000, True), (600, 3, 4500, True), (800, 3, 4500, False)])
def test_the_line_for_observers_in_no_block_order(native, oracle, n, roi, count, local):
    """Intervis, one block: 80 circles on the raster, the share of cells, the bins' size."""
    side = int(np.ceil(np.sqrt(count)))
    i = np.arange(count)
    jitter = np.random.default_rng(n).random((2, count)) * 0.9
    x = ((i // side + jitter[0]) * (n / side)).astype(int)  # one in each square of a grid
    y = ((i % side + jitter[1]) * (n / side)).astype(int)
    obs = (np.clip(x, 0, n - 1) * n + np.clip(y, 0, n - 1)).astype(np.int32)
    dem = native.fbm_dem(n, seed=n, octaves=7, range_max=6000)
    sheds = oracle.sheds(dem, n, roi, 20, 20, obs)
    want, used, area, order = oracle.site(n, roi, 1, obs, sheds, want_order=True)
    with native.Context(0) as ctx:
        sel, res = ctx.site_it(n, roi, 1, obs, sheds)
        assert np.array_equal(ctx.last_pick_order(count), order)
        # the clock of the cut runs in the global order alone
        assert (ctx.last_site_phase_cycles()[12] == 0) == local
    assert np.array_equal(sel, want)
    assert (res.nusedsheds, res.cumarea) == (used, area)


@pytest.mark.parametrize("n, roi, count, top", [(700, 3, 6000, 6000), (1000, 3, 9000, 6000), (1600, 35, 4000, 9000), (330, 1, 20000, 1),
                                                (900, 12, 9000, 3000), (520, 4, 1030, 6000)])
@pytest.mark.parametrize("intervis", [0, 1])
def test_the_order_of_many_picks(native, oracle, n, roi, count, top, intervis):
    """More than 8192 picks, 1024 with intervis, are put in order by buckets: small and large
    areas, equal ones."""
    dem = native.fbm_dem(n, seed=n, octaves=7, range_max=top)
    obs = np.random.default_rng(n).integers(0, n * n, count).astype(np.int32)
    sheds = oracle.sheds(dem, n, roi, 3, 3, obs)
    want, used, area, order = oracle.site(n, roi, intervis, obs, sheds, want_order=True)
    for ctas in (0, 5):
        with native.Context(0) as ctx:
            ctx.set_site_ctas(ctas)
            ctx.set_site_order(2)
            sel, res = ctx.site_it(n, roi, intervis, obs, sheds)
            assert np.array_equal(ctx.last_pick_order(count), order), f"{ctas} CTAs"
        assert np.array_equal(sel, want)
        assert (res.nusedsheds, res.cumarea) == (used, area)


@pytest.mark.parametrize("ctas, local", [(4, True), (8, True), (32, False), (0, False)])
def test_the_line_for_narrow_groups(native, oracle, ctas, local):
    """Two circles on the raster: a group of few CTAs goes by local dominance."""
    n, roi, count = 300, 120, 1100
    dem = native.fbm_dem(n, seed=5, octaves=7, range_max=9000)
    obs = np.random.default_rng(5).integers(0, n * n, count).astype(np.int32)
    sheds = oracle.sheds(dem, n, roi, 20, 20, obs)
    want, used, area, order = oracle.site(n, roi, 0, obs, sheds, want_order=True)
    with native.Context(0) as ctx:
        ctx.set_site_ctas(ctas)
        sel, res = ctx.site_it(n, roi, 0, obs, sheds)
        assert np.array_equal(ctx.last_pick_order(count), order)
        assert (ctx.last_site_phase_cycles()[12] == 0) == local
    assert np.array_equal(sel, want) and (res.nusedsheds, res.cumarea) == (used, area)
