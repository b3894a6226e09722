"""VIEWSHED on device buffers with observers outside the DEM, and the largest quarters.

The device entry does not see the indices: its kernels write an empty shed for each bad
observer, whatever the form of the launch and the place in it, and read no cell for it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheds_dev(native, ctx, n, dem, roi, oht, tht, obs):
    torch = pytest.importorskip("torch")
    d_dem = torch.from_numpy(dem.view(np.int16)).cuda()
    d_obs = torch.from_numpy(obs).cuda()
    out = torch.full((len(obs) * native.shed_words(roi),), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.calc_sheds_dev(n, d_dem, roi, oht, tht, len(obs), d_obs, out)
    ctx.sync()
    return out.cpu().numpy().view(np.uint64).reshape(len(obs), -1)


@pytest.mark.parametrize("roi, count", [(5, 400), (12, 6000), (60, 300), (90, 300), (140, 300),
                                        (212, 700), (216, 1300), (256, 1300), (320, 40)])
def test_bad_observers_have_empty_sheds(native, oracle, roi, count):
    n = 2 * roi + 37
    rng = np.random.default_rng(roi)
    dem = native.fbm_dem(n, seed=roi, octaves=7, range_max=30000)
    obs = rng.integers(0, n * n, count).astype(np.int32)
    want = oracle.sheds(dem, n, roi, 60, 5, obs).reshape(count, -1).copy()
    bad = np.unique(np.r_[0, 1, 5, 6, count // 2, count // 2 + 1, count - 2, count - 1])
    values = [n * n, -1, n * n + 7, -5, 2**31 - 1, -2**31]
    wrong = obs.copy()
    wrong[bad] = [values[i % len(values)] for i in range(len(bad))]
    with native.Context(0) as ctx:
        for plan in (-1, 1, 2, 0):
            ctx.autotune_clear()
            if plan >= 0:
                ctx.autotune_set(roi, 1, native.Plan(0, -1, plan, 0))
            got = _sheds_dev(native, ctx, n, dem, roi, 60, 5, wrong)
            assert not got[bad].any(), f"plan {plan}"
            good = np.setdiff1d(np.arange(count), bad)
            assert np.array_equal(got[good], want[good]), f"plan {plan}"
            assert np.array_equal(_sheds_dev(native, ctx, n, dem, roi, 60, 5, obs), want), f"plan {plan}"


@pytest.mark.parametrize("roi", [254, 255, 256, 288, 289, 303, 304])
def test_quarters_of_two_boxes(native, oracle, roi):
    """A quarter has roi + 1 rows: two boxes from radius 256 on; 48 near steps end at 288
    and quarters at 303.  Enough observers for clusters that take several halves."""
    n = roi + 150
    dem = native.fbm_dem(n, seed=roi, octaves=7, range_max=40000)
    rng = np.random.default_rng(roi)
    obs = np.r_[[0, n - 1, n * (n - 1), n * n - 1, (n // 2) * n + n // 2],
                rng.integers(0, n * n, 1300)].astype(np.int32)
    want = oracle.sheds(dem, n, roi, 40, 8, obs)
    with native.Context(0) as ctx:
        for plan in (1, -1):
            ctx.autotune_clear()
            if plan >= 0:
                ctx.autotune_set(roi, 1, native.Plan(0, -1, plan, 0))
            assert np.array_equal(ctx.calc_sheds(n, dem, roi, 40, 8, obs), want), f"plan {plan}"


@pytest.mark.parametrize("n, roi, count", [(128, 110, 400), (128, 100, 400), (448, 216, 400), (512, 209, 151),
                                           (512, 209, 152), (384, 240, 400), (200, 180, 400), (20, 16, 300)])
def test_windows_through_l1_and_the_pitch_of_the_dem(native, oracle, n, roi, count):
    """Large radii and rasters smaller than a window: through L1 from one observer an SM on,
    from a copy of the DEM where its rows are whole cache lines; without one in a budget."""
    dem = native.fbm_dem(n, seed=n + roi, octaves=6, range_max=20000)
    obs = np.random.default_rng(n).integers(0, n * n, count).astype(np.int32)
    want = oracle.sheds(dem, n, roi, 30, 10, obs)
    for budget in (0, 1 << 30):
        with native.Context(0, hbm_budget=budget) as ctx:
            assert np.array_equal(ctx.calc_sheds(n, dem, roi, 30, 10, obs), want)
            got = _sheds_dev(native, ctx, n, dem, roi, 30, 10, obs)
            assert np.array_equal(got.ravel(), want)


def test_jobs_whose_dem_is_copied(native, oracle):
    torch = pytest.importorskip("torch")
    job = dict(nrows=320, roi=212, height=40, ntests=8, bw=16, nwanted0=400, intervis=1)
    dem = native.fbm_dem(320, seed=2, octaves=7, range_max=20000)
    ref = oracle.run(dem, *(job[k] for k in ("nrows", "roi", "height", "ntests", "bw", "nwanted0", "intervis")))
    p = native.Params(**job)
    d_dem = torch.from_numpy(dem.view(np.int16)).cuda()
    d_obs = [torch.empty(len(ref["obs"]), dtype=torch.int32, device="cuda") for _ in range(2)]
    d_sel = [torch.empty(len(ref["obs"]), dtype=torch.uint8, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()

    def same(obs, sel, res):
        assert np.array_equal(obs, ref["obs"]) and np.array_equal(sel, ref["selected"])
        assert (res.nusedsheds, res.cumarea) == (ref["nused"], ref["cumarea"])

    with native.Context(0) as ctx:
        same(*ctx.run(p, dem))
        res = ctx.run_dev(p, d_dem, d_obs[0], d_sel[0])
        same(d_obs[0].cpu().numpy(), d_sel[0].cpu().numpy(), res)
        for got in ctx.run_batch([p, p], [dem, dem]):
            same(*got)
        for _ in range(2):  # captured, then replayed
            rs = ctx.run_batch_dev([p, p], [d_dem, d_dem], d_obs, d_sel)
            for o, s, res in zip(d_obs, d_sel, rs):
                same(o.cpu().numpy(), s.cpu().numpy(), res)
    with native.Server(0) as srv:
        obs, sel, info = srv.wait(srv.submit(p, dem))
        same(obs, sel, info.result)


@pytest.mark.parametrize("roi", [7, 12, 80, 130, 215, 216, 320])
@pytest.mark.parametrize("oht, tht", [(-3, 5), (1500000, 0)])
def test_heights_that_divide_in_every_form(native, oracle, roi, oht, tht):
    """Observer heights outside 0..10^6 divide: whole and half windows, and through L1."""
    n = 2 * roi + 45
    dem = native.fbm_dem(n, seed=roi, octaves=7, range_max=60000)
    obs = np.random.default_rng(roi).integers(0, n * n, 160).astype(np.int32)
    want = oracle.sheds(dem, n, roi, oht, tht, obs)
    with native.Context(0) as ctx:
        for plan in (-1, 1, 2, 0):
            ctx.autotune_clear()
            if plan >= 0:
                ctx.autotune_set(roi, 1, native.Plan(0, -1, plan, 0))
            assert np.array_equal(ctx.calc_sheds(n, dem, roi, oht, tht, obs), want), f"plan {plan}"
