"""VIX at small radii and few targets, and many small jobs with large radii in one grid.

Radii up to 2 and 8 unroll one and three samples; with one or two targets a cell and a large
radius only the tile is staged; few targets keep 32x32 tiles on a small raster.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, roi, ntests", [
    (70, 1, 5), (71, 2, 40), (72, 3, 5), (97, 4, 12), (130, 8, 9), (131, 9, 9), (300, 120, 1),
    (301, 130, 2), (302, 130, 3), (64, 200, 1), (450, 104, 2), (200, 60, 6), (200, 60, 7), (840, 5, 3),
])
def test_default_plan_matches_oracle(native, oracle, n, roi, ntests):
    dem = native.fbm_dem(n, seed=n + roi, octaves=7, range_max=9000)
    dem[:: 5] = 0
    with native.Context(0) as ctx:
        for oht, tht in ((0, 0), (25, 900)):
            want = oracle.vix(dem, n, roi, oht, tht, ntests)
            got = ctx.calc_vix(n, dem, roi, oht, tht, ntests)
            assert int(np.count_nonzero(got != want)) == 0


@pytest.mark.parametrize("mode", [1, 2])
def test_jobs_of_all_forms_in_one_batch(native, oracle, mode):
    jobs = [dict(nrows=n, roi=roi, height=15, ntests=nt, bw=bw, nwanted0=nw, intervis=iv) for
            n, roi, nt, bw, nw, iv in ((200, 2, 6, 10, 300, 0), (260, 110, 1, 20, 100, 1),
                                       (300, 120, 2, 20, 200, 0), (310, 130, 40, 20, 150, 1),
                                       (180, 8, 30, 8, 400, 1), (257, 150, 9, 16, 256, 0))]
    dems = [native.fbm_dem(j["nrows"], seed=i, octaves=7, range_max=8000) for i, j in enumerate(jobs)]
    refs = [oracle.run(d, *(j[k] for k in ("nrows", "roi", "height", "ntests", "bw", "nwanted0", "intervis")))
            for d, j in zip(dems, jobs)]
    with native.Context(0) as ctx:
        ctx.set_batch_mode(mode)
        for ref, (obs, sel, res) in zip(refs, ctx.run_batch([native.Params(**j) for j in jobs], dems)):
            assert np.array_equal(obs, ref["obs"])
            assert np.array_equal(sel, ref["selected"])
            assert (res.nusedsheds, res.cumarea) == (ref["nused"], ref["cumarea"])
