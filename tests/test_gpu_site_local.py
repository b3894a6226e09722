"""SITE by local dominance, pick by pick against the sequential greedy.

With intervis it takes over at 16 384 candidates (4096 in no block order, as here),
unless they are dense: both sides of these lines; window widths of one word and two; candidates in any order
and on the same cell; one CTA, a few, and the default.  Every result is a whole
number, so all are compared exactly.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, roi, count, intervis, height", [
    (256, 5, 16384, 1, 10), (256, 5, 16383, 1, 10), (256, 1, 20000, 1, 0), (257, 12, 16641, 1, 60),
    (600, 12, 17000, 1, 60),
    (200, 4, 4096, 1, 10), (200, 4, 4095, 1, 10), (200, 12, 4096, 1, 10),
    (700, 31, 16400, 1, 150), (700, 32, 16400, 1, 40), (331, 2, 17000, 1, 5),
    (64, 3, 300, 0, 10), (97, 40, 60, 0, 100), (33, 16, 500, 0, 50), (50, 1, 2500, 0, 0),
    (40, 5, 1, 0, 10), (300, 63, 700, 0, 200), (300, 64, 700, 0, 200), (256, 5, 16384, 0, 10),
])
def test_picks_match_the_sequential_greedy(native, oracle, n, roi, count, intervis, height):
    rng = np.random.default_rng(n + roi + count)
    dem = native.fbm_dem(n, seed=n + roi, octaves=7, range_max=6000)
    obs = rng.integers(0, n * n, count).astype(np.int32)  # any order, some cells twice
    sheds = oracle.sheds(dem, n, roi, height, height, obs)
    want, used, area, order = oracle.site(n, roi, intervis, obs, sheds, want_order=True)
    for ctas in (0, 1, 7):
        if ctas and -(-count // ctas) > 4096:
            continue  # more than a CTA takes
        with native.Context(0) as ctx:
            ctx.set_site_ctas(ctas)
            sel, res = ctx.site_it(n, roi, intervis, obs, sheds)
            got = ctx.last_pick_order(count)
        assert np.array_equal(got, order), f"{ctas} CTAs"
        assert np.array_equal(sel, want)
        assert (res.nusedsheds, res.cumarea) == (used, area)


def test_noalloc_scratch_holds_a_local_selection(native, oracle):
    torch = pytest.importorskip("torch")
    n, roi, count = 256, 5, 16384
    dem = native.fbm_dem(n, seed=9, octaves=7, range_max=6000)
    obs = np.random.default_rng(9).permutation(n * n)[:count].astype(np.int32)
    sheds = oracle.sheds(dem, n, roi, 10, 10, obs)
    d_obs = torch.from_numpy(obs).cuda()
    d_sheds = torch.from_numpy(sheds.view(np.int64)).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    for intervis in (1, 0, 1):
        want, used, area = oracle.site(n, roi, intervis, obs, sheds)
        sel = torch.full((count,), 7, dtype=torch.uint8, device="cuda")
        res = native._ResultC()
        rc = native.load().siting_site_it_noalloc(n, roi, intervis, count, d_obs.data_ptr(),
                                                  d_sheds.data_ptr(), sel.data_ptr(), C.c_void_p(stream),
                                                  C.byref(res))
        assert rc == 0
        assert np.array_equal(sel.cpu().numpy(), want)
        assert (res.nusedsheds, res.cumarea) == (used, area)


@pytest.mark.parametrize("ctas", [1, 42, 43, 85, 86, 152])
def test_global_order_takes_picks_by_one_warp_or_by_ranking(native, oracle, ctas):
    # 3 published keys a CTA: up to 256 are taken by one warp, more are ranked
    n, roi, count = 180, 9, 1500
    dem = native.fbm_dem(n, seed=4, octaves=7, range_max=6000)
    obs = np.random.default_rng(4).integers(0, n * n, count).astype(np.int32)
    sheds = oracle.sheds(dem, n, roi, 15, 15, obs)
    want, used, area, order = oracle.site(n, roi, 1, obs, sheds, want_order=True)
    with native.Context(0) as ctx:
        ctx.set_site_ctas(ctas)
        sel, res = ctx.site_it(n, roi, 1, obs, sheds)
        assert np.array_equal(ctx.last_pick_order(count), order)
    assert np.array_equal(sel, want)
    assert (res.nusedsheds, res.cumarea) == (used, area)
