"""VIX launch forms at the edges of their ranges, bit for bit against the oracle.

The number of unrolled samples changes at roi 32, 64 and 128; the far form reads
samples at offsets 128, 256, ... through L1; a tile takes the unchecked path only
where the whole radius lies inside the DEM.  Every plan must give the oracle's
bytes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLANS = [(0, -1), (16, 1), (32, 1), (64, 1), (16, 0), (32, 0)]


@pytest.mark.parametrize("n,roi,ntests,oht,tht", [
    (65, 1, 3, 0, 0), (130, 16, 9, 5, 0), (131, 32, 33, 0, 7), (200, 33, 5, 20, 3),
    (257, 64, 8, 0, 900000), (258, 65, 8, 1000000, 0), (330, 102, 71, 9, 9),
    (331, 104, 72, 9, 9), (400, 128, 5, 50, 0), (401, 129, 5, 50, 0), (620, 257, 4, 300, 40),
    (150, 600, 6, 3, 3),
])
def test_vix_plans_match_oracle(native, oracle, n, roi, ntests, oht, tht):
    dem = native.fbm_dem(n, seed=n + roi, octaves=7, range_max=12000)
    dem[:: 7] = 0
    want = oracle.vix(dem, n, roi, oht, tht, ntests)
    with native.Context(0) as ctx:
        for tile, smem in PLANS:
            ctx.autotune_clear()
            if tile:
                ctx.autotune_set(roi, ntests, native.Plan(tile, smem, -1, 0))
            got = ctx.calc_vix(n, dem, roi, oht, tht, ntests)
            bad = int(np.count_nonzero(got != want))
            assert bad == 0, f"plan {(tile, smem)}: {bad} of {n * n} cells differ"
