"""SITE with windows of many words, against the sequential greedy.

A row of a window spans up to 33 words from radius 993 on (1987 columns at bit 62 or 63)
and 64 at radius 2000, more than a warp has lanes.  VIEWSHED ends at radius 475, so the
viewsheds are made here: discs, whole or with random cells missing.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _disc_sheds(n, roi, obs, seed):
    """Packed viewsheds: the cells within roi of each observer, every other shed thinned."""
    rng = np.random.default_rng(seed)
    nr = 2 * roi + 1
    d = np.arange(nr) - roi
    disc = d[:, None] ** 2 + d[None, :] ** 2 <= roi * roi
    out = np.zeros((len(obs), nr, (nr + 63) // 64 * 64), np.uint8)
    for i, o in enumerate(obs):
        x, y = divmod(int(o), n)
        r, c = x + d, y + d
        inside = ((r >= 0) & (r < n))[:, None] & ((c >= 0) & (c < n))[None, :]
        cells = disc & inside
        if i % 2:
            cells &= rng.random((nr, nr)) < 0.7
            cells[roi, roi] = True
        out[i, :, :nr] = cells
    words = np.packbits(out, axis=-1).reshape(len(obs), nr, -1, 8)
    return np.ascontiguousarray(words[..., ::-1]).view(np.uint64).ravel()


@pytest.mark.parametrize("intervis", [0, 1])
@pytest.mark.parametrize("n, roi", [(2100, 991), (2300, 992), (4500, 993), (4500, 1023), (4500, 1024),
                                    (4500, 1500), (4600, 2000)])
def test_windows_of_more_words_than_lanes(native, oracle, n, roi, intervis):
    rng = np.random.default_rng(roi)
    # columns at every kind of bit, pairs that share nearly whole rows, and distant ones
    x = rng.integers(0, n, 12)
    y = np.clip(n // 2 + np.r_[0, 1, 5, 31, 62, 63, 64, 65, rng.integers(-n // 2, n // 2, 4)], 0, n - 1)
    obs = (x * n + y).astype(np.int32)
    sheds = _disc_sheds(n, roi, obs, roi)
    want, used, area, order = oracle.site(n, roi, intervis, obs, sheds, want_order=True)
    assert used > 1  # later picks' areas have lost the earlier ones' cells
    with native.Context(0) as ctx:
        for how in (2, 1):
            ctx.set_site_order(how)
            sel, res = ctx.site_it(n, roi, intervis, obs, sheds)
            assert np.array_equal(ctx.last_pick_order(len(obs)), order), f"order {how}"
            assert np.array_equal(sel, want)
            assert (res.nusedsheds, res.cumarea) == (used, area)
