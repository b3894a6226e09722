"""SITE on viewsheds with bits farther than roi from their observer.

The packed form has room for the whole square about an observer.  Two picks that are more
than 2*roi apart can then cover one cell, which the selection by local dominance rules
out: such a job is taken in the global key order, whichever order is asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROI = 20


def _groups(count, side):
    """Groups of three: two whole squares that overlap at their corners, and a candidate in
    the overlap, seen by both and of neither's neighbourhood in its own cells."""
    n = side * 100
    nr = 2 * ROI + 1
    obs, sheds = [], []
    for g in range(count):
        x, y = 30 + 100 * (g // side), 30 + 100 * (g % side)
        for k, (dx, dy) in enumerate(((0, 0), (30, 30), (15, 15))):
            cells = np.zeros((nr, 64), np.uint8)
            if k < 2:
                cells[:, :nr] = 1
                cells[ROI, ROI + 1:ROI + 1 + 2 * g + k] = 0  # no two areas alike
            else:
                cells[:15 - g, ROI + 6:] = 1  # beyond the first's columns, before the second's rows
                cells[:, nr:] = 0
            obs.append((x + dx) * n + y + dy)
            sheds.append(np.packbits(cells, axis=-1)[:, ::-1].copy().view(np.uint64).ravel())
    return n, np.array(obs, np.int32), np.concatenate(sheds)


@pytest.mark.parametrize("intervis", [0, 1])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_squares_that_overlap_at_their_corners(native, oracle, order, intervis):
    n, obs, sheds = _groups(9, 3)
    want, used, area, picks = oracle.site(n, ROI, intervis, obs, sheds, want_order=True)
    assert used == len(obs)
    with native.Context(0) as ctx:
        ctx.set_site_order(order)
        sel, res = ctx.site_it(n, ROI, intervis, obs, sheds)
        assert np.array_equal(ctx.last_pick_order(len(obs)), picks)
        assert (res.nusedsheds, res.cumarea) == (used, area)
        assert np.array_equal(sel, want)
        # within roi again: the same context, by local dominance where asked
        dem = np.zeros(n * n, np.uint16)
        flat = oracle.sheds(dem, n, ROI, 5, 5, obs)
        want, used, area, picks = oracle.site(n, ROI, intervis, obs, flat, want_order=True)
        sel, res = ctx.site_it(n, ROI, intervis, obs, flat)
        assert np.array_equal(ctx.last_pick_order(len(obs)), picks)
        assert np.array_equal(sel, want)


@pytest.mark.parametrize("roi", [1, 2, 3, 31, 32, 40, 127, 200])
@pytest.mark.parametrize("inside", [True, False])
def test_one_bit_at_the_rim(native, oracle, roi, inside):
    """The disc's outermost cells are within roi; the nearest cells beyond it are not."""
    n, nr = 4 * roi + 9, 2 * roi + 1
    nw = (nr + 63) // 64
    d = np.arange(nr) - roi
    far = d[:, None] ** 2 + d[None, :] ** 2
    rim = far[far <= roi * roi].max() if inside else far[far > roi * roi].min()
    cells = np.argwhere(far == rim)
    obs = np.full(len(cells) + 1, (n // 2) * n + n // 2, np.int32)
    bits = np.zeros((len(obs), nr, nw * 64), np.uint8)
    bits[:, roi, roi] = 1
    for i, (r, c) in enumerate(cells):
        bits[i, r, c] = 1
    sheds = np.packbits(bits, axis=-1).reshape(len(obs), nr, nw, 8)[..., ::-1].copy().view(np.uint64).ravel()
    want, used, area, picks = oracle.site(n, roi, 0, obs, sheds, want_order=True)
    with native.Context(0) as ctx:
        rounds = []
        for order in (1, 2):
            ctx.set_site_order(order)
            sel, res = ctx.site_it(n, roi, 0, obs, sheds)
            assert np.array_equal(ctx.last_pick_order(len(obs)), picks)
            assert np.array_equal(sel, want)
            rounds.append(ctx.last_site_phase_cycles()[12])
        # the clock of the cut runs in the global order alone
        assert rounds[0] > 0
        assert (rounds[1] == 0) == inside
