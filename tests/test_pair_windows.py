"""The pairs of rays of VIEWSHED's forms, checked on the CPU against the oracle.

`shed_kernel` and `shed_quad_kernel` (siting_gb300/csrc/viewshed.cu) give a thread two
perimeter rays (siting.cpp:291-304) that mirror each other: about the observer's column in
whole and half windows, about the quadrant's diagonal in quarters.  This module restates
which pairs each CTA of a form takes and in which order, sweeps them (siting.cpp:252-360)
and checks for each observer that
* the pairs of a form are the 8*roi perimeter rays, and only straight and diagonal rays come
  twice;
* every sample of a CTA lies in the window that it stages;
* the marks that a CTA drops, on the observer's row (lower side) and column (left side of
  quarters), are among those of the CTA that writes them;
* the kept marks together are the oracle's shed.
The restatement is test infrastructure; the GPU tests check the kernels themselves.
"""
import numpy as np
import pytest

F32 = np.float32


def _ordered(count):
    """Lanes take every second ray: the even numbers, then the odd ones."""
    evens = (count + 1) // 2
    return [2 * t if t < evens else 2 * (t - evens) + 1 for t in range(count)]


def ctas(form, roi):
    """The CTAs of a form: rows and columns of the window, targets of the pairs, and which
    marks are kept, by the signs of row and column distance."""
    up, down, left, right = (-1, 0), (0, 1), (-1, 0), (0, 1)
    if form == "quarters":
        for sx, rows in ((-1, up), (1, down)):
            for sy, cols in ((1, right), (-1, left)):
                pairs = []
                for m in _ordered(roi + 1):
                    pairs += [(sx * roi, sy * m), (sx * m, sy * roi)]
                yield rows, cols, pairs, (lambda dx, dy, sx=sx, sy=sy:
                                          (sx < 0 or dx > 0) and (sy > 0 or dy < 0))
        return
    halves = []
    for sx in (-1, 1):
        pairs = []
        for m in _ordered(roi + 1):
            pairs += [(sx * roi, m), (sx * roi, -m)]
        first = 1 if form == "one warp" or sx > 0 else 0  # the observer's row: the upper side's
        for m in _ordered(roi - first):
            pairs += [(sx * (m + first), roi), (sx * (m + first), -roi)]
        halves.append(pairs)
    if form == "halves":
        yield up, (-1, 1), halves[0], lambda dx, dy: True
        yield down, (-1, 1), halves[1], lambda dx, dy: dx > 0
    else:
        row = [(0, roi), (0, -roi)] if form == "one warp" else []
        yield (-1, 1), (-1, 1), halves[0] + halves[1] + row, lambda dx, dy: True


def sweep(dem, n, roi, oht, tht, ox, oy, dx, dy):
    """Offsets from the observer of a ray's samples and of those that it marks."""
    y_major = abs(dx) < abs(dy)
    major, minor = (dy, dx) if y_major else (dx, dy)
    slope = abs(F32(minor) / F32(major))
    foalt, ftht = F32(int(dem[ox * n + oy]) + oht), F32(tht)
    hs, seen, marks = F32(-99999.0), [], []
    for k in range(1, roi + 1):
        off = int(np.floor(float(F32(k) * slope) + 0.5)) * (1 if minor >= 0 else -1)
        x, y = (off, k if dy > 0 else -k) if y_major else (k if dx > 0 else -k, off)
        if x * x + y * y > roi * roi or not (0 <= ox + x < n and 0 <= oy + y < n):
            break
        seen.append((x, y))
        fe = F32(int(dem[(ox + x) * n + oy + y]))
        hs = max(hs, (fe - foalt) / F32(k))
        if fe + ftht >= foalt + hs * F32(k):
            marks.append((x, y))
    return seen, marks


@pytest.mark.parametrize("form", ["whole", "one warp", "halves", "quarters"])
@pytest.mark.parametrize("roi,n,seed", [(1, 24, 1), (2, 30, 2), (3, 40, 3), (8, 50, 4), (15, 64, 5)])
def test_pairs_cover_the_perimeter_and_give_the_oracle_shed(native, oracle, form, roi, n, seed):
    if form == "one warp" and roi < 8:
        pytest.skip("radii 8 to 15")
    dem = native.fbm_dem(n, seed, octaves=6, range_max=3000)
    dem.reshape(n, n)[n // 3:n // 2, n // 4:n // 2] = 1200  # a plateau: ties along straight rays
    rng = np.random.default_rng(seed)
    obs = np.array(list(rng.choice(n * n, 4, replace=False)) +
                   [0, n - 1, n * n - 1, n // 2, (n // 2) * n, (n // 3 + 1) * n + n // 3], np.int32)
    want = oracle.sheds(dem, n, roi, 20, 20, obs)
    nr, nwpr = 2 * roi + 1, (2 * roi + 64) // 64
    rays = [p for _, _, pairs, _ in ctas(form, roi) for p in pairs]
    assert set(rays) == {(x, y) for x in range(-roi, roi + 1) for y in range(-roi, roi + 1)
                         if max(abs(x), abs(y)) == roi}
    twice = {p for p in rays if rays.count(p) > 1}
    assert all(0 in p or abs(p[0]) == abs(p[1]) for p in twice)
    for i, ob in enumerate(obs):
        ox, oy = divmod(int(ob), n)
        kept, dropped = {(0, 0)}, set()  # the observer's own cell (siting.cpp:279)
        for rows, cols, pairs, keeps in ctas(form, roi):
            for dx, dy in pairs:
                seen, marks = sweep(dem, n, roi, 20, 20, ox, oy, dx, dy)
                assert all(rows[0] * roi <= x <= rows[1] * roi and cols[0] * roi <= y <= cols[1] * roi
                           for x, y in seen), f"ray {dx, dy} leaves its window"
                for m in marks:
                    (kept if keeps(*m) else dropped).add(m)
        assert dropped <= kept
        got = np.zeros(nr * nwpr, np.uint64)
        for x, y in kept:
            got[(x + roi) * nwpr + (y + roi) // 64] |= np.uint64(1) << np.uint64(63 - (y + roi) % 64)
        assert np.array_equal(got, want[i * nr * nwpr:(i + 1) * nr * nwpr]), f"observer {ob}"
