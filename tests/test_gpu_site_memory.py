"""SITE under a memory budget that has no room for the scratch of local dominance.

The selection is then taken in the global order, so that a budget which was enough for it
stays enough; the picks are the same.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JOBS = [dict(nrows=600, roi=12, height=60, ntests=16, bw=5, nwanted0=17000, intervis=1),
        dict(nrows=700, roi=10, height=30, ntests=16, bw=10, nwanted0=5000, intervis=0),
        dict(nrows=300, roi=20, height=30, ntests=16, bw=10, nwanted0=900, intervis=1)]


def _oracle_of(native, oracle, jobs):
    dems = [native.fbm_dem(j["nrows"], seed=j["nrows"], octaves=7, range_max=6000) for j in jobs]
    refs = [oracle.run(d, *(j[k] for k in ("nrows", "roi", "height", "ntests", "bw", "nwanted0", "intervis")))
            for d, j in zip(dems, jobs)]
    return dems, refs


def _same(ref, obs, sel, res):
    assert np.array_equal(obs, ref["obs"])
    assert np.array_equal(sel, ref["selected"])
    assert (res.nusedsheds, res.cumarea) == (ref["nused"], ref["cumarea"])


@pytest.mark.parametrize("job", JOBS[:2])
def test_a_single_job(native, oracle, job):
    (dem,), (ref,) = _oracle_of(native, oracle, [job])
    p = native.Params(**job)
    held = []
    for order in (0, 1):
        with native.Context(0) as ctx:
            ctx.set_site_order(order)
            _same(ref, *ctx.run(p, dem))
            held.append(ctx.workspace_bytes())
    assert held[1] + (1 << 18) < held[0]
    with native.Context(0, hbm_budget=held[1]) as ctx:
        _same(ref, *ctx.run(p, dem))
        assert ctx.last_site_phase_cycles()[12] > 0  # the clock of the cut: in the global order
        assert ctx.workspace_bytes() <= held[1]
    with native.Context(0, hbm_budget=held[1] - 4096) as ctx:
        with pytest.raises(native.SitingError):
            ctx.run(p, dem)


def test_a_batch_and_a_server(native, oracle):
    # the last job's SITE takes 1024 threads a CTA, in one launch with the others
    jobs = JOBS + [dict(nrows=420, roi=130, height=60, ntests=8, bw=20, nwanted0=900, intervis=1)]
    dems, refs = _oracle_of(native, oracle, jobs)
    params = [native.Params(**j) for j in jobs]
    with native.Context(0) as ctx:
        usual = ctx.batch_workspace_bytes(params)
        one = ctx.batch_workspace_bytes(params[:1])
    for budget in (0, usual - (1 << 20)):
        with native.Context(0, hbm_budget=budget) as ctx:
            for _ in range(2):
                for ref, got in zip(refs, ctx.run_batch(params, dems)):
                    _same(ref, *got)
            assert budget == 0 or ctx.workspace_bytes() < usual
    for budget in (1 << 30, one - (1 << 20)):
        with native.Server(0, hbm_budget=budget) as srv:
            tickets = [srv.submit(p, d) for p, d in zip(params[:3], dems)]
            for ref, t in zip(refs, tickets):
                obs, sel, info = srv.wait(t)
                _same(ref, obs, sel, info.result)


def test_noalloc_takes_what_does_not_fit_in_the_global_order(native, oracle):
    torch = pytest.importorskip("torch")
    n, roi, count = 10800, 60, 700  # 14.6 MB of coverage; past 16 MiB with the other's scratch
    xy = np.random.default_rng(1).integers(0, n, (count, 2))
    obs = (xy[:, 0] * n + xy[:, 1]).astype(np.int32)
    sheds = oracle.sheds(np.zeros(n * n, np.uint16), n, roi, 5, 5, obs)
    want, used, area = oracle.site(n, roi, 0, obs, sheds)
    d_obs, d_sheds = torch.from_numpy(obs).cuda(), torch.from_numpy(sheds.view(np.int64)).cuda()
    sel = torch.full((count,), 7, dtype=torch.uint8, device="cuda")
    res = native._ResultC()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = native.load().siting_site_it_noalloc(n, roi, 0, count, d_obs.data_ptr(), d_sheds.data_ptr(),
                                              sel.data_ptr(), stream, C.byref(res))
    assert rc == 0
    assert np.array_equal(sel.cpu().numpy(), want)
    assert (res.nusedsheds, res.cumarea) == (used, area)
