"""Workloads of the siting pipeline for timing, through the package's public entry points.

Each case is one kind of call that a program makes: a whole job on device or
host buffers, one stage on device buffers, a batch of unlike jobs, or a burst
of requests to a server.  Terrain is seeded value-noise fBm (smoothstep
lattices, persistence 0.5, lacunarity 2), made on the GPU; parameters follow
the command line (roi, height, targets, block width, number of observers,
intervisibility).
"""
import atexit
import math
import random

import numpy as np
import torch

import siting_gb300 as sg

_kept = {}


def _context():
    """The context that a program keeps for its jobs."""
    if "ctx" not in _kept:
        _kept["ctx"] = sg.Context(0)
        atexit.register(_kept["ctx"].close)
    return _kept["ctx"]


def _server():
    """The server that a program keeps for its requests."""
    if "srv" not in _kept:
        _kept["srv"] = sg.Server(0, hbm_budget=8 << 30, max_batch_jobs=64)
        atexit.register(_kept["srv"].close)
    return _kept["srv"]


# ---- the cases ---------------------------------------------------------------


def _job(kind, n, roi, height, targets, bw, nwanted, intervis, octaves=10, top=30000):
    return {"kind": kind, "n": n, "roi": roi, "height": height, "targets": targets, "bw": bw,
            "nwanted": nwanted, "intervis": intervis, "octaves": octaves, "top": top}


def listed():
    return [
        # the smallest request of a service: a tile of a few hundred cells, where the launches and
        # the selection's dependent rounds are all there is
        dict(_job("job", 256, 20, 20, 32, 8, 512, 1, 8, 10000), name="job_256"),
        # the command line's own job: a 1000x1000 raster in host memory, its default parameters
        dict(_job("job_host", 1000, 50, 100, 50, 10, 10000, 0, 8, 10000), name="job_host_1000"),
        # an odd side (rows that cannot be tiled by 16 bytes) and a radius whose VIX halo is large
        dict(_job("job", 1537, 137, 150, 77, 16, 1537 * 1537 // 128, 0, 10, 20000), name="job_1537"),
        # the benchmark's headline job
        dict(_job("job", 4096, 100, 200, 100, 16, 65536, 1, 10, 30000), name="job_4096"),
        # the largest single raster: 268 M cells, radius 200
        dict(_job("job", 16384, 200, 150, 64, 32, 262144, 0, 10, 40000), name="job_16384"),
        # the first two stages alone (visibility index and block maxima), a moderate radius
        dict(_job("vix", 2048, 45, 50, 128, 8, 32768, 0, 10, 20000), name="vix_2048"),
        # the same on an odd raster with a large radius
        dict(_job("vix", 2001, 180, 120, 64, 16, 31250, 0, 10, 30000), name="vix_2001"),
        # viewsheds alone: many observers with a small radius
        dict(_job("sheds", 2048, 30, 60, 0, 16, 16384, 0, 10, 20000), name="sheds_2048"),
        # viewsheds alone: the service's largest radius, an odd raster
        dict(_job("sheds", 2999, 200, 150, 0, 32, 6000, 0, 10, 30000), name="sheds_2999"),
        # the selection alone, over viewsheds that the caller holds
        dict(_job("site", 1500, 60, 80, 0, 16, 8836, 1, 10, 20000), name="site_1500"),
        # sixteen unlike jobs in one call: sides 512 to 2048, radii 25 to 150
        {"kind": "batch", "name": "batch_16", "jobs": 16, "lo": 512, "hi": 2048, "per": 64, "mix": 3},
        # a burst of requests to the server: sides 256 to 2048, radii 20 to 200, host buffers
        {"kind": "serve", "name": "serve_24", "jobs": 24, "lo": 256, "hi": 2048, "per": 128, "mix": 5},
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_job(rng, kind, n, per):
    roi = _logu(rng, 20, 200)
    return _job(kind, n, roi, rng.randint(20, 300), rng.randint(32, 128), rng.choice([8, 16, 32]),
                max(64, n * n // per), rng.randint(0, 1), rng.randint(7, 11),
                rng.randint(2000, 40000))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "job_host", "vix", "vix", "sheds", "sheds", "site",
                       "batch", "serve"])
    if kind in ("batch", "serve"):
        lo = _logu(rng, 256, 700)
        return {"kind": kind, "jobs": rng.randint(2, 24), "lo": lo,
                "hi": _logu(rng, lo + 1, 2200), "per": rng.choice([64, 100, 128]),
                "mix": rng.randrange(1 << 20)}
    n = _logu(rng, 256, 4500)
    c = _draw_job(rng, kind, n, _logu(rng, 64, 400))
    if kind in ("sheds", "site"):
        # viewsheds of at most 2 GB
        words = (2 * c["roi"] + 1) * ((2 * c["roi"] + 64) // 64)
        c["nwanted"] = min(c["nwanted"], (2 << 30) // (8 * words), 20000)
    return c


def _mix(case):
    """The jobs of a batch or a burst: unlike sizes and parameters."""
    rng = random.Random(case["mix"])
    jobs = []
    for _ in range(case["jobs"]):
        n = _logu(rng, case["lo"], case["hi"])
        if case["kind"] == "batch":  # sides a multiple of 32, as the batched benchmark has them
            n = max(256, n // 32 * 32)
            roi = rng.randint(25, 150)
        else:
            roi = rng.randint(20, 200)
        jobs.append(_job("job", n, roi, rng.randint(20, 300), rng.choice([32, 64, 128]),
                         rng.choice([8, 16, 32]), n * n // case["per"], rng.randint(0, 1), 9,
                         rng.randint(2000, 30000)))
    return jobs


# ---- inputs --------------------------------------------------------------------


def _terrain(n, seed, octaves, top):
    """uint16[n*n] fBm elevations 0..top on the GPU (held as int16 bits)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h = torch.zeros(n, n, device="cuda")
    i = torch.arange(n, device="cuda", dtype=torch.float32)
    amp, wave = 1.0, 256.0
    for _ in range(octaves):
        m = int(n / wave) + 2
        if m > n:  # a lattice finer than the cells is white noise
            h.add_(torch.rand(n, n, device="cuda", generator=g), alpha=amp)
        else:
            lattice = torch.rand(m, m, device="cuda", generator=g)
            x = i / wave
            k = x.floor()
            f = x - k
            f = f * f * (3 - 2 * f)
            k = k.long()
            rows = torch.lerp(lattice[k], lattice[k + 1], f[:, None])
            h.add_(torch.lerp(rows[:, k], rows[:, k + 1], f[None, :]), alpha=amp)
            del rows
        amp *= 0.5
        wave *= 0.5
    lo, hi = torch.aminmax(h)
    h.sub_(lo).mul_(top / (hi - lo))
    return h.to(torch.int32).to(torch.int16).reshape(-1)


def _params(c):
    return sg.Params(nrows=c["n"], roi=c["roi"], height=c["height"], ntests=max(c["targets"], 1),
                     bw=c["bw"], nwanted0=c["nwanted"], intervis=c["intervis"])


def _jittered(n, count, seed):
    """`count` cells, one at a random place in each square of a grid over the raster, in grid order."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    side = math.ceil(math.sqrt(count))
    i = torch.arange(count, device="cuda")
    r = torch.rand(2, count, device="cuda", generator=g)
    x = (((i // side) + r[0]) * (n / side)).long().clamp_(0, n - 1)
    y = (((i % side) + r[1]) * (n / side)).long().clamp_(0, n - 1)
    return (x * n + y).to(torch.int32)


def _job_buffers(c, seed):
    p = _params(c)
    nw = sg.block_geometry(p.nrows, p.bw, p.nwanted0).nwanted
    return {"p": p, "dem": _terrain(c["n"], seed, c["octaves"], c["top"]),
            "obs": torch.empty(nw, dtype=torch.int32, device="cuda"),
            "sel": torch.empty(nw, dtype=torch.uint8, device="cuda")}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "serve":
        s["srv"] = _server()
        s["reqs"] = [(_params(j), _terrain(j["n"], seed * 1000 + k, j["octaves"], j["top"])
                      .cpu().numpy().view(np.uint16)) for k, j in enumerate(_mix(case))]
        return s
    s["ctx"] = _context()
    if kind == "batch":
        s["jobs"] = [_job_buffers(j, seed * 1000 + k) for k, j in enumerate(_mix(case))]
    elif kind == "job_host":
        s["p"] = _params(case)
        s["dem"] = _terrain(case["n"], seed, case["octaves"], case["top"]).cpu().numpy().view(np.uint16)
    elif kind == "job":
        s.update(_job_buffers(case, seed))
    elif kind == "vix":
        s.update(_job_buffers(case, seed))
        s["geo"] = sg.block_geometry(case["n"], case["bw"], case["nwanted"])
        s["vix"] = torch.empty(case["n"] ** 2, dtype=torch.uint8, device="cuda")
    else:
        n, roi, nw = case["n"], case["roi"], case["nwanted"]
        s.update(n=n, roi=roi, height=case["height"], intervis=case["intervis"],
                 dem=_terrain(n, seed, case["octaves"], case["top"]), obs=_jittered(n, nw, seed),
                 sheds=torch.empty(nw * sg.shed_words(roi), dtype=torch.int64, device="cuda"))
        if kind == "site":
            s["sel"] = torch.empty(nw, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            s["ctx"].calc_sheds_dev(n, s["dem"], roi, case["height"], case["height"], nw, s["obs"],
                                    s["sheds"])
            s["ctx"].sync()
    torch.cuda.synchronize()  # the context's stream is not torch's
    return s


# ---- one pass --------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "serve":
        tickets = [s["srv"].submit(p, dem) for p, dem in s["reqs"]]
        done = [s["srv"].wait(t) for t in tickets]
        return [[obs, sel] for obs, sel, _ in done] + \
            [np.array([[d.result.nusedsheds, d.result.cumarea] for _, _, d in done])]
    ctx = s["ctx"]
    if kind == "job":
        r = ctx.run_dev(s["p"], s["dem"], s["obs"], s["sel"])
        return [s["obs"], s["sel"], r.nusedsheds, r.cumarea]
    if kind == "job_host":
        obs, sel, r = ctx.run(s["p"], s["dem"])
        return [obs, sel, r.nusedsheds, r.cumarea]
    if kind == "vix":
        p, g = s["p"], s["geo"]
        ctx.calc_vix_dev(p.nrows, s["dem"], p.roi, p.height, p.height, p.ntests, s["vix"])
        ctx.find_max_dev(p.nrows, s["vix"], g.blocksize, g.nwanted, g.nblocks, g.nwantedperblock,
                         s["obs"])
        return [s["vix"], s["obs"]]
    if kind == "sheds":
        ctx.calc_sheds_dev(s["n"], s["dem"], s["roi"], s["height"], s["height"], len(s["obs"]),
                           s["obs"], s["sheds"])
        return [s["sheds"]]
    if kind == "site":
        r = ctx.site_it_dev(s["n"], s["roi"], s["intervis"], len(s["obs"]), s["obs"], s["sheds"],
                            s["sel"])
        return [s["sel"], r.nusedsheds, r.cumarea]
    jobs = s["jobs"]
    rs = ctx.run_batch_dev([j["p"] for j in jobs], [j["dem"] for j in jobs],
                           [j["obs"] for j in jobs], [j["sel"] for j in jobs])
    return [[j["obs"], j["sel"]] for j in jobs] + [np.array([[r.nusedsheds, r.cumarea] for r in rs])]


def exact(case, seed):
    """None: every output is a whole number (counts, indices, bits) and has to stay as it is."""
    return None


# ---- what a pass cannot do without --------------------------------------------------


def _vix_flops(n, roi, targets):
    # a target: two draws scaled and two products; a sample on its line of sight: two products,
    # a sum and a comparison, at offsets 1, 2, 4, ... up to the target
    return n * n * targets * (4.0 + 4.0 * math.log2(max(roi, 2)))


def _shed_flops(roi, count):
    # 8*roi rays that end at the circle (0.88 roi steps on average); a step: the position, the
    # slope and its maximum, the sight line's height and the comparison
    return count * 8.0 * roi * 0.88 * roi * 7


def _job_work(c):
    n, nw = c["n"], c["nwanted"]
    shed = nw * sg.shed_words(c["roi"]) * 8
    # elevations in, observers and selection out; the viewsheds are written and read back once
    return {"bytes": 2.0 * n * n + 5.0 * nw + 2.0 * shed,
            "flops": _vix_flops(n, c["roi"], c["targets"]) + _shed_flops(c["roi"], nw)}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        parts = [_job_work(j) for j in _mix(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind in ("job", "job_host"):
        return _job_work(case)
    n, roi, nw = case["n"], case["roi"], case["nwanted"]
    shed = nw * sg.shed_words(roi) * 8.0
    if kind == "vix":
        return {"bytes": 3.0 * n * n + 4.0 * nw, "flops": _vix_flops(n, roi, case["targets"])}
    if kind == "sheds":
        return {"bytes": 2.0 * n * n + 4.0 * nw + shed, "flops": _shed_flops(roi, nw)}
    # the viewsheds read once, a bit of coverage a cell
    return {"bytes": shed + 5.0 * nw + n * n / 8.0, "flops": shed / 8.0}
