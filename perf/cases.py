"""The calls whose time counts: what a user of this package has it do, over the range of sizes.

Every case is one call (or one short sequence) of the package's public Python
surface on inputs that are already on the GPU.  The sizes are those of the
repository's own scenes: Sentinel-1 IW bursts of about 1500 x 21000 samples
(synth.CONFIGS "c1", the frame of bench.py), the 512 x 2048 and 160 x 640
scenes of the tests ("c0", "small"), and odd sizes between them.

``listed()`` are the fixed cases, ``draw(rng)`` makes others of the same kinds
and ranges.  ``exact`` restates each result in float64 with torch and numpy.
"""
import dataclasses
import math

import numpy as np
import torch
import torch.nn.functional as F

from sentinel_gpu_processor_b200 import chain, geo2rdr, interfere, kernels, plan, refine, stitch, synth

DEV = "cuda:0"
GEOMETRY = 20261203  # the seed of orbits, burst sizes and terrain: products keep their shapes from seed to seed
EXACT_PIXELS = 300_000_000  # exact() of whole frames and stacks up to this many burst samples


def listed():
    return [
        # one small burst geocoded by itself, as the smallest scenes and unit tests do: launches and host work count
        {"name": "geocode_small", "kind": "geocode", "lines": 512, "samples": 2048, "ci16": False},
        # one full IW burst straight from the measurement TIFF (complex int16): what the geo2rdr executable does per burst
        {"name": "geocode_burst_ci16", "kind": "geocode", "lines": 1500, "samples": 21000, "ci16": True},
        # the whole single-pair chain on a small scene of odd size, host read of the crop rows included
        {"name": "pair_small", "kind": "pair", "lines": 331, "samples": 1187, "rowlook": 2, "collook": 8},
        # the headline: a full IW frame, 3 subswaths x 9 burst pairs of uneven size, complex64, replayed from its graph
        {"name": "frame_iw", "kind": "frame", "swaths": 3, "bursts": 9, "scale": 1.0, "ci16": False, "rowlook": 4,
         "collook": 20},
        # time-series processing: one reference date against several, every burst geocoded once (windows form)
        {"name": "stack_dates", "kind": "stack", "dates": 4, "bursts": 2, "lines": 1500, "samples": 21000},
        # radar-grid coregistration, stage 1: sample offsets of a full burst
        {"name": "offsets_burst", "kind": "offsets", "lines": 1500, "samples": 21000},
        # stage 2: the 8-tap sinc resampler on a full burst
        {"name": "resample_burst", "kind": "resample", "lines": 1500, "samples": 21000, "interp": "sinc8"},
        # stage 3: full-resolution 5 x 5 coherence of a burst of odd width
        {"name": "boxcoh_burst", "kind": "box", "lines": 1497, "samples": 20991, "win": 5},
        # crossmul with looks, amplitudes and coherence of two geocoded bursts (the crossmul_daemon's task)
        {"name": "crossmul_burst", "kind": "crossmul", "lines": 1500, "samples": 21000, "rowlook": 4, "collook": 20},
        # Goldstein filter of a stitched frame interferogram
        {"name": "goldstein_frame", "kind": "goldstein", "rows": 3217, "cols": 1391, "alpha": 0.5},
        # the adjoint: objective and gradient of the coregistration refinement (forward and backward in one call)
        {"name": "adjoint_bursts", "kind": "adjoint", "bursts": 2, "lines": 1468, "samples": 20968, "rowlook": 4,
         "collook": 20, "grad": True},
        # the 27 burst interferograms of a frame stitched into one raster
        {"name": "stitch_frame", "kind": "stitch", "swaths": 3, "bursts": 9, "rows": 430, "cols": 470,
         "out_float": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["geocode", "pair", "frame", "stack", "offsets", "resample", "box", "crossmul", "goldstein",
                       "adjoint", "stitch"])
    lines, samples = _log(rng, 160, 1530), _log(rng, 640, 25500)
    rl, cl = rng.choice([(2, 4), (2, 8), (3, 12), (4, 20), (5, 20), (8, 40)])
    if kind == "geocode":
        return {"kind": kind, "lines": lines, "samples": samples, "ci16": rng.random() < 0.5}
    if kind == "pair":
        return {"kind": kind, "lines": lines, "samples": samples, "rowlook": rl, "collook": cl}
    if kind == "frame":
        return {"kind": kind, "swaths": rng.randint(1, 3), "bursts": rng.randint(1, 4),
                "scale": round(math.exp(rng.uniform(math.log(0.12), 0.0)), 3), "ci16": rng.random() < 0.5,
                "rowlook": rl, "collook": cl}
    if kind == "stack":
        return {"kind": kind, "dates": rng.randint(1, 5), "bursts": rng.randint(1, 2), "lines": lines,
                "samples": samples}
    if kind == "offsets":
        return {"kind": kind, "lines": lines, "samples": samples}
    if kind == "resample":
        return {"kind": kind, "lines": lines, "samples": samples, "interp": rng.choice(["sinc8", "sinc8", "bilinear"])}
    if kind == "box":
        return {"kind": kind, "lines": lines, "samples": samples, "win": rng.choice([3, 5, 5, 7, 9])}
    if kind == "crossmul":
        return {"kind": kind, "lines": lines, "samples": samples, "rowlook": rl, "collook": cl}
    if kind == "goldstein":
        return {"kind": kind, "rows": _log(rng, 64, 4200), "cols": _log(rng, 64, 2000),
                "alpha": rng.choice([0.2, 0.5, 0.6, 0.9])}
    if kind == "adjoint":
        return {"kind": kind, "bursts": rng.randint(1, 2), "lines": lines, "samples": samples, "rowlook": rl,
                "collook": cl, "grad": rng.random() < 0.7}
    return {"kind": kind, "swaths": rng.randint(1, 3), "bursts": rng.randint(2, 9), "rows": _log(rng, 60, 800),
            "cols": _log(rng, 80, 1000), "out_float": rng.random() < 0.3}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _pair_scene(c, seed):
    """A burst pair (reference speckle seen by both dates, TOPS-modulated) on fractal terrain."""
    sc = synth.make_pair("c1" if c["lines"] > 700 else "c0", seed=GEOMETRY, device=DEV, lines=c["lines"],
                         samples=c["samples"], rowlook=c.get("rowlook"), collook=c.get("collook"))
    sc.ref_slc, sc.sec_slc = ([x] for x in _date_pair(sc.ref[0], sc.sec[0], seed, 0.7))
    return sc


def _date_pair(ref, sec, seed, coherence):
    g, L, S = _gen(seed), ref.radar.lines_per_burst, ref.radar.samples_per_burst
    s = synth.speckle(L, S, g, DEV)
    t = coherence * s + math.sqrt(1 - coherence ** 2) * synth.speckle(L, S, g, DEV)
    return (synth.tops_modulate(z, a, a.bursts[0]).contiguous() for z, a in ((s, ref), (t, sec)))


def _frame_scene(c, with_dem=True):
    return synth.make_frame(seed=GEOMETRY, device=DEV if with_dem else "cpu", n_swaths=c["swaths"],
                            n_bursts=c["bursts"], scale=c["scale"], rowlook=c["rowlook"], collook=c["collook"],
                            slc_pairs=0, with_dem=with_dem)


def _frame_slcs(sc, c, seed):
    """The frame's SLCs pair by pair, as its sample format holds them."""
    for i, (r, s) in enumerate(zip(sc.ref, sc.sec)):
        pair = _date_pair(r, s, seed * 64 + i, sc.extra["coherence"][i])
        yield tuple(synth.cint16(z) if c["ci16"] else z for z in pair)


def _stack_scene(c, with_dem=True):
    return synth.make_stack(seed=GEOMETRY, device=DEV if with_dem else "cpu", n_sec=c["dates"], n_bursts=c["bursts"],
                            lines=c["lines"], samples=c["samples"], overlap=min(100, c["lines"] // 4),
                            with_dem=with_dem)


def _radar_pair(c):
    """Reference and secondary acquisitions (150 m baseline) of one burst, for the radar-grid calls."""
    L, S, t_c = c["lines"], c["samples"], synth.ORBIT_T0 + 50.0
    orbit = synth.make_orbit(t_c=t_c)
    off = synth.secondary_offset(orbit, t_c, synth.NEAR_RANGE + S * synth.RANGE_SPACING / 2, 150.0)
    radar = synth.make_radar(L, S)
    fm, dc = synth.tops_tables(radar, t_c, -1500.0)
    b = synth.burst_meta(t_c - L * synth.AZIMUTH_INTERVAL / 2, L, S, margin_l=4, margin_s=4)
    ref = synth.Acquisition(radar=radar, orbit=orbit, fm=fm, dc=dc, bursts=[b])
    sec = synth.Acquisition(radar=radar, orbit=synth.make_orbit(t_c=t_c, offset=off), fm=fm.copy(), dc=dc.copy(),
                            bursts=[b])
    return ref, sec


def _relief(L, S, seed, cell=24):
    """Smooth zero-mean unit-range field [L, S] (float32): noise on a coarse lattice, bicubic between."""
    n0, n1 = max(4, -(-L // cell) + 2), max(4, -(-S // cell) + 2)
    z = torch.randn((1, 1, n0, n1), generator=_gen(seed), device=DEV)
    z = F.avg_pool2d(F.pad(z, (2, 2, 2, 2), mode="replicate"), 5, 1)
    z = F.interpolate(z, size=(L, S), mode="bicubic", align_corners=True)[0, 0]
    return z / z.abs().max().clamp_min(1e-6)


def _llh_rasters(acq, seed):
    """float64 latitude, longitude, height of every sample, bilinear between solved points of the burst's grid."""
    r, b = acq.radar, acq.bursts[0]
    L, S, ka, kr = r.lines_per_burst, r.samples_per_burst, 12, 20
    n0, n1 = -(-(L - 1) // ka) + 1, -(-(S - 1) // kr) + 1
    coarse = dataclasses.replace(r, lines_per_burst=n0, samples_per_burst=n1, prf=r.prf / ka,
                                 range_sampling_rate=r.range_sampling_rate / kr)
    g = synth.rdr2geo_grid(acq.orbit, coarse, b, lambda la, lo: synth.fbm_height(la, lo, seed & 0xFFFF, 3000.0),
                           device=DEV, outer=2, steps=40)
    size = ((n0 - 1) * ka + 1, (n1 - 1) * kr + 1)
    return [F.interpolate(x[None, None], size=size, mode="bilinear", align_corners=True)[0, 0, :L, :S].contiguous()
            for x in g]


def _offset_rasters(L, S, seed):
    """Coregistration offsets as a 150 m baseline gives them: a drift across the burst plus the terrain's share."""
    y = torch.linspace(0, 1, L, device=DEV)[:, None]
    x = torch.linspace(0, 1, S, device=DEV)[None, :]
    h = _relief(L, S, seed)
    return (-1.4 + 0.1 * y + 0.3 * x + 0.02 * h).contiguous(), (3.3 + 0.2 * y + 5.5 * x + 0.4 * h).contiguous()


def _ifg(rows, cols, seed, noise=0.6):
    """A multilooked interferogram: fringes, speckle amplitude, decorrelation noise."""
    g = _gen(seed)
    ph = 9.0 * _relief(rows, cols, seed + 1, cell=40) + torch.linspace(0, 21, cols, device=DEV)[None, :]
    amp = 0.3 + torch.rand((rows, cols), generator=g, device=DEV)
    z = torch.polar(amp, ph) + noise * synth.speckle(rows, cols, g, DEV)
    return (z * 1.7).contiguous()


def _stitch_layout(c):
    """Boxes (left, top, right, bottom), subswath, group of the bursts of a frame on its multilooked grid."""
    h, w, out = c["rows"], c["cols"], []
    step, shift = max(1, int(h * 0.62)), max(0, h // 40)
    for s in range(c["swaths"]):
        for b in range(c["bursts"]):
            left, top = s * int(w * 0.9) + (c["bursts"] - 1 - b) * shift, b * step + 7 * s
            out.append(((left, top, left + w, top + h), s + 1, b))
    return out, max(b[3] for b, _, _ in out) + 3, max(b[2] for b, _, _ in out) + 5


def prepare(case, seed):
    c, k = case, case["kind"]
    st = {"kind": k}
    if k == "geocode":
        sc = _pair_scene(c, seed)
        a = sc.ref[0]
        st["plan"] = plan.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc)
        st["slc"] = synth.cint16(sc.ref_slc[0]) if c["ci16"] else sc.ref_slc[0]
        st["dem"] = sc.dem
    elif k == "pair":
        sc = _pair_scene(c, seed)
        st["chain"] = chain.PairChain(sc.ref[0], sc.sec[0], sc.rsc, sc.rowlook, sc.collook, sc.alpha, device=DEV)
        st["in"] = (sc.ref_slc[0], sc.sec_slc[0], sc.dem)
    elif k in ("frame", "stack"):
        if k == "frame":
            sc = _frame_scene(c)
            ch = chain.BatchedFrameChain(sc.ref, sc.sec, sc.rsc, sc.rowlook, sc.collook, sc.alpha, device=DEV,
                                         sample_format="ci16" if c["ci16"] else "c64")
            for r, t, pair in zip(ch.ref_views, ch.sec_views, _frame_slcs(sc, c, seed)):
                r.copy_(pair[0])
                t.copy_(pair[1])
        else:
            sc = _stack_scene(c)
            nb, acqs = c["bursts"], sc.ref + [a for s in sc.sec for a in s]
            ch = chain.BatchedFrameChain(acqs, None, sc.rsc, sc.rowlook, sc.collook, sc.alpha, device=DEV,
                                         crossmul_fused=False,
                                         pairs=[(b, nb + d * nb + b) for d in range(c["dates"]) for b in range(nb)])
            for v, s in zip(ch.views, _stack_slcs(sc, c, seed)):
                v.copy_(s)
        for o in (ch.ifg, ch.amp1, ch.amp2, ch.coh, ch.filt):
            o.zero_()  # product slots are as large as a pair can get; the rest of a slot stays as it is
        st["chain"], st["dem"] = ch, sc.dem
        if k == "frame":
            ch.capture(sc.dem)
        else:
            ch.run(sc.dem)
        res = ch.results() if ch.n_pairs <= 10 else None
        st["out"] = {"pairs": ch.pairs_dev, "ifg": ch.ifg, "amp1": ch.amp1, "amp2": ch.amp2, "coh": ch.coh,
                     "filt": ch.filt} if res is None else _pair_views(res)
    elif k == "offsets":
        ref, sec = _radar_pair(c)
        st["plan"] = plan.burst_plan(sec.radar, sec.orbit, sec.fm, sec.dc, sec.bursts[0], None)
        st["llh"] = _llh_rasters(ref, seed)
    elif k == "resample":
        _, sec = _radar_pair(c)
        st["plan"] = plan.burst_plan(sec.radar, sec.orbit, sec.fm, sec.dc, sec.bursts[0], None)
        w = synth.speckle(c["lines"], c["samples"], _gen(seed), DEV)
        st["sec"] = synth.tops_modulate(w, sec, sec.bursts[0]).contiguous()
        st["off"], st["interp"] = _offset_rasters(c["lines"], c["samples"], seed + 1), c["interp"]
    elif k in ("box", "crossmul"):
        g, L, S = _gen(seed), c["lines"], c["samples"]
        ref = synth.speckle(L, S, g, DEV) * 40.0
        fringe = torch.polar(torch.ones((L, S), device=DEV), 6.0 * _relief(L, S, seed + 1))
        sec = (0.7 * ref * fringe + 28.0 * synth.speckle(L, S, g, DEV)).contiguous()
        sec[:4] = 0  # lines and samples that the coregistration leaves empty
        sec[:, -7:] = 0
        st["ref"], st["sec"] = ref.contiguous(), sec
        if k == "box":
            st["win"] = c["win"]
        else:
            st["looks"] = (c["rowlook"], c["collook"])
            st["hdr"] = _crossmul_headers(c)
    elif k == "goldstein":
        st["img"], st["alpha"] = _ifg(c["rows"], c["cols"], seed), c["alpha"]
    elif k == "adjoint":
        p = _adjoint_inputs(c, seed)
        st["problem"] = refine.CoregProblem([p["plan"]] * c["bursts"], p["ref"], p["sec"], p["az0"], p["rg0"], p["daz"],
                                            p["drg"], c["rowlook"], c["collook"])
        st["params"], st["dh"], st["grad"] = p["params"], p["dh"], c["grad"]
    else:
        boxes, nrow, ncol = _stitch_layout(c)
        data = _stitch_data(c, boxes, nrow, ncol, seed)
        st["bursts"] = [(b, d, sw, grp) for (b, sw, grp), d in zip(boxes, data)]
        st["shape"], st["out_float"] = (nrow, ncol), c["out_float"]
    return st


def _pair_views(res):
    return [None if r is None else {"ifg": r.ifg, "amp1": r.amp1, "amp2": r.amp2, "coh": r.coh, "filt": r.filt,
                                    "header": r.header} for r in res]


def _stack_slcs(sc, c, seed):
    """The stack's SLCs in acquisition order: the reference's speckle decorrelating with time, TOPS-modulated."""
    for d, acqs in enumerate([sc.ref] + sc.sec):
        for b, a in enumerate(acqs):
            s = synth.speckle(c["lines"], c["samples"], _gen(seed * 31 + b), DEV)
            if d:
                g = sc.coherence[d - 1]
                s = g * s + math.sqrt(1 - g * g) * synth.speckle(c["lines"], c["samples"], _gen(seed * 31 + 100 * d + b), DEV)
            yield synth.tops_modulate(s, a, a.bursts[0])


def _crossmul_headers(c):
    """Headers of two geocoded rasters on one frame grid; both rasters are whole, the overlap is aligned to the looks."""
    h = [c["lines"] + 50, c["samples"] + 90, 41, 23, 41 + c["samples"], 23 + c["lines"]]
    return np.array(h, dtype=np.int32)


def _adjoint_inputs(c, seed):
    """White speckle seen by both dates a whole number of samples apart, at parameters off the optimum."""
    n, L, S, m = c["bursts"], c["lines"], c["samples"], 16
    big = dict(c, lines=L + 2 * m, samples=S + 2 * m)
    _, acq = _radar_pair(big)
    g = _gen(seed)
    sec = torch.empty((n, L + 2 * m, S + 2 * m), dtype=torch.complex64, device=DEV)
    ref = torch.empty((n, L, S), dtype=torch.complex64, device=DEV)
    for b in range(n):
        sec[b] = synth.tops_modulate(synth.speckle(L + 2 * m, S + 2 * m, g, DEV), acq, acq.bursts[0])
        ref[b] = 0.8 * sec[b, m + 1:m + 1 + L, m - 2:m - 2 + S] + 0.6 * synth.speckle(L, S, g, DEV)
    rel = _relief(L, S, seed + 3)
    one = torch.ones((n, 1, 1), device=DEV)
    az0 = (one * (m + 1 + 0.05 * rel)).contiguous()
    rg0 = (one * (m - 2 + 0.1 * rel)).contiguous()
    daz = (one * (2e-6 * (1 + 0.3 * rel))).contiguous()
    drg = (one * (1.2e-4 * (1 + 0.1 * rel))).contiguous()
    rng = np.random.Generator(np.random.PCG64(seed & 0x7FFFFFFF))
    p = 0.15 * rng.choice([-1.0, 1.0], (n, 6)) * rng.uniform(0.6, 1.4, (n, 6))
    dh = 10.0 * torch.stack([_relief(L, S, seed + 7 + b, cell=64) for b in range(n)])
    return {"plan": plan.burst_plan(acq.radar, acq.orbit, acq.fm, acq.dc, acq.bursts[0], None), "acq": acq, "ref": ref,
            "sec": sec, "az0": az0, "rg0": rg0, "daz": daz, "drg": drg,
            "params": torch.tensor(p, dtype=torch.float32, device=DEV), "dh": dh.contiguous()}


def _stitch_data(c, boxes, nrow, ncol, seed):
    """Burst interferograms cut from one frame, each with its own phase offset, decorrelation and slanted empty edges."""
    frame = _ifg(nrow, ncol, seed, noise=0.2)
    g, out = _gen(seed + 5), []
    for i, ((l, t, r, b), _, _) in enumerate(boxes):
        d = frame[t:b, l:r] * complex(math.cos(0.4 * i), math.sin(0.4 * i))
        d = d + 0.2 * synth.speckle(b - t, r - l, g, DEV)
        y = torch.arange(b - t, device=DEV)[:, None] - 0.05 * torch.arange(r - l, device=DEV)[None, :]
        d = torch.where((y < 4) & (y > -0.04 * (r - l) + 4), torch.zeros_like(d), d)
        out.append((torch.where(d == 0, 0.0, torch.angle(d)) if c["out_float"] else d).contiguous())
    return out


# --------------------------------------------------------------------- run

def run(state):
    k = state["kind"]
    if k == "geocode":
        r = geo2rdr.geocode_burst(state["plan"], state["slc"], state["dem"])
        return {"header": r[0], "gslc": r[1]}
    if k == "pair":
        r = state["chain"].run(*state["in"])
        return {"header": r.header, "ifg": r.ifg, "amp1": r.amp1, "amp2": r.amp2, "coh": r.coh, "filt": r.filt}
    if k == "frame":
        state["chain"].replay()
        return state["out"]
    if k == "stack":
        state["chain"].run(state["dem"])
        return state["out"]
    if k == "offsets":
        return kernels.geo2rdr_offsets(state["plan"], *state["llh"])
    if k == "resample":
        return kernels.resample(state["plan"], state["sec"], *state["off"], state["interp"])
    if k == "box":
        return kernels.box_coherence(state["ref"], state["sec"], state["win"])
    if k == "crossmul":
        r = interfere.crossmul_pair(state["hdr"], state["ref"], state["hdr"], state["sec"], *state["looks"])
        return {"header": r["header"], "ifg": r["ifg"], "amp1": r["amp1"], "amp2": r["amp2"], "coh": r["coh"]}
    if k == "goldstein":
        return kernels.goldstein(state["img"], state["alpha"])
    if k == "adjoint":
        p = state["problem"]
        if not state["grad"]:
            return p.objective(state["params"], state["dh"])
        return p.gradient(state["params"], state["dh"])
    return stitch.stitch_bursts(state["bursts"], *state["shape"], state["out_float"])


# -------------------------------------------------------------------- work

def _window_pixels(acq, rsc):
    p = plan.burst_plan(acq.radar, acq.orbit, acq.fm, acq.dc, acq.bursts[0], rsc)
    return p.nrow * p.ncol


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: those of the interpolation sums and transforms."""
    c, k = case, case["kind"]
    if k in ("geocode", "pair"):
        t_c = synth.ORBIT_T0 + 50.0
        ref, _ = _radar_pair(c)
        rsc = synth.footprint_rsc([ref], 0.0, 3000.0)
        w, n = _window_pixels(ref, rsc), c["lines"] * c["samples"]
        if k == "geocode":
            return {"bytes": (4 if c["ci16"] else 8) * n + 10 * w, "flops": 200 * w}
        m = w // (c["rowlook"] * c["collook"])
        return {"bytes": 16 * n + 2 * w + 28 * m, "flops": 400 * w + 16 * 1300 * m}
    if k in ("frame", "stack"):
        sc = _frame_scene(c, False) if k == "frame" else _stack_scene(c, False)
        acqs = sc.ref + (sc.sec if k == "frame" else [a for s in sc.sec for a in s])
        npair = len(acqs) - len(sc.ref)
        w = _window_pixels(acqs[0], sc.rsc)
        n = sum(a.radar.lines_per_burst * a.radar.samples_per_burst for a in acqs)
        m = npair * w // (sc.rowlook * sc.collook)
        return {"bytes": (4 if c.get("ci16") else 8) * n + 2 * sc.rsc.nlat * sc.rsc.nlon + 28 * m,
                "flops": 200 * w * len(acqs) + 16 * 1300 * m}
    n = c.get("lines", 0) * c.get("samples", 0)
    if k == "offsets":
        return {"bytes": 32 * n, "flops": 250 * n}
    if k == "resample":
        return {"bytes": 24 * n, "flops": (288 if c["interp"] == "sinc8" else 12) * n}
    if k == "box":
        return {"bytes": 20 * n, "flops": 14 * n}
    if k == "crossmul":
        return {"bytes": 16 * n + 20 * (n // (c["rowlook"] * c["collook"])), "flops": 16 * n}
    if k == "goldstein":
        m = c["rows"] * c["cols"]
        return {"bytes": 16 * m, "flops": 16 * m * 1300}
    if k == "adjoint":
        n *= c["bursts"]
        return {"bytes": (36 + (4 if c["grad"] else 0)) * n, "flops": (3 if c["grad"] else 1) * 288 * n}
    boxes, nrow, ncol = _stitch_layout(c)
    es = 4 if c["out_float"] else 8
    return {"bytes": es * (len(boxes) * c["rows"] * c["cols"] + nrow * ncol), "flops": 20 * nrow * ncol}


# ------------------------------------------------------------------- exact

RA, RE2, SOL = 6378137.0, 0.00669437999015, 299792458.0


def _hermite(orbit, w):
    """Degree-7 polynomial (8 x 3, in t - tc) through the state vectors w-1 .. w+2 and their velocities."""
    tt, xx, vv = (np.asarray(a, dtype=np.longdouble) for a in orbit)
    tc = float(tt[w])
    z = np.repeat(tt[w - 1:w + 3] - tc, 2)
    out = np.zeros((8, 3), dtype=np.longdouble)
    for k in range(3):
        d = np.repeat(xx[w - 1:w + 3, k], 2)
        coef = [d[0]]
        for order in range(1, 8):
            nd = np.empty(8 - order, dtype=np.longdouble)
            for i in range(8 - order):
                if z[i] == z[i + order]:
                    nd[i] = vv[w - 1 + i // 2, k]
                else:
                    nd[i] = (d[i + 1] - d[i]) / (z[i + order] - z[i])
            d = nd
            coef.append(d[0])
        poly, basis = np.zeros(8, dtype=np.longdouble), np.zeros(8, dtype=np.longdouble)
        basis[0] = 1
        for i in range(8):
            poly += coef[i] * basis
            basis = np.concatenate([[np.longdouble(0)], basis[:-1]]) - z[i] * basis
        out[:, k] = poly
    return tc, out.astype(np.float64)


class _Orbit:
    def __init__(self, orbit, t_lo, t_hi):
        self.t0, self.dt, n = float(orbit[0][0]), float(orbit[0][1] - orbit[0][0]), len(orbit[0])
        pick = lambda t: min(max(int((t - self.t0) / self.dt), 1), n - 3)  # noqa: E731
        self.n, self.win = n, {w: _hermite(orbit, w) for w in range(pick(t_lo), pick(t_hi) + 1)}

    def at(self, t):
        """Position and velocity (lists of 3) at t (tensor)."""
        idx = ((t - self.t0) / self.dt).trunc().clamp(1, self.n - 3)
        x, v = [0.0] * 3, [0.0] * 3
        for w, (tc, c) in self.win.items():
            h, on = t - tc, idx == w
            for k in range(3):
                p = torch.full_like(h, float(c[7, k]))
                d = torch.zeros_like(h)
                for i in range(6, -1, -1):
                    d = d * h + p
                    p = p * h + float(c[i, k])
                x[k] = torch.where(on, p, x[k]) if len(self.win) > 1 else p
                v[k] = torch.where(on, d, v[k]) if len(self.win) > 1 else d
        return x, v


def _ecef(lat, lon, h):
    la, lo = torch.deg2rad(lat), torch.deg2rad(lon)
    re = RA / torch.sqrt(1 - RE2 * torch.sin(la) ** 2)
    return [(re + h) * torch.cos(la) * torch.cos(lo), (re + h) * torch.cos(la) * torch.sin(lo),
            (re * (1 - RE2) + h) * torch.sin(la)]


def _zero_doppler(orb, xyz, t):
    """Zero-Doppler time and range of ground points."""
    for it in range(25):
        x, v = orb.at(t)
        f = sum((p - a) * b for p, a, b in zip(xyz, x, v))
        step = f / -sum(b * b for b in v)
        t = t - step
        if it > 2 and float(step.abs().max()) < 1e-12:
            break
    x, _ = orb.at(t)
    return t, torch.sqrt(sum((p - a) ** 2 for p, a in zip(xyz, x)))


def _table_at(tab, tc):
    i = int(np.argmin(np.abs(tab[:, 0] - tc)))
    if tab[i, 0] < tc and i < len(tab) - 1:
        return tab[i, 1:] + (tc - tab[i, 0]) / (tab[i + 1, 0] - tab[i, 0]) * (tab[i + 1, 1:] - tab[i, 1:])
    if tab[i, 0] > tc and i > 0:
        return tab[i - 1, 1:] + (tc - tab[i - 1, 0]) / (tab[i, 0] - tab[i - 1, 0]) * (tab[i, 1:] - tab[i - 1, 1:])
    return tab[i, 1:]


class _Tops:
    """TOPS phase of an acquisition's burst at any line and range time."""

    def __init__(self, acq):
        r, b = acq.radar, acq.bursts[0]
        self.r, self.L, self.ati = r, r.lines_per_burst, r.azimuth_time_interval
        self.dtaz, self.t0 = 1.0 / r.prf, b.azimuth_time
        tc = b.azimuth_time + self.L * self.ati / 2
        self.orb = _Orbit(acq.orbit, b.azimuth_time - 10, b.azimuth_time + self.L * self.ati + 10)
        _, v = self.orb.at(torch.tensor([tc], dtype=torch.float64))
        self.ks = 2 * math.sqrt(sum(float(a) ** 2 for a in v)) * r.radar_frequency / SOL * r.azimuth_steering_rate * math.pi / 180
        self.fm, self.dc = _table_at(acq.fm, tc), _table_at(acq.dc, tc)
        self.etac0 = 0.0
        self.etac0 = float(self.rate(torch.tensor(r.slant_range_time, dtype=torch.float64))[1])

    def rate(self, tr):
        d = tr - self.fm[0]
        ka = self.fm[1] + d * (self.fm[2] + self.fm[3] * d)
        d = tr - self.dc[0]
        fnc = self.dc[1] + d * (self.dc[2] + self.dc[3] * d)
        return ka * self.ks / (ka - self.ks), -fnc / ka - self.etac0

    def half_cycles(self, az, rg):
        """-kt (eta - etaref)^2 (the deramp phase over pi) at fractional line az and sample rg."""
        kt, er = self.rate(self.r.slant_range_time + rg / self.r.range_sampling_rate)
        return -kt * (-self.L * self.ati / 2 + az * self.ati - er) ** 2


def _turn(h):
    """exp(i pi h)."""
    h = torch.remainder(h, 2.0) * math.pi
    return torch.polar(torch.ones_like(h), h)


def _deramped(acq, slc):
    r = acq.radar
    rows = torch.arange(r.lines_per_burst, dtype=torch.float64, device=DEV)[:, None]
    cols = torch.arange(r.samples_per_burst, dtype=torch.float64, device=DEV)[None, :]
    s = torch.complex(slc[..., 0].double(), slc[..., 1].double()) if slc.dtype == torch.int16 else slc.to(torch.complex128)
    return s.reshape(r.lines_per_burst, -1) * _turn(_Tops(acq).half_cycles(rows, cols))


def _geocoded(acq, slc, dem, rsc):
    """The burst on its DEM window, complex128, and the plan that says which window."""
    p = plan.burst_plan(acq.radar, acq.orbit, acq.fm, acq.dc, acq.bursts[0], rsc)
    tops, r, b = _Tops(acq), acq.radar, acq.bursts[0]
    der = _deramped(acq, slc)
    S, out = r.samples_per_burst, torch.zeros((p.nrow, p.ncol), dtype=torch.complex128, device=DEV)
    r0, dr = r.slant_range_time * SOL / 2, SOL / 2 / r.range_sampling_rate
    lat0, lon0 = rsc.latmax + rsc.dlat * p.win_top, rsc.lonmin + rsc.dlon * p.win_left
    lon = lon0 + torch.arange(p.ncol, dtype=torch.float64, device=DEV)[None, :] * rsc.dlon
    step = max(1, 4_000_000 // p.ncol)
    for y in range(0, p.nrow, step):
        n = min(step, p.nrow - y)
        lat = lat0 + torch.arange(y, y + n, dtype=torch.float64, device=DEV)[:, None] * rsc.dlat
        h = dem[p.win_top + y:p.win_top + y + n, p.win_left:p.win_right].double()
        la, lo = torch.broadcast_tensors(lat, lon)
        xyz = _ecef(la, lo, h)
        t, R = _zero_doppler(tops.orb, xyz, torch.full_like(h, b.azimuth_time + r.lines_per_burst * tops.dtaz / 2))
        rg, az = (R - r0) / dr, (t - b.azimuth_time) / tops.dtaz
        ok = (rg > b.first_valid_sample) & (rg < b.last_valid_sample - 1) & (az >= b.first_valid_line + 5) & (
            az < b.last_valid_line - 5)
        R, t, rg, az = R[ok], t[ok], rg[ok], az[ok]
        i, j = az.trunc().long(), rg.trunc().long()
        fa, fr = az - i, rg - j
        q = der.reshape(-1)
        v = (q[i * S + j] * (1 - fr) + q[i * S + j + 1] * fr) * (1 - fa) + (
            q[(i + 1) * S + j] * (1 - fr) + q[(i + 1) * S + j + 1] * fr) * fa
        kt, er = tops.rate(R * 2 / SOL)
        eta = -tops.L * tops.dtaz / 2 + t - tops.t0
        out[y:y + n][ok] = v * _turn(4 / r.wvl * R + kt * (eta - er) ** 2)
    return out, p


def _crop(g, p):
    """First and last non-zero row, as rows of the RSC grid."""
    nz = torch.nonzero((g != 0).any(1)).reshape(-1)
    return p.win_top + int(nz[0]), p.win_top + int(nz[-1]) + 1


def _looked(a, b, rl, cl):
    n0, n1 = a.shape[0] // rl, a.shape[1] // cl
    box = lambda z: z[:n0 * rl, :n1 * cl].reshape(n0, rl, n1, cl).mean((1, 3))  # noqa: E731
    ifg, p1, p2 = box(a.conj() * b), box(a.abs() ** 2), box(b.abs() ** 2)
    a1, a2 = p1.sqrt(), p2.sqrt()
    den = a1 * a2
    return {"ifg": ifg, "amp1": a1, "amp2": a2, "coh": torch.where(den > 0, ifg.abs() / den.clamp_min(1e-300), 0.0)}


GAUSS = [[4e-6, 8.8e-5, 5.43e-4, 9.48e-4], [8.8e-5, 1.915e-3, 1.1776e-2, 2.0584e-2],
         [5.43e-4, 1.1776e-2, 7.241e-2, 1.26584e-1], [9.48e-4, 2.0584e-2, 1.26584e-1, 2.21141e-1]]


def _goldstein(img, alpha, n=32):
    z, (h, w) = img.to(torch.complex128), img.shape
    ys, xs = ([min(k * 8, m - n) for k in range(max(1, -(-m // 8) - 3))] for m in (h, w))
    tri = torch.tensor([float(t if t < n // 2 else n - 1 - t) for t in range(n)], dtype=torch.float64, device=DEV)
    wt = tri[:, None] + tri[None, :]
    acc, ws = torch.zeros_like(z), torch.zeros((h, w), dtype=torch.float64, device=DEV)
    for y in ys:
        p = torch.stack([z[y:y + n, x:x + n] for x in xs])
        f = torch.fft.fft2(p)
        m, s = f.abs(), 0.0
        for ky in range(-3, 4):
            for kx in range(-3, 4):
                s = s + torch.roll(m, (-ky, -kx), (1, 2)) * float(np.float32(GAUSS[3 - abs(ky)][3 - abs(kx)]))
        mean = s.mean((1, 2), keepdim=True)
        s = torch.where(mean > 1e-8, s / mean.clamp_min(1e-300), 0.0) ** float(np.float32(alpha))
        f = torch.fft.ifft2(torch.where(s > 0, f * s, f)) * wt
        for k, x in enumerate(xs):
            acc[y:y + n, x:x + n] += f[k]
            ws[y:y + n, x:x + n] += wt
    return torch.where(ws > 0, acc / ws.clamp_min(1e-300), acc)


def _pair_exact(a1, s1, a2, s2, dem, rsc, rl, cl, alpha):
    g1, p1 = _geocoded(a1, s1, dem, rsc)
    g2, p2 = _geocoded(a2, s2, dem, rsc)
    (t1, b1), (t2, b2) = _crop(g1, p1), _crop(g2, p2)
    left = -(-max(p1.win_left, p2.win_left) // cl) * cl
    right = min(p1.win_right, p2.win_right) // cl * cl
    top, bottom = -(-max(t1, t2) // rl) * rl, min(b1, b2) // rl * rl
    cut = lambda g, p: g[top - p.win_top:bottom - p.win_top, left - p.win_left:right - p.win_left]  # noqa: E731
    out = _looked(cut(g1, p1), cut(g2, p2), rl, cl)
    out["filt"] = _goldstein(out["ifg"], alpha) if min(out["ifg"].shape) >= 32 else out["ifg"]
    return out


def _sinc8(f):
    """Weights and their slopes (8 tensors each) of the normalised windowed sinc at the fractions f."""
    w, d = [], []
    for k in range(-3, 5):
        x = k - f
        sx = torch.where(x.abs() < 1e-9, torch.ones_like(x), torch.sin(math.pi * x) / (math.pi * x.where(x.abs() >= 1e-9, torch.ones_like(x))))
        ds = torch.where(x.abs() < 1e-6, -math.pi ** 2 / 3 * x, (torch.cos(math.pi * x) - sx) / x.where(x.abs() >= 1e-6, torch.ones_like(x)))
        c, dc = 0.5 + 0.5 * torch.cos(math.pi * x / 4), -math.pi / 8 * torch.sin(math.pi * x / 4)
        w.append(sx * c)
        d.append(-(ds * c + sx * dc))
    sw, sd = sum(w), sum(d)
    return [a / sw for a in w], [(b - a / sw * sd) / sw for a, b in zip(w, d)]


def _interpolated(acq, der, az, rg, interp="sinc8", slopes=False):
    """The burst at (az, rg), reramped; with slopes also its derivatives along az and rg."""
    tops = _Tops(acq)
    L, S = der.shape
    lo, hi = (3, 4) if interp == "sinc8" else (0, 1)
    n, m = az.floor().long(), rg.floor().long()
    ok = (n >= lo) & (n + hi < L) & (m >= lo) & (m + hi < S)
    n, m, fa, fr = n.clamp(lo, L - 1 - hi), m.clamp(lo, S - 1 - hi), az - n, rg - m
    if interp == "sinc8":
        wa, da = _sinc8(fa)
        wr, dr = _sinc8(fr)
    else:
        wa, wr, da, dr = [1 - fa, fa], [1 - fr, fr], None, None
    s = sa = sr = 0.0
    q = der.reshape(-1)
    for i in range(hi + lo + 1):
        row = rowd = 0.0
        for j in range(hi + lo + 1):
            v = q[(n + (i - lo)) * S + m + (j - lo)]
            row = row + wr[j] * v
            rowd = rowd + dr[j] * v if slopes else 0.0
        s = s + wa[i] * row
        if slopes:
            sa, sr = sa + da[i] * row, sr + wa[i] * rowd
    ph = _turn(-tops.half_cycles(az, rg))
    s = torch.where(ok, s * ph, 0.0)
    if not slopes:
        return s
    kt, er = tops.rate(acq.radar.slant_range_time + rg / acq.radar.range_sampling_rate)
    e = 1e-3  # central difference of the smooth TOPS phase in range
    u = -tops.L * tops.ati / 2 + az * tops.ati - er
    pa = 2 * kt * u * tops.ati * math.pi
    pr = -(tops.half_cycles(az, rg + e) - tops.half_cycles(az, rg - e)) / (2 * e) * math.pi
    return s, torch.where(ok, sa * ph, 0.0) + 1j * pa * s, torch.where(ok, sr * ph, 0.0) + 1j * pr * s


def _adjoint_exact(c, seed):
    p = _adjoint_inputs(c, seed)
    n, L, S, rl, cl = c["bursts"], c["lines"], c["samples"], c["rowlook"], c["collook"]
    nr, nc = L // rl, S // cl
    J, gp = 0.0, torch.zeros((n, 6), dtype=torch.float64, device=DEV)
    gh = torch.zeros((n, L, S), dtype=torch.float64, device=DEV)
    step = max(1, 2_000_000 // (rl * S)) * rl
    xr = (torch.arange(S, dtype=torch.float64, device=DEV)[None, :] - 0.5 * S) / S
    for b in range(n):
        der, q = _deramped(p["acq"], p["sec"][b]), p["params"][b].double()
        for y in range(0, nr * rl, step):
            z = slice(y, min(y + step, nr * rl))
            rows = torch.arange(z.start, z.stop, dtype=torch.float64, device=DEV)[:, None]
            xa, dh = (rows - 0.5 * L) / L, p["dh"][b, z].double()
            az = rows + p["az0"][b, z].double() + q[0] + q[1] * xa + q[2] * xr + p["daz"][b, z].double() * dh
            rg = torch.arange(S, dtype=torch.float64, device=DEV)[None, :] + p["rg0"][b, z].double() + q[3] + q[4] * xa \
                + q[5] * xr + p["drg"][b, z].double() * dh
            s, sa, sr = (v[:, :nc * cl] for v in _interpolated(p["acq"], der, az, rg, slopes=True))
            r = p["ref"][b, z, :nc * cl].to(torch.complex128)
            box = lambda v: v.reshape(-1, rl, nc, cl).sum((1, 3))  # noqa: E731
            full = lambda v: v.repeat_interleave(rl, 0).repeat_interleave(cl, 1)  # noqa: E731
            I, P1, P2 = box(r.conj() * s), box(r.abs() ** 2), box(s.abs() ** 2)
            ok = (P1 * P2 > 0) & (I.abs() > 0)
            gam = torch.where(ok, I.abs() / (P1 * P2).clamp_min(1e-300).sqrt(), 0.0)
            J = J + gam.sum()
            if not c["grad"]:
                continue
            ci = torch.where(ok, gam * I / (I.abs() ** 2).clamp_min(1e-300), 0.0)
            cp = torch.where(ok, gam / P2.clamp_min(1e-300), 0.0)
            g = full(ci) * r - full(cp) * s
            ga, gr = (g.conj() * sa).real, (g.conj() * sr).real
            x = xr[:, :nc * cl]
            gp[b] += torch.stack([ga.sum(), (ga * xa).sum(), (ga * x).sum(), gr.sum(), (gr * xa).sum(), (gr * x).sum()])
            gh[b, z, :nc * cl] = p["daz"][b, z, :nc * cl].double() * ga + p["drg"][b, z, :nc * cl].double() * gr
    k = -1.0 / (n * nr * nc)
    return (J * k, gp * k, gh * k) if c["grad"] else J * k


def _stitch_exact(c, seed):
    boxes, nrow, ncol = _stitch_layout(c)
    data = _stitch_data(c, boxes, nrow, ncol, seed)
    fl = c["out_float"]
    data = [d.double() if fl else d.to(torch.complex128) for d in data]
    frame = torch.zeros((nrow, ncol), dtype=data[0].dtype, device=DEV)
    real = (lambda z: z) if fl else (lambda z: z.real)
    for sw in range(1, c["swaths"] + 1):
        mos, off, prev = torch.zeros_like(frame), 0.0, None
        one = sorted(((b, d, g) for (b, s, g), d in zip(boxes, data) if s == sw), key=lambda q: q[0][1] + q[0][3])
        lo, hi = (min(one[0][0][i], one[-1][0][i]) for i in (0, 1)), (max(one[0][0][i], one[-1][0][i]) for i in (2, 3))
        (left, top), (right, bottom) = lo, hi
        for b, d, grp in one:
            l, t, r, u = max(b[0], left), max(b[1], top), min(b[2], right), min(b[3], bottom)
            new, old = d[t - b[1]:u - b[1], l - b[0]:r - b[0]], mos[t:u, l:r]
            if prev is not None and grp != prev:
                both = (real(old) != 0) & (real(new) != 0)
                if bool(both.any()):
                    pd = torch.polar(torch.ones_like(old[both]), new[both] - old[both]) if fl else old[both].conj() * new[both]
                    off = float(torch.angle(pd.mean()))
                    a = torch.sort(torch.angle(pd * complex(math.cos(off), -math.sin(off)))).values
                    off += float(0.5 * (a[(a.numel() - 1) // 2] + a[a.numel() // 2]))
            if off != 0.0:
                if fl:
                    put = new - off
                    put = torch.where(put > math.pi, put - 2 * math.pi, torch.where(put < -math.pi, put + 2 * math.pi, put))
                else:
                    put = new * complex(math.cos(off), -math.sin(off))
            else:
                put = new
            mos[t:u, l:r] = new if prev is None else torch.where((real(old) == 0) & (real(new) != 0), put, old)
            prev = grp
        frame = torch.where(real(mos) != 0, mos, frame)
    return frame


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "geocode":
        sc = _pair_scene(c, seed)
        slc = synth.cint16(sc.ref_slc[0]) if c["ci16"] else sc.ref_slc[0]
        g, p = _geocoded(sc.ref[0], slc, sc.dem, sc.rsc)
        top, bottom = _crop(g, p)
        return {"header": None, "gslc": g[top - p.win_top:bottom - p.win_top]}
    if k == "pair":
        sc = _pair_scene(c, seed)
        return {"header": None, **_pair_exact(sc.ref[0], sc.ref_slc[0], sc.sec[0], sc.sec_slc[0], sc.dem, sc.rsc,
                                              sc.rowlook, sc.collook, sc.alpha)}
    if k == "frame":
        if c["swaths"] * c["bursts"] > 10 or 2 * c["swaths"] * c["bursts"] * 3.4e7 * c["scale"] ** 2 > EXACT_PIXELS:
            return None
        sc = _frame_scene(c)
        return [{"header": None, **_pair_exact(sc.ref[i], r, sc.sec[i], t, sc.dem, sc.rsc, sc.rowlook, sc.collook,
                                               sc.alpha)} for i, (r, t) in enumerate(_frame_slcs(sc, c, seed))]
    if k == "stack":
        nb = c["bursts"]
        if nb * c["dates"] > 10 or 2 * nb * c["dates"] * c["lines"] * c["samples"] > 2 * EXACT_PIXELS:
            return None
        sc = _stack_scene(c)
        slcs, out = list(_stack_slcs(sc, c, seed)), []
        for d in range(c["dates"]):
            for b in range(nb):
                out.append({"header": None, **_pair_exact(sc.ref[b], slcs[b], sc.sec[d][b], slcs[nb + d * nb + b], sc.dem,
                                                          sc.rsc, sc.rowlook, sc.collook, sc.alpha)})
        return out
    if k == "offsets":
        ref, sec = _radar_pair(c)
        la, lo, h = _llh_rasters(ref, seed)
        tops, r = _Tops(sec), sec.radar
        az, rg = torch.empty_like(la), torch.empty_like(la)
        cols = torch.arange(c["samples"], dtype=torch.float64, device=DEV)[None, :]
        for y in range(0, c["lines"], 128):
            z = slice(y, min(y + 128, c["lines"]))
            rows = torch.arange(z.start, z.stop, dtype=torch.float64, device=DEV)[:, None]
            t, R = _zero_doppler(tops.orb, _ecef(la[z], lo[z], h[z]), torch.full_like(h[z], tops.t0 + c["lines"] * tops.dtaz / 2))
            az[z] = (t - tops.t0) / tops.dtaz - rows
            rg[z] = (R - r.slant_range_time * SOL / 2) / (SOL / 2 / r.range_sampling_rate) - cols
        return az, rg
    if k == "resample":
        _, sec = _radar_pair(c)
        w = synth.speckle(c["lines"], c["samples"], _gen(seed), DEV)
        der = _deramped(sec, synth.tops_modulate(w, sec, sec.bursts[0]))
        az, rg = _offset_rasters(c["lines"], c["samples"], seed + 1)
        out = torch.empty(der.shape, dtype=torch.complex128, device=DEV)
        cols = torch.arange(c["samples"], dtype=torch.float64, device=DEV)[None, :]
        for y in range(0, c["lines"], 128):
            z = slice(y, min(y + 128, c["lines"]))
            rows = torch.arange(z.start, z.stop, dtype=torch.float64, device=DEV)[:, None]
            out[z] = _interpolated(sec, der, rows + az[z].double(), cols + rg[z].double(), c["interp"])
        return out
    if k == "box":
        st, w = prepare(c, seed), c["win"]
        a, b = st["ref"].to(torch.complex128), st["sec"].to(torch.complex128)
        box = lambda v: F.avg_pool2d(v[None, None], w, 1, w // 2, divisor_override=1)[0, 0]  # noqa: E731
        p = a.conj() * b
        num, den = torch.hypot(box(p.real), box(p.imag)), (box(a.abs() ** 2) * box(b.abs() ** 2)).sqrt()
        return torch.where(den > 0, num / den.clamp_min(1e-300), 0.0)
    if k == "crossmul":
        st, (rl, cl) = prepare(c, seed), (c["rowlook"], c["collook"])
        h = [int(v) for v in st["hdr"][:6]]
        left, top = -(-h[2] // cl) * cl, -(-h[3] // rl) * rl
        z = (slice(top - h[3], h[5] // rl * rl - h[3]), slice(left - h[2], h[4] // cl * cl - h[2]))
        return {"header": None, **_looked(st["ref"][z].to(torch.complex128), st["sec"][z].to(torch.complex128), rl, cl)}
    if k == "goldstein":
        return _goldstein(_ifg(c["rows"], c["cols"], seed), c["alpha"])
    if k == "adjoint":
        return _adjoint_exact(c, seed)
    return _stitch_exact(c, seed)
