"""The workloads this framework's speed is judged by, as a user's program
runs them: visibility simulation (host and device-resident calls, both
tensor-core forms, the plain FP32 and the FP64 form, several simulations as
one batch), Omnical calibration and median filtering.

    listed()            the cases, each a dict of plain values
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call
    run(state)          one pass through the public entry points
    work(case)          the bytes and operations a pass cannot do without
    exact(case, seed)   what run() returns, evaluated in 64 bits by plain torch

Sizes are those of the benchmark, the configurations and the tests of this
repository; inputs are synthetic with the distributions of
``hera_gpu_gb300.synth`` (hexagonal arrays, sphere-uniform power-law sources,
Airy beams, redundant arrays), made on the GPU from the seed.
"""
import ctypes
import random

import numpy as np
import torch

from hera_gpu_gb300 import default_context, omnical, sky, synth, vis_gpu, vis_gpu_multifreq
from hera_gpu_gb300._native import Batch

LAT = np.radians(sky.HERA_LATITUDE_DEG)
C_LIGHT = 299792458.0
# A drawn case is kept below these: the largest listed cases' operations.
MAX_FLOPS = {"tc": 4.0e12, "tc_fp16": 4.0e12, "plain": 1.0e11, "fp64": 8.0e10}


def listed():
    return [
        # one notebook-sized call with host arrays: launches and latency
        dict(name="call-small", kind="vis", method="auto", host=True, nant=16, nsrc=1000,
             ntimes=10, nfreq=1, px=31),
        # a host call of the shape the reference's speed test times
        dict(name="call-512", kind="vis", method="auto", host=True, nant=512, nsrc=3072,
             ntimes=10, nfreq=1, px=31),
        # an hour of LSTs at one frequency, arrays resident on the device
        dict(name="hour", kind="vis", method="auto", host=False, nant=350, nsrc=100_000,
             ntimes=60, nfreq=1, px=63),
        # the deep sky over a band: the benchmark's arrays and sources
        dict(name="band", kind="vis", method="auto", host=False, nant=350, nsrc=1_048_576,
             ntimes=2, nfreq=8, px=63),
        # the FP16 + FP8 form on a smaller array of ragged sizes
        dict(name="band-fp16", kind="vis", method="tc_fp16", host=False, nant=203,
             nsrc=150_001, ntimes=5, nfreq=7, px=63),
        # the plain FP32 form: results to 1e-5, for checks of the other forms
        dict(name="plain", kind="vis", method="plain", host=False, nant=350, nsrc=100_000,
             ntimes=8, nfreq=1, px=63),
        # double precision, the form validation runs use
        dict(name="fp64", kind="vis", method="fp64", host=False, nant=350, nsrc=100_000,
             ntimes=3, nfreq=1, px=63),
        # several uneven simulations planned once and replayed from a graph
        dict(name="batch", kind="batch", nsims=12, sizes=3, maxsrc=50_000),
        # redundant calibration of a big array, data resident on the device
        dict(name="omnical", kind="omnical", host=False, nants=180, ndata=2000, precision=1,
             maxiter=12),
        # the same in double precision through the drop-in call, host arrays
        dict(name="omnical-f64", kind="omnical", host=True, nants=54, ndata=1000, precision=2,
             maxiter=24),
        # the default 3 x 3 median filter of a large waterfall
        dict(name="median", kind="median", nimg=1, rows=7000, cols=7000, k0=3, k1=3),
        # a wider window on a stack of ragged images
        dict(name="median-wide", kind="median", nimg=2, rows=2003, cols=1501, k0=5, k1=5),
    ]


def _between(rng, lo, hi):
    """A whole number, spread over the logarithm of [lo, hi]."""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["vis", "vis", "vis", "vis", "vis", "batch", "omnical", "omnical",
                       "median", "median"])
    if kind == "vis":
        method = rng.choice(["auto", "auto", "tc_fp16", "plain", "fp64"])
        small = method in ("plain", "fp64")
        while True:
            c = dict(kind="vis", method=method, host=rng.random() < 0.3,
                     nant=_between(rng, 16, 512), nsrc=_between(rng, 1000, 100_000 if small else 1_048_576),
                     ntimes=_between(rng, 1, 60), nfreq=_between(rng, 1, 3 if small else 8),
                     px=rng.choice([31, 63]))
            if c["host"]:
                c["nsrc"] = min(c["nsrc"], 20_000)
            if _vis_flops(c) <= MAX_FLOPS.get(method, 4.0e12) and c["ntimes"] * c["nfreq"] * c["nant"] ** 2 <= 2e7:
                return c
    if kind == "batch":
        return dict(kind="batch", nsims=rng.randint(4, 12), sizes=rng.randint(4, 1 << 20),
                    maxsrc=_between(rng, 5000, 50_000))
    if kind == "omnical":
        precision = rng.choice([1, 2])
        nants = _between(rng, 12, 180 if precision == 1 else 90)
        nbls = nants * (nants - 1) // 2
        most = (3.2e7 if precision == 1 else 2.8e6) / nbls
        ndata = min(4000, _between(rng, max(1, most / 64), most))
        return dict(kind="omnical", host=rng.random() < 0.5, nants=nants, ndata=max(1, ndata),
                    precision=precision, maxiter=rng.choice([8, 12] if precision == 1 else [8, 16, 24]))
    k0, k1 = rng.choice([(3, 3), (3, 3), (5, 5), (7, 7), (9, 9), (9, 5), (5, 9), (3, 5), (1, 11), (11, 1)])
    rows, cols = _between(rng, 29, 7000), _between(rng, 29, 7000)
    while rows * cols * k0 * k1 > 9 * 4.9e7:
        rows = (rows + 1) // 2
    return dict(kind="median", nimg=rng.choice([1, 1, 3]) if rows * cols < 4_000_000 else 1,
                rows=rows, cols=cols, k0=k0, k1=k1)


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sky_arrays(nsrc, gen):
    """Sphere-uniform unit vectors and power-law fluxes (index -2, 0.05-50 Jy), FP64."""
    r = torch.rand(3, nsrc, generator=gen, device="cuda", dtype=torch.float64)
    z = 2 * r[0] - 1
    phi = 2 * np.pi * r[1]
    xy = torch.sqrt(1 - z * z)
    crd = torch.stack([xy * torch.cos(phi), xy * torch.sin(phi), z])
    flux = 1 / (1 / 0.05 + r[2] * (1 / 50.0 - 1 / 0.05))
    return crd, flux


def _beams(nant, px, freqs, gen, dtype):
    """Airy power beams of a 14 m dish (2 % diameter scatter), (nfreq, nant, px, px)."""
    g = torch.linspace(-1, 1, px, device="cuda", dtype=torch.float64)
    st = torch.clamp(torch.hypot(g[None, :], g[:, None]), max=1.0)
    dish = 14.0 * (1 + 0.02 * (2 * torch.rand(nant, generator=gen, device="cuda",
                                              dtype=torch.float64) - 1))
    out = torch.empty(len(freqs), nant, px, px, device="cuda", dtype=dtype)
    for i, f in enumerate(freqs):
        x = (np.pi * float(f) / C_LIGHT) * dish[:, None, None] * st
        safe = torch.where(x == 0, torch.ones_like(x), x)
        out[i] = torch.where(x == 0, torch.ones_like(x),
                             (2 * torch.special.bessel_j1(safe) / safe) ** 2)
    return out


def _sim_arrays(nant, nsrc, ntimes, nfreq, px, seed, dtype):
    gen, rng = _gen(seed), np.random.default_rng(seed)
    if nant > 350:
        antpos = synth.hex_array(nant, 14.6, 0.01, rng)
    else:   # a random part of the 350-antenna array
        antpos = synth.hex_array(350, 14.6, 0.01, rng)[np.sort(rng.choice(350, nant, replace=False))]
    freqs = np.linspace(100e6, 200e6, nfreq) if nfreq > 1 else np.array([150e6])
    e2t = sky.eq2tops(sky.lst_grid(ntimes, 1.0, start_rad=rng.uniform(0, 2 * np.pi)), LAT)
    crd, flux = _sky_arrays(nsrc, gen)
    to = lambda a: torch.as_tensor(a, device="cuda").to(dtype).contiguous()  # noqa: E731
    return dict(antpos=to(antpos), freqs=freqs, eq2tops=to(e2t), crd_eq=to(crd), I_sky=to(flux),
                bm_cubes=_beams(nant, px, freqs, gen, dtype))


def _vis_precision(case):
    return 2 if case["method"] == "fp64" else 1


def _vis_arrays(case, seed):
    dtype = torch.float64 if _vis_precision(case) == 2 else torch.float32
    return _sim_arrays(case["nant"], case["nsrc"], case["ntimes"], case["nfreq"], case["px"], seed,
                       dtype)


def _batch_specs(case):
    """Sizes of the batched form: antennas 16-350 and sources 1e3-maxsrc (log-uniform), 1-60
    times, 1-16 channels, beams of 31 or 63 pixels a side."""
    r = random.Random(case["sizes"])
    return [dict(nant=_between(r, 16, 350), nsrc=_between(r, 1000, case["maxsrc"]),
                 ntimes=r.randint(1, 60), nfreq=r.randint(1, 16), px=r.choice([31, 63]))
            for _ in range(case["nsims"])]


def _batch_arrays(case, seed):
    return [_sim_arrays(s["nant"], s["nsrc"], s["ntimes"], s["nfreq"], s["px"], seed * 1000 + i,
                        torch.float32) for i, s in enumerate(_batch_specs(case))]


def _omnical_arrays(case, seed):
    """A hexagonal redundant array: gains 1 + noise, unit-variance unique baselines, data with
    2 % noise, weights of unflagged and flagged samples, a start a few percent off."""
    gen = _gen(seed)
    ggu, nubls = synth.hex_redundant_layout(case["nants"])
    idx = torch.as_tensor(ggu.astype(np.int64), device="cuda")
    n, nants, nbls = case["ndata"], case["nants"], len(ggu)
    cplx = lambda *s: torch.complex(  # noqa: E731
        *torch.randn(2, *s, generator=gen, device="cuda", dtype=torch.float64).unbind(0))
    g = 1 + 0.1 * cplx(n, nants)
    u = cplx(n, nubls)
    d = g[:, idx[:, 0]] * g[:, idx[:, 1]].conj() * u[:, idx[:, 2]] + 0.02 * cplx(n, nbls)
    w = 1.0 - (torch.rand(n, nbls, generator=gen, device="cuda", dtype=torch.float64) < 0.01).double()
    g0 = g * (1 + 0.05 * cplx(n, nants))
    u0 = u * (1 + 0.05 * cplx(n, nubls))
    rt, ct = (torch.float32, torch.complex64) if case["precision"] == 1 else (torch.float64, torch.complex128)
    return dict(ggu=ggu, gains=g0.to(ct), ubls=u0.to(ct), data=d.to(ct), wgts=w.to(rt))


def _median_images(case, seed):
    """Noise waterfalls with interference spikes and flagged (zero) samples."""
    gen = _gen(seed)
    shape = (case["nimg"], case["rows"], case["cols"])
    x = torch.randn(shape, generator=gen, device="cuda")
    r = torch.rand(shape, generator=gen, device="cuda")
    x[r < 0.01] *= 1000.0
    x[r > 0.98] = 0.0
    return x


def prepare(case, seed):
    ctx = default_context()
    if case["kind"] == "vis":
        a = _vis_arrays(case, seed)
        if case["host"]:
            a = {k: v.cpu().numpy() if torch.is_tensor(v) else v for k, v in a.items()}
            return dict(case=case, a=a)
        ct = torch.complex128 if _vis_precision(case) == 2 else torch.complex64
        out = torch.empty(case["nfreq"], case["ntimes"], case["nant"], case["nant"], dtype=ct,
                          device="cuda")
        return dict(case=case, a=a, out=out, ctx=ctx)
    if case["kind"] == "batch":
        sims, outs, arrays = [], [], _batch_arrays(case, seed)
        for s, a in zip(_batch_specs(case), arrays):
            outs.append(torch.empty(s["nfreq"], s["ntimes"], s["nant"], s["nant"],
                                    dtype=torch.complex64, device="cuda"))
            sims.append(dict({k: a[k].data_ptr() for k in ("antpos", "eq2tops", "crd_eq", "I_sky",
                                                           "bm_cubes")},
                             freqs=a["freqs"], vis_out=outs[-1].data_ptr(), nant=s["nant"],
                             ntimes=s["ntimes"], nsrc=s["nsrc"], beam_px=s["px"]))
        torch.cuda.synchronize()
        return dict(case=case, arrays=arrays, outs=outs, batch=Batch(ctx, sims, graph=True))
    if case["kind"] == "omnical":
        a = _omnical_arrays(case, seed)
        if case["host"]:
            return dict(case=case, a={k: v.cpu().numpy() if torch.is_tensor(v) else v
                                      for k, v in a.items()})
        n = case["ndata"]
        a.update(g=torch.empty_like(a["gains"]), u=torch.empty_like(a["ubls"]),
                 chisq=torch.empty(n, dtype=a["wgts"].dtype, device="cuda"),
                 conv=torch.empty(n, dtype=a["wgts"].dtype, device="cuda"),
                 iters=torch.empty(n, dtype=torch.int32, device="cuda"))
        return dict(case=case, a=a, ctx=ctx)
    x = _median_images(case, seed)
    return dict(case=case, x=x, out=torch.empty_like(x), ctx=ctx)


# -------------------------------------------------------------------- runs --
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    case = state["case"]
    if case["kind"] == "vis":
        a, precision = state["a"], _vis_precision(case)
        method = "auto" if case["method"] == "fp64" else case["method"]
        if case["host"]:
            if case["nfreq"] == 1:
                return vis_gpu(a["antpos"], float(a["freqs"][0]), a["eq2tops"], a["crd_eq"],
                               a["I_sky"], a["bm_cubes"][0], precision=precision, method=method)
            return vis_gpu_multifreq(a["antpos"], a["freqs"], a["eq2tops"], a["crd_eq"],
                                     a["I_sky"], a["bm_cubes"], precision=precision, method=method)
        state["ctx"].vis_multifreq_device(
            precision, method, a["antpos"].data_ptr(), case["nant"], a["freqs"],
            a["eq2tops"].data_ptr(), case["ntimes"], a["crd_eq"].data_ptr(),
            a["I_sky"].data_ptr(), case["nsrc"], a["bm_cubes"].data_ptr(), case["px"],
            state["out"].data_ptr())
        return state["out"]
    if case["kind"] == "batch":
        state["batch"].launch()
        return state["outs"]
    if case["kind"] == "omnical":
        a = state["a"]
        if case["host"]:
            return omnical(a["ggu"], a["gains"], a["ubls"], a["data"], a["wgts"], 1e-10,
                           case["maxiter"], precision=case["precision"])
        ctx = state["ctx"]
        # the solver overwrites its starting point: a pass starts from a copy of it
        for dst, src in ((a["g"], a["gains"]), (a["u"], a["ubls"])):
            ctx.check(ctx.lib.hv_memcpy_async(ctx.h, _ptr(dst), _ptr(src),
                                              dst.numel() * dst.element_size(), 3))
        ctx.check(ctx.lib.hv_omnical_device(
            ctx.h, case["precision"], ctypes.c_void_p(a["ggu"].ctypes.data), len(a["ggu"]),
            _ptr(a["g"]), case["nants"], _ptr(a["u"]), a["u"].shape[1], _ptr(a["data"]),
            _ptr(a["wgts"]), case["ndata"], 1e-10, case["maxiter"], 4, 1, 0.3, _ptr(a["chisq"]),
            _ptr(a["iters"]), _ptr(a["conv"]), None))
        return {"gains": a["g"], "ubls": a["u"], "chisq": a["chisq"], "iters": a["iters"],
                "conv": a["conv"]}
    ctx, x = state["ctx"], state["x"]
    ctx.check(ctx.lib.hv_median_filter_device(ctx.h, _ptr(x), _ptr(state["out"]), case["nimg"],
                                              case["rows"], case["cols"], case["k0"], case["k1"],
                                              None))
    return state["out"]


# -------------------------------------------------------------------- work --
def _vis_flops(c):
    """8 flops per source above the horizon (half of them) and antenna pair of the upper
    triangle."""
    return 4.0 * c["nant"] * (c["nant"] + 1) * (c["nsrc"] / 2) * c["ntimes"] * c["nfreq"]


def _vis_bytes(c, rs):
    return rs * (4.0 * c["nsrc"] + 9 * c["ntimes"] + 3 * c["nant"]
                 + c["nfreq"] * c["nant"] * c["px"] ** 2
                 + 2 * c["nfreq"] * c["ntimes"] * c["nant"] ** 2)


def work(case):
    if case["kind"] == "vis":
        return {"bytes": _vis_bytes(case, 4 * _vis_precision(case)), "flops": _vis_flops(case)}
    if case["kind"] == "batch":
        specs = _batch_specs(case)
        return {"bytes": sum(_vis_bytes(s, 4) for s in specs),
                "flops": sum(_vis_flops(s) for s in specs)}
    if case["kind"] == "omnical":
        rs, nants = 4 * case["precision"], case["nants"]
        nbls = nants * (nants - 1) // 2
        nubls = synth.hex_redundant_layout(nants)[1]
        checks = case["maxiter"] // 4
        return {"bytes": float(case["ndata"]) * rs * (3 * nbls + 4 * (nants + nubls) + 3),
                # per iteration and baseline: three complex products and three complex sums;
                # per check: the model and the weighted squared difference
                "flops": float(case["ndata"]) * nbls * (24 * case["maxiter"] + 20 * checks)}
    return {"bytes": 8.0 * case["nimg"] * case["rows"] * case["cols"], "flops": 0.0}


# ------------------------------------------------------------------- exact --
def _exact_vis(a, block=16384):
    """V[f, t, a, b] = sum_s v[a, s] conj(v[b, s]) in complex128: rotation, horizon, bilinear
    beam (clamped at the grid's edge) and phasors of every source."""
    f64 = {k: (v if torch.is_tensor(v) else torch.as_tensor(v)).to("cuda", torch.float64)
           for k, v in a.items()}
    pos, e2t, crd, beams = f64["antpos"], f64["eq2tops"], f64["crd_eq"], f64["bm_cubes"]
    nf, nant, px, _ = beams.shape
    nt = e2t.shape[0]
    flat = beams.reshape(nf, nant, px * px)
    out = torch.zeros(nf, nt, nant, nant, dtype=torch.complex128, device="cuda")
    for t in range(nt):
        top = e2t[t] @ crd
        up = top[2] > 0
        top, amp = top[:, up], torch.sqrt(f64["I_sky"][up])
        for s in range(0, top.shape[1], block):
            tp = top[:, s:s + block]
            b = (px - 1) * (0.5 * tp[:2] + 0.5)
            lo = torch.clamp(torch.floor(b), 0, px - 2)
            w = torch.clamp(b - lo, 0, 1)
            i = (lo[1] * px + lo[0]).long()
            tau = (pos @ tp) / C_LIGHT
            for f in range(nf):
                bf = flat[f]
                top_row = bf[:, i] * (1 - w[0]) + bf[:, i + 1] * w[0]
                bot_row = bf[:, i + px] * (1 - w[0]) + bf[:, i + px + 1] * w[0]
                A = (top_row * (1 - w[1]) + bot_row * w[1]) * amp[s:s + block]
                ph = 2 * np.pi * torch.remainder(tau * f64["freqs"][f], 1.0)
                v = torch.polar(A.abs(), ph) * torch.sign(A)
                out[f, t] += v @ v.conj().T
    return out


def _exact_omnical(a, maxiter, check_every=4, check_after=1, crit=1e-10, step=0.3):
    """The Omnical iteration in 64 bits: weights every check_every iterations, a step of
    float32(step) toward the new estimate, a problem stopped (keeping its old solution) at a
    check where it has converged or its chi^2 has risen."""
    to = lambda x, t: torch.as_tensor(x).to("cuda", t)  # noqa: E731
    g, u, d = (to(a[k], torch.complex128).clone() for k in ("gains", "ubls", "data"))
    w = to(a["wgts"], torch.float64)
    idx = torch.as_tensor(a["ggu"].astype(np.int64), device="cuda")
    i, j, k = idx[:, 0], idx[:, 1], idx[:, 2]
    nants, nubls, n = g.shape[1], u.shape[1], g.shape[0]
    hot = lambda x, m: torch.nn.functional.one_hot(x, m).to(torch.float64)  # noqa: E731
    Ai, Aj, Ak = hot(i, nants), hot(j, nants), hot(k, nubls)
    csum = lambda x, A: torch.complex(x.real @ A, x.imag @ A)  # noqa: E731
    model = lambda g, u: g[:, i] * g[:, j].conj() * u[:, k]  # noqa: E731
    chi = lambda g, u: ((d - model(g, u)).abs() ** 2 * w).sum(1)  # noqa: E731
    chisq, live = chi(g, u), torch.ones(n, dtype=torch.bool, device="cuda")
    conv = torch.zeros(n, dtype=torch.float64, device="cuda")
    iters = torch.zeros(n, dtype=torch.int64, device="cuda")
    gs = float(np.float32(step))
    one_m = float(np.float32(1.0) - np.float32(step))
    for it in range(1, maxiter + 1):
        m = model(g, u)
        m2 = m.real ** 2 + m.imag ** 2
        if it % check_every == 1:
            dw = m2 * w
            gw, uw = dw @ Ai + dw @ Aj, dw @ Ak
        z = d * m.conj() * (dw / m2)
        gb = csum(z, Ai) + csum(z.conj(), Aj)
        ng, nu = g * (one_m + gs * gb / gw), u * (one_m + gs * csum(z, Ak) / uw)
        ok = live
        if not (it < maxiter and (it < check_after or it % check_every != 0)):
            nchi = chi(ng, nu)
            num = ((ng - g).abs() ** 2).sum(1) + ((nu - u).abs() ** 2).sum(1)
            den = (ng.abs() ** 2).sum(1) + (nu.abs() ** 2).sum(1)
            c = torch.sqrt(num / den)
            conv = torch.where(live, c, conv)
            ok = live & ~((c < crit) | (nchi > chisq))
            chisq = torch.where(ok, nchi, chisq)
            iters = torch.where(ok, torch.full_like(iters, it), iters)
        g = torch.where(ok[:, None], ng, g)
        u = torch.where(ok[:, None], nu, u)
        live = ok
    # iters is a count, compared as such: no 64-bit value stands for it
    return {"gains": g, "ubls": u, "chisq": chisq, "iters": None, "conv": conv}


def _exact_median(x, k0, k1):
    """Rank k0 k1 // 2 of each zero-padded window (which starts k // 2 before its pixel)."""
    p = torch.nn.functional.pad(x, (k1 // 2, k1 - 1 - k1 // 2, k0 // 2, k0 - 1 - k0 // 2))
    out = torch.empty(x.shape, dtype=torch.float64, device="cuda")
    rows = max(1, 20_000_000 // (x.shape[2] * k0 * k1))
    for m in range(x.shape[0]):
        for r in range(0, x.shape[1], rows):
            win = p[m, r:r + rows + k0 - 1].unfold(0, k0, 1).unfold(1, k1, 1)
            win = win.reshape(win.shape[0], win.shape[1], k0 * k1)
            out[m, r:r + rows] = torch.sort(win, dim=-1).values[..., (k0 * k1) // 2].double()
    return out


def exact(case, seed):
    if case["kind"] == "vis":
        v = _exact_vis(_vis_arrays(case, seed))
        return v[0] if case["host"] and case["nfreq"] == 1 else v
    if case["kind"] == "batch":
        return [_exact_vis(a) for a in _batch_arrays(case, seed)]
    if case["kind"] == "omnical":
        a = _omnical_arrays(case, seed)
        parts = [_exact_omnical({k: (v if k == "ggu" else v[s:s + 250]) for k, v in a.items()},
                                case["maxiter"]) for s in range(0, case["ndata"], 250)]
        return {k: None if k == "iters" else torch.cat([p[k] for p in parts]) for k in parts[0]}
    return _exact_median(_median_images(case, seed), case["k0"], case["k1"])
