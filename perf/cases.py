"""Workloads of the transit search, for timing it.

A case is one call (or one short sequence of calls) that a program makes
through this package's entry points:

  kind "search"   ``core.CurveOnDevice.search``: the chi2 of every trial period
                  of one light curve, main pass (starts thinned by the skip
                  rule) or all-starts pass, FP64 or FP32
  kind "spectra"  ``_lib.spectra``: chi2 spectrum -> SR, power and SDE
  kind "adjoint"  ``refine.model_chi2_function``: chi2 of the unfolded transit
                  model and its gradient (one forward and one backward)
  kind "power"    ``gtls(t, y, dy).power()`` from host arrays
  kind "batch"    ``batch.gtls_batch(curves).power()`` from host arrays

Sizes are those of the repository's own configurations (a 19,728-sample
2-minute sector, a 70,000-sample multi-year curve with up to 187,850 periods, survey
curves of 5,000 to 70,000 samples, 1,024 curves of 20,000 samples) and odd
ones between them.  Inputs are synthetic, made from the seed: regular cadence
with gaps, white noise (or, with errors given per sample, white and red noise),
a limb-darkened transit train.
"""
import numpy as np
import torch

from gtls_b200 import _lib, batch, core, grid, ldmodel, refine, template, validate
from gtls_b200 import gtls

DAY_MIN = 1440.0
PLANET = (12.9, 0.03, 23.1, 89.21, 0, 90, [0.4804, 0.1867], "quadratic")   # the default template
DEPTH_MIN = 10e-6
SKIP = 8


def listed():
    return [
        # the smallest search: one visit of a few days, latency and launches
        dict(name="search_short", kind="search", n=1499, cadence=5.6, gap_days=0.4, dy=False, pmin=0.5, pmax=3.0,
             periods=350, precision="fp64", all=False, batch=12),
        # the main pass of a one-sector search, every period of its grid
        dict(name="search_sector", kind="search", n=19728, cadence=2.0, gap_days=1.0, dy=False, pmin=0.5, pmax=13.7,
             periods=2592, precision="fp64", all=False, batch=86),
        # the main pass over a multi-year curve with per-sample errors
        dict(name="search_long_fp64", kind="search", n=70000, cadence=29.4, gap_days=41.0, dy=True, pmin=0.5,
             pmax=735.0, periods=1500, precision="fp64", all=False, batch=50),
        # the same in the survey's FP32 form, an odd length
        dict(name="search_long_fp32", kind="search", n=65321, cadence=29.4, gap_days=41.0, dy=True, pmin=0.5,
             pmax=650.0, periods=1501, precision="fp32", all=False, batch=50),
        # the re-search of the 200 candidates of a multi-year curve at every start
        dict(name="research_long_fp64", kind="search", n=70000, cadence=29.4, gap_days=41.0, dy=True, pmin=0.5,
             pmax=735.0, periods=200, precision="fp64", all=True, batch=200),
        # a curve above 2^17 samples (20-second cadence over a month and more)
        dict(name="search_dense", kind="search", n=160001, cadence=0.3333, gap_days=1.0, dy=True, pmin=0.5, pmax=18.0,
             periods=300, precision="fp64", all=False, batch=30),
        # the statistics of a spectrum: the multi-year grid, and a sector's
        dict(name="spectra_long", kind="spectra", periods=187850, osf=3, masked=True),
        dict(name="spectra_sector", kind="spectra", periods=2592, osf=3, masked=False),
        # one gradient step of the peak refinement of 1,024 curves
        dict(name="adjoint_set", kind="adjoint", curves=1024, n=20000),
        # whole calls: a sector from host arrays, a multi-year curve, a handful of survey curves in FP32
        dict(name="power_sector", kind="power", n=19728, cadence=2.0, gap_days=1.0, dy=False, pmin=0.5, pmax=13.7,
             batch=86),
        dict(name="power_long", kind="power", n=70000, cadence=29.4, gap_days=41.0, dy=True, pmin=0.7, pmax=735.0,
             batch=1024),
        dict(name="batch_survey", kind="batch", curves=6, n_min=5003, n_max=24000, cadence=10.0, precision="fp32",
             batch=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "spectra", "adjoint", "power", "batch"])
    if kind == "spectra":
        return dict(kind=kind, periods=_log_int(rng, 300, 187850), osf=rng.choice([1, 2, 3, 5]),
                    masked=rng.random() < 0.5)
    if kind == "adjoint":
        n = _log_int(rng, 1000, 40000)
        return dict(kind=kind, curves=_log_int(rng, 1, min(1024, 20_480_000 // n)), n=n)
    if kind == "batch":
        lo = _log_int(rng, 1500, 8000)
        return dict(kind=kind, curves=rng.randint(2, 7), n_min=lo, n_max=_log_int(rng, lo + 1000, 24000),
                    cadence=rng.choice([2.0, 10.0]), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    batch=rng.randint(20, 100))
    n = _log_int(rng, 1000, 60000 if kind == "power" else 200000)
    # spans of 5 days to 4 years; the cadence follows, between 20 seconds and 30 minutes
    span = float(np.exp(rng.uniform(np.log(max(5.0, n * 0.3333 / DAY_MIN)), np.log(max(6.0, min(1470.0, n * 30.0 / DAY_MIN))))))
    c = dict(kind=kind, n=n, cadence=round(span * DAY_MIN / n, 4), gap_days=round(0.03 * span, 3),
             dy=rng.random() < 0.5, pmin=0.5, pmax=round(span / 2, 3))
    if kind == "power":
        if span > 300.0:
            c["pmin"] = 5.0   # a shorter grid
        c["batch"] = rng.randint(20, 200)
        return c
    c["all"] = rng.random() < 0.3
    c["periods"] = max(3, _log_int(rng, 5, 200) if c["all"] else _log_int(rng, 20, max(21, min(4000, 100_000_000 // n))))
    c["precision"] = rng.choice(["fp64", "fp64", "fp32"])
    c["batch"] = c["periods"] if c["all"] else rng.randint(10, 100)
    return c


# ---------------------------------------------------------------- inputs
def _curve(case, seed, n=None, cadence=None):
    """(t, y, dy or None) on the host: regular cadence, three gaps, white noise
    and one transit train."""
    rng = np.random.default_rng(seed)
    n = int(case["n"] if n is None else n)
    cad = (case["cadence"] if cadence is None else cadence) / DAY_MIN
    t = 1000.0 + np.arange(n) * cad
    gap = case.get("gap_days", 0.03 * n * cad)
    for f in np.sort(rng.uniform(0.1, 0.9, 3)):
        t[int(f * n):] += gap / 3.0
    span = t[-1] - t[0]
    sigma = np.full(n, 1e-3)
    if case.get("dy"):
        sigma = rng.uniform(50e-6, 500e-6, n)
    period = float(np.exp(rng.uniform(np.log(min(2.0, span / 4)), np.log(span / 2.5))))
    depth = float(np.exp(rng.uniform(np.log(300e-6), np.log(2000e-6))))
    rp, a, inc = ldmodel.transit_params_from_shape(period, depth, 0.12 * (period / 4.0) ** (1.0 / 3.0), [0.45, 0.2])
    y = 1.0 + sigma * rng.standard_normal(n)
    if case.get("dy"):   # red noise on top: correlation 0.9 from sample to sample, 100 ppm
        y += 100e-6 * np.sqrt(1 - 0.9 ** 2) * np.convolve(rng.standard_normal(n + 127), 0.9 ** np.arange(128), "valid")
    y *= ldmodel.light_curve(t, t[0] + rng.uniform(0, 1) * period, period, rp, a, inc, [0.45, 0.2])
    return t, y, (sigma if case.get("dy") else None)


def _search_inputs(case, seed):
    """Cleaned curve, trial periods spread over its Ofir grid, and the template
    tables, all on the host."""
    t, y, dy = validate.validate_inputs(*_curve(case, seed))
    p = np.sort(grid.period_grid(1, 1, t.max() - t.min(), period_min=case["pmin"], period_max=case["pmax"],
                                 oversampling_factor=3))
    durs = grid.duration_grid(p, shortest=1 / len(t))
    width = int(np.max(durs) * len(y))
    overview, lc = template.get_cache(durs, width + width % 2, *PLANET)
    p = p[np.linspace(0, len(p) - 1, min(case["periods"], len(p))).astype(int)]
    return t, y, dy, np.ascontiguousarray(p), lc, overview


def _spectra_inputs(case, seed):
    """A chi2 spectrum: noise below a baseline, a slow trend and one peak."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n = case["periods"]
    x = torch.arange(n, dtype=torch.float64, device="cuda") / n
    chi2 = 70000.0 - 20.0 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g).square() - 30.0 * x
    at = int(torch.randint(n // 10, n - n // 10, (1,), device="cuda", generator=g))
    chi2[at - 2:at + 3] -= torch.tensor([100.0, 300.0, 500.0, 320.0, 90.0], dtype=torch.float64, device="cuda")
    mask = None
    if case["masked"]:   # periods whose chi2 is an outlier (over 100 medians)
        mask = torch.rand(n, device="cuda", generator=g) < 0.002
        chi2[mask] = 1e8
        mask = mask.to(torch.uint8)
    return chi2, mask


def _adjoint_inputs(case, seed):
    """Device tensors (t, y, w, off, params): 2-minute curves with a transit
    each and parameters beside the truth."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    C, n = case["curves"], case["n"]
    f64 = dict(dtype=torch.float64, device="cuda")

    def uni(a, b):
        return a + (b - a) * torch.rand(C, 1, generator=g, **f64)

    t = (100.0 + torch.arange(n, **f64) * (2.0 / DAY_MIN)).repeat(C, 1)
    P = torch.exp(uni(0.0, float(np.log(13.0))))
    depth = torch.exp(uni(float(np.log(100e-6)), float(np.log(2000e-6))))
    T0 = 100.0 + uni(0.2, 0.8) * P
    D = 0.13 * P ** (1.0 / 3.0) / 3.0
    x = (t - T0) / P
    x = (x - torch.round(x)) * P / (0.5 * D)
    y = 1.0 - depth * torch.sqrt((1.0 - x * x).clamp(min=0.0)).sqrt()
    y += 1e-3 * torch.randn(C, n, generator=g, **f64)
    dy = torch.full((C, n), 1e-3, **f64)
    off = torch.arange(C + 1, device="cuda") * n
    params = torch.cat([P * (1 + uni(-1e-5, 1e-5)), T0 + uni(-7e-4, 7e-4), D * uni(0.95, 1.05), depth * uni(0.9, 1.1),
                        torch.full_like(P, 0.4804), torch.full_like(P, 0.1867)], dim=1)
    return t.reshape(-1), y.reshape(-1), (1.0 / (dy * dy)).reshape(-1), off, params


def _batch_lengths(case):
    return [int(v) for v in np.geomspace(case["n_min"], case["n_max"], case["curves"])]


def prepare(case, seed):
    k = case["kind"]
    if k == "search":
        t, y, dy, p, lc, overview = _search_inputs(case, seed)
        return dict(case=case, cur=core.CurveOnDevice(t, y, dy, lc, overview), periods=torch.from_numpy(p).cuda())
    if k == "spectra":
        chi2, mask = _spectra_inputs(case, seed)
        return dict(case=case, chi2=chi2, mask=mask)
    if k == "adjoint":
        return dict(case=case, inputs=_adjoint_inputs(case, seed))
    if k == "power":
        return dict(case=case, curve=_curve(case, seed))
    return dict(case=case, curves=[_curve({"n": n, "cadence": case["cadence"]}, 1000 * seed + i)[:2]
                                   for i, n in enumerate(_batch_lengths(case))])


# ---------------------------------------------------------------- the calls
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "search":
        chi2, _ = state["cur"].search(state["periods"], DEPTH_MIN, SKIP, case["batch"],
                                      _lib.GTLS_PASS_ALL if case["all"] else _lib.GTLS_PASS_MAIN, case["precision"])
        return chi2
    if k == "spectra":
        return _lib.spectra(state["chi2"], state["mask"], case["osf"])
    if k == "adjoint":
        t, y, w, off, params = state["inputs"]
        p = params.clone().requires_grad_(True)
        chi2 = refine.model_chi2_function().apply(p, t, y, w, off)
        chi2.sum().backward()
        return chi2.detach(), p.grad
    if k == "power":
        t, y, dy = state["curve"]
        r = gtls(t, y, dy, verbose=False).power(period_min=case["pmin"], period_max=case["pmax"],
                                                oversampling_factor=3, use_threads=1, batch_periods=case["batch"])
        return dict(periods=np.ma.getdata(r.periods), chi2=np.ma.getdata(r.chi2), power=np.ma.getdata(r.power),
                    chi2_main=r.diagnostics["chi2_main"], transit_times=np.asarray(r.transitTimes[:2]),
                    index=int(r.diagnostics["period_index"]), width=int(r.durationPoints),
                    best=np.array([r.period, r.duration, r.depth, r.T0, r.SDE, r.snr, r.snrPink, r.snrFit]))
    out = batch.gtls_batch(state["curves"]).power(precision=case["precision"], use_threads=1,
                                                  batch_periods=case["batch"])
    return dict(best=np.array([[r.period, r.duration, r.depth, r.T0, r.SDE] for r in out]),
                index=np.array([r.period_index for r in out]), width=np.array([r.width for r in out]),
                power=np.concatenate([np.ma.getdata(r.power) for r in out]),
                chi2=np.concatenate([np.ma.getdata(r.chi2) for r in out]))


def work(case):
    """Inputs once, outputs once; per trial period the fold of every sample and
    the prefix of the folded flux (two operations a sample), and for a
    gradient step the forward model and its derivatives in transit."""
    k = case["kind"]
    if k == "spectra":
        n = case["periods"]
        return dict(bytes=8.0 * n * 4 + n * bool(case["masked"]), flops=12.0 * n)
    if k == "adjoint":
        m = float(case["curves"]) * case["n"]
        # about 2% of the samples are in transit: 96 quadrature nodes, some 30 operations a node, value and gradient
        return dict(bytes=24.0 * m + 14 * 8.0 * case["curves"], flops=10.0 * m + 0.02 * m * 96 * 30 * 3)
    if k == "search":
        n, p = float(case["n"]), float(case["periods"])
    elif k == "power":
        n, p = float(case["n"]), _grid_size(case["n"] * case["cadence"] / DAY_MIN + case["gap_days"], case)
    else:
        b = f = 0.0
        for n in _batch_lengths(case):
            p = _grid_size(1.03 * n * case["cadence"] / DAY_MIN, dict(pmin=0.0, pmax=float("inf")))
            b += 24.0 * n + 24.0 * p
            f += 2.0 * n * p
        return dict(bytes=b, flops=f)
    return dict(bytes=24.0 * n + 16.0 * p, flops=2.0 * n * p)


def _grid_size(span, case):
    return float(len(grid.period_grid(1, 1, span, period_min=case["pmin"], period_max=case["pmax"],
                                      oversampling_factor=3)))


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    k = case["kind"]
    if k == "search":
        passes = 9.0 if case["all"] else 1.0
        if case["n"] * float(case["periods"]) * passes > 1.5e8:
            return None   # too long to work out
        return _exact_search(case, seed)
    if k == "spectra":
        return _exact_spectra(case, seed)
    if k == "adjoint":
        return _exact_adjoint(case, seed)
    return None


def _duration_limits(p, span, n):
    """Shortest and longest width (samples) searched at each period."""
    ps = p * 86400.0
    nt = span / p
    tmin = 695508000 * 0.05 * (4.0 * ps / (20848 * 1e15)) ** (1.0 / 3.0)
    tmax = (695508000 * 4.0 + 69911000 * 2.0) * (4.0 * ps / (416970 * 1e15)) ** (1.0 / 3.0)
    lo = np.floor(np.minimum(tmin / ps, 0.15) * n)
    hi = np.ceil(np.minimum(tmax / ps, 0.15) * n * ((nt + 1.0) / nt))
    return lo.astype(int), hi.astype(int)


def _exact_search(case, seed):
    """chi2 of every period from its definition: fold, stable sort, and for
    every duration of the period's batch and every start whose mean depth
    passes, the template's sums over the window."""
    t_h, y_h, dy_h, p_h, lc, overview = _search_inputs(case, seed)
    widths, first = np.unique(overview["width_in_samples"], return_index=True)
    n = len(t_h)
    maxd = int(widths.max()) + int(widths.max()) % 2
    lo, hi = _duration_limits(p_h, float(np.float32(t_h.max() - t_h.min())), n)
    ok = (widths[None, :] >= lo[:, None]) & (widths[None, :] <= hi[:, None])
    t, v0 = torch.from_numpy(t_h).cuda(), torch.from_numpy(y_h - 1.0).cuda()
    w0 = torch.from_numpy(1.0 / (dy_h * dy_h)).cuda()
    E = (v0 * v0 * w0).sum()
    rows = []
    for d in range(len(widths)):
        s = torch.ones(int(widths[d]), dtype=torch.float64)
        m = min(len(lc[first[d]]), len(s))
        s[:m] = 1.0 - torch.from_numpy(np.asarray(lc[first[d]][:m], dtype=np.float64))
        s = s.cuda()
        rows.append(torch.stack([s, s * s]))
    out = torch.empty(len(p_h), dtype=torch.float64, device="cuda")
    for i, P in enumerate(p_h):
        b = i // case["batch"]
        union = np.nonzero(ok[b * case["batch"]:(b + 1) * case["batch"]].any(axis=0))[0]
        x = t / float(P)
        o = torch.argsort(x - torch.trunc(x), stable=True)
        v, w = v0[o], w0[o]
        v, w = torch.cat([v, v[:maxd]]), torch.cat([w, w[:maxd]])
        uw = torch.stack([v * w, w])
        V = torch.cat([v.new_zeros(1), torch.cumsum(v, 0)])
        best = torch.full((), float("inf") if len(union) else float("nan"), dtype=torch.float64, device="cuda")
        for d in union:
            W = int(widths[d])
            s = 1 if case["all"] or W <= SKIP else W // SKIP
            k = torch.arange(0, n, s, device="cuda")
            mean = -(V[k + W] - V[k]) / W
            on = mean > DEPTH_MIN
            if s > 1 or not bool(on.all()):
                best = torch.minimum(best, torch.full_like(best, float(n)))
            k, c = k[on], 2.0 * float(overview["overshoot"][first[d]]) * mean[on]
            step = max(1, 30_000_000 // W)
            for j in range(0, len(k), step):
                win = uw.unfold(1, W, 1)[:, k[j:j + step]]
                B, C = win[0] @ rows[d][0], win[1] @ rows[d][1]
                cj = c[j:j + step]
                best = torch.minimum(best, (E + cj * (2.0 * B + cj * C)).min())
        out[i] = best
    return out


def _exact_spectra(case, seed):
    chi2, mask = _spectra_inputs(case, seed)
    n, k = case["periods"], int(case["osf"] * 30)
    k += 1 - k % 2
    on = torch.ones(n, dtype=torch.bool, device="cuda") if mask is None else mask == 0
    sr = chi2[on].min() / chi2
    mean, std = sr[on].mean(), sr[on].std(correction=0)
    sde_raw = (1.0 - mean) / std
    raw = (sr - mean) * (sde_raw / (sr[on] - mean).max())
    if n <= 2 * k:
        return sr, raw, raw, float(sde_raw), float(sde_raw)
    v = torch.where(on, raw, torch.full_like(raw, float("inf"))).unfold(0, k, 1).sort(dim=1).values
    c = on.to(torch.int64).unfold(0, k, 1).sum(1, keepdim=True)
    med = 0.5 * (v.gather(1, ((c - 1) // 2).clamp(min=0)) + v.gather(1, (c // 2).clamp(max=k - 1)))[:, 0]
    front = (n - len(med)) // 2
    med = torch.cat([med[:1].expand(front), med, med[-1:].expand(n - len(med) - front)])
    p = raw - med
    p = p - p[on].mean()
    sde = (p[on] / p[on].std(correction=0)).max()
    return sr, raw, p * (sde / p[on].max()), float(sde_raw), float(sde)


def _exact_adjoint(case, seed):
    """The transit model by its definition (a disk of radius p across a
    quadratically limb-darkened star, 96-point quadrature) and torch's own
    gradient of it; out of transit the model is 1."""
    t, y, w, off, params = _adjoint_inputs(case, seed)
    C, n = case["curves"], case["n"]
    gx, gw = np.polynomial.legendre.leggauss(96)
    node = torch.from_numpy(np.sin(0.5 * np.pi * gx)).cuda()
    jac = torch.from_numpy(np.cos(0.5 * np.pi * gx) * 0.5 * np.pi * gw).cuda()
    chi2, grad = torch.empty(C, dtype=torch.float64, device="cuda"), torch.empty_like(params)
    step = max(1, 1_000_000 // n)
    for a in range(0, C, step):
        b = min(C, a + step)
        th = params[a:b].clone().requires_grad_(True)
        P, T0, D, depth, u1, u2 = (th[:, j:j + 1].expand(-1, n).reshape(-1) for j in range(6))
        tt, yy, ww = (x[a * n:b * n] for x in (t, y, w))
        with torch.no_grad():   # the samples in transit
            q = (tt - T0) / P
            q = q - torch.round(q)
            K = 1 - u1 / 3 - u2 / 6
            r0 = torch.sqrt(depth * K)
            z = (1 + r0) / torch.sin(np.pi * D / P) * torch.sin(2 * np.pi * q).abs()
            hit = (torch.cos(2 * np.pi * q) >= 0) & (z < 1 + r0)
        rest = (ww * (yy - 1.0) ** 2 * ~hit).reshape(b - a, n).sum(1)
        at = torch.nonzero(hit)[:, 0]
        P, T0, D, depth, u1, u2, tt, yy, ww = (x[at] for x in (P, T0, D, depth, u1, u2, tt, yy, ww))
        K = 1 - u1 / 3 - u2 / 6
        r0 = torch.sqrt(depth * K)
        x = (tt - T0) / P
        z = (1 + r0) / torch.sin(np.pi * D / P) * torch.sin(2 * np.pi * (x - torch.round(x).detach())).abs()

        def integral(lo, hi, length, z, r0, u1, u2):
            m, h = 0.5 * (lo + hi)[:, None], 0.5 * (hi - lo)[:, None]
            r = m + h * node
            om = 1 - torch.sqrt((1 - r * r).clamp(min=0.0))
            return (length(r, z, r0) * (1 - u1[:, None] * om - u2[:, None] * om * om) * h * jac).sum(1)

        def arc(r, z, r0):
            c = (r * r + (z * z - r0 * r0)[:, None]) / (2 * r * z[:, None])
            return 2 * r * torch.arccos(c.clamp(-1.0, 1.0))

        inside = torch.nonzero(r0 - z > 0)[:, 0]
        ring = torch.nonzero(torch.minimum(z + r0, torch.ones_like(z)) > (z - r0).abs())[:, 0]
        f = torch.zeros_like(z)
        zi, ri = z[inside], r0[inside]
        f = f.index_add(0, inside, integral(torch.zeros_like(zi), (ri - zi).clamp(max=1.0),
                                            lambda r, z, r0: 2 * np.pi * r, zi, ri, u1[inside], u2[inside]))
        zr, rr = z[ring], r0[ring]
        f = f.index_add(0, ring, integral((zr - rr).abs(), torch.minimum(zr + rr, torch.ones_like(zr)), arc, zr, rr,
                                          u1[ring], u2[ring]))
        res = ww * (yy - 1.0 + f / (np.pi * K)) ** 2
        c2 = rest.index_add(0, at // n, res)
        c2.sum().backward()
        chi2[a:b] = c2.detach()
        grad[a:b] = th.grad
    return chi2, grad
