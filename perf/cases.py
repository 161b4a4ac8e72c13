"""Timed cases of the periodogram framework: what a survey's programs have it do.

A case is one pass through a public entry point: `calc()` and `peaks()` on
lists of numpy curves (host data in, host results out), `periodograms_device`
and batch plans on curves that are already on the GPU, the frequency-grid
call of the C ABI, and the differentiable Lomb-Scargle power.  Curves have a
survey's seasonal cadence (a 240-day gap each year) and are a third
sinusoids, a third box eclipses and a third noise around magnitude 15;
trial periods are log-spaced, as a search over unknown periods takes them.
"""

import math

import numpy as np
import torch

from periodfind_b200 import _native, gpu, ls_grad
from periodfind_b200.plan import BatchPlan

N_PEAKS = 32


def _case(name, kind, algo, n_curves, n_points, ragged, n_per, n_pdt, p_min, p_max, baseline,
          n_phase=10, n_mag=10, errs=False):
    c = dict(kind=kind, algo=algo, n_curves=n_curves, n_points=n_points, ragged=ragged,
             n_per=n_per, n_pdt=n_pdt, p_min=p_min, p_max=p_max, baseline=baseline,
             n_phase=n_phase, n_mag=n_mag, errs=errs)
    return dict(c, name=name) if name else c


def listed():
    return [
        # A look at one star: latency of the whole call.
        _case("aov_stats_one_curve", "stats", "aov", 1, 500, False, 1000, 1, 0.5, 10.0, 100.0),
        # A small field: the reference benchmark's 100 x 1024 x 1000 row.
        _case("ce_stats_100x1024", "stats", "ce", 100, 1024, False, 1000, 1, 0.5, 10.0, 100.0),
        # The default output ('stats') over a survey's whole period range.
        _case("aov_stats_survey", "stats", "aov", 400, 300, True, 20000, 1, 0.05, 500.0, 2500.0,
              n_phase=15),
        # A survey's ragged batch (20-2000 points) with its top-32 peaks, the
        # pipeline replayed from a plan: CE and AOV.
        _case("ce_survey_plan", "plan", "ce", 3000, 300, True, 20000, 1, 0.05, 500.0, 2500.0),
        _case("aov_survey_plan", "plan", "aov", 3000, 300, True, 20000, 1, 0.05, 500.0, 2500.0,
              n_phase=15),
        # The same ragged batch, Lomb-Scargle periodograms left on the GPU.
        _case("ls_survey_device", "device", "ls", 3000, 300, True, 20000, 1, 0.05, 500.0, 2500.0),
        # Well-sampled curves with period derivatives (a 1000 x 4096 batch's
        # shape), periodograms left on the GPU.
        _case("ce_4096_pdt_device", "device", "ce", 200, 4096, False, 10000, 2, 0.1, 100.0,
              2000.0),
        # The same shape from host arrays to the peaks of each curve.
        _case("aov_4096_pdt_peaks", "peaks", "aov", 250, 4096, False, 10000, 2, 0.1, 100.0,
              2000.0, n_phase=15),
        # Weighted statistics with per-point uncertainties.
        _case("fpw_4096_errs", "pgram", "fpw", 100, 4096, False, 10000, 2, 0.1, 100.0, 2000.0,
              errs=True),
        _case("bls_1500_errs", "pgram", "bls", 150, 1500, False, 10000, 1, 0.1, 100.0, 2000.0,
              n_phase=50, errs=True),
        # Lomb-Scargle on a uniform frequency grid, 64 to 16384 points.
        _case("ls_frequency_grid", "fgrid", "ls", 300, 1024, True, 50000, 1, 0.05, 100.0, 3000.0),
        # A fit through the Lomb-Scargle power: forward and both gradients.
        _case("ls_power_gradients", "grad", "ls", 100, 2048, False, 20000, 1, 0.05, 100.0,
              3000.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# Evaluations (points x trial parameters) a drawn case may have, by kind.
_MOST = {"stats": 2.5e9, "plan": 2.0e10, "device": 1.6e10, "peaks": 2.0e10, "pgram": 4.0e9,
         "fgrid": 2.5e10, "grad": 4.0e9}


def draw(rng):
    kind, algo = rng.choice([
        ("stats", "ce"), ("stats", "aov"), ("stats", "ls"), ("plan", "ce"), ("plan", "aov"),
        ("device", "ce"), ("device", "aov"), ("device", "ls"), ("peaks", "ce"), ("peaks", "aov"),
        ("pgram", "fpw"), ("pgram", "bls"), ("fgrid", "ls"), ("grad", "ls")])
    ragged = rng.random() < 0.5
    n_points = _log_int(rng, 100, 1200) if ragged else _log_int(rng, 33, 5000)
    n_pdt = 2 if kind in ("device", "peaks", "pgram") and rng.random() < 0.4 else 1
    n_per = _log_int(rng, 500, 50000 if kind == "fgrid" else 20000)
    room = _MOST[kind] / (n_points * (1.45 if ragged else 1.0) * n_per * n_pdt)
    n_curves = max(1, _log_int(rng, max(1.0, room / 50.0), max(1.0, room / 1.5)))
    n_curves = min(n_curves, 4000, int(4.0e8 / (n_per * n_pdt)))
    p_min = rng.choice([0.05, 0.1, 0.5])
    if algo == "bls":
        n_phase = rng.choice([30, 50, 64])
    else:
        n_phase = rng.choice([8, 10, 10, 12, 15, 20])
    return _case(None, kind, algo, n_curves, n_points, ragged, n_per, n_pdt, p_min,
                 p_min * rng.choice([20.0, 1000.0, 10000.0]), rng.choice([100.0, 2000.0, 3000.0]),
                 n_phase, rng.choice([8, 10, 10, 12]),
                 algo in ("fpw", "bls") and rng.random() < 0.7)


def _lengths(case):
    # The same for every seed, so that outputs keep their shapes.
    n, m = case["n_curves"], case["n_points"]
    rng = np.random.default_rng([n, m])
    if not case["ragged"]:
        return np.full(n, m, np.int64)
    if case["kind"] == "fgrid":  # log-uniform over a factor of 256 around n_points
        lens = m / 16.0 * np.exp(rng.uniform(0.0, math.log(256.0), n))
        return np.maximum(np.round(lens), 20).astype(np.int64)
    lens = rng.lognormal(math.log(m), 0.8, n)
    return np.clip(np.round(lens), max(20, m // 15), m * 7).astype(np.int64)


def _curves(case, seed):
    """(times, magnitudes, uncertainties, offsets): flat float32 arrays of the
    curves back to back, and int64 offsets."""
    rng = np.random.default_rng([seed, 17])
    lens = _lengths(case)
    n, total = len(lens), int(lens.sum())
    off = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    cid = np.repeat(np.arange(n), lens)
    base = case["baseline"]
    if base > 365.25:
        t = (rng.integers(0, math.ceil(base / 365.25), total) * 365.25
             + rng.uniform(0.0, 125.25, total))
        t = np.minimum(t, base)
    else:
        t = rng.uniform(0.0, base, total)
    t = t[np.argsort(cid * (2.0 * base) + t, kind="stable")].astype(np.float32)
    period = np.exp(rng.uniform(math.log(case["p_min"]), math.log(case["p_max"]), n))[cid]
    ph = np.mod(t / period + rng.uniform(0, 1, n)[cid], 1.0)
    kind = (np.arange(n) % 3)[cid]
    y = np.where(kind == 0, 0.3 * np.sin(2 * np.pi * ph),
                 np.where((kind == 1) & (ph < 0.05), -0.5, 0.0))
    err = rng.uniform(0.02, 0.1, total).astype(np.float32)
    m = (15.0 + y + rng.normal(0.0, 1.0, total) * err).astype(np.float32)
    return t, m, err, off


def _grid(case):
    p = np.exp(np.linspace(math.log(case["p_min"]), math.log(case["p_max"]), case["n_per"]))
    return p.astype(np.float32), np.array([0.0, 1e-6][:case["n_pdt"]], np.float32)


def _freqs(case):
    """(f_min, df) of the uniform frequency grid, cycles per day."""
    lo, hi = 1.0 / case["p_max"], 1.0 / case["p_min"]
    return lo, (hi - lo) / case["n_per"]


def _split(flat, off):
    return [flat[a:b] for a, b in zip(off[:-1], off[1:])]


def _normalized(m, off):
    lens = np.diff(off)
    lo = np.repeat(np.minimum.reduceat(m, off[:-1]), lens)
    hi = np.repeat(np.maximum.reduceat(m, off[:-1]), lens)
    return ((m - lo) / (hi - lo)) * np.float32(0.999) + np.float32(5e-4)


def _centered(m, off):
    mean = np.add.reduceat(m.astype(np.float64), off[:-1]) / np.diff(off)
    return (m - np.repeat(mean, np.diff(off))).astype(np.float32)


def _object(case):
    a = case["algo"]
    if a == "ce":
        return gpu.ConditionalEntropy(case["n_phase"], case["n_mag"])
    if a == "aov":
        return gpu.AOV(case["n_phase"])
    if a == "fpw":
        return gpu.FPW(case["n_phase"])
    if a == "bls":
        return gpu.BoxLeastSquares(case["n_phase"], 0.01, 0.5)
    return gpu.LombScargle()


def prepare(case, seed):
    kind, algo = case["kind"], case["algo"]
    t, m, err, off = _curves(case, seed)
    periods, pdts = _grid(case)
    st = dict(kind=kind, off=off, periods=periods, pdts=pdts)
    if kind in ("stats", "peaks", "pgram"):
        if kind == "peaks" and algo == "ce":
            m = _normalized(m, off)
        st.update(obj=_object(case), times=_split(t, off), mags=_split(m, off),
                  errs=_split(err, off) if case["errs"] else None)
        return st
    if kind == "plan" and algo == "ce":
        m = _normalized(m, off)
    if kind in ("fgrid", "grad"):
        m = _centered(m, off)
    dev = "cuda"
    st.update(t=torch.from_numpy(t).to(dev), m=torch.from_numpy(m).to(dev))
    cells = (case["n_curves"], case["n_per"] * case["n_pdt"])
    if kind == "device":
        st.update(obj=_object(case))
    elif kind == "plan":
        out = torch.empty(cells, device=dev)
        idx = torch.empty((cells[0], N_PEAKS), dtype=torch.int64, device=dev)
        val = torch.empty((cells[0], N_PEAKS), device=dev)
        plan = BatchPlan(algo, st["t"], st["m"], off, torch.from_numpy(periods).to(dev),
                         torch.from_numpy(pdts).to(dev), out, n_phase=case["n_phase"],
                         n_mag=case["n_mag"] if algo == "ce" else 1, n_peaks=N_PEAKS,
                         peak_idx=idx, peak_val=val)
        st.update(plan=plan, out=out, idx=idx, val=val)
    elif kind == "fgrid":
        st.update(ctx=_native.default_context(0), out=torch.empty(cells, device=dev),
                  grid=_freqs(case), n_freq=case["n_per"])
    else:
        rng = np.random.default_rng([seed, 23])
        g = rng.uniform(0.0, 1.0, cells).astype(np.float32) / cells[1]
        w = 2.0 * np.pi / periods.astype(np.float64)
        st.update(m=st["m"].requires_grad_(),
                  omega=torch.from_numpy(w).to(dev).requires_grad_(),
                  g=torch.from_numpy(g).to(dev))
    return st


def run(st):
    kind = st["kind"]
    if kind == "stats":
        found = st["obj"].calc(st["times"], st["mags"], st["periods"], st["pdts"])
        rows = np.array([(s.params[0], s.value, s.mean, s.std, s.median, s.mad) for s in found],
                        np.float32)
        return tuple(rows.T)
    if kind == "peaks":
        return st["obj"].peaks(st["times"], st["mags"], st["periods"], st["pdts"], N_PEAKS)
    if kind == "pgram":
        return st["obj"].periodograms(st["times"], st["mags"], st["periods"], st["pdts"],
                                      errs=st["errs"])
    if kind == "device":
        return st["obj"].periodograms_device(st["t"], st["m"], st["off"], st["periods"],
                                             st["pdts"])
    if kind == "plan":
        st["plan"].launch()
        return st["out"], st["idx"], st["val"]
    if kind == "fgrid":
        ctx, out = st["ctx"], st["out"]
        with ctx.lock:
            ctx.check(ctx.lib.pf_ls_fgrid_dev(
                ctx.handle, st["t"].data_ptr(), st["m"].data_ptr(), st["off"].ctypes.data,
                len(st["off"]) - 1, *st["grid"], st["n_freq"], _native.PF_MODE_CHOSEN,
                out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return out
    st["m"].grad = st["omega"].grad = None
    power = ls_grad.ls_power(st["t"], st["m"], st["omega"], st["off"])
    power.backward(st["g"])
    return power.detach(), st["m"].grad, st["omega"].grad


def _points(case):
    """Expected number of points of the case's curves."""
    mean = case["n_points"] * 1.0
    if case["ragged"]:
        mean *= (256.0 - 1.0) / (16.0 * math.log(256.0)) if case["kind"] == "fgrid" else 1.35
    return mean * case["n_curves"]


def work(case):
    pts, cells = _points(case), case["n_per"] * case["n_pdt"]
    n_out = case["n_curves"] * cells
    # Arithmetic of one evaluation: the fold (product and fraction), then the
    # bin and its update, or the trigonometric sums.  On a uniform frequency
    # grid the sums follow from two transforms of the grid's length.
    per = {"ce": 4.0, "aov": 5.0, "fpw": 5.0, "bls": 5.0, "ls": 14.0}[case["algo"]]
    if case["kind"] == "fgrid":
        flops = case["n_curves"] * 2.0 * 5.0 * cells * math.log2(cells) + pts * 100.0
    elif case["kind"] == "grad":
        flops = pts * cells * (22.0 + 12.0)
    else:
        flops = pts * cells * per
        if case["algo"] == "bls":
            flops += n_out * case["n_phase"] ** 2 / 2.0 * 8.0
    if case["kind"] == "stats":
        n_out = 6.0 * case["n_curves"]
    elif case["kind"] == "peaks":
        n_out = 3.0 * N_PEAKS * case["n_curves"]
    elif case["kind"] == "plan":
        n_out += 3.0 * N_PEAKS * case["n_curves"]
    elif case["kind"] == "grad":
        n_out = 2.0 * n_out + pts + 4.0 * cells
    return {"bytes": 4.0 * (pts * (3.0 if case["errs"] else 2.0) + n_out), "flops": flops}


# ------------------------------------------------ the same values in 64 bits

def _phase(t, periods, pdt):
    """Folded phase [points, periods] of one curve."""
    if pdt:
        q = (t[:, None] - (0.5 * pdt / periods)[None, :] * (t * t)[:, None]) / periods[None, :]
    else:
        q = t[:, None] / periods[None, :]
    return q - torch.floor(q)


def _sums(index, n_bins, n_per, weight=None):
    """Per-period sums over bins, [n_bins, n_per]; index [points, periods]."""
    out = torch.zeros(n_bins * n_per, dtype=torch.float64, device=index.device)
    flat = index * n_per + torch.arange(n_per, device=index.device)[None, :]
    src = torch.ones(1, 1, dtype=torch.float64, device=index.device)
    src = src if weight is None else weight[:, None]
    out.scatter_add_(0, flat.reshape(-1), src.expand(flat.shape).reshape(-1))
    return out.view(n_bins, n_per)


def _one_exact(case, t, m, err, periods, pdt):
    """One curve's periodogram [n_per] in float64."""
    n, n_per, nb = len(t), len(periods), case["n_phase"]
    algo = case["algo"]
    if algo == "ls":
        th = (2.0 * math.pi) * _phase(t, periods, pdt)
        c, s = torch.cos(th), torch.sin(th)
        C, S = m @ c, m @ s
        CC, CS = (c * c).sum(0), (c * s).sum(0)
        SS = n - CC
        return 0.5 * (SS * C * C - 2.0 * CS * C * S + CC * S * S) / (CC * SS - CS * CS)
    b = torch.clamp((_phase(t, periods, pdt) * nb).to(torch.int64), max=nb - 1)
    if algo == "ce":
        k = case["n_mag"]
        col = torch.clamp((m * k).to(torch.int64), 0, k - 1)
        c = _sums(b * k + col[:, None], nb * k, n_per).view(nb, k, n_per)
        row = c.sum(1)
        return (torch.xlogy(row, row).sum(0) - torch.xlogy(c, c).sum((0, 1))) / n
    if algo == "aov":
        x = m - m.mean()
        c, y = _sums(b, nb, n_per), _sums(b, nb, n_per, x)
        s1 = (y * y / torch.clamp(c, min=1.0)).sum(0)
        return (n - nb) / (nb - 1.0) * s1 / ((x * x).sum() - s1)
    w = 1.0 / (err * err) if err is not None else torch.ones_like(t)
    if algo == "bls":
        m = m - (w * m).sum() / w.sum()
    v, y = _sums(b, nb, n_per, w), _sums(b, nb, n_per, w * m)
    if algo == "fpw":
        return torch.where(v > 0, y * y / (2.0 * torch.clamp(v, min=1e-300)), 0.0).sum(0)
    best = torch.zeros(n_per, dtype=torch.float64, device=t.device)
    cum = lambda a: torch.cumsum(torch.cat([torch.zeros_like(a[:1]), a, a]), 0)
    cv, cy, W = cum(v), cum(y), v.sum(0)
    for width in range(max(int(0.01 * nb), 1), min(math.ceil(0.5 * nb), nb - 1) + 1):
        r, sy = cv[width:width + nb] - cv[:nb], cy[width:width + nb] - cy[:nb]
        ok = (v > 0).to(torch.float64)
        filled = cum(ok)
        inside = filled[width:width + nb] - filled[:nb]
        ok = (inside > 0) & (inside < ok.sum(0))
        sc = torch.where(ok, sy * sy / torch.where(ok, r * (W - r), 1.0), 0.0)
        best = torch.maximum(best, sc.amax(0))
    return best


def _exact_grad(t, m, off, omega, g):
    power = torch.empty_like(g)
    gm, gw = torch.empty_like(m), torch.zeros_like(omega)
    for c, (a, b) in enumerate(zip(off[:-1], off[1:])):
        tc = t[a:b] - 0.5 * (t[a:b].min() + t[a:b].max())
        y, n = m[a:b], int(b - a)
        th = tc[:, None] * omega[None, :]
        co, si = torch.cos(th), torch.sin(th)
        C, S, CC, CS = y @ co, y @ si, (co * co).sum(0), (co * si).sum(0)
        C1, S1 = -((y * tc) @ si), (y * tc) @ co
        CC1 = -2.0 * (tc @ (co * si))
        CS1 = tc @ (co * co) - tc @ (si * si)
        SS = n - CC
        det = CC * SS - CS * CS
        al, be = (SS * C - CS * S) / det, (CC * S - CS * C) / det
        power[c] = 0.5 * (al * C + be * S)
        gm[a:b] = co @ (g[c] * al) + si @ (g[c] * be)
        gw += g[c] * (al * C1 + be * S1 - 0.5 * ((al * al - be * be) * CC1 + 2.0 * al * be * CS1))
    return power, gm, gw


def exact(case, seed):
    kind, algo = case["kind"], case["algo"]
    if kind == "peaks":
        return None
    if kind == "stats":
        return _exact_stats(case, seed)
    t, m, err, off = _curves(case, seed)
    if algo == "ce":
        m = _normalized(m, off)
    elif kind in ("fgrid", "grad") or algo == "ls":
        m = _centered(m, off)
    dev = "cuda"
    t, m, err = (torch.from_numpy(a).to(dev, torch.float64) for a in (t, m, err))
    periods, pdts = _grid(case)
    if kind == "grad":
        rng = np.random.default_rng([seed, 23])
        cells = (case["n_curves"], case["n_per"])
        g = rng.uniform(0.0, 1.0, cells).astype(np.float32) / cells[1]
        w = torch.from_numpy(2.0 * np.pi / periods.astype(np.float64)).to(dev)
        return _exact_grad(t, m, off, w, torch.from_numpy(g).to(dev, torch.float64))
    if kind == "fgrid":
        lo, df = _freqs(case)
        pd = 1.0 / (lo + df * torch.arange(case["n_per"], dtype=torch.float64, device=dev))
    else:
        pd = torch.from_numpy(periods).to(dev, torch.float64)
    out = torch.empty((case["n_curves"], case["n_per"], case["n_pdt"]), dtype=torch.float64,
                      device=dev)
    for c, (a, b) in enumerate(zip(off[:-1], off[1:])):
        step = max(1, int(4.0e8) // int(b - a))
        for k in range(0, case["n_per"], step):
            for d in range(case["n_pdt"]):
                out[c, k:k + step, d] = _one_exact(
                    case, t[a:b], m[a:b], err[a:b] if case["errs"] else None, pd[k:k + step],
                    float(pdts[d]))
    if kind == "plan":
        return out.view(case["n_curves"], -1), None, None
    if kind == "fgrid":
        return out.view(case["n_curves"], -1)
    return out.cpu().numpy() if kind == "pgram" else out


def _exact_stats(case, seed):
    """Best value, mean, std, median and MAD (the best period is one of the
    grid's, picked by the float32 periodogram: no value here)."""
    t, m, _, off = _curves(case, seed)
    if case["algo"] == "ce":
        m = _normalized(m, off)
    elif case["algo"] == "ls":
        m = _centered(m, off)
    t, m = (torch.from_numpy(a).to("cuda", torch.float64) for a in (t, m))
    periods = torch.from_numpy(_grid(case)[0]).to("cuda", torch.float64)
    rows = []
    for a, b in zip(off[:-1], off[1:]):
        x = _one_exact(case, t[a:b], m[a:b], None, periods, 0.0)
        best = x.min() if case["algo"] == "ce" else x.max()
        med = x.quantile(0.5)
        rows.append(torch.stack([best, x.mean(), x.std(correction=0), med,
                                 (x - med).abs().quantile(0.5)]))
    return (None, *torch.stack(rows).cpu().numpy().T)
