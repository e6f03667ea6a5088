"""The workloads that the framework's speed is measured on: what its users have it do.

Every case goes through public entry points on synthetic light curves of the surveys' shapes
(Kepler's 29.4-min and TESS's 2-min cadence, contiguous gaps with time -1000 and zig-zag filled
flux, stellar trends, noise, transits in a part of the curves).  A case's ``kind`` names the
path, its other entries the sizes; ``listed`` holds one of each kind, ``draw`` gives others of
the same ranges.
"""
import math

import numpy as np
import torch

from gtrap_gb300 import api, batch, serve, synth, tls
from gtrap_gb300.detect_peaks import detect_peaks

TESS, KEPLER = 2.0 / 1440.0, 29.4 / 1440.0   # cadences in days
CADENCE = {"tess": TESS, "kepler": KEPLER}
QMI, QMA = 0.005, 0.1                         # shortest and longest transit in units of the period
NW, NL = 8, 16                                # GTLS widths and ingress widths
FOLD_W = np.linspace(0.5, 8.0, 8, dtype=np.float32) / np.float32(24.0)   # days
REFINED = ("freq", "period", "phase", "duration", "t0", "depth", "sr")


def listed():
    return [
        # One short curve asked for by itself, from the raw flux to the best period: latency.
        dict(name="curve_bls", kind="curve_bls", n=3001, cadence="kepler", r=24),
        # One TESS sector curve through the single-event search and the reference's peak finder.
        dict(name="curve_tls", kind="curve_tls", n=20011, r=24, mpd=10),
        # A batch of evenly sampled curves on one time axis: the plain BLS configuration.
        dict(name="plain_bls", kind="plain_bls", n=4096, nq=64, nf=4096, nb=1024),
        # Whole Kepler-mission curves with gaps as an [n, nq] image: detrend, offset, BLS, statistics.
        dict(name="kepler_bls", kind="kepler_bls", n=65536, nq=8, nf=16384, nb=2048, r=24),
        # What follows a BLS search of many curves: statistics and the refined best peak of each.
        dict(name="bls_peaks", kind="bls_peaks", n=18000, nq=64, nf=4096),
        # The running-median detrend of an image by itself, and its offsets.
        dict(name="detrend", kind="detrend", n=65536, nq=128, r=24),
        # A TESS sector image through the single-event search.
        dict(name="tess_tls", kind="tess_tls", n=18000, nq=96, mode=0),
        # Peak statistics of many single-event S/N series.
        dict(name="tls_peaks", kind="tls_peaks", n=18000, nq=96, mpd=10, ntop=4, k=8),
        # The folded trapezoid search of a TESS sector image.
        dict(name="fold", kind="fold", n=18000, nq=16, nf=8192, nb=2048, dmax=1024),
        # Curves of every length, cadence and grid as one packed batch: the production path.
        dict(name="ragged", kind="ragged", curves=160, n_max=70000, r=24),
        # The trapezoid grid fit in 64 bits of one curve held by the host.
        dict(name="grid_fit", kind="grid_fit", n=18000, nw=8, nl=8, nt=4211),
        # A dozen requests handed to the server at once, results on the host.
        dict(name="served", kind="served", requests=12, n_max=70000, r=24),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["curve_bls", "curve_tls", "plain_bls", "kepler_bls", "bls_peaks", "detrend", "tess_tls",
                       "tls_peaks", "fold", "ragged", "grid_fit", "served"])
    r = rng.choice([_log(rng, 5, 64), 16, 24, 32, 128])
    if kind == "curve_bls":
        return dict(kind=kind, n=_log(rng, 1000, 70000), cadence=rng.choice(["tess", "kepler"]), r=r)
    if kind == "curve_tls":
        return dict(kind=kind, n=_log(rng, 2000, 30000), r=r, mpd=rng.choice([1, 10, 100]))
    if kind == "plain_bls":
        return dict(kind=kind, n=_log(rng, 500, 4096), nq=_log(rng, 1, 64), nf=_log(rng, 500, 4096),
                    nb=rng.choice([256, 512, 1000, 1024, 2048]))
    if kind == "kepler_bls":
        return dict(kind=kind, n=_log(rng, 8000, 65536), nq=_log(rng, 1, 8), nf=_log(rng, 2000, 16384),
                    nb=rng.choice([1024, 2048]), r=r)
    if kind == "bls_peaks":
        return dict(kind=kind, n=_log(rng, 2000, 18000), nq=_log(rng, 1, 64), nf=_log(rng, 1000, 4096))
    if kind == "detrend":
        return dict(kind=kind, n=_log(rng, 1000, 65536), nq=_log(rng, 1, 128), r=r)
    if kind == "tess_tls":
        return dict(kind=kind, n=_log(rng, 1000, 18000), nq=_log(rng, 1, 96), mode=rng.choice([0, 1]))
    if kind == "tls_peaks":
        return dict(kind=kind, n=_log(rng, 1000, 18000), nq=_log(rng, 1, 96), mpd=rng.choice([1, 10, 30]),
                    ntop=4, k=rng.choice([4, 8, 16]))
    if kind == "fold":
        nb = rng.choice([512, 1024, 2048, 4096])
        return dict(kind=kind, n=_log(rng, 1000, 18000), nq=_log(rng, 1, 16), nf=_log(rng, 200, 4096), nb=nb,
                    dmax=nb // rng.choice([2, 4]))
    if kind == "ragged":
        return dict(kind=kind, curves=_log(rng, 3, 100), n_max=_log(rng, 4000, 70000), r=24)
    if kind == "grid_fit":
        return dict(kind=kind, n=_log(rng, 1000, 18000), nw=rng.randint(2, 8), nl=rng.randint(2, 8),
                    nt=_log(rng, 100, 4000))
    return dict(kind=kind, requests=rng.randint(1, 12), n_max=_log(rng, 4000, 70000), r=24)


# ------------------------------------------------------------------------------------ inputs

def _image(n, nq, cadence, seed, gaps, trends, noise, flip=False):
    """Curves ``[n, nq]`` on the GPU: (flux, times), float32.  ``gaps``: fraction of the samples
    in gaps of 0.5 to 3 days (time -1000, zig-zag filled flux)."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def uni(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    t = (torch.arange(n, device="cuda", dtype=torch.float64)[:, None] + 0.5) * cadence
    t = t + uni(-1.0, 1.0, n, nq) / 86400.0
    span = n * cadence
    f = torch.ones(n, nq, device="cuda", dtype=torch.float64)
    if trends:
        for _ in range(3):
            f += uni(2e-4, 2e-3, nq) * torch.sin(2 * math.pi * t / uni(5.0, 50.0, nq) + uni(0, 2 * math.pi, nq))
        f += uni(-1e-3, 1e-3, nq) * (t / span) ** 2 + uni(-1e-3, 1e-3, nq) * (t / span)
    # a transit in a quarter of the curves, with an ingress of up to half its width
    per, width = uni(1.0, min(12.0, max(1.5, span / 2)), nq), uni(0.5, 6.0, nq) / 24.0
    ph = torch.remainder(t - uni(0.0, 1.0, nq) * per + 0.5 * per, per) - 0.5 * per
    ramp = uni(0.05, 0.5, nq) * width
    depth = uni(3e-4, 3e-3, nq) * (uni(0.0, 1.0, nq) < 0.25)
    f -= depth * torch.clamp((0.5 * width - ph.abs()) / ramp, 0.0, 1.0)
    f += noise * torch.randn(n, nq, generator=g, device="cuda", dtype=torch.float64)
    if flip:
        f = 2.0 - f
    count = max(1, int(round(gaps * span / 1.75))) if gaps else 0
    mask = torch.zeros(n, nq, dtype=torch.bool, device="cuda")
    rows = torch.arange(n, device="cuda")[:, None]
    for _ in range(count):
        a = uni(0, n, nq)
        mask |= (rows >= a) & (rows < a + uni(0.5, 3.0, nq) / cadence)
    big = torch.finfo(torch.float64).max
    lo = torch.where(mask, big, f).amin(0)
    hi = torch.where(mask, -big, f).amax(0)
    fill = torch.where(rows % 2 == 0, lo, hi)
    f = torch.where(mask, fill, f)
    t = torch.where(mask, torch.full_like(t, synth.INVALID_T), t)
    return f.float().contiguous(), t.float().contiguous()


def _centred(n, nq, seed):
    """TESS curves of flipped, centred flux with a gap in the middle, as gtls takes them."""
    lc, tu = _image(n, nq, TESS, seed, 0.0, False, 1e-3, flip=True)
    g = min(int(1.0 / TESS), n // 10)
    rows = torch.arange(n, device="cuda")[:, None]
    gap = (rows >= n // 2 - g // 2) & (rows < n // 2 - g // 2 + g)
    lc = lc - torch.where(gap, 0.0, lc.double()).sum(0).div(n - g).float()
    return (torch.where(gap, torch.zeros((), device="cuda"), lc).contiguous(),
            torch.where(gap, torch.full((), -1000.0, device="cuda"), tu).contiguous())


def _bls_grid(n, span, nb=2048, nf=None):
    """The frequency grid of a curve: about eight per day of baseline, up to two cycles a day."""
    nf = nf or int(min(32768, max(2048, synth.next_pow2(8.0 * span))))
    fmin = float(np.float32(2.0 / span))
    return dict(nf=nf, nb=nb, kma=int(QMA * nb) + 1, kmi=int(QMI * nb), kkmi=int(n * QMI), fmin=fmin,
                df=float(np.float32((2.0 - fmin) / (nf - 1))))


def _tls_grid(cadence):
    g = synth.tls_grid(nw=NW, nl=NL, deltat=cadence)
    return g["nsc"], g["wmax"], g["dw"], g["deltat"]


def _curves(case, seed, count):
    """Requests of the uneven mix: lengths log-uniform up to n_max, both cadences, BLS and GTLS.
    The lengths and grids are the case's own; times and flux are the seed's."""
    out = []
    for k in range(count):
        c = synth.ragged_curve(k, n_range=(2000, case["n_max"]))
        rng = np.random.default_rng((seed, k))
        shift = rng.uniform(0.0, 0.01) + rng.uniform(-1.0, 1.0, c["n"]) / 86400.0
        c["t"] = np.where(c["t"] < 0, c["t"], c["t"] + shift).astype(np.float32)
        c["x"] = (c["x"] + rng.normal(0.0, 5e-4, c["n"])).astype(np.float32)
        out.append(c)
    return out


def _fit_inputs(case, seed):
    lc, tu = _centred(case["n"], 1, seed)
    t, x = tu[:, 0].double().cpu().numpy(), -lc[:, 0].double().cpu().numpy()
    keep = t >= 0
    W = np.linspace(0.5, 8.0, case["nw"]) / 24.0
    L = np.linspace(2.0, 30.0, case["nl"]) / 1440.0
    return t[keep], x[keep], W, L, np.linspace(t[keep][0], t[keep][-1], case["nt"])


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind in ("curve_bls", "kepler_bls"):
        cad = CADENCE[case.get("cadence", "kepler")]
        nq = case.get("nq", 1)
        s["lc"], s["tu"] = _image(case["n"], nq, cad, seed, 0.1 if kind == "curve_bls" else 0.05, True, 5e-4)
        s["ntrue"] = (s["tu"] >= 0).sum(0).int()
        s["grid"] = _bls_grid(case["n"], case["n"] * cad, case.get("nb", 2048), case.get("nf"))
    elif kind == "curve_tls":
        s["lc"], s["tu"] = _image(case["n"], 1, TESS, seed, 0.05, True, 1e-3, flip=True)
    elif kind == "plain_bls":
        lc, _ = _image(case["n"], case["nq"], KEPLER, seed, 0.0, False, 1e-3)
        s["lc"] = (lc - lc.double().mean(0).float()).contiguous()
        s["tu"] = (0.02043 * torch.arange(case["n"], device="cuda", dtype=torch.float64)).float()
        s["grid"] = _bls_grid(case["n"], 60.0, case["nb"], case["nf"])
    elif kind == "bls_peaks":
        s["lc"], s["tu"] = _image(case["n"], case["nq"], KEPLER, seed, 0.05, False, 5e-4)
        s["ntrue"] = (s["tu"] >= 0).sum(0).int()
        s["grid"] = _bls_grid(case["n"], case["n"] * KEPLER, 2048, case["nf"])
        s["lc"] = api.gfilter(s["lc"], 24)
        s["off"] = api.offset(s["lc"], s["tu"])
        s["spectra"] = api.geebls(s["lc"], s["tu"], s["off"], s["ntrue"], **s["grid"])
    elif kind == "detrend":
        s["lc"], s["tu"] = _image(case["n"], case["nq"], KEPLER, seed, 0.05, True, 5e-4)
    elif kind == "tess_tls":
        s["lc"], s["tu"] = _centred(case["n"], case["nq"], seed)
    elif kind == "tls_peaks":
        lc, tu = _centred(case["n"], case["nq"], seed)
        nsc, wmax, dw, deltat = _tls_grid(TESS)
        s["sn"] = api.gtls(lc, tu, case["n"], 4, 8, nsc, wmax, dw, deltat)[0]
    elif kind == "fold":
        s["lc"], s["tu"] = _centred(case["n"], case["nq"], seed)
        s["off"] = torch.zeros(case["nq"], dtype=torch.float32, device="cuda")
        span = case["n"] * TESS
        s["fmin"] = float(np.float32(min(0.5, 2.0 / span)))
        s["df"] = float(np.float32((2.0 - s["fmin"]) / (case["nf"] - 1)))
    elif kind == "ragged":
        b = batch.RaggedBatch(batch.BlsSpec(2048, 205, 10), batch.TlsSpec(NW, NL), detrend_r=case["r"])
        for c in _curves(case, seed, case["curves"]):
            if c["kind"] == "bls":
                b.add_bls(c["t"], c["x"], c["nf"], c["fmin"], c["df"], kkmi=c["kkmi"])
            else:
                b.add_tls(c["t"], c["x"], c["nsc"], c["wmax"], c["dw"], c["deltat"])
        s["batch"] = b.build()
    elif kind == "grid_fit":
        s["fit"] = _fit_inputs(case, seed)
    else:
        s["requests"] = [serve.Request.from_curve(c) for c in _curves(case, seed, case["requests"])]
        s["server"] = serve.TransitServer(detrend_r=case["r"], hbm_budget=2e9)
    return s


# ------------------------------------------------------------------------------------ one pass

def run(s):
    kind, case = s["kind"], s["case"]
    if kind in ("curve_bls", "kepler_bls"):
        res = api.gfilter(s["lc"], case["r"])
        off = api.offset(res, s["tu"])
        g = s["grid"]
        sr, p1, p2 = api.geebls(res, s["tu"], off, s["ntrue"], **g)
        pest, sde, b1, b2 = api.blsstat(sr, p1, p2, g["df"], g["fmin"])
        return dict(sr=sr, p1=p1, p2=p2, pest=pest, sde=sde, b1=b1, b2=b2)
    if kind == "curve_tls":
        n = case["n"]
        nsc, wmax, dw, deltat = _tls_grid(TESS)
        out = api.gtls(api.gfilter(s["lc"], case["r"]), s["tu"], n, NW, NL, nsc, wmax, dw, deltat)
        peaks = np.zeros(n, np.int8)   # their number differs from curve to curve: marked in the series
        peaks[detect_peaks(out[0], mpd=case["mpd"])] = 1
        return dict(zip(("sn", "w", "t0", "l", "h"), out), peaks=peaks)
    if kind == "plain_bls":
        return dict(zip(("sr", "p1", "p2"), api.geebls_simple(s["lc"], s["tu"], with_phase=True, **s["grid"])))
    if kind == "bls_peaks":
        g = s["grid"]
        pest, sde, b1, b2 = api.blsstat(*s["spectra"], g["df"], g["fmin"])
        grid = {k: g[k] for k in ("nb", "kma", "kmi", "kkmi", "fmin", "df")}
        rec = api.refined_to_numpy(api.bls_refine(*s["spectra"], s["lc"], s["tu"], s["off"], s["ntrue"], **grid))
        return dict({k: rec[k] for k in rec.dtype.names}, pest=pest, sde=sde, b1=b1, b2=b2)
    if kind == "detrend":
        res = api.gfilter(s["lc"], case["r"])
        return dict(residual=res, offset=api.offset(res, s["tu"]))
    if kind == "tess_tls":
        nsc, wmax, dw, deltat = _tls_grid(TESS)
        out = api.gtls(s["lc"], s["tu"], case["n"], NW, NL, nsc, wmax, dw, deltat, mode=case["mode"])
        return dict(zip(("sn", "w", "t0", "l", "h"), out))
    if kind == "tls_peaks":
        stats, idx, val = api.tls_peakstat(s["sn"], case["mpd"], case["ntop"], case["k"])
        rec = api.stats_to_numpy(stats)
        return dict({k: rec[k] for k in rec.dtype.names}, idx=idx, val=val)
    if kind == "fold":
        out = api.tls_fold(s["lc"], s["tu"], s["off"], case["nf"], case["nb"], s["fmin"], s["df"], FOLD_W,
                           lfrac=0.2, dmax=case["dmax"])
        return dict(zip(("tsr", "start", "dur", "depth"), out))
    if kind == "ragged":
        b = s["batch"]
        b.launch()
        out = dict(tls=list(b.tls_outs)) if b.n_tls else {}
        if b.n_bls:
            out.update(bls=[b.blsp, b.ph1, b.ph2], stats=list(b.bls_stats()))
        return out
    if kind == "grid_fit":
        t, x, W, L, T = s["fit"]
        model, H, w, l, t0, off = tls.tlsfit(t, x, W, L, T)
        return dict(model=model, best=[H, w, l, t0, off])
    rids = [s["server"].submit(q) for q in s["requests"]]
    got = {r.rid: r.outputs for r in s["server"].run_until_idle()}
    return [got[k] for k in rids]


# ------------------------------------------------------------------- what a pass cannot do without

def _searches(kind, case):
    """(samples, BLS (sample, frequency) pairs, GTLS epochs, output values) of a case, of the
    uneven mix by its expectation (half of each kind, lengths log-uniform)."""
    count = case.get("curves") or case.get("requests")
    ratio = case["n_max"] / 2000.0
    mean = (case["n_max"] - 2000.0) / math.log(ratio)
    mean2 = (case["n_max"] ** 2 - 2000.0 ** 2) / (2 * math.log(ratio))
    nf = max(2048.0, 4.3 * KEPLER * mean + 1024.0)     # mean of the two cadences' grids
    return count * mean, 0.5 * count * max(2048.0 * mean, 6.0 * KEPLER * mean2), 0.5 * count * mean, \
        count * (1.5 * nf + 2.5 * mean)


def work(case):
    """Bytes: inputs read once and outputs written once.  Operations: two additions a (sample,
    trial frequency) of a fold, some 16 a trapezoid template, a few a sample of the rest."""
    kind = case["kind"]
    n, nq = case.get("n", 0), case.get("nq", 1)
    if kind in ("curve_bls", "kepler_bls"):
        nf = _bls_grid(n, n * CADENCE[case.get("cadence", "kepler")], case.get("nb", 2048), case.get("nf"))["nf"]
        return dict(bytes=nq * (8 * n + 12 * nf), flops=2.0 * nq * n * nf)
    if kind == "plain_bls":
        return dict(bytes=nq * (4 * n + 12 * case["nf"]) + 4 * n, flops=2.0 * nq * n * case["nf"])
    if kind in ("curve_tls", "tess_tls"):
        return dict(bytes=28 * n * nq, flops=16.0 * n * nq * NW * NL)
    if kind == "bls_peaks":
        return dict(bytes=nq * (8 * n + 4 * case["nf"] + 96), flops=2.0 * 65 * n * nq)
    if kind == "detrend":
        return dict(bytes=12 * n * nq, flops=n * nq * 2.0 * math.log2(2 * case["r"] + 1))
    if kind == "tls_peaks":
        return dict(bytes=4 * n * nq, flops=8.0 * n * nq)
    if kind == "fold":
        pairs = float(nq * case["nf"])
        return dict(bytes=nq * (8 * n + 16 * case["nf"]), flops=pairs * (2.0 * n + 8 * 16 * case["nb"]))
    if kind == "grid_fit":
        W = np.linspace(0.5, 8.0, case["nw"]) / 24.0
        return dict(bytes=16 * n + 8 * n, flops=10.0 * case["nl"] * case["nt"] * float((W / TESS).sum()))
    samples, pairs, epochs, outs = _searches(kind, case)
    return dict(bytes=8 * samples + 4 * outs, flops=2.0 * pairs + 16.0 * epochs * NW * NL)


# ------------------------------------------------------------------------ the same in 64 bits

def _median64(x, r):
    """x[n, nq] less its running median over 2r + 1 rows, zeros outside, in 64 bits."""
    n, nq = x.shape
    p = torch.nn.functional.pad(x.double().t(), (r, r))
    out = torch.empty(nq, n, dtype=torch.float64, device=x.device)
    step = max(1, (1 << 26) // (2 * r + 1))
    for q in range(nq):
        for a in range(0, n, step):
            b = min(n, a + step)
            out[q, a:b] = p[q, r + a:r + b] - p[q, a:b + 2 * r].unfold(0, 2 * r + 1, 1).median(-1)[0]
    return out.t().contiguous()


def _offset64(res, tu):
    return torch.where(tu < 0, 0.0, res).sum(0) / res.shape[0]


def _bls64(t, x, N, g):
    """The BLS spectrum of one curve's valid samples (float64), without ties."""
    nf, nb, kma, kmi = g["nf"], g["nb"], g["kma"], max(g["kmi"], 1)
    kkmi = max(g["kkmi"], 5)
    a = torch.frac(t.double() * g["fmin"])
    b = torch.frac(t.double() * g["df"])
    out = torch.empty(nf, dtype=torch.float64, device=t.device)
    rows = max(1, min(512, (1 << 25) // max(t.numel(), nb)))
    for j0 in range(0, nf, rows):
        j = torch.arange(j0, min(nf, j0 + rows), device=t.device, dtype=torch.float64)[:, None]
        bins = (torch.frac(a + j * b) * nb).long().clamp_(max=nb - 1)
        m = j.numel()
        S = torch.zeros(m, nb, dtype=torch.float64, device=t.device).scatter_add_(1, bins, x.expand(m, -1))
        C = torch.zeros(m, nb, dtype=torch.float64, device=t.device).scatter_add_(
            1, bins, torch.ones_like(x).expand(m, -1))
        zero = torch.zeros(m, 1, dtype=torch.float64, device=t.device)
        S = torch.cat([zero, torch.cat([S, S[:, :kma]], 1).cumsum(1)], 1)
        C = torch.cat([zero, torch.cat([C, C[:, :kma]], 1).cumsum(1)], 1)
        best = torch.zeros(m, dtype=torch.float64, device=t.device)
        for k in range(kmi + 1, kma + 1):
            s, c = S[:, k:k + nb] - S[:, :nb], C[:, k:k + nb] - C[:, :nb]
            p = torch.where(c > kkmi, s * s / (c * (N - c)), 0.0)
            best = torch.maximum(best, p.amax(1))
        out[j0:j0 + m] = best.sqrt()
    return out


def _stat64(sr, df, fmin):
    m, at = sr.max(1)
    mean = sr.mean(1)
    return 1.0 / (at.double() * df + fmin), (m - mean) / ((sr * sr).mean(1) - mean * mean).sqrt()


def _tls64(lc, tu, grid, mode=0):
    """The best S/N of every epoch of one curve: lc (64 bits), tu (float32).  Times and region
    bounds are the search's float32 ones, every sum is in 64 bits."""
    nsc, wmax, dw, deltat = grid
    n, dev = tu.numel(), tu.device
    ts = ((tu + 1000.0) - 1000.0)
    ok = ts >= 0
    last = torch.where(ok, torch.arange(n, device=dev), -1).cummax(0)[0]
    filled = torch.where(last >= 0, ts[last.clamp(min=0)].double(), -math.inf)
    flux = torch.where(ok, lc, 0.0)
    f32 = np.float32
    out = torch.zeros(n, dtype=torch.float64, device=dev)
    for e0 in range(0, n, 16384):
        e = torch.arange(e0, min(n, e0 + 16384), device=dev)
        idx = e[:, None] - nsc // 2 + torch.arange(nsc, device=dev)[None, :]
        inside = (idx >= 0) & (idx < n)
        idx = idx.clamp(0, n - 1)
        tt = (filled[idx] - float(f32(deltat)) * e[:, None].double()).float()
        v = ok[idx] & inside
        x = torch.where(v, flux[idx], 0.0)
        first = (~inside & (torch.arange(nsc, device=dev)[None, :] < nsc // 2)).sum(1)   # slots before the series
        vd, td = v.double(), tt.double()
        best = torch.zeros(e.numel(), dtype=torch.float64, device=dev)
        for w in range(NW):
            W = f32(float(f32(wmax)) - float(f32(dw)) * w)
            dl = f32(float(W) / 4.0 / NL) if mode else f32(float(W) * 0.45 / NL)
            hw, qw = float(f32(0.5) * W), float(f32(0.25) * W)
            full = v & (tt > -hw) & (tt <= hw)
            N = full.sum(1).double()
            good = N.float() / (torch.tensor(W, device=dev) / torch.tensor(f32(deltat), device=dev)) > 0.75
            closed = v & (tt >= -hw) & (tt <= hw)
            m = torch.where(closed, x, 0.0).sum(1) / closed.sum(1)
            xc = x - m[:, None]
            SS = torch.where(full, xc * xc, 0.0).sum(1)
            # slot s of region A against the flux of scoop slot s - nS, as the search sums it
            ubS = first + (inside & (tt <= -hw)).sum(1)
            at = ubS[:, None] + torch.arange(nsc, device=dev)[None, :]
            va = torch.gather(v, 1, at.clamp(max=nsc - 1)) & (at < nsc)
            QA = torch.where(va, x, 0.0).cumsum(1)
            pos = inside & (tt > -hw)
            for i in range(NL):
                L = f32(f32(i + 1 if mode else i) * dl)
                if L == 0:
                    continue
                tab, tbc = float(f32(-qw) - f32(0.5) * L), float(f32(-qw) + f32(0.5) * L)
                A = v & (tt > -hw) & (tt <= tab)
                B = v & (tt > tab) & (tt <= tbc)
                C = v & (tt > tbc) & (tt <= -tbc)
                D = v & (tt > -tbc) & (tt <= -tab)
                E = v & (tt > -tab) & (tt <= hw)
                nA, nB, nC, nD = (z.sum(1).double() for z in (A, B, C, D))
                nE = E.sum(1).double()
                sA, sC, sE = (torch.where(z, xc, 0.0).sum(1) for z in (A, C, E))
                u = torch.where(B, td + qw, 0.0)
                z = torch.where(D, td - qw, 0.0)
                XU, XV = (xc * u).sum(1), (xc * z).sum(1)
                uu = (u * u).sum(1) + (z * z).sum(1)
                nAx = (pos & (tt <= tab)).sum(1)
                q = torch.where(nAx > 0, torch.gather(QA, 1, (nAx - 1).clamp(min=0)[:, None])[:, 0], 0.0)
                l = float(L)
                den = 4.0 * l * l * (nA + nE - nC) + 16.0 * uu
                H = -(8.0 * l * l * (q - m * nA + sC + sE) + 16.0 * l * (XV - XU)) / den
                hl = H / l
                chi2 = SS + H * (sA + sE - sC) + 0.25 * H * H * (nA + nC + nE) + 2.0 * hl * (XV - XU) + hl * hl * uu
                sn = (H.abs() if mode else H) / (chi2 / (N - 3)).sqrt()
                best = torch.maximum(best, torch.where(good & (chi2 > 0) & ~sn.isnan(), sn, 0.0))
        out[e] = best
    return out


def _fold64(t, x, case, fmin, df):
    """TSR of the folded trapezoid search of one curve's valid samples."""
    nf, nb, dmax = case["nf"], case["nb"], case["dmax"]
    a, b = torch.frac(t.double() * fmin), torch.frac(t.double() * df)
    N, mean = float(t.numel()), x.mean()
    out = torch.empty(nf, dtype=torch.float64, device=t.device)
    rows = max(1, min(512, (1 << 25) // max(t.numel(), nb + dmax)))
    f0 = (np.float64(np.float32(df)) * np.arange(nf) + np.float64(np.float32(fmin))).astype(np.float32)
    D = np.rint(FOLD_W[None, :] * f0[:, None] * np.float32(nb)).astype(np.int64)
    L = np.minimum(np.maximum(1, np.rint(np.float32(0.2) * D.astype(np.float32)).astype(np.int64)), D // 2)
    ok = (D >= 2) & (D <= dmax)
    arange = torch.arange(nb, device=t.device)
    for j0 in range(0, nf, rows):
        j = torch.arange(j0, min(nf, j0 + rows), device=t.device, dtype=torch.float64)[:, None]
        bins = (torch.frac(a + j * b) * nb).long().clamp_(max=nb - 1)
        m = j.numel()

        def ramps(v):   # prefix of the prefix, and the sums that the templates' squares need
            h = torch.zeros(m, nb, dtype=torch.float64, device=t.device).scatter_add_(1, bins, v.expand(m, -1))
            h = torch.cat([torch.zeros(m, 1, dtype=torch.float64, device=t.device), h, h[:, :dmax]], 1)
            at = torch.arange(nb + dmax + 1, device=t.device, dtype=torch.float64) - 0.5   # the bin's centre
            return h.cumsum(1), (h * at).cumsum(1), (h * at * at).cumsum(1)

        c0, c1, c2 = ramps(torch.ones_like(x))
        s0, s1, _ = ramps(x - mean)
        best = torch.zeros(m, dtype=torch.float64, device=t.device)
        for d in range(D.shape[1]):
            Dd, Ld, okd = (torch.from_numpy(v[j0:j0 + m, d]).to(t.device)[:, None] for v in (D, L, ok))
            Dd, Ld = torch.where(okd, Dd, 2), torch.where(okd, Ld, 1)
            e0 = arange[None, :].expand(m, -1)
            e1, e2, e3 = e0 + Ld, e0 + Dd - Ld, e0 + Dd
            g = lambda p, i, k: torch.gather(p, 1, k) - torch.gather(p, 1, i)   # noqa: E731
            i0, i3, Lf = e0.double(), e3.double(), Ld.double()
            flat = g(s0, e1, e2) + (g(s1, e0, e1) - i0 * g(s0, e0, e1) + i3 * g(s0, e2, e3) - g(s1, e2, e3)) / Lf
            cw = g(c0, e1, e2) + (g(c1, e0, e1) - i0 * g(c0, e0, e1) + i3 * g(c0, e2, e3) - g(c1, e2, e3)) / Lf
            up = g(c2, e0, e1) - 2 * i0 * g(c1, e0, e1) + i0 * i0 * g(c0, e0, e1)
            dn = g(c2, e2, e3) - 2 * i3 * g(c1, e2, e3) + i3 * i3 * g(c0, e2, e3)
            cww = g(c0, e1, e2) + (up + dn) / (Lf * Lf)
            den = N * cww - cw * cw
            p = torch.where(okd & (den > 1e-9 * N), flat * flat / den, 0.0)
            best = torch.maximum(best, p.amax(1))
        out[j0:j0 + m] = best.sqrt()
    return out


def _refine64(t, x, N, sr, p1, p2, g, K=32, S=8, M=8):
    """The refined best peak of one curve's valid samples: the fields of REFINED."""
    nb, kma, kmi, kkmi = g["nb"], g["kma"], max(g["kmi"], 1), max(g["kkmi"], 5)
    j = int(sr.argmax())
    a, b = int(p1[j]), int(p2[j])
    if not float(sr[j]) > 0:
        return [0.0] * len(REFINED)
    while M > 0 and b - a + 1 + 2 * M > nb:
        M -= 1
    Lc = b - a + 1 + 2 * M
    dev, LS = t.device, Lc * S
    td = t.double()
    tref = float(np.float32(np.float32(float(t.min()) + float(t.max())) * np.float32(0.5)))
    dfk = g["df"] / K
    k = torch.arange(-K, K + 1, device=dev, dtype=torch.float64)[:, None]
    start = (a - M) % nb
    step = torch.frac(td * dfk) - (tref * dfk) % 1.0
    ph = torch.frac(td * g["fmin"]) + torch.remainder(torch.frac(td * dfk) * (j * K), 1.0) + k * step - start / nb
    fb = (torch.remainder(ph, 1.0) * (nb * S)).long()
    fb = torch.where(fb < LS, fb, LS)
    z = lambda v: torch.zeros(2 * K + 1, LS + 1, dtype=torch.float64, device=dev).scatter_add_(   # noqa: E731
        1, fb, v.expand(2 * K + 1, -1))[:, :LS].cumsum(1)
    pad = torch.zeros(2 * K + 1, 1, dtype=torch.float64, device=dev)
    Ps, Pc = torch.cat([pad, z(x)], 1), torch.cat([pad, z(torch.ones_like(x))], 1)

    def best(u, v):
        """Best window [u, v) of each trial (fine bins, [trials, windows])."""
        good = (u >= 0) & (v <= LS) & (v - u > kmi * S) & (v - u <= kma * S)
        u, v = u.clamp(0, LS), v.clamp(0, LS)
        s, c = torch.gather(Ps, 1, v) - torch.gather(Ps, 1, u), torch.gather(Pc, 1, v) - torch.gather(Pc, 1, u)
        p = torch.where(good & (c > kkmi) & (N - c > 0), s * s / (c * (N - c)), -1.0)
        m, at = p.max(1)
        return m, torch.gather(u, 1, at[:, None]), torch.gather(v, 1, at[:, None])

    u = (torch.arange(Lc, device=dev)[:, None] * S).expand(Lc, min(kma, Lc)).reshape(1, -1)
    w = (torch.arange(1, min(kma, Lc) + 1, device=dev)[None, :] * S).expand(Lc, -1).reshape(1, -1)
    _, u1, v1 = best(u.expand(2 * K + 1, -1), (u + w).expand(2 * K + 1, -1))
    near = torch.arange(-S, S + 1, device=dev)
    m, u2, v2 = best(u1 + near.repeat_interleave(2 * S + 1)[None, :], v1 + near.repeat(2 * S + 1)[None, :])
    i = int(m.argmax())
    ua, vb, dk = int(u2[i]), int(v2[i]), i - K
    s, c = float(Ps[i, vb] - Ps[i, ua]), float(Pc[i, vb] - Pc[i, ua])
    f = g["fmin"] + (j * K + dk) * dfk
    phase = (start / nb + ua / (nb * S) + tref * dk * dfk) % 1.0
    dur = (vb - ua) / (nb * S)
    mid = phase + 0.5 * dur
    return [f, 1.0 / f, phase, dur, (round(tref * f - mid) + mid) / f,
            (float(x.sum()) - s) / (t.numel() - c) - s / c, math.sqrt(float(m[i]))]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ragged", "served"):
        return None   # minutes: every curve's whole search in 64 bits
    s = prepare(case, seed)
    if kind in ("curve_bls", "kepler_bls"):
        g = s["grid"]
        if case["n"] * g["nf"] * case.get("nq", 1) > 1e10:
            return None   # the folds alone take over 20 seconds in 64 bits
        res = _median64(s["lc"], case["r"])
        off = _offset64(res, s["tu"])
        sr = []
        for q in range(res.shape[1]):
            v = s["tu"][:, q] >= 0
            sr.append(_bls64(s["tu"][v, q], res[v, q] - off[q], float(v.sum()), g))
        sr = torch.stack(sr)
        pest, sde = _stat64(sr, g["df"], g["fmin"])
        return dict(sr=sr, p1=None, p2=None, pest=pest, sde=sde, b1=None, b2=None)
    if kind == "curve_tls":
        res = _median64(s["lc"], case["r"])
        sn = _tls64(res[:, 0], s["tu"][:, 0], _tls_grid(TESS))
        return dict(sn=sn[:, None], w=None, t0=None, l=None, h=None, peaks=None)
    if kind == "plain_bls":
        g = s["grid"]
        return dict(sr=torch.stack([_bls64(s["tu"], s["lc"][:, q].double(), float(case["n"]), g)
                                    for q in range(case["nq"])]), p1=None, p2=None)
    if kind == "bls_peaks":
        g = s["grid"]
        sr, p1, p2 = s["spectra"]
        got = []
        for q in range(case["nq"]):
            v = s["tu"][:, q] >= 0
            x = s["lc"][v, q].double() - float(s["off"][q])
            got.append(_refine64(s["tu"][v, q], x, float(v.sum()), sr[q], p1[q], p2[q], g))
        pest, sde = _stat64(sr.double(), g["df"], g["fmin"])
        out = {k: np.array([r[i] for r in got]) for i, k in enumerate(REFINED)}
        return dict(out, sr_grid=sr.max(1)[0].double(), pest=pest, sde=sde)
    if kind == "detrend":
        res = _median64(s["lc"], case["r"])
        return dict(residual=res, offset=_offset64(res, s["tu"]))
    if kind == "tess_tls":
        sn = [_tls64(s["lc"][:, q].double(), s["tu"][:, q], _tls_grid(TESS), case["mode"])
              for q in range(case["nq"])]
        return dict(sn=torch.stack(sn, 1), w=None, t0=None, l=None, h=None)
    if kind == "tls_peaks":
        sn = s["sn"].double()
        pos = sn > 0
        cnt = pos.sum(0)
        mean = torch.where(pos, sn, 0.0).sum(0) / cnt
        std = (torch.where(pos, (sn - mean) ** 2, 0.0).sum(0) / cnt).sqrt()
        top = sn.max(0)[0]
        order = sn.sort(0)[0]
        med = 0.5 * (order[(len(sn) - 1) // 2] + order[len(sn) // 2])
        return dict(maxsn=top, median=med, std=std, far=(top - med) / std)
    if kind == "fold":
        tsr = []
        for q in range(case["nq"]):
            v = s["tu"][:, q] >= 0
            tsr.append(_fold64(s["tu"][v, q], s["lc"][v, q].double(), case, s["fmin"], s["df"]))
        return dict(tsr=torch.stack(tsr), start=None, dur=None, depth=None)
    t, x, W, L, T = s["fit"]
    dev = "cuda"
    td, xd, T0 = (torch.from_numpy(v).to(dev) for v in (t, x, T))
    top = (-1.0,)
    for w in W:
        for l in L:
            for a in range(0, T0.numel(), 512):
                tn = td[None, :] - T0[a:a + 512, None]
                inside = (tn >= -w / 2) & (tn <= w / 2)
                cnt = inside.sum(1)
                m = torch.where(inside, xd, 0.0).sum(1) / cnt
                xc = xd[None, :] - m[:, None]
                A = (tn >= -w / 2) & (tn < -w / 4 - l / 2)
                B = (tn >= -w / 4 - l / 2) & (tn < -w / 4 + l / 2)
                C = (tn >= -w / 4 + l / 2) & (tn < w / 4 - l / 2)
                D = (tn >= w / 4 - l / 2) & (tn < w / 4 + l / 2)
                E = (tn >= w / 4 + l / 2) & (tn < w / 2)
                AE = A | E
                tu_, tv = tn + w / 4, tn - w / 4
                ramp = torch.where(B, tu_, 0.0) - torch.where(D, tv, 0.0)
                # the depth as the reference defines it (the flat bottom's count enters with a minus)
                flat = torch.where(AE | C, xc, 0.0).sum(1)
                den = 4 * l * l * (AE.sum(1) - C.sum(1)) + 16 * (ramp * ramp).sum(1)
                H = -(8 * l * l * flat - 16 * l * (ramp * xc).sum(1)) / den
                # its template: -1/2 outside, +1/2 in the middle, ramps between
                tmpl = torch.where(C, 0.5, 0.0) - torch.where(AE, 0.5, 0.0) + ramp / l
                used = AE | B | C | D
                res = torch.where(used, (xc - H[:, None] * tmpl) ** 2, 0.0).sum(1)
                sn = -H / (res / (used.sum(1) - 3)).sqrt()
                sn = torch.where(sn.isnan() | sn.isinf(), -math.inf, sn)
                i = int(sn.argmax())
                if float(sn[i]) > top[0]:
                    top = (float(sn[i]), float(H[i]), w, l, T[a + i], float(m[i]))
    _, H, w, l, t0, off = top
    tn = t - t0
    model = np.where((tn <= -w / 4 - l / 2) | (tn >= w / 4 + l / 2), -H / 2, 0.0)
    model = np.where((tn < w / 4 - l / 2) & (tn >= -w / 4 + l / 2), H / 2, model)
    model = np.where((tn > -w / 4 - l / 2) & (tn <= -w / 4 + l / 2), H / l * (tn + w / 4), model)
    model = np.where((tn < w / 4 + l / 2) & (tn >= w / 4 - l / 2), -H / l * (tn - w / 4), model)
    return dict(model=model + off, best=[H, w, l, t0, off])
