"""BLS (geebls / geebls_simple) on the GPU against the FP64 oracle.

Tolerances: SR relative error <= 1e-4 against FP64 (observed ~1e-6: exact integer bin
sums, float32 prefix sums and powers); best bins identical, or -- for near-ties only --
the oracle's FP64 power at the GPU's window within 1e-5 of the oracle's maximum.
"""
import numpy as np
import pytest
import torch

import oracle
from gtrap_gb300 import api, synth

pytestmark = pytest.mark.gpu

SR_RTOL = 1e-4


def _check_spectrum(sr, p1, p2, osr, op1, op2, opmax, lc, tu, wl_grid, offset=None, ntrue=None,
                    pow_tie=1e-5):
    # kma = nb lets a window hold every sample: kk = N, power s^2/0 = inf in both
    np.testing.assert_array_equal(np.isinf(sr), np.isinf(osr))
    fin = np.isfinite(osr)
    rel = np.abs(sr[fin] - osr[fin]) / np.maximum(osr[fin], 1e-30)
    assert rel.size == 0 or rel.max() <= SR_RTOL, "max SR rel err %g" % rel.max()
    if p1 is None:
        return
    # every differing best window must be a tie in FP64 (windows whose complement is also
    # admissible, kma > nb/2, tie with it up to rounding)
    bad = np.argwhere(((p1 != op1) | (p2 != op2)) & np.isfinite(osr))
    for q, j in bad[:400]:
        pw = oracle.bls_window_power(lc, tu, q, j, int(p1[q, j]), int(p2[q, j]), wl_grid["nb"],
                                     wl_grid["fmin"], wl_grid["df"], offset=offset, ntrue=ntrue)
        assert abs(pw - opmax[q, j]) <= pow_tie * opmax[q, j], (q, j, pw, opmax[q, j])


def test_simple_config1_subset(cuda):
    wl = synth.plain_bls(nq=8, n=4096, nf=512, nb=1024)
    lc, tu = torch.from_numpy(wl.lc).to(cuda), torch.from_numpy(wl.tu).to(cuda)
    sr, p1, p2 = api.geebls_simple(lc, tu, wl.nf, wl.nb, wl.kma, wl.kmi, wl.kkmi, wl.fmin, wl.df,
                                   with_phase=True)
    osr, op1, op2, opmax = oracle.bls(wl.lc, wl.tu, wl.nf, wl.nb, wl.kma, wl.kmi, wl.kkmi, wl.fmin, wl.df)
    grid = dict(nb=wl.nb, fmin=wl.fmin, df=wl.df)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax,
                    wl.lc, wl.tu, grid)


@pytest.mark.parametrize("nb,kma,kmi,kkmi", [(256, 30, 2, 5), (1000, 90, 5, 10), (64, 64, 1, 3), (64, 63, 1, 3),
                                             (4096, 200, 10, 50), (8192, 300, 8, 20)])
def test_simple_grid_shapes(cuda, nb, kma, kmi, kkmi):
    wl = synth.plain_bls(nq=3, n=3000, nf=37, nb=nb, seed=nb)
    lc, tu = torch.from_numpy(wl.lc).to(cuda), torch.from_numpy(wl.tu).to(cuda)
    sr, p1, p2 = api.geebls_simple(lc, tu, wl.nf, nb, kma, kmi, kkmi, wl.fmin, wl.df, with_phase=True)
    osr, op1, op2, opmax = oracle.bls(wl.lc, wl.tu, wl.nf, nb, kma, kmi, kkmi, wl.fmin, wl.df)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax,
                    wl.lc, wl.tu, dict(nb=nb, fmin=wl.fmin, df=wl.df))


def _masked_case(nq=6, n=6000, nf=200, nb=2048, seed=21):
    lc, tu, ntrue, g, inj = synth.kepler_like(nq=nq, n=n, nf=nf, nb=nb, seed=seed, transit_frac=0.5)
    resid = oracle.medfilt_residual(lc, 24)
    off = oracle.offset(resid, tu).astype(np.float32)
    return resid, tu, ntrue, off, g


def test_full_masked_offset_ntrue(cuda):
    resid, tu, ntrue, off, g = _masked_case()
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    sr, p1, p2 = api.geebls(d(resid), d(tu), d(off), d(ntrue.astype(np.int32)), g["nf"], g["nb"],
                            g["kma"], g["kmi"], g["kkmi"], g["fmin"], g["df"])
    osr, op1, op2, opmax = oracle.bls(resid, tu, g["nf"], g["nb"], g["kma"], g["kmi"], g["kkmi"],
                                      g["fmin"], g["df"], offset=off, ntrue=ntrue)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy().view(np.uint32), p2.cpu().numpy().view(np.uint32),
                    osr, op1, op2, opmax, resid, tu, g, offset=off, ntrue=ntrue)


def test_full_fp32_reference_phase_and_tail_drop(cuda):
    resid, tu, ntrue, off, g = _masked_case(nq=3, n=5000, nf=64, nb=1024, seed=5)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    for f0_fma in (True, False):
        sr, p1, p2 = api.geebls(d(resid), d(tu), d(off), d(ntrue.astype(np.int32)), g["nf"], g["nb"],
                                min(g["kma"], 512), g["kmi"], g["kkmi"], g["fmin"], g["df"],
                                phase="fp32", ref_nthread=512, f0_fma=f0_fma)
        osr, op1, op2, opmax = oracle.bls(resid, tu, g["nf"], g["nb"], min(g["kma"], 512), g["kmi"],
                                          g["kkmi"], g["fmin"], g["df"], offset=off, ntrue=ntrue,
                                          phase="fp32", n_eff=(5000 // 512) * 512, f0_fma=f0_fma)
        rel = np.abs(sr.cpu().numpy() - osr) / np.maximum(osr, 1e-30)
        assert rel.max() <= SR_RTOL


def test_edge_cases(cuda):
    rng = np.random.default_rng(0)
    n, nq = 300, 2
    tu = np.sort(rng.uniform(0, 50, n)).astype(np.float32)
    lc = rng.normal(size=(n, nq)).astype(np.float32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    # kmi >= kma: no admissible width -> SR = 0 everywhere
    sr, p1, p2 = api.geebls_simple(d(lc), d(tu), 10, 64, 5, 5, 5, 0.1, 0.01, with_phase=True)
    assert float(sr.abs().max()) == 0.0 and int(p1.abs().max()) == 0
    # everything masked -> zeros
    tuf = np.full((n, nq), -1000.0, np.float32)
    sr, p1, p2 = api.geebls(d(lc), d(tuf), d(np.zeros(nq, np.float32)), d(np.zeros(nq, np.int32)), 10,
                            64, 8, 1, 5, 0.1, 0.01)
    assert float(sr.abs().max()) == 0.0
    # nf = 1 and nq = 1
    sr1 = api.geebls_simple(d(lc[:, :1]), d(tu), 1, 128, 12, 1, 5, 0.37, 0.0)
    o = oracle.bls(lc[:, :1], tu, 1, 128, 12, 1, 5, 0.37, 0.0)[0]
    np.testing.assert_allclose(sr1.cpu().numpy(), o, rtol=SR_RTOL)


def test_deterministic_and_batch_invariant(cuda):
    """Integer bin sums make a curve's spectrum bit-identical run to run and alone vs batched."""
    resid, tu, ntrue, off, g = _masked_case(nq=5, n=4000, nf=150, nb=1024, seed=8)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    args = (g["nf"], g["nb"], g["kma"], g["kmi"], g["kkmi"], g["fmin"], g["df"])
    a = [t.cpu().numpy() for t in api.geebls(d(resid), d(tu), d(off), d(ntrue.astype(np.int32)), *args)]
    b = [t.cpu().numpy() for t in api.geebls(d(resid), d(tu), d(off), d(ntrue.astype(np.int32)), *args)]
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
    q = 3
    solo = [t.cpu().numpy() for t in api.geebls(d(resid[:, q:q + 1]), d(tu[:, q:q + 1]), d(off[q:q + 1]),
                                                 d(ntrue[q:q + 1].astype(np.int32)), *args)]
    for x, y in zip(a, solo):
        np.testing.assert_array_equal(x[q], y[0])


def test_injected_transit_recovered(cuda):
    wl = synth.plain_bls(nq=16, n=4096, nf=4096, nb=1024, n_transit=16, seed=77)
    lc, tu = torch.from_numpy(wl.lc).to(cuda), torch.from_numpy(wl.tu).to(cuda)
    sr, p1, p2 = api.geebls_simple(lc, tu, wl.nf, wl.nb, wl.kma, wl.kmi, wl.kkmi, wl.fmin, wl.df,
                                   with_phase=True)
    pest, sde, _, _ = api.blsstat(sr, p1, p2, wl.df, wl.fmin)
    pest, sde = pest.cpu().numpy(), sde.cpu().numpy()
    per, depth = wl.injected[:, 1], wl.injected[:, 3]
    strong = depth > 1.5e-3
    ok = 0
    for q in np.nonzero(strong)[0]:
        ratio = pest[q] / per[q]
        ok += any(abs(ratio - m) < 0.01 * m for m in (1.0, 0.5, 2.0, 1 / 3, 3.0))
    assert ok >= 0.8 * strong.sum()


def test_concentrated_bins_use_exact_fallback(cuda):
    """A frequency so low that each bin receives ~1000 samples exceeds the 32-bit fold
    format's per-bin limit; the kernel must detect it and re-fold in 64 bits."""
    rng = np.random.default_rng(12)
    n, nq, nb = 8192, 2, 512
    tu = (0.02 * np.arange(n)).astype(np.float32)
    lc = rng.normal(size=(n, nq)).astype(np.float32)
    lc -= lc.mean(axis=0)
    fmin, df, nf = np.float32(1e-4), np.float32(2e-3), 40   # the first frequencies cover < 1 cycle
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    sr, p1, p2 = api.geebls_simple(d(lc), d(tu), nf, nb, 52, 2, 5, fmin, df, with_phase=True)
    osr, op1, op2, opmax = oracle.bls(lc, tu, nf, nb, 52, 2, 5, fmin, df)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax,
                    lc, tu, dict(nb=nb, fmin=fmin, df=df))


@pytest.mark.parametrize("nb,kma,kmi", [(20, 10, 1), (31, 15, 1), (33, 7, 3), (96, 48, 30), (512, 33, 31), (1000, 499, 1),
                                        (2048, 205, 204), (2048, 64, 1)])
@pytest.mark.parametrize("n", [1500, 3001])
def test_scan_chunks_at_their_edges(cuda, n, nb, kma, kmi):
    """Units of 32 starts by 32 ends: bin counts under, at and off a multiple of 32, windows of one
    width, of every width and across several chunks, sparse and full bins, a strong transit (few
    units survive) and none (many do)."""
    wl = synth.plain_bls(nq=4, n=n, nf=25, nb=nb, seed=nb + n, n_transit=2)
    lc, tu = torch.from_numpy(wl.lc).to(cuda), torch.from_numpy(wl.tu).to(cuda)
    sr, p1, p2 = api.geebls_simple(lc, tu, wl.nf, nb, kma, kmi, 1, wl.fmin, wl.df, with_phase=True)
    osr, op1, op2, opmax = oracle.bls(wl.lc, wl.tu, wl.nf, nb, kma, kmi, 1, wl.fmin, wl.df)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax,
                    wl.lc, wl.tu, dict(nb=nb, fmin=wl.fmin, df=wl.df))


@pytest.mark.parametrize("nf,nb", [(3, 2048), (1000, 2048), (3644, 2048), (3654, 2048), (4100, 1024), (700, 1000)])
def test_lone_curve_takes_smaller_blocks(cuda, nf, nb):
    """A launch of few blocks takes fewer frequencies a block: the same bits as the curve gets in a
    batch that fills the GPU, at both ends of the rule."""
    rng = np.random.default_rng(nf + nb)
    n, nq = 1500, 40
    tu = torch.from_numpy(np.sort(rng.uniform(0, 60, (n, 1)), axis=0).astype(np.float32)).to(cuda)
    lc = torch.from_numpy(rng.normal(0, 1e-3, (n, 1)).astype(np.float32)).to(cuda)
    kw = dict(nf=nf, nb=nb, kma=nb // 10, kmi=nb // 200, kkmi=8, fmin=0.05, df=2.0 / nf)

    def run(k):
        return api.geebls(lc.expand(n, k).contiguous(), tu.expand(n, k).contiguous(), torch.zeros(k, device=cuda),
                          torch.full((k,), n, dtype=torch.int32, device=cuda), **kw)
    for one, many in zip(run(1), run(nq)):
        assert torch.equal(one[0].view(torch.int32), many[0].view(torch.int32))
        assert torch.equal(one[0].view(torch.int32), many[-1].view(torch.int32))


@pytest.mark.parametrize("nb,kma", [(256, 27), (1024, 103)])
def test_kmi_past_the_range_of_widths(cuda, nb, kma):
    """kmi from kma on leaves no window; negative numbers, which the binding wraps to 2^31 and more, all pass every
    width from one bin on (the kernels index from kmi: none of these may reach them)."""
    n, nf = 1500, 40
    rng = np.random.default_rng(nb)
    t = np.tile((np.arange(n) * np.float32(0.0204)).astype(np.float32)[:, None], (1, 2))
    lc = rng.normal(0, 1e-3, (n, 2)).astype(np.float32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    T, X, off, nt = d(t), d(lc), torch.zeros(2, device=cuda), torch.full((2,), n, dtype=torch.int32, device=cuda)
    run = lambda kmi: [v.cpu().numpy() for v in api.geebls(X, T, off, nt, nf, nb, kma, kmi, 5, 0.05, 0.02)]
    for kmi in (kma, kma + 1, 2 ** 31 - 1):
        assert not run(kmi)[0].any()
    one, low = run(1), run(-1)
    assert np.all(low[0] >= one[0])
    for kmi in (-2, -40, -100000, -2 ** 31):
        for a, b in zip(run(kmi), low):
            np.testing.assert_array_equal(a, b)
    sr, p1, p2 = (d(v) for v in one)
    for kmi in (kma, 2 ** 31 - 1, -1, -100000, -2 ** 31):
        rec = api.refined_to_numpy(api.bls_refine(sr, p1, p2, X, T, off, nt, nb, kma, kmi, 5, 0.05, 0.02, K=8, S=4, M=4))
        assert not rec["sr"].any() and not rec["kk"].any()


@pytest.mark.parametrize("nb,kma", [(100, 10), (100, 40), (256, 25), (300, 101), (512, 51), (512, 160), (512, 161), (1024, 102),
                                    (1000, 33)])
@pytest.mark.parametrize("kind", ["trend", "transit", "steps"])
def test_units_with_many_windows_left(cuda, nb, kma, kind):
    """Slow trends, deep transits and a flux of few values leave most windows of many units: the starts are then
    bounded in blocks of eight up to the largest width that does so, all at once past it."""
    n, nq, nf = 1200, 3, 12
    rng = np.random.default_rng(nb + kma)
    t = np.tile(((np.arange(n) + 0.3) * np.float32(0.0204)).astype(np.float32)[:, None], (1, nq))
    x = rng.normal(0, 1e-3, (n, nq))
    if kind == "trend":
        x = 0.05 * x + np.sin(t / (2.0 + np.arange(nq)))
    if kind == "transit":
        x = x - 5e-2 * (np.mod(t + 0.1 * np.arange(nq), 3.3) < 0.25)
    if kind == "steps":
        x = np.round(x * 500) / 500
    x = x.astype(np.float32)
    off, ntrue = np.zeros(nq, np.float32), np.full(nq, n, np.uint32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    sr, p1, p2 = api.geebls(d(x), d(t), d(off), d(ntrue.astype(np.int32)), nf, nb, kma, 1, 5, 0.05, 0.05)
    osr, op1, op2, opmax = oracle.bls(x, t, nf, nb, kma, 1, 5, np.float32(0.05), np.float32(0.05), offset=off, ntrue=ntrue)
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax, x, t,
                    dict(nb=nb, fmin=0.05, df=0.05), off, ntrue)


@pytest.mark.parametrize("n,nb,kma", [(300, 96, 95), (300, 256, 120), (3000, 1024, 500), (2000, 100, 45)])
def test_windows_that_hold_every_sample(cuda, n, nb, kma):
    """Fewer cycles than a window is wide: a window holds every sample, and where the flux does not sum to zero its
    power is infinite, as in FP64; at the other frequencies the spectrum is finite."""
    rng = np.random.default_rng(nb)
    nq, nf = 2, 24
    t = np.tile((np.arange(n) * np.float32(0.02)).astype(np.float32)[:, None], (1, nq))
    x = (0.01 + rng.normal(0, 1e-3, (n, nq))).astype(np.float32)
    off, ntrue = np.zeros(nq, np.float32), np.full(nq, n, np.uint32)
    fmin = df = float(np.float32(0.06 / (n * 0.02)))     # 0.06, 0.12, ... 1.44 cycles
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    sr, p1, p2 = api.geebls(d(x), d(t), d(off), d(ntrue.astype(np.int32)), nf, nb, kma, 1, 5, fmin, df)
    osr, op1, op2, opmax = oracle.bls(x, t, nf, nb, kma, 1, 5, np.float32(fmin), np.float32(df), offset=off, ntrue=ntrue)
    assert np.isinf(osr).any() and np.isfinite(osr).any()
    _check_spectrum(sr.cpu().numpy(), p1.cpu().numpy(), p2.cpu().numpy(), osr, op1, op2, opmax, x, t,
                    dict(nb=nb, fmin=fmin, df=df), off, ntrue)
