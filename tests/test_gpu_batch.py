"""Packed (ragged) batches: one persistent BLS launch and one GTLS launch over device work
queues, against the plain per-curve entry points (bit-identical) and the FP64 oracle.

Tolerances as for the plain kernels: SR relative error <= 1e-4 and best bins identical up to
FP64 near-ties (1e-5 of the maximum power); GTLS S/N within 1e-4 (relative, absolute below 1).
"""
import numpy as np
import pytest
import torch

import oracle
from gtrap_gb300 import batch as B, synth
from gtrap_gb300 import api

pytestmark = pytest.mark.gpu

R = 8  # detrend window 17
BLS = B.BlsSpec(nb=256, kma=27, kmi=1)
TLS = B.TlsSpec(nw=4, nl=8)


def _mix(count=10, seed=4100):
    mix = synth.ragged_mix(count, seed=seed, n_range=(400, 4000))
    bat = B.RaggedBatch(BLS, TLS, detrend_r=R)
    for k, c in enumerate(mix):
        if c["kind"] == "bls":
            nf = min(c["nf"], 120 + 37 * k)  # uneven grids, small enough for the oracle
            bat.add_bls(c["t"], c["x"], nf, c["fmin"], c["df"], kkmi=c["kkmi"])
        else:
            bat.add_tls(c["t"], c["x"], c["nsc"], c["wmax"], c["dw"], c["deltat"])
    return mix, bat


def _results(bat):
    bls = [bat.bls_result(k) for k in range(bat.n_bls)]
    tls = [bat.tls_result(k) for k in range(bat.n_tls)]
    return bls, tls


def _same(a, b):
    for x, y in zip(a[0], b[0]):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)
    for x, y in zip(a[1], b[1]):
        for u, v in zip(x, y):
            np.testing.assert_array_equal(u, v)


@pytest.fixture(scope="module")
def ragged(cuda):
    mix, bat = _mix()
    assert bat.n_bls >= 2 and bat.n_tls >= 2
    bat.build()
    bat.launch()
    torch.cuda.synchronize()
    return mix, bat, _results(bat)


def test_ragged_equals_plain_per_curve(ragged):
    mix, bat, got = ragged
    B.run_plain(bat)
    torch.cuda.synchronize()
    _same(got, _results(bat))


def test_ragged_bls_against_oracle(ragged):
    mix, bat, got = ragged
    dev_table = np.frombuffer(bat.bls_curves.cpu().numpy().tobytes(), B.BLS_CURVE)
    k = 0
    for c in mix:
        if c["kind"] != "bls":
            continue
        row = bat.bls_table[k]
        x, t = c["x"].astype(np.float32), c["t"].astype(np.float32)
        resid = oracle.medfilt_residual(x[:, None], R)
        np.testing.assert_array_equal(bat.resid[int(row["off"]):int(row["off"]) + x.size].cpu().numpy(),
                                      resid[:, 0])
        off64 = oracle.offset(resid, t[:, None])
        off = np.array([dev_table[k]["offset"]], np.float32)  # get_offset on the device
        assert abs(off[0] - off64[0]) <= 1e-6 * max(1e-3, abs(off64[0])), (off[0], off64[0])
        assert dev_table[k]["nv"] == row["ntrue"]
        nf = int(row["nf"])
        osr, op1, op2, opmax = oracle.bls(resid, t[:, None], nf, BLS.nb, BLS.kma, BLS.kmi,
                                          int(row["kkmi"]), float(row["fmin"]), float(row["df"]),
                                          offset=off, ntrue=np.array([row["ntrue"]], np.uint32))
        sr, p1, p2 = got[0][k]
        fin = np.isfinite(osr[0])
        rel = np.abs(sr[fin] - osr[0][fin]) / np.maximum(osr[0][fin], 1e-30)
        assert rel.max() <= 1e-4, (k, rel.max())
        for j in np.flatnonzero(((p1 != op1[0]) | (p2 != op2[0])) & fin):
            pw = oracle.bls_window_power(resid, t[:, None], 0, j, int(p1[j]), int(p2[j]), BLS.nb,
                                         float(row["fmin"]), float(row["df"]), offset=off,
                                         ntrue=np.array([row["ntrue"]], np.uint32))
            assert abs(pw - opmax[0, j]) <= 1e-5 * opmax[0, j], (k, j)
        k += 1


def test_ragged_tls_against_oracle(ragged):
    mix, bat, got = ragged
    k = 0
    for c in mix:
        if c["kind"] != "tls":
            continue
        x, t = c["x"].astype(np.float32), c["t"].astype(np.float32)
        resid = oracle.medfilt_residual(x[:, None], R)
        n = x.size
        ref = oracle.gtls(resid, t[:, None], n, TLS.nw, TLS.nl, c["nsc"], c["wmax"], c["dw"], c["deltat"])
        sn = got[1][k][0]
        osn = ref[0][:, 0]
        err = np.abs(sn - osn) / np.maximum(np.abs(osn), 1.0)
        assert err.max() <= 1e-4, (k, err.max())
        np.testing.assert_array_equal(got[1][k][2], ref[2][:, 0])
        k += 1


def test_graph_replay_and_in_place_update(ragged, cuda):
    mix, bat, got = ragged
    g = bat.capture()
    g.replay()
    torch.cuda.synchronize()
    _same(got, _results(bat))
    # new flux of the same layout: the replay must follow the arrays' contents
    x0 = bat.x.clone()
    bat.x.mul_(1.25).add_(0.001)
    g.replay()
    torch.cuda.synchronize()
    replayed = _results(bat)
    bat.launch()
    torch.cuda.synchronize()
    _same(replayed, _results(bat))
    assert not np.array_equal(replayed[0][0][0], got[0][0][0])
    bat.x.copy_(x0)
    g.replay()
    torch.cuda.synchronize()
    _same(got, _results(bat))


def test_autotune_and_partial_segments_keep_results(ragged):
    mix, bat, got = ragged
    F, bb, tb = B.autotune(bat, F_candidates=(2, 5), bps_candidates=(1, 2), sample=3)
    assert F in (2, 5)
    bat.launch()
    torch.cuda.synchronize()
    _same(got, _results(bat))
    # a segment may start at any tile: only frequencies [F*tile0, F*(tile0+count)) are written
    bat.blsp.fill_(-1.0)
    segs = np.zeros(1, B.SEGMENT)
    segs["curve"], segs["tile0"] = 1, 1
    cum = np.array([0, 2], np.uint32)
    bat.launch_bls(queue=bat._upload_segments(segs, cum))
    sr = bat.bls_result(1)[0]
    nf = sr.size
    lo, hi = min(F, nf), min(3 * F, nf)
    np.testing.assert_array_equal(sr[lo:hi], got[0][1][0][lo:hi])
    assert (sr[:lo] == -1.0).all() and (sr[hi:] == -1.0).all()
    bat.launch()


def test_fp32_reference_phase_batch(cuda):
    mix, bat = _mix(count=6, seed=4200)
    bat.bls_spec = B.BlsSpec(nb=256, kma=27, kmi=1, phase="fp32")
    bat.build()
    bat.launch()
    torch.cuda.synchronize()
    got = _results(bat)
    B.run_plain(bat)
    torch.cuda.synchronize()
    _same(got, _results(bat))


def test_degenerate_curves_equal_plain(cuda):
    """Curves of one sample, one frequency, all samples masked and fewer samples than bins,
    mixed with ordinary ones, in every request kind: the batch equals the plain per-curve
    path."""
    rng = np.random.default_rng(4600)
    bat = B.RaggedBatch(BLS, TLS, detrend_r=R, fold=B.FoldSpec(nb=256, durations=(0.05, 0.1), dmax=128))
    ordinary_t = (np.arange(900) * 0.02).astype(np.float32)
    ordinary_x = (1.0 + rng.normal(0, 1e-3, 900)).astype(np.float32)
    masked_t = np.full(300, -1000.0, np.float32)
    for t, x, nf in ((ordinary_t[:1], ordinary_x[:1], 5), (ordinary_t, ordinary_x, 1), (masked_t, ordinary_x[:300], 7),
                     (ordinary_t[:40], ordinary_x[:40], 33), (ordinary_t, ordinary_x, 61)):
        bat.add_bls(t, x, nf, 0.05, 0.01, kkmi=1)
        bat.add_fold(t, x, nf, 0.05, 0.01)
        bat.add_tls(t, x, 40, 0.3, 0.05, 0.02)
    bat.build()
    bat.launch()
    torch.cuda.synchronize()
    got = ([bat.bls_result(k) for k in range(bat.n_bls)], [bat.fold_result(k) for k in range(bat.n_fold)],
           [bat.tls_result(k) for k in range(bat.n_tls)])
    B.run_plain(bat)
    torch.cuda.synchronize()
    want = ([bat.bls_result(k) for k in range(bat.n_bls)], [bat.fold_result(k) for k in range(bat.n_fold)],
            [bat.tls_result(k) for k in range(bat.n_tls)])
    for g_kind, w_kind in zip(got, want):
        for g, w in zip(g_kind, w_kind):
            for a, b in zip(g, w):
                np.testing.assert_array_equal(a, b)
    assert np.all(got[0][2][0] == 0) and np.all(got[1][2][0] == 0)  # all masked: no window


def test_tile_plan_keeps_two_blocks_per_sm(cuda):
    """At the benchmark's grid (nb 2048, kma 205) a tile holds six frequencies and two blocks
    share an SM: the tile budget counts the kernels' static shared memory and the per-block
    reservation (a few hundred more static bytes once cost the second block)."""
    from gtrap_gb300 import _native as N
    # the plan subtracts the kernels' queried static shared memory and the reservation from
    # half an SM: more static bytes would drop F to 5 here
    assert int(N.fn("gtrap_bls_tile_frequencies")(2048, 205)) == 6


@pytest.mark.parametrize("nb,nf,phase", [(1024, 1, "exact"), (1024, 5, "exact"), (1024, 131, "exact"), (1000, 64, "exact"),
                                         (2048, 45, "fp32"), (8192, 13, "exact"), (8192, 7, "fp32"), (64, 200, "exact")])
def test_spread_and_consecutive_tiles_give_the_same_bits(cuda, nb, nf, phase):
    """Few segments of whole curves take every tiles-th frequency a tile, many segments and parts of a curve
    consecutive ones; an image of long curves the former, of short ones in a big launch the latter.  Grids of one
    frequency, of less than a tile, of whole tiles and of a remainder; nothing but the curve's spectrum written."""
    rng = np.random.default_rng(nb + nf)
    n = 8200
    t = np.sort(rng.uniform(0, 160, n)).astype(np.float32)
    x = rng.normal(0, 1e-3, n).astype(np.float32)
    spec = B.BlsSpec(nb=nb, kma=max(2, nb // 10), kmi=1, phase=phase)

    def batch(count):
        bat = B.RaggedBatch(spec)
        for _ in range(count):
            bat.add_bls(t, x, nf, 0.05, 0.004, kkmi=10)
        bat.build()
        bat.launch()
        return bat

    few, many = batch(1), batch(20)
    ref = [v.copy() for v in few.bls_result(0)]
    assert ref[0].any()
    for k in (0, 7, 19):
        for a, b in zip(ref, many.bls_result(k)):
            np.testing.assert_array_equal(a, b)
    # the first tiles alone, and the curve in two segments
    F = few.F
    tiles = (nf + F - 1) // F
    for parts in ([(0, tiles - 1)], [(0, tiles // 2), (tiles // 2, tiles)]):
        few.blsp.fill_(-1.0)
        segs = np.zeros(len(parts), B.SEGMENT)
        segs["tile0"] = [a for a, _ in parts]
        cum = np.cumsum([0] + [b - a for a, b in parts]).astype(np.uint32)
        if cum[-1] == 0:
            continue
        few.launch_bls(queue=few._upload_segments(segs, cum))
        got, end = few.bls_result(0)[0], min(nf, F * parts[-1][1])
        np.testing.assert_array_equal(got[:end], ref[0][:end])
        assert (got[end:] == -1.0).all()
    # the image forms: one curve, and enough of them to fill the GPU several times
    img = [np.ascontiguousarray(v)[:, None] for v in (x, t)]
    d = lambda a, k: torch.from_numpy(a).to(cuda).expand(n, k).contiguous()
    off = float(np.frombuffer(few.bls_curves.cpu().numpy().tobytes(), B.BLS_CURVE)[0]["offset"])
    for k in (1, 40 if nb >= 1000 else 3):
        sr, p1, p2 = api.geebls(d(img[0], k), d(img[1], k), torch.full((k,), off, device=cuda),
                                torch.full((k,), n, dtype=torch.int32, device=cuda), nf, nb, spec.kma, 1, 10, 0.05,
                                0.004, phase=phase)
        for a, b in zip(ref, (sr, p1, p2)):
            for q in (0, k - 1):
                np.testing.assert_array_equal(a, b[q].cpu().numpy().view(a.dtype))
