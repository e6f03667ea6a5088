"""GTLS peak statistics on the device (gtrap_peakstat) against the oracle restatement of
detect_peaks and gtrap/gtls.py:245-273.  Peak index sets, heights, max/argmax, medians and
counts are exact (the oracle ranks equal heights by index as the kernel does); the FP64
standard deviations and the ratios built on them agree to 1e-9 relative."""
import numpy as np
import pytest
import torch

from oracle import peaks as P
from gtrap_gb300 import api, batch as B, synth

pytestmark = pytest.mark.gpu

STAT_KEYS = ("maxsn", "argmax", "lent", "npeaks", "median")
FLOAT_KEYS = ("std", "far", "pssn", "diff", "medc", "stdc")


def _series(k, n=None):
    rng = np.random.default_rng(9000 + k)
    n = int(rng.integers(3, 5000)) if n is None else n
    kind = k % 3
    if kind == 0:
        x = np.abs(rng.normal(0, 1, n)).astype(np.float32)
        x[rng.uniform(size=n) < 0.3] = 0.0
    elif kind == 1:
        x = (np.sin(np.arange(n) / rng.uniform(2, 40)) + 0.2 * rng.normal(size=n)).astype(np.float32)
    else:
        x = np.round(rng.normal(0, 2, n)).astype(np.float32)  # many equal heights
    return x


def _check(rec, idx, val, x, mpd, ntop, k):
    ref = P.peakstat(x, mpd, ntop)
    for key in STAT_KEYS:
        assert rec[key] == pytest.approx(ref[key], abs=0, rel=0), key
    for key in FLOAT_KEYS:
        a, b = float(rec[key]), float(ref[key])
        if np.isfinite(b):
            assert a == pytest.approx(b, rel=1e-9, abs=1e-12), (key, a, b)
        else:
            assert (np.isnan(a) and np.isnan(b)) or a == b, (key, a, b)
    m = min(k, ref["npeaks"])
    np.testing.assert_array_equal(idx[:m], ref["peaks"][:m])
    np.testing.assert_array_equal(val[:m], x[ref["peaks"][:m]])
    assert np.all(idx[m:] == -1)


@pytest.mark.parametrize("mpd,ntop,k", [(10, 4, 8), (1, 4, 4), (3, 0, 16), (25, 2, 3)])
def test_peakstat_packed_series(cuda, mpd, ntop, k):
    xs = [_series(j) for j in range(12)] + [_series(20, 3), _series(21, 4), _series(22, 70000)]
    lens = np.array([x.size for x in xs])
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
    flat = torch.from_numpy(np.concatenate(xs)).to(cuda)
    st, idx, val = api.peakstat(flat, torch.from_numpy(offs.astype(np.int64)).to(cuda),
                                torch.from_numpy(lens.astype(np.int32)).to(cuda), 1, int(lens.max()),
                                mpd, ntop, k)
    st = api.stats_to_numpy(st)
    idx, val = idx.cpu().numpy(), val.cpu().numpy()
    for q, x in enumerate(xs):
        _check(st[q], idx[q], val[q], x, mpd, ntop, k)


def test_peakstat_of_gtls_image(cuda):
    lc, tu, inj = synth.tess_like(nq=6, n=3000, seed=3100, transit_frac=0.5)
    g = synth.tls_grid()
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    sn = api.gtls(d(lc), d(tu), 3000, g["nw"], g["nl"], g["nsc"], g["wmax"], g["dw"], g["deltat"])[0]
    st, idx, val = api.tls_peakstat(sn, mpd=10, ntop=4, k=8)
    st = api.stats_to_numpy(st)
    s = sn.cpu().numpy()
    for q in range(6):
        _check(st[q], idx.cpu().numpy()[q], val.cpu().numpy()[q], s[:, q], 10, 4, 8)


def test_peakstat_of_packed_batch(cuda):
    mix = synth.ragged_mix(8, seed=4300, n_range=(500, 3000), tls_frac=1.0)
    bat = B.RaggedBatch(B.BlsSpec(nb=256, kma=27, kmi=1), B.TlsSpec(nw=4, nl=8), detrend_r=8)
    for c in mix:
        bat.add_tls(c["t"], c["x"], c["nsc"], c["wmax"], c["dw"], c["deltat"])
    bat.build()
    bat.launch()
    st, idx, val = bat.tls_peakstat(mpd=10, ntop=4, k=6)
    st = api.stats_to_numpy(st)
    for q in range(bat.n_tls):
        _check(st[q], idx.cpu().numpy()[q], val.cpu().numpy()[q], bat.tls_result(q)[0], 10, 4, 6)


@pytest.mark.parametrize("mpd,ntop,k", [(10, 4, 8), (0, 2, 5), (1, 3, 4), (1000, 1, 2)])
def test_staged_and_long_series_agree(cuda, mpd, ntop, k):
    """Series that fit in shared memory run on one kernel, a launch with a longer one on another:
    the same series through both, with NaN, infinities, constants, ramps, every sample a peak and
    the shortest lengths.  Counts, indices, heights and order statistics equal; the FP64 sums
    differ by their order only."""
    rng = np.random.default_rng(11)
    xs = [_series(j) for j in range(3)]
    y = rng.normal(size=4097).astype(np.float32)
    y[[5, 100, 4096]] = np.nan
    y[200:203] = np.inf
    y[300] = -np.inf
    xs += [y, np.zeros(50, np.float32), np.arange(3000, dtype=np.float32), np.arange(3000, 0, -1).astype(np.float32),
           np.tile([0, 1], 1500).astype(np.float32), np.ones(1, np.float32), np.ones(2, np.float32),
           np.array([0, 2, 1], np.float32), rng.normal(size=30000).astype(np.float32), -np.ones(9, np.float32)]

    def run(series):
        lens = np.array([x.size for x in series])
        offs = np.concatenate([[0], np.cumsum(lens)[:-1]])
        st, idx, val = api.peakstat(torch.from_numpy(np.concatenate(series)).to(cuda),
                                    torch.from_numpy(offs.astype(np.int64)).to(cuda),
                                    torch.from_numpy(lens.astype(np.int32)).to(cuda), 1, int(lens.max()), mpd, ntop, k)
        return api.stats_to_numpy(st), idx.cpu().numpy(), val.cpu().numpy()

    a, ai, av = run(xs)
    b, bi, bv = run(xs + [np.zeros(60000, np.float32)])
    np.testing.assert_array_equal(ai, bi[:-1])
    np.testing.assert_array_equal(av, bv[:-1])
    for key in STAT_KEYS + ("medc",):
        np.testing.assert_array_equal(a[key], b[key][:-1], err_msg=key)
    for key in ("std", "far", "pssn", "diff", "stdc"):
        np.testing.assert_allclose(a[key], b[key][:-1], rtol=1e-11, atol=1e-13, err_msg=key)


@pytest.mark.parametrize("n", [3, 63, 64, 65, 66, 129, 4095, 8193, 35001])
def test_states_at_word_edges(cuda, n):
    """A lone series whose candidates just fill or just pass a word of states, odd and even lengths (the words
    lie behind the series), windows of masks (up to 16 samples) and of lists, long chains of decisions."""
    zigzag = np.zeros(n, np.float32)
    zigzag[1::2] = 1.0 + np.arange(n // 2, dtype=np.float32) / 64.0
    for x in (_series(60 + n, n), _series(61 + n, n), zigzag):
        for mpd in (1, 2, 16, 17, 40):
            st, idx, val = api.peakstat(torch.from_numpy(x).to(cuda), torch.zeros(1, dtype=torch.int64, device=cuda),
                                        torch.full((1,), n, dtype=torch.int32, device=cuda), 1, n, mpd, 3, 16)
            _check(api.stats_to_numpy(st)[0], idx.cpu().numpy()[0], val.cpu().numpy()[0], x, mpd, 3, 16)


@pytest.mark.parametrize("bits", [0x7fc00000, 0x7fffffff, 0x7f800001, 0xffc00000, 0xffffffff])
@pytest.mark.parametrize("n,count,shift", [(4097, 3, 0.5), (4096, 3, -0.5), (4097, 2500, -0.5), (4096, 2500, 0.5)])
def test_median_of_a_series_with_nan(cuda, bits, n, count, shift):
    """A NaN ranks as -0 (sign bit clear) or below all (set) in the median, by itself or beside a longer series,
    which takes another kernel."""
    rng = np.random.default_rng(n + count)
    x = (rng.normal(size=n) + shift).astype(np.float32)
    x.view(np.uint32)[rng.choice(n, count, replace=False)] = bits
    ranked = np.sort(np.where(np.isnan(x), np.float32(-np.inf if bits >> 31 else -0.0), x)).astype(np.float64)
    ref = 0.5 * (ranked[(n - 1) // 2] + ranked[n // 2])
    for xs in ([x], [x, np.zeros(60000, np.float32)]):
        lens = np.array([a.size for a in xs])
        st, _, _ = api.peakstat(torch.from_numpy(np.concatenate(xs)).to(cuda),
                                torch.from_numpy(np.cumsum(lens) - lens).to(cuda),
                                torch.from_numpy(lens.astype(np.int32)).to(cuda), 1, int(lens.max()), 10, 4, 8)
        got = api.stats_to_numpy(st)[0]["median"]
        assert np.isnan(got) if np.isinf(ref) else got == ref, (len(xs), got, ref)


@pytest.mark.parametrize("n,nq,mpd", [(512, 700, 17), (513, 700, 17), (200, 700, 100), (200, 600, 100), (40, 2000, 16), (40, 2000, 40)])
def test_many_short_series_with_wide_windows(cuda, n, nq, mpd):
    """At both ends of the rule that takes them to the kernel of the longest series."""
    xs = [_series(3000 + q % 9, n) for q in range(9)]
    img = np.stack([xs[q % 9] for q in range(nq)], axis=1)
    st, idx, val = api.tls_peakstat(torch.from_numpy(img).to(cuda), mpd=mpd, ntop=3, k=6)
    st, idx, val = api.stats_to_numpy(st), idx.cpu().numpy(), val.cpu().numpy()
    for q in list(range(9)) + [nq - 1]:
        _check(st[q], idx[q], val[q], img[:, q], mpd, 3, 6)
