"""gfilter on the GPU: bit-exact against scipy.signal.medfilt (the oracle) and the
drop-in get_detrend / get_offset surface."""
import numpy as np
import pytest
import torch

import oracle
from gtrap_gb300 import api, driver, gfilter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,r", [(1000, 1, 16), (777, 33, 24), (64, 5, 40), (2048, 64, 0),
                                    (3000, 2, 128), (500, 70, 3)])
def test_gfilter_bit_exact(cuda, n, nq, r):
    rng = np.random.default_rng(n + nq + r)
    x = rng.normal(1.0, 1e-3, size=(n, nq)).astype(np.float32)
    x[n // 3: n // 3 + 20] = 1.002            # plateau (ties)
    x[:, 0] = np.round(x[:, 0] * 1000) / 1000  # heavy duplicates
    got = api.gfilter(torch.from_numpy(x).to(cuda), r).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.medfilt_residual(x, r))


def test_gfilter_constant_and_zero_padding(cuda):
    x = np.full((100, 3), 2.5, np.float32)
    got = api.gfilter(torch.from_numpy(x).to(cuda), 10).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.medfilt_residual(x, 10))
    # first and last rows see the zero padding exactly as medfilt does
    assert got[50, 0] == 0.0


def test_gfilter_large_window_vs_n(cuda):
    rng = np.random.default_rng(1)
    x = rng.normal(size=(30, 4)).astype(np.float32)
    got = api.gfilter(torch.from_numpy(x).to(cuda), 40).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.medfilt_residual(x, 40))


def test_get_detrend_dropin(cuda):
    rng = np.random.default_rng(2)
    lc = rng.normal(1.0, 1e-3, size=(4000, 4)).astype(np.float32)
    out = gfilter.get_detrend(np.array(lc.T.tolist()).T, nby=1000, nbx=1, r=16, isw=0, osw=0)
    np.testing.assert_array_equal(out, oracle.medfilt_residual(lc, 16))
    dev = gfilter.get_detrend(lc, nby=1000, nbx=1, r=16, osw=1)
    host = np.zeros(lc.size, np.float32)
    driver.memcpy_dtoh(host, dev)
    np.testing.assert_array_equal(host.reshape(lc.shape), out)


def test_get_offset_dropin(cuda):
    rng = np.random.default_rng(3)
    n, nq = 5000, 7
    resid = rng.normal(0, 1e-3, size=(n, nq)).astype(np.float32)
    tu = np.tile(np.arange(n, dtype=np.float32)[:, None], (1, nq))
    tu[100:900, 2] = -1000.0
    dev = driver.mem_alloc(resid.nbytes)
    driver.memcpy_htod(dev, resid)
    off, img = gfilter.get_offset(n, nq, dev, tu)
    np.testing.assert_allclose(off, oracle.offset(resid, tu), rtol=1e-5, atol=1e-10)
    ref_img = resid.copy()
    ref_img[tu < 0] = 0.0
    np.testing.assert_array_equal(img, ref_img)


@pytest.mark.parametrize("lens,r", [((10000,), 24), ((50000,), 24), ((300, 7000, 1, 65), 24), ((2000,) * 40, 12)])
def test_gfilter_packed_bit_exact(cuda, lens, r):
    """The packed detrend (one flat array, curve q = [off[q], off[q] + n[q])) from a lone curve
    (short runs spread over many lanes) to a batch (long runs) equals medfilt per curve."""
    from gtrap_gb300 import _native as N
    from gtrap_gb300._dev import as_ptr
    rng = np.random.default_rng(sum(lens) + r)
    xs = [rng.normal(1.0, 1e-3, size=n).astype(np.float32) for n in lens]
    flat = torch.from_numpy(np.concatenate(xs)).to(cuda)
    out = torch.empty_like(flat)
    off = torch.tensor(np.concatenate([[0], np.cumsum(lens)[:-1]]), dtype=torch.int64, device=cuda)
    n = torch.tensor(lens, dtype=torch.int32, device=cuda)
    N.call("gtrap_gfilter_packed", as_ptr(flat), as_ptr(out), as_ptr(off), as_ptr(n), len(lens), max(lens), r,
           torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    o = 0
    for x in xs:
        np.testing.assert_array_equal(got[o:o + x.size], oracle.medfilt_residual(x[:, None], r)[:, 0])
        o += x.size


def _packed(cuda, xs, r):
    from gtrap_gb300 import _native as N
    from gtrap_gb300._dev import as_ptr
    lens = [x.size for x in xs]
    flat = torch.from_numpy(np.concatenate(xs)).to(cuda)
    out = torch.empty_like(flat)
    off = torch.tensor(np.concatenate([[0], np.cumsum(lens)[:-1]]), dtype=torch.int64, device=cuda)
    n = torch.tensor(lens, dtype=torch.int32, device=cuda)
    N.call("gtrap_gfilter_packed", as_ptr(flat), as_ptr(out), as_ptr(off), as_ptr(n), len(lens), max(lens), r,
           torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    return np.split(got, np.cumsum(lens)[:-1])


@pytest.mark.parametrize("kind", ["duplicates", "signed_zeros", "nan"])
def test_gfilter_ties_zeros_and_nan(cuda, kind):
    """Windows full of equal values, of +0 and -0, and with NaN, in the packed detrend (lone
    curves: short runs) and the image detrend.  Windows that never held a NaN take binary
    searches and block moves, the others the element-by-element loops.  Equal values: both
    equal medfilt bit for bit.  Signed zeros: equal medfilt in value (which zero a window
    holds depends on where its run started, as it always has).  NaN: every row whose window
    and run have not yet met the first NaN equals medfilt."""
    rng = np.random.default_rng({"duplicates": 1, "signed_zeros": 2, "nan": 3}[kind])
    lens = (7000, 300, 41, 2500)
    xs = []
    for m in lens:
        x = rng.integers(-3, 4, size=m).astype(np.float32)
        if kind == "signed_zeros":
            x[rng.random(m) < 0.4] = np.float32(-0.0)
        if kind == "nan":
            x = rng.normal(size=m).astype(np.float32)
            x[int(m * 0.6):][rng.random(m - int(m * 0.6)) < 0.01] = np.nan
        xs.append(x)
    r = 24
    got = _packed(cuda, xs, r)
    for x, g in zip(xs, got):
        img = api.gfilter(torch.from_numpy(x).to(cuda).view(-1, 1), r).cpu().numpy()[:, 0]
        ref = oracle.medfilt_residual(np.nan_to_num(x)[:, None], r)[:, 0]
        if kind == "duplicates":
            np.testing.assert_array_equal(g, ref)
            np.testing.assert_array_equal(img, ref)
        elif kind == "signed_zeros":
            assert np.array_equal(g, ref) and np.array_equal(img, ref)   # -0 == +0
        else:
            nan_at = np.flatnonzero(np.isnan(x))
            clean = (nan_at[0] if nan_at.size else x.size) - r
            if clean > 0:
                np.testing.assert_array_equal(g[:clean], ref[:clean])
                np.testing.assert_array_equal(img[:clean], ref[:clean])


@pytest.mark.parametrize("r", [3, 4, 7, 8, 15, 16, 23, 31, 32, 47, 48, 63, 64])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 130, 2065])
def test_gfilter_groups_at_their_edges(cuda, n, r):
    """Every group size and core of the grouped medians, at the ends of its range of radii and
    just past it, on series shorter and longer than a window, a group and a block, with ties and
    infinities: image (one, three and 40 curves) and packed, bit-exact against medfilt."""
    rng = np.random.default_rng(64 * n + r)
    x = rng.normal(1.0, 1e-3, size=(n, 40)).astype(np.float32)
    x[:, 1] = rng.integers(0, 3, n)
    x[rng.random((n, 40)) < 0.002] = np.inf
    want = oracle.medfilt_residual(x, r)
    for cols in (slice(0, 1), slice(0, 3), slice(0, 40)):
        got = api.gfilter(torch.from_numpy(np.ascontiguousarray(x[:, cols])).to(cuda), r).cpu().numpy()
        np.testing.assert_array_equal(got, want[:, cols])
    for q, got in enumerate(_packed(cuda, [x[:, q].copy() for q in range(5)] + [x[:n // 2 + 1, 5].copy()], r)[:5]):
        np.testing.assert_array_equal(got, want[:, q])


@pytest.mark.parametrize("n,r", [(1, 64), (17, 71), (130, 72), (700, 65), (700, 128), (2065, 100), (2065, 128),
                                 (5000, 300), (1500, 888), (1500, 900)])
def test_gfilter_merged_cores(cuda, n, r):
    """Radii past the grouped medians (cores that move by merging, and at the largest the
    sliding windows), with cores of every remainder of 16, runs of one and of several groups, series
    shorter and longer than a window, ties, equal series and infinities: image (one, three and 40
    curves) and packed, equal to medfilt."""
    rng = np.random.default_rng(64 * n + r)
    x = rng.normal(1.0, 1e-3, size=(n, 40)).astype(np.float32)
    x[:, 1] = rng.integers(-1, 2, n)
    x[:, 2] = 0.5
    x[:, 3] = np.sin(np.arange(n) / 50.0)
    x[rng.random((n, 40)) < 0.002] = np.inf
    x[rng.random((n, 40)) < 0.002] = -np.inf
    want = oracle.medfilt_residual(x, r)
    for cols in (slice(0, 1), slice(0, 3), slice(0, 40)):
        got = api.gfilter(torch.from_numpy(np.ascontiguousarray(x[:, cols])).to(cuda), r).cpu().numpy()
        np.testing.assert_array_equal(got, want[:, cols])
    for q, got in enumerate(_packed(cuda, [x[:, q].copy() for q in range(5)] + [x[:n // 2 + 1, 5].copy()], r)[:5]):
        np.testing.assert_array_equal(got, want[:, q])


def test_gfilter_merged_cores_long_runs(cuda):
    """Runs of many groups (both directions of the pass) and a last run cut short."""
    rng = np.random.default_rng(9)
    x = rng.normal(1.0, 1e-3, size=(6001, 1500)).astype(np.float32)
    got = api.gfilter(torch.from_numpy(x).to(cuda), 200).cpu().numpy()
    cols = [0, 31, 32, 777, 1499]
    np.testing.assert_array_equal(got[:, cols], oracle.medfilt_residual(np.ascontiguousarray(x[:, cols]), 200))


def _median_by_keys(x, r):
    """x minus the median of its zero-padded windows in the order -NaN, -inf, ..., -0, +0, ..., inf, NaN."""
    b = x.view(np.int32)
    key = np.clip(b ^ ((b >> 31) & 0x7fffffff), -2 ** 31 + 1, 2 ** 31 - 2).astype(np.int32)
    win = np.lib.stride_tricks.sliding_window_view(np.pad(key, ((r, r), (0, 0))), 2 * r + 1, axis=0)
    med = np.partition(win, r, axis=-1)[..., r]
    with np.errstate(invalid="ignore"):
        return x - (med ^ ((med >> 31) & 0x7fffffff)).astype(np.int32).view(np.float32)


@pytest.mark.parametrize("r", [4, 7, 8, 15, 16, 24, 31, 32, 47, 48, 63, 64, 65, 128])
@pytest.mark.parametrize("frac", [0.001, 0.05, 0.6])
def test_gfilter_windows_with_nan(cuda, r, frac):
    """NaN of either sign, scattered and as a gap, beside infinities: a window's median is that of the order with
    NaN past the infinity of its sign, whatever came before the window: image (one, three and 40 curves) and
    packed."""
    n = 1300
    rng = np.random.default_rng(int(1000 * frac) + r)
    x = rng.normal(1.0, 1e-3, size=(n, 40)).astype(np.float32)
    x[rng.random(x.shape) < frac] = np.nan
    x.view(np.uint32)[rng.random(x.shape) < frac / 4] = 0xffc00000
    x[rng.random(x.shape) < 0.002] = np.inf
    x[rng.random(x.shape) < 0.002] = -np.inf
    x[500:700, 1] = np.nan
    x[:, 2] = rng.normal(size=n)          # a curve without
    want = _median_by_keys(x, r)
    for cols in (slice(0, 1), slice(0, 3), slice(0, 40)):
        got = api.gfilter(torch.from_numpy(np.ascontiguousarray(x[:, cols])).to(cuda), r).cpu().numpy()
        np.testing.assert_array_equal(got, want[:, cols])
    for q, got in enumerate(_packed(cuda, [x[:, q].copy() for q in range(5)], r)):
        np.testing.assert_array_equal(got, want[:, q])
