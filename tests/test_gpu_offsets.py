"""get_offset in images and in packed batches: the same summation order, so a curve's offset
is bit-identical in an [n, nq] image (gtrap_offset) and in a packed batch
(gtrap_bls_offsets), and within FP32 rounding of the FP64 mean (gtrap/gfilter.py:94-101)."""
import numpy as np
import pytest
import torch

import oracle
from gtrap_gb300 import _native as N, api
from gtrap_gb300._dev import as_ptr
from gtrap_gb300.batch import BLS_CURVE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [(1,), (255, 256, 257), (70000,), (3000, 65536, 17, 40000), (2000,) * 37])
def test_packed_offsets_equal_image_offsets(cuda, lens):
    rng = np.random.default_rng(sum(lens))
    ts, xs = [], []
    for n in lens:
        t = np.arange(n, dtype=np.float32) * np.float32(0.0204)
        if n > 100:   # a masked gap and a few isolated masked samples
            g = int(rng.integers(0, n - 50))
            t[g:g + 40] = -1000.0
            t[rng.integers(0, n, 5)] = -1000.0
        x = (rng.normal(0.0, 1e-3, n) + rng.uniform(-5e-3, 5e-3)).astype(np.float32)
        ts.append(t)
        xs.append(x)
    off = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    tab = np.zeros(len(lens), BLS_CURVE)
    tab["off"] = off
    tab["n"] = lens
    tab_d = torch.from_numpy(tab.view(np.uint8)).to(cuda)
    t_d = torch.from_numpy(np.concatenate(ts)).to(cuda)
    x_d = torch.from_numpy(np.concatenate(xs)).to(cuda)
    N.call("gtrap_bls_offsets", as_ptr(tab_d), len(lens), as_ptr(t_d), as_ptr(x_d),
           torch.cuda.current_stream(cuda).cuda_stream)
    packed = tab_d.cpu().numpy().view(BLS_CURVE)["offset"]
    for q, n in enumerate(lens):
        img = api.offset(torch.from_numpy(xs[q]).to(cuda).view(n, 1),
                         torch.from_numpy(ts[q]).to(cuda).view(n, 1)).cpu().numpy()[0]
        assert packed[q].tobytes() == np.float32(img).tobytes(), (n, packed[q], img)
        ref = oracle.offset(xs[q][:, None], ts[q][:, None])[0]
        assert abs(img - ref) <= 2e-7 * max(abs(ref), 1e-6), (n, img, ref)


def test_image_offsets_many_curves(cuda):
    """32-curve blocks with ragged tails of rows: every curve of a wide image against FP64."""
    rng = np.random.default_rng(5)
    n, nq = 4097, 70
    resid = rng.normal(0.0, 1e-3, size=(n, nq)).astype(np.float32)
    tu = np.tile(np.arange(n, dtype=np.float32)[:, None], (1, nq))
    tu[rng.random((n, nq)) < 0.05] = -1000.0
    got = api.offset(torch.from_numpy(resid).to(cuda), torch.from_numpy(tu).to(cuda)).cpu().numpy()
    ref = oracle.offset(resid, tu)
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=1e-12)


def _offset_in_order(x, t):
    """One curve's offset in the documented order, float32 Neumaier partials step by step."""
    n = x.size
    pad = (-n) % 256
    v = np.concatenate([x, np.zeros(pad, np.float32)]).reshape(-1, 256)
    skip = np.concatenate([t < 0, np.ones(pad, bool)]).reshape(-1, 256)
    s, c = np.zeros(256, np.float32), np.zeros(256, np.float32)
    for row, no in zip(v, skip):
        a = np.where(no, 0, row).astype(np.float32)
        u = s + a
        e = np.where(np.abs(s) >= np.abs(a), (s - u) + a, (a - u) + s).astype(np.float32)
        s, c = np.where(no, s, u), np.where(no, c, c + e)
    part = (s.astype(np.float64) + c.astype(np.float64)).reshape(8, 32)
    sr = np.zeros(32)
    for u in range(8):
        sr = sr + part[u]
    acc = 0.0
    for r in range(32):
        acc += sr[r]
    return np.float32(acc / n)


@pytest.mark.parametrize("nq", [1, 3, 15, 16, 17, 33])
@pytest.mark.parametrize("n", [1, 256, 4096, 4097, 12289])
def test_image_offsets_keep_the_order(cuda, n, nq):
    """The clustered kernel at the edges of its blocks (lanes) and load batches (16 x 256 rows)."""
    rng = np.random.default_rng(n + nq)
    resid = rng.normal(1e-3, 1e-3, size=(n, nq)).astype(np.float32)
    tu = np.tile(np.arange(n, dtype=np.float32)[:, None], (1, nq))
    tu[rng.random((n, nq)) < 0.1] = -1000.0
    resid[(tu < 0) & (rng.random((n, nq)) < 0.2)] = np.nan   # masked samples are not looked at
    got = api.offset(torch.from_numpy(resid).to(cuda), torch.from_numpy(tu).to(cuda)).cpu().numpy()
    want = np.array([_offset_in_order(resid[:, q], tu[:, q]) for q in range(nq)], np.float32)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nq", [600, 700, 1003])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 4096, 4097])
def test_offsets_of_many_short_curves_keep_the_order(cuda, n, nq):
    """Many curves of up to 4096 samples take one block a group, longer or fewer ones a cluster: the same order."""
    rng = np.random.default_rng(n + nq)
    resid = rng.normal(1e-3, 1e-3, size=(n, nq)).astype(np.float32)
    tu = np.tile(np.arange(n, dtype=np.float32)[:, None], (1, nq))
    tu[rng.random((n, nq)) < 0.1] = -1000.0
    resid[(tu < 0) & (rng.random((n, nq)) < 0.2)] = np.nan
    got = api.offset(torch.from_numpy(resid).to(cuda), torch.from_numpy(tu).to(cuda)).cpu().numpy()
    for q in (0, 1, 15, 16, 31, 300, nq - 2, nq - 1):
        assert got[q] == _offset_in_order(resid[:, q], tu[:, q]), q
