"""detect_peaks on the device (gtrap_gb300.detect_peaks) against the reference's own
detect_peaks over option sets (mph, mpd, threshold, edge, kpsh, valley) and series with
distinct values, plateaus, NaNs and infinities: identical index arrays."""
from pathlib import Path

import numpy as np
import pytest

from gtrap_gb300 import detect_peaks as D

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).parent / "golden" / "detect_peaks_opts_golden.npz"
EDGE = {0: None, 1: "rising", 2: "falling", 3: "both"}


def test_matches_reference_over_options(cuda):
    g = np.load(GOLDEN)
    off, allind = g["ind_off"], g["ind_all"]
    for k in range(int(g["ncases"])):
        x = g["series_%d" % g["series_of_case"][k]]
        has_mph, mph, mpd, thr, edge, kpsh, valley = g["opts"][k]
        got = D.detect_peaks(x, mph=mph if has_mph else None, mpd=int(mpd), threshold=thr, edge=EDGE[int(edge)],
                             kpsh=bool(kpsh), valley=bool(valley))
        np.testing.assert_array_equal(got, allind[off[k]:off[k + 1]], err_msg=str(g["opts"][k]))


def test_device_tensor_input_and_other_edge(cuda):
    import torch
    x = np.sin(np.arange(300) * 0.2)
    ref = D.detect_peaks(x, mpd=5)
    np.testing.assert_array_equal(D.detect_peaks(torch.from_numpy(x).cuda(), mpd=5), ref)
    assert ref.size > 5 and D.detect_peaks(x, edge="sideways").size == 0


def _greedy(x, mpd, edge, kpsh):
    """Candidates by the edge rule, then in decreasing height (lower index first) each kept one
    deletes the others within +-mpd (the strictly lower ones with kpsh)."""
    d = np.diff(x)
    l, r = d[:-1], d[1:]
    c = np.zeros(x.size, bool)
    if edge is None:
        c[1:-1] = (r < 0) & (l > 0)
    if edge in ("rising", "both"):
        c[1:-1] |= (r <= 0) & (l > 0)
    if edge in ("falling", "both"):
        c[1:-1] |= (r < 0) & (l >= 0)
    ind = np.flatnonzero(c)
    if mpd <= 1:
        return ind
    alive = np.ones(ind.size, bool)
    for k in np.lexsort((ind, -x[ind])):
        if alive[k]:
            a, b = np.searchsorted(ind, [ind[k] - mpd, ind[k] + mpd + 1])
            near = np.ones(b - a, bool) if not kpsh else x[ind[a:b]] < x[ind[k]]
            near[k - a] = False
            alive[a:b] &= ~near
    return ind[alive]


@pytest.mark.parametrize("n", [63, 64, 65, 257, 8193, 40000])
@pytest.mark.parametrize("edge", [None, "rising", "falling", "both"])
def test_clusters_at_their_edges(cuda, n, edge):
    """One block and a cluster, series shorter than a run of a block and longer than a step of the
    compaction, windows at either side of the masks' reach (16 neighbours: 33 samples, 16 where
    neighbouring samples can both be peaks), plateaus, ramps that decide one peak a round."""
    rng = np.random.default_rng(n)
    noise = rng.normal(size=n)
    steps = np.round(rng.normal(size=n) * 2)
    ramp = np.tile([0.0, 1.0], n // 2 + 1)[:n] * np.arange(n)
    for x in (noise, steps, ramp):
        for mpd in (1, 2, 10, 16, 17, 33, 34, 700):
            if x is ramp and mpd > 34 and n > 10000:
                continue   # a round a peak: minutes of rounds for the plain statement's sake
            for kpsh in (False, True):
                got = D.detect_peaks(x, mpd=mpd, edge=edge, kpsh=kpsh)
                np.testing.assert_array_equal(got, _greedy(x, mpd, edge, kpsh), err_msg=str((n, edge, mpd, kpsh)))
