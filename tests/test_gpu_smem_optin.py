"""Launches whose dynamic shared memory fits 48 KB and whose static does not fit beside it: the opt-in is theirs
too.  Each in a process of its own, as an earlier larger launch of the same kernel would have opted in for it."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PEAKS = """
import numpy as np, torch
from gtrap_gb300 import api
from oracle import peaks
x = np.abs(np.random.default_rng(1).normal(size=({n}, 2))).astype(np.float32)
st, idx, val = api.tls_peakstat(torch.from_numpy(x).cuda(), mpd=10, ntop=4, k=8)
ref = peaks.peakstat(x[:, 1], 10, 4)
assert api.stats_to_numpy(st)[1]["npeaks"] == ref["npeaks"]
assert (idx.cpu().numpy()[1] == ref["peaks"][:8]).all()
"""

GTLS = """
import numpy as np, torch
from gtrap_gb300 import api, synth
lc, tu, _ = synth.tess_like(nq=1, n=4000, seed=3)
g = synth.tls_grid(nw=4, nl=4)
out = api.gtls(torch.from_numpy(lc).cuda(), torch.from_numpy(tu).cuda(), 4000, 4, 4, {n}, g["wmax"], g["dw"], g["deltat"])
assert float(out[0].max()) > 0
"""


@pytest.mark.parametrize("code,n", [(PEAKS, 6400), (PEAKS, 7000), (PEAKS, 7700), (PEAKS, 7900), (GTLS, 1400), (GTLS, 1650)])
def test_first_launch_near_48_kb(cuda, code, n):
    res = subprocess.run([sys.executable, "-c", code.format(n=n)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-800:]


def test_threads_launching_one_kernel_at_different_sizes(cuda):
    """Four threads, each on its own stream, with series of lengths of their own: no launch is refused for the size
    that another thread has just asked for, and the results are those of each alone."""
    import threading

    import numpy as np
    import torch
    from gtrap_gb300 import api
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    errors = []

    def work(n):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                x = torch.from_numpy(np.abs(np.random.default_rng(n).normal(size=(n, 1))).astype(np.float32)).cuda()
                ref = [v.clone() for v in api.tls_peakstat(x)[1:]]
                for _ in range(1500):
                    got = api.tls_peakstat(x)[1:]
                assert all(torch.equal(a, b) for a, b in zip(ref, got))
                s.synchronize()
        except Exception as exc:   # (a thread's exception would not fail the test)
            errors.append((n, exc))

    try:
        threads = [threading.Thread(target=work, args=(n,)) for n in (9000, 30000, 12000, 34000)]
        [t.start() for t in threads]
        [t.join() for t in threads]
    finally:
        sys.setswitchinterval(interval)
    assert not errors, errors[0]
