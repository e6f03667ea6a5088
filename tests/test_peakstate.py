"""The peak suppression's states (gtrap_gb300/csrc/peakstate.cuh, built here for the CPU): warps decide
32 candidates each while others write their words, and a reader may see any value that a word has had
since the last barrier.  Whatever it sees, the kept set is the greedy one; with the two bits of a state in
words of their own, read one after the other without an order, it is not."""
import ctypes
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "gtrap_gb300" / "csrc"

HARNESS = """
#include "peakstate.cuh"
#define DECIDE(R) \\
  extern "C" unsigned decide##R(uint64_t b, uint64_t m, uint64_t a, uint32_t higher, int lane) { \\
    bool d, w; gtrap::peak_decide<R>(b, m, a, higher, lane, d, w); return (d ? 1u : 0u) | (w ? 2u : 0u); }
DECIDE(8)
DECIDE(16)
extern "C" uint64_t word(uint32_t u, uint32_t k) { return gtrap::peak_word(u, k); }
extern "C" uint32_t und(uint64_t s) { return gtrap::undecided_of(s); }
extern "C" uint32_t kept(uint64_t s) { return gtrap::kept_of(s); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("peakstate")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), str(d / "h.cpp"), "-o",
                    str(d / "h.so")], check=True)
    h = ctypes.CDLL(str(d / "h.so"))
    for f in (h.decide8, h.decide16):
        f.argtypes = [ctypes.c_uint64] * 3 + [ctypes.c_uint32, ctypes.c_int]
        f.restype = ctypes.c_uint
    h.word.argtypes, h.word.restype = [ctypes.c_uint32] * 2, ctypes.c_uint64
    for f in (h.und, h.kept):
        f.argtypes, f.restype = [ctypes.c_uint64], ctypes.c_uint32
    return h


def _masks(pos, val, w, reach):
    """Bit j < reach: entry c - reach + j ranks above c within w samples; bit reach + j: entry c + 1 + j."""
    out = []
    for c, (p, v) in enumerate(zip(pos, val)):
        m = 0
        for j in range(2 * reach):
            o = c - reach + j if j < reach else c + 1 + j - reach
            if 0 <= o < len(pos) and abs(pos[o] - p) <= w and (val[o], -pos[o]) > (v, -p):
                m |= 1 << j
        out.append(m)
    return out


def _greedy(pos, val, w):
    alive = np.ones(len(pos), bool)
    for c in sorted(range(len(pos)), key=lambda c: (-val[c], pos[c])):
        if alive[c]:
            near = np.abs(pos - pos[c]) <= w
            near[c] = False
            alive &= ~near
    return set(np.flatnonzero(alive))


def _rounds(h, reach, masks, rng, torn):
    """Rounds of the kernels, one word after another in any order; a word next to the one decided is seen as it
    is or as it was before any of its writes of this round (torn: each half so, by itself)."""
    decide = h.decide8 if reach == 8 else h.decide16
    M = len(masks)
    nword = (M + 31) // 32
    now = {-1: h.word(0, 0), nword: h.word(0, 0)}
    for i in range(nword):
        u = k = 0
        for lane in range(min(32, M - 32 * i)):
            if masks[32 * i + lane]:
                u |= 1 << lane
            else:
                k |= 1 << lane
        now[i] = h.word(u, k)
    for _ in range(M + 1):
        old = dict(now)
        for i in rng.sample(range(nword), nword):
            u0, k0 = h.und(now[i]), h.kept(now[i])

            def see(j):
                a = rng.choice([old, now])[j]
                b = rng.choice([old, now])[j] if torn else a
                return h.word(h.und(a), h.kept(b))

            before, behind = see(i - 1), see(i + 1)
            u, k = u0, k0
            for lane in range(32):
                if u0 >> lane & 1:
                    r = decide(before, now[i], behind, masks[32 * i + lane], lane)
                    if r & 1:
                        u &= ~(1 << lane)
                    elif not r & 2:
                        u &= ~(1 << lane)
                        k |= 1 << lane
            now[i] = h.word(u, k)
        if not any(h.und(now[i]) for i in range(nword)):
            return {32 * i + b for i in range(nword) for b in range(32) if h.kept(now[i]) >> b & 1}
    raise AssertionError("a round decided nothing")


def _case(rng, reach):
    n = 200
    pos = np.cumsum([rng.randint(1 if reach == 16 else 2, 4) for _ in range(n)])
    val = [rng.choice([rng.random(), 0.5, 0.25]) for _ in range(n)]   # ties among them
    return pos, val, rng.randint(2, 16)


@pytest.mark.parametrize("reach", [8, 16])
def test_any_view_of_the_words_gives_the_greedy_set(lib, reach):
    rng = random.Random(reach)
    for _ in range(60):
        pos, val, w = _case(rng, reach)
        masks = _masks(pos, val, w, reach)
        assert _rounds(lib, reach, masks, rng, torn=False) == _greedy(pos, val, w)


def test_halves_seen_apart_would_not(lib):
    rng = random.Random(3)
    cases = [(_masks(p, v, w, 16), _greedy(p, v, w)) for p, v, w in (_case(rng, 16) for _ in range(60))]
    assert any(_rounds(lib, 16, m, rng, torn=True) != g for m, g in cases)
