"""Pair lists that narrow sweeps do not pay for: unrelated reads, whose 8-mers
say nothing about the alignment any more, and reads that share their 8-mers
but not their order, whose narrow sweeps prove nothing (once an eighth of a
list has failed the rest goes to the whole-band sweeps unswept).  The results
are the whole bands'."""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle

pytestmark = pytest.mark.gpu

_ACGT = np.frombuffer(b"ACGT", np.uint8)


def _mutated(rng, s, rate):
    s = s.copy()
    hit = rng.random(len(s)) < rate
    s[hit] = (s[hit] + rng.integers(1, 4, int(hit.sum()))) % 4
    return s


def _reads(kind, n, length, rng):
    root = rng.integers(0, 4, length + 30)
    out = []
    for i in range(n):
        if kind == "unrelated":
            s = rng.integers(0, 4, length + 30)
        else:
            s = _mutated(rng, root, 0.01)
        s = s[:int(rng.integers(length - 30, length + 30))]
        if kind == "rotated" and i % 2:
            s = np.concatenate([s[len(s) // 2:], s[:len(s) // 2]])
        if kind == "mixed" and i % 5 == 0:
            s = rng.integers(0, 4, len(s))
        out.append(_ACGT[s])
    lens = np.array([len(s) for s in out], np.int32)
    offs = np.zeros(n, np.int64)
    np.cumsum(lens[:-1], out=offs[1:])
    return np.concatenate(out), offs, lens


@pytest.mark.parametrize("kind,length,pairs,bands", [
    ("similar", 250, 20000, (10, 2)),      # the sample agrees: narrow sweeps
    ("unrelated", 250, 20000, (10, 2)),    # the sample says no
    ("unrelated", 250, 6000, (2,)),        # no sample: each pair by itself
    ("rotated", 250, 20000, (2,)),         # half of the pairs fail the proof
    ("rotated", 400, 9000, (2, 1)),
    ("mixed", 250, 17000, (5, 2)),
    ("rotated", 1850, 1200, (5,)),         # beyond the 16-bit range: twice listed
])
def test_lists_without_gain(engine, monkeypatch, kind, length, pairs, bands):
    monkeypatch.setenv("CRISPY_GEN_NARROW", "1")
    rng = np.random.default_rng(length + pairs)
    buf, offs, lens = _reads(kind, 300, length, rng)
    a = rng.integers(0, 300, pairs)
    b = (a + rng.integers(1, 300, pairs)) % 300
    pr = np.stack([a, b], 1).astype(np.int32)
    engine.gen_prepare(buf, offs, lens)
    for band in bands:
        got = engine.gen_align(pr, band, cg.MODE_BATCHED)
        st = engine.stats()
        want = oracle.gen_all(buf, offs, lens, pr, band)
        for g, w in zip(got[1:], want[1:]):
            assert np.array_equal(g, w)
        assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))
        share = st["gen_swept_cells"] / st["gen_cells"]
        if kind == "similar":
            assert share < 0.9
        elif kind == "unrelated":
            assert share == 1.0
