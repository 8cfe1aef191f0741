"""Narrow sweeps of large batched genDist runs against the oracle.

Large runs (CRISPY_GEN_NARROW=1: every run) sweep each pair over the diagonals
it is likely to need and prove the result by its score, or sweep the whole
band again.
Score, ML, AL and distance must be the whole band's for similar reads (nearly
all proved), for unrelated ones (nearly all swept again), for reads whose
repeats make far diagonals score as well as the main one, at odd and even
lengths and length differences on either side, and for bands from 10 to the
unbanded alignment.
"""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def narrow(monkeypatch):
    monkeypatch.setenv("CRISPY_GEN_NARROW", "1")


def _check(engine, reads, pairs, bands):
    buf, offs, lens = synth.pack_reads(reads)
    engine.gen_prepare(buf, offs, lens)
    for band in bands:
        got = engine.gen_align(pairs, band, cg.MODE_BATCHED)
        want = oracle.gen_all(buf, offs, lens, pairs, band)
        for g, w in zip(got[1:], want[1:]):
            bad = np.nonzero(g != w)[0]
            assert len(bad) == 0, (band, pairs[bad[:4]].tolist(), g[bad[:4]], w[bad[:4]])
        assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))


def _random_pairs(n, m, seed):
    return np.random.default_rng(seed).integers(0, n, (m, 2)).astype(np.int32)


@pytest.mark.parametrize("spec", [
    (120, 2, 260, "normal", 250, 30),        # one of two OTUs: similar pairs
    (120, 60, 260, "uniform", 100, 260),     # mostly unrelated
    (120, 3, 420, "uniform", 200, 400),      # length differences beyond the band
    (120, 4, 90, "uniform", 1, 90),          # short
])
def test_narrow_read_sets(engine, spec):
    n, cents, root, dist, a, b = spec
    reads = synth.make_read_set(synth.ReadSetSpec(n, cents, root, dist, a, b, 6, 800 + cents))
    _check(engine, reads, _random_pairs(len(reads), 4300, cents), (10, 5, 3, 2, 1))


def test_narrow_repeats(engine):
    # tandem repeats of 1 to 24 bases: shifting by a period costs only the
    # overhang, so scores off the main diagonal come close to it
    rng = np.random.default_rng(31)
    reads = []
    for i in range(160):
        unit = rng.choice(np.frombuffer(b"ACGT", np.uint8), 1 + i % 24)
        s = np.resize(unit, int(rng.integers(120, 300)))
        for p in rng.integers(0, len(s), int(rng.integers(0, 6))):
            s[p] = b"ACGT"[rng.integers(0, 4)]
        reads.append(s.astype(np.uint8).tobytes())
    same = np.array([[i, (i + 24 * k) % 160] for i in range(160) for k in range(1, 6)], np.int32)
    pairs = np.concatenate([same, _random_pairs(160, 4100 - len(same) + 200, 32)])
    _check(engine, reads, pairs, (10, 4, 2, 1))


def test_narrow_planted_shifts(engine):
    # copies with a stretch removed near one end: the path leaves the main
    # diagonal by the stretch's length, within or beyond the estimate
    rng = np.random.default_rng(33)
    base = [rng.choice(np.frombuffer(b"ACGT", np.uint8), 300).tobytes() for _ in range(20)]
    reads = list(base)
    for k, s in enumerate(base):
        for cut in (1, 2, 3, 5, 8, 13, 21, 34):
            at = int(rng.integers(5, 250))
            reads.append(s[:at] + s[at + cut:])
            reads.append(s[cut:] + rng.choice(np.frombuffer(b"ACGT", np.uint8), cut).tobytes())
    n = len(reads)
    own = np.array([[k, 20 + 16 * k + c] for k in range(20) for c in range(16)], np.int32)
    pairs = np.concatenate([own, own[:, ::-1], _random_pairs(n, 4200, 34)])
    _check(engine, reads, pairs, (10, 5, 2))


@pytest.mark.parametrize("k,thr", [(5, 0.3), (6, 0.45), (7, 0.5), (8, 0.5)])
def test_narrow_from_kmer(engine, k, thr):
    # the estimate from kmerDist's distances, close pairs and loose ones
    reads = synth.make_read_set(synth.ReadSetSpec(500, 6, 320, "uniform", 150, 300, k, 840 + k))
    buf, offs, lens = synth.pack_reads(reads)
    engine.kmer_prepare(buf, offs, lens, k)
    cnt = engine.kmer_run(thr, cg.MODE_BATCHED, False)
    pairs, _ = engine.kmer_fetch(cnt, False)
    assert cnt > 2000
    engine.gen_prepare_from_kmer()
    for band in (10, 5, 2):
        d, _, _, _ = oracle.gen_all(buf, offs, lens, pairs, band)
        want = oracle.gen_chunks(pairs, d, 0.2)
        got = engine.gen_run_from_kmer(band, 0.2, cg.MODE_BATCHED)
        assert len(got) == len(want)
        for (ci, p, x), (wi, wp, wx) in zip(got, want):
            assert ci == wi and np.array_equal(p, wp)
            assert np.array_equal(x.view(np.uint32), wx.view(np.uint32))


@pytest.mark.parametrize("count", [1, 7, 200, 1300, 1900, 2600, 3700])
def test_few_pairs_shapes(engine, monkeypatch, count):
    # runs of few pairs take the shapes with 16 and 32 lanes per pair
    monkeypatch.setenv("CRISPY_GEN_NARROW", "0")
    reads = synth.make_read_set(synth.ReadSetSpec(90, 5, 330, "uniform", 1, 330, 6, 850))
    _check(engine, reads, _random_pairs(len(reads), count, count), (10, 5, 3, 2))


def test_narrow_after_whole_bands_were_tuned(engine, monkeypatch):
    # the shape tuned for a bin of whole bands may be the 32-bit kernel's,
    # which sweeps nothing else; narrow sweeps have their own choice.  Short
    # reads fill the small bins that longer reads' narrow sweeps fall into.
    rng = np.random.default_rng(41)
    short = [rng.choice(np.frombuffer(b"ACGT", np.uint8), int(rng.integers(30, 300))).tobytes() for _ in range(200)]
    monkeypatch.setenv("CRISPY_GEN_NARROW", "0")
    _check(engine, short, _random_pairs(200, 30000, 42), (10, 5))
    monkeypatch.setenv("CRISPY_GEN_NARROW", "1")
    reads = synth.make_read_set(synth.ReadSetSpec(150, 2, 330, "uniform", 290, 320, 6, 860))
    _check(engine, reads, _random_pairs(len(reads), 20000, 43), (10, 5))


@pytest.mark.parametrize("narrow_on", ["0", "1"])
def test_long_reads_extended_keys(engine, monkeypatch, narrow_on):
    # L1 + L2 around and beyond 3,600: similar pairs are proved by their
    # score, unrelated ones and reads that share no symbol are swept again
    monkeypatch.setenv("CRISPY_GEN_NARROW", narrow_on)
    reads = synth.make_read_set(synth.ReadSetSpec(60, 3, 2100, "uniform", 1750, 2048, 6, 870))
    rng = np.random.default_rng(45)
    reads += [rng.choice(np.frombuffer(b"ACGT", np.uint8), int(L)).tobytes() for L in (1801, 2000, 2047, 2048)]
    reads += [b"A" * 2048, b"C" * 2048, b"G" * 2001, b"A" * 1800, b"AC" * 1024, reads[0], reads[1][:1799] + b"T"]
    n = len(reads)
    fixed = [[n - 7, n - 6], [n - 7, n - 5], [n - 7, n - 7], [n - 3, n - 7], [n - 3, n - 6], [n - 2, 0], [n - 1, 1]]
    pairs = np.concatenate([np.array(fixed, np.int32), _random_pairs(n, 240, 46)])
    _check(engine, reads, pairs, (40, 20, 10))
    _check(engine, reads, pairs[:60], (5,))


@pytest.mark.parametrize("narrow_on", ["0", "1"])
def test_bands_beyond_256_slots(engine, monkeypatch, narrow_on):
    # kBand 250 to 520: the 384- and 512-slot shapes, and the wide-band kernel
    # beyond them; short runs, and one pair
    monkeypatch.setenv("CRISPY_GEN_NARROW", narrow_on)
    reads = synth.make_read_set(synth.ReadSetSpec(70, 3, 1650, "uniform", 1200, 1600, 6, 880))
    pairs = _random_pairs(len(reads), 120, 47)
    _check(engine, reads, pairs, (5, 4, 3))
    _check(engine, reads, pairs[:1], (5,))
    longr = synth.make_read_set(synth.ReadSetSpec(30, 2, 2100, "uniform", 1850, 2048, 6, 881))
    _check(engine, longr, _random_pairs(len(longr), 60, 48), (6, 4))
    short = synth.make_read_set(synth.ReadSetSpec(60, 3, 520, "uniform", 300, 500, 6, 882))
    _check(engine, short, _random_pairs(len(short), 300, 49), (1,))


@pytest.mark.parametrize("narrow_on", ["0", "1", None])
def test_bands_beyond_512_slots(engine, monkeypatch, narrow_on):
    # kBand 500 to 1,023: the 768- and 1,024-slot shapes at their edges (a band
    # of one slot more or less on either side of 768 and 1,024), and bands
    # beyond them, which sweep narrow diagonals first unless told not to
    if narrow_on is None:
        monkeypatch.delenv("CRISPY_GEN_NARROW")
    else:
        monkeypatch.setenv("CRISPY_GEN_NARROW", narrow_on)
    rng = np.random.default_rng(883)
    base = rng.integers(0, 4, 1700)
    fixed = []
    for n in (510, 511, 512, 766, 767, 768, 769, 1022, 1023, 1024, 1025):
        s = base[:n].copy()
        hit = rng.random(n) < 0.04
        s[hit] = rng.integers(0, 4, int(hit.sum()))
        fixed.append(bytes(b"AGTC"[c] for c in s))
    pairs = np.array([(i, j) for i in range(len(fixed)) for j in range(len(fixed)) if abs(i - j) <= 1], np.int32)
    _check(engine, fixed, pairs, (1,))
    reads = synth.make_read_set(synth.ReadSetSpec(60, 3, 1650, "uniform", 1200, 1600, 6, 884))
    _check(engine, reads, _random_pairs(len(reads), 200, 50), (2,))
    _check(engine, reads, _random_pairs(len(reads), 1, 51), (2, 1))
    longr = synth.make_read_set(synth.ReadSetSpec(24, 1, 2100, "uniform", 1850, 2048, 6, 885))
    _check(engine, longr, _random_pairs(len(longr), 40, 52), (3, 2))


def test_server_estimate_wide_bands(monkeypatch):
    # a few reads whose bands take the widest shapes: the run stays within the
    # bytes it was admitted with
    monkeypatch.delenv("CRISPY_GEN_NARROW")
    reads = synth.make_read_set(synth.ReadSetSpec(40, 2, 1000, "uniform", 800, 1000, 6, 886))
    buf, offs, lens = synth.pack_reads(reads)
    with cg.Server(0, 0, 1) as srv:
        jid = srv.submit(buf, offs, lens, 6, 1, 0.5, 0.5)
        assert srv.wait(jid) == cg.JOB_DONE
        mem = srv.job_memory(jid)
        assert 0 < mem["needed"] <= mem["reserved"], mem


@pytest.mark.parametrize("narrow_on", ["0", "1"])
def test_long_unrelated_reads(engine, monkeypatch, narrow_on):
    # L1 + L2 > 3,600 and scores too low to prove anything: exact because no
    # cell was raised to the floor, or left to the 32-bit kernel; among them
    # reads without a symbol in common, whose scores fall the furthest
    monkeypatch.setenv("CRISPY_GEN_NARROW", narrow_on)
    rng = np.random.default_rng(887)
    reads = [bytes(b"AGTC"[c] for c in rng.integers(0, 4, n)) for n in
             (1801, 1850, 1903, 1957, 2000, 2031, 2047, 2048)]
    reads += [b"A" * 1900, b"C" * 2048, b"G" * 1999, b"AC" * 1000, b"GT" * 1024, b"A" * 1024 + b"C" * 1024]
    n = len(reads)
    pairs = np.array([(i, j) for i in range(n) for j in range(n) if i != j], np.int32)
    _check(engine, reads, pairs, (40, 10, 5))
    _check(engine, reads, pairs[::7], (2,))
