"""The tensor-core candidate filter of the batched k-mer run (K >= 5, cut
<= 0.3) against the oracle: pairs, order and distances bit for bit.

Sizes sit at the edges of the 128-row panels, the 224-column tiles and the
256-dimension chunks of the signatures (resident and streamed rows); reads
with folded counts beyond 36 (homopolymers), reads in no length order, reads
without a k-mer, K = 8 reads with and without an H half, and sets whose
candidates outgrow their buffer, which the tile kernels then take.
"""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


def _reads(n, seed, k=6, root=260, dist="normal", a=250, b=15, cents=None):
    spec = synth.ReadSetSpec(n + n // 8 + 8, cents or max(2, n // 20), root, dist, a, b, k, seed)
    return synth.make_read_set(spec)[:n]


def _check(engine, monkeypatch, reads, k, thr):
    buf, offs, lens = synth.pack_reads(reads)
    got = {}
    for on in ("1", "0"):
        monkeypatch.setenv("CRISPY_KMER_FILTER", on)
        engine.kmer_prepare(buf, offs, lens, k)
        cnt = engine.kmer_run(thr, cg.MODE_BATCHED, True)
        got[on] = engine.kmer_fetch(cnt, True)
    op, od = oracle.kmer_all(buf, offs, lens, k, thr)
    for pairs, d in got.values():
        assert np.array_equal(pairs, op)
        assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
    return len(op)


@pytest.mark.parametrize("n", [10, 127, 128, 129, 223, 225, 449, 1025])
def test_filter_tile_edges(engine, monkeypatch, n):
    assert _check(engine, monkeypatch, _reads(n, 900 + n), 6, 0.2) > 0


@pytest.mark.parametrize("k", [5, 6, 7, 8])
@pytest.mark.parametrize("thr", [0.0, 0.1, 0.2, 0.3])
def test_filter_k_and_cut(engine, monkeypatch, k, thr):
    reads = _reads(700, 910 + k, k=k, root=520, dist="uniform", a=300, b=500)
    _check(engine, monkeypatch, reads, k, thr)


@pytest.mark.parametrize("length", [40, 128, 400, 700, 1100, 2048])
def test_filter_signature_lengths(engine, monkeypatch, length):
    # one chunk of 256 dimensions to the most (4,096, streamed)
    reads = _reads(300, 920 + length, root=2100, dist="uniform", a=max(20, length - 30), b=length)
    assert _check(engine, monkeypatch, reads, 6, 0.2) > 0


@pytest.mark.parametrize("k", [6, 8])
def test_filter_repeats_and_order(engine, monkeypatch, k):
    rng = np.random.default_rng(k)
    reads = _reads(260, 930, k=k)
    for i in range(60):     # runs of one base: folded counts far beyond 36
        s = bytearray(reads[i])
        run = 40 + 3 * (i % 30)
        s[20:20 + run] = b"ACGT"[i % 4:i % 4 + 1] * run
        reads.append(bytes(s))
    reads += [b"A" * (300 + i) for i in range(6)] + [b"CT" * (150 + i) for i in range(6)]
    reads += [b"ACGTACG"[:k - 1 + (i & 1)] for i in range(2)]
    reads = [reads[i] for i in rng.permutation(len(reads))]
    assert _check(engine, monkeypatch, reads, k, 0.2) > 0


def test_filter_heavy_h_reads(engine, monkeypatch):
    # K = 8 reads rich in T and C: pairs of different H keys can pass
    rng = np.random.default_rng(5)
    reads = _reads(200, 940, k=8)
    base = rng.choice(np.frombuffer(b"TC", np.uint8), 260).tobytes()
    for i in range(80):
        s = bytearray(base)
        for p in rng.integers(0, 260, 3):
            s[p] = b"TC"[rng.integers(0, 2)]
        reads.append(bytes(s[:200 + i // 2]))
    assert _check(engine, monkeypatch, synth.preprocess_order(reads), 8, 0.25) > 0


def test_filter_gives_up(engine, monkeypatch):
    # one centroid: nearly every pair is a candidate, more than the buffer holds
    reads = _reads(1800, 950, cents=1)
    assert _check(engine, monkeypatch, reads, 6, 0.3) > 300000


@pytest.mark.parametrize("n,length", [(12000, 120), (12000, 250), (12000, 400), (9000, 550), (9000, 1100)])
def test_filter_many_tiles(engine, monkeypatch, n, length):
    # several tiles per block, so that every ring and both accumulators wrap
    # (1 to 4 chunks with resident rows, more streamed), against the tile
    # kernels, twice
    reads = _reads(n, 960 + length, root=length + 20, dist="uniform", a=length - 20, b=length, cents=n // 40)
    buf, offs, lens = synth.pack_reads(reads)
    got = []
    for on in ("0", "1", "1"):
        monkeypatch.setenv("CRISPY_KMER_FILTER", on)
        engine.kmer_prepare(buf, offs, lens, 6)
        got.append(engine.kmer_fetch(engine.kmer_run(0.15, cg.MODE_BATCHED, True), True))
    assert len(got[0][0]) > n
    for pairs, d in got[1:]:
        assert np.array_equal(pairs, got[0][0])
        assert np.array_equal(d.view(np.uint32), got[0][1].view(np.uint32))


# below 0: every block's loader gives up at its first wait; small limits: somewhere on
# the way, with copies and matrix instructions in flight, or not at all
@pytest.mark.parametrize("length", [250, 1400])
@pytest.mark.parametrize("wait", [-1, 0, 300, 1000, 3000, 10000])
def test_filter_wait_limit(engine, monkeypatch, wait, length):
    n, cents = (4000, 100) if length == 250 else (1500, 40)
    reads = _reads(n, 970 + length, root=length + 20, dist="uniform", a=length - 20, b=length, cents=cents)
    buf, offs, lens = synth.pack_reads(reads)

    def run():
        engine.kmer_prepare(buf, offs, lens, 6)
        return engine.kmer_fetch(engine.kmer_run(0.15, cg.MODE_BATCHED, True), True)

    want = run()
    monkeypatch.setenv("CRISPY_KMER_WAIT", str(wait))
    for _ in range(3):
        try:
            got = run()
        except cg.CrispyError as e:
            assert e.code == cg.E_TIMEOUT
        else:
            assert wait >= 0
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    monkeypatch.delenv("CRISPY_KMER_WAIT")
    got = run()         # the context is as usable as before
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


# reads of few bases over and over: more repeats than the count's table takes
# at once (128, 256 or 512 entries), so that it is filled part by part
@pytest.mark.parametrize("k,length", [(5, 450), (6, 300), (6, 900), (7, 500), (7, 2048), (8, 700), (8, 2048)])
def test_filter_rows_of_many_repeats(engine, monkeypatch, k, length):
    rng = np.random.default_rng(k + length)
    reads = []
    for unit in (1, 2, 3, 5, 9, 40):
        base = np.resize(rng.choice(np.frombuffer(b"ACGT", np.uint8), unit), length)
        for _ in range(30):
            s = base[:int(rng.integers(length - length // 8, length + 1))].copy()
            for p in rng.integers(0, len(s), int(rng.integers(0, 6))):
                s[p] = b"ACGT"[int(rng.integers(0, 4))]
            reads.append(s.tobytes())
    reads = [reads[i] for i in rng.permutation(len(reads))]
    for thr in (0.05, 0.3):
        assert _check(engine, monkeypatch, reads, k, thr) > 100
