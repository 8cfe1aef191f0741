"""The tile kernels' bound pass and the tuner of its split (K <= 6), with the
candidate filter off: read sets that the filter gives up, runs without memory
for it and cuts above 0.3 take them.  Survivors, their order and distances must
not depend on the split, the threshold or the read order."""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _tiles(monkeypatch):
    monkeypatch.setenv("CRISPY_KMER_FILTER", "0")
    monkeypatch.delenv("CRISPY_KMER_SPLIT", raising=False)
    monkeypatch.delenv("CRISPY_AUTOTUNE", raising=False)


def _reads(n, seed, k=6, cents=None):
    return synth.make_read_set(synth.ReadSetSpec(n, cents or max(4, n // 60), 520, "uniform", 300, 500, k, seed))


def _check(engine, reads, k, thr):
    buf, offs, lens = synth.pack_reads(reads)
    engine.kmer_prepare(buf, offs, lens, k)
    cnt = engine.kmer_run(thr, cg.MODE_BATCHED, True)
    st = engine.stats()
    pairs, d = engine.kmer_fetch(cnt, True)
    op, od = oracle.kmer_all(buf, offs, lens, k, thr)
    assert np.array_equal(pairs, op)
    assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
    return cnt, st


@pytest.mark.parametrize("thr", [0.0, 0.02, 0.08, 0.3, 1.0])
def test_thresholds(engine, thr):
    _, st = _check(engine, _reads(900, 602), 6, thr)
    assert st["kmer_bound_entries"] > 0


@pytest.mark.parametrize("k", [4, 5, 6])
def test_unsorted_reads(engine, k):
    reads = _reads(1300, 603 + k, k)
    rng = np.random.default_rng(k)
    reads = [reads[i] for i in rng.permutation(len(reads))]
    cnt, st = _check(engine, reads, k, cg.default_threshold(len(reads), -1.0, 0))
    assert cnt > 0 and st["kmer_bound_entries"] > 0


def test_many_alive_columns(engine):
    reads = _reads(2500, 604, cents=3)
    cnt, st = _check(engine, reads, 6, cg.default_threshold(len(reads), -1.0, 0))
    assert cnt > 10000 and st["kmer_rounds"] > 0 and st["kmer_full_columns"] > 0


def test_split_tuned_from_the_second_run(engine):
    reads = _reads(9100, 620)
    assert len(reads) >= 8192
    buf, offs, lens = synth.pack_reads(reads)
    t = cg.default_threshold(len(reads), -1.0, 0)

    def entries():
        return [e for e in cg.tune_report() if e.get("stage") == "kmer" and e["reads"] == len(reads)]

    first = None
    for i in range(3):
        engine.kmer_prepare(buf, offs, lens, 6)
        got = engine.kmer_fetch(engine.kmer_run(t, cg.MODE_BATCHED, True), True)
        first = first or got
        assert np.array_equal(got[0], first[0]) and np.array_equal(got[1], first[1])
        e = entries()
        assert len(e) == (1 if i else 0)
        if i:
            assert e[0]["split"] in (0, 96, 112, 128, 144, 160) and 0 < e[0]["ms"] <= e[0]["default_ms"]


def test_filter_note_names_the_tuned_split(engine, monkeypatch):
    # the same set tuned by the tile kernels, then taken by the filter: both
    # entries of the report give one split
    reads = _reads(8700, 621)
    buf, offs, lens = synth.pack_reads(reads)
    for on in ("0", "0", "1", "1"):
        monkeypatch.setenv("CRISPY_KMER_FILTER", on)
        engine.kmer_prepare(buf, offs, lens, 6)
        engine.kmer_run(0.1, cg.MODE_BATCHED, False)
    e = [x for x in cg.tune_report() if x.get("stage") == "kmer" and x["reads"] == len(reads)]
    assert len(e) == 2 and e[0]["split"] == e[1]["split"]
    assert sum("candidates" in x for x in e) == 1
