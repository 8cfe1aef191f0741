"""Read sets whose candidates are too many for the tensor-core filter: the tile
kernels take them, with the same survivors.  CRISPY_KMER_CAND sets the room for
candidates, so that small sets reach every way the filter is given up: by the
probe before the rest, by a round whose candidates outgrow the room, and in a
later range of a run whose survivors spill.  kmer_launches counts the rounds of
the attempt and the tile launch behind it."""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


def _reads(n, k, seed, cents, length=250):
    spec = synth.ReadSetSpec(n + n // 8 + 8, cents, length + 10, "normal", length, 15, k, seed)
    return synth.make_read_set(spec)[:n]


def _run(engine, thr):
    got = engine.kmer_fetch(engine.kmer_run(thr, cg.MODE_BATCHED, True), True)
    return got, engine.stats()


def _same(got, want):
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("k", [5, 6, 7, 8])
def test_round_outgrows_its_room(engine, monkeypatch, k):
    # fewer tiles than the probe is for: the one round overflows
    reads = _reads(900, k, 80 + k, 6)
    buf, offs, lens = synth.pack_reads(reads)
    want = oracle.kmer_all(buf, offs, lens, k, 0.2)
    engine.kmer_prepare(buf, offs, lens, k)
    got, st = _run(engine, 0.2)
    _same(got, want)
    assert st["kmer_launches"] == 1                     # the filter alone
    engine.kmer_prepare(buf, offs, lens, k)
    monkeypatch.setenv("CRISPY_KMER_CAND", str(max(1, len(want[0]) // 2)))
    got, st = _run(engine, 0.2)
    _same(got, want)
    assert st["kmer_launches"] == 2                     # an attempt, then the tiles
    got, st = _run(engine, 0.25)                        # looser: no second attempt
    _same(got, oracle.kmer_all(buf, offs, lens, k, 0.25))
    assert st["kmer_launches"] == 1
    monkeypatch.delenv("CRISPY_KMER_CAND")
    got, st = _run(engine, 0.05)                        # tighter: another attempt
    _same(got, oracle.kmer_all(buf, offs, lens, k, 0.05))
    engine.kmer_prepare(buf, offs, lens, k)             # new reads: as at first
    got, st = _run(engine, 0.2)
    _same(got, want)
    assert st["kmer_launches"] == 1


@pytest.mark.parametrize("k", [6, 8])
def test_probe_gives_up(engine, monkeypatch, k):
    # k = 8: runs of equal H keys wide enough for as many tiles
    n = 12000 if k == 6 else 14000
    reads = _reads(n, k, 90 + k, 60 if k == 6 else 2)
    buf, offs, lens = synth.pack_reads(reads)
    thr = 0.1 if k == 6 else 0.05
    monkeypatch.setenv("CRISPY_KMER_FILTER", "0")
    engine.kmer_prepare(buf, offs, lens, k)
    want, _ = _run(engine, thr)
    monkeypatch.setenv("CRISPY_KMER_FILTER", "1")
    for room in (50, len(want[0]) // 2, 1 << 22):
        monkeypatch.setenv("CRISPY_KMER_CAND", str(room))
        engine.kmer_prepare(buf, offs, lens, k)
        got, st = _run(engine, thr)
        _same(got, want)
        if room < len(want[0]):
            assert st["kmer_launches"] == 2
        # genDist behind either: its reads come packed or not
        engine.gen_prepare_from_kmer()
    assert len(want[0]) > n


@pytest.mark.parametrize("k", [6, 8])
def test_second_range_gives_up(engine, monkeypatch, k):
    # survivors beyond the device share, the last reads all of one OTU: the
    # first pass and the first ranges of stage rows have few candidates for
    # their pairs, the last range many
    sparse = _reads(2000, k, 100 + k, 1000)
    dense = _reads(620, k, 110 + k, 1, 270)      # longer: behind the others
    reads = [r for r in sparse if len(r) < 262] + [r for r in synth.preprocess_order(dense) if len(r) > 262]
    buf, offs, lens = synth.pack_reads(reads)
    thr = 0.15
    want = oracle.kmer_all(buf, offs, lens, k, thr)
    monkeypatch.setenv("CRISPY_KMER_DEVICE_PAIRS", str(len(want[0]) * 9 // 10))
    launches = {}
    # room for any number; for one in 20 of a pass's pairs, which the last
    # reads' own rows outgrow; for one in 1,000, which the first pass does
    for room in ("100000000", "-20", "-1000"):
        monkeypatch.setenv("CRISPY_KMER_CAND", room)
        engine.kmer_prepare(buf, offs, lens, k)
        got, st = _run(engine, thr)
        assert st["kmer_spilled"] == 1
        _same(got, want)
        launches[room] = st["kmer_launches"]
    passes = launches["100000000"]               # the filter in every pass
    assert passes >= 3
    # one attempt more than passes, after which no other pass tries (at K = 8
    # every pass bounds all pairs: what the first one fits fits the others)
    assert launches["-20"] == (passes + 1 if k == 6 else passes)
    assert launches["-1000"] == passes + 1


def test_tuner_behind_a_gave_up_filter(engine, monkeypatch):
    # the bound pass's split is tuned from the second batched run on, as for
    # sets the filter never takes
    monkeypatch.delenv("CRISPY_AUTOTUNE", raising=False)
    monkeypatch.setenv("CRISPY_KMER_CAND", "1000")
    reads = _reads(8900, 6, 120, 100)
    buf, offs, lens = synth.pack_reads(reads)

    def tuned():
        return [e for e in cg.tune_report()
                if e.get("stage") == "kmer" and e["reads"] == len(reads) and "candidates" not in e]

    want = None
    for i in range(3):
        engine.kmer_prepare(buf, offs, lens, 6)
        got, st = _run(engine, 0.1)
        assert st["kmer_launches"] == 2 and (i or st["kmer_bound_entries"] > 0)   # (a tuned split may be 0)
        want = want or got
        _same(got, want)
        assert len(tuned()) == (1 if i else 0)
    monkeypatch.setenv("CRISPY_KMER_FILTER", "0")
    engine.kmer_prepare(buf, offs, lens, 6)
    _same(_run(engine, 0.1)[0], want)


@pytest.mark.parametrize("k,length", [(5, 300), (6, 500), (8, 400)])
def test_lists_built_again_after_giving_up(engine, monkeypatch, k, length):
    # reads over two bases: nearly every K-mer is a repeat, so the lists of
    # repeats fill their room; a round gives up behind them, and tighter cuts
    # with as many dimensions build them again, time after time
    rng = np.random.default_rng(k)
    base = rng.choice(np.frombuffer(b"TC", np.uint8), length)
    reads = []
    for _ in range(400):
        s = base[:int(rng.integers(length - 20, length + 1))].copy()
        for p in rng.integers(0, len(s), int(rng.integers(0, 4))):
            s[p] = b"TC"[int(rng.integers(0, 2))]
        reads.append(s.tobytes())
    buf, offs, lens = synth.pack_reads(synth.preprocess_order(reads))
    engine.kmer_prepare(buf, offs, lens, k)
    for i, thr in enumerate((0.15, 0.14, 0.13, 0.12, 0.11, 0.1, 0.09)):
        # given up at all cuts but the last (the room is what it is for them)
        monkeypatch.setenv("CRISPY_KMER_CAND", "50" if i < 6 else "100000000")
        got, _ = _run(engine, thr)
        _same(got, oracle.kmer_all(buf, offs, lens, k, thr))
