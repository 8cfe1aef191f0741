"""Runs that only just have the memory for the forms that need least: the
candidate filter, narrow sweeps and wide 16-bit shapes give way, and the results
are the same.  A server admits a job whose lean forms fit its budget."""
import numpy as np
import pytest

import crispy_gb300 as cg
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu

_LEAN = {"CRISPY_KMER_FILTER": "0", "CRISPY_GEN_NARROW": "0", "CRISPY_GEN_EXT": "0"}
_KINDS = {   # reads, root, distribution, a, b, K, band, cut
    "short": (3000, 260, "normal", 250, 15, 6, 10, 0.2),
    "short8": (3000, 260, "normal", 250, 15, 8, 5, 0.2),
    "uneven": (1500, 520, "uniform", 60, 500, 5, 3, 0.2),
    "long": (300, 2100, "uniform", 1800, 2048, 6, 10, 0.2),      # beyond the 16-bit range
    "wide": (250, 1650, "uniform", 1200, 1600, 7, 2, 0.2),       # bands beyond 256 slots
}


def _reads(kind):
    n, root, dist, a, b, k, band, cut = _KINDS[kind]
    reads = synth.make_read_set(synth.ReadSetSpec(n, max(4, n // 40), root, dist, a, b, k, 11))
    return synth.pack_reads(reads), k, band, cut


def _run(eng, kind):
    (buf, offs, lens), k, band, cut = _reads(kind)
    eng.kmer_prepare(buf, offs, lens, k)
    n = eng.kmer_run(cut, cg.MODE_BATCHED, True)
    pairs, dists = eng.kmer_fetch(n, True)
    eng.gen_prepare_from_kmer()
    chunks = eng.gen_run_from_kmer(band, 0.3, cg.MODE_BATCHED)
    few = np.ascontiguousarray(pairs[:: max(1, len(pairs) // 150)])
    aligned = eng.gen_align(few, band)
    out = [pairs, dists.view(np.uint32)]
    for _, p, d in chunks:
        out += [p, np.asarray(d).view(np.uint32)]
    return out + [np.asarray(x).view(np.uint32) for x in aligned]


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("kind", list(_KINDS))
def test_caps_below_the_full_need(monkeypatch, kind):
    monkeypatch.setenv("CRISPY_AUTOTUNE", "0")
    with cg.Engine(0) as eng:
        want = _run(eng, kind)
        full = eng.mem_in_use()
    with monkeypatch.context() as m:
        for name, value in _LEAN.items():
            m.setenv(name, value)
        with cg.Engine(0) as eng:
            _same(_run(eng, kind), want)
            lean = eng.mem_in_use()
    # all that the plain forms took is enough, as is anything between
    for cap in sorted({full - 1, (full + lean) // 2, lean}):
        if cap < lean:
            continue
        with cg.Engine(0) as eng:
            eng.set_mem_cap(cap)
            _same(_run(eng, kind), want)
            assert eng.mem_in_use() <= cap
            _same(_run(eng, kind), want)        # and again in buffers that are there
    with cg.Engine(0) as eng:                   # too little for any form
        eng.set_mem_cap(1 << 20)
        with pytest.raises(cg.CrispyError) as e:
            _run(eng, kind)
        assert e.value.code == cg.E_OOM
        eng.set_mem_cap(0)
        _same(_run(eng, kind), want)            # no error is left behind


@pytest.mark.parametrize("kind", ["short", "short8", "long"])
def test_server_admits_lean_jobs(kind):
    (buf, offs, lens), k, band, _ = _reads(kind)
    full = cg.server_job_bytes(lens, k)
    with cg.Server(0, 0, 1) as srv:
        jid = srv.submit(buf, offs, lens, k=k, band=band)
        assert srv.wait(jid) == cg.JOB_DONE
        want = srv.result(jid)
    for budget in (full - 1, full - full // 50):
        with cg.Server(0, budget, 1) as srv:
            jid = srv.submit(buf, offs, lens, k=k, band=band)
            assert srv.wait(jid) == cg.JOB_DONE
            mem = srv.job_memory(jid)
            assert 0 < mem["needed"] <= mem["reserved"] <= budget
            got = srv.result(jid)
        assert got[0] == want[0] and len(got[1]) == len(want[1])
        for (i1, p1, d1), (i2, p2, d2) in zip(got[1], want[1]):
            assert i1 == i2 and np.array_equal(p1, p2) and np.array_equal(d1.view(np.uint32), d2.view(np.uint32))
    with cg.Server(0, full // 8, 1) as srv:
        with pytest.raises(cg.CrispyError) as e:
            srv.submit(buf, offs, lens, k=k, band=band)
        assert e.value.code == cg.E_OOM


@pytest.mark.parametrize("length", [30, 250])
def test_preprocess_needs_no_more_than_before_the_keys(tmp_path, length):
    # the sort keys lie where the raw reads were: beside reads, padded reads and
    # the index lists (43 bytes a record) there is nothing of any size
    n = 20000
    rng = np.random.default_rng(length)
    rows = np.full((n, length + 3), 10, np.uint8)
    rows[:, 0] = ord(">")
    rows[:, 2:-1] = rng.choice(np.frombuffer(b"ACGT", np.uint8), (n, length))
    path = str(tmp_path / "raw.fa")
    rows.tofile(path)
    raw = cg.RawReads(path)
    with cg.Engine(0) as eng:
        index, _, _ = eng.preprocess(raw)
        used = eng.mem_in_use()
    raw.close()
    seqs = [r.tobytes() for r in rows[:, 2:-1]]
    assert index.tolist() == sorted({s: i for i, s in enumerate(seqs)}.values(), key=lambda i: seqs[i])
    short = max(0, 40 - length + 8) * n          # reads of under 40 bytes leave too little room
    assert used <= n * (length + (length + 15) // 16 * 16 + 43) + short + (1 << 16)
