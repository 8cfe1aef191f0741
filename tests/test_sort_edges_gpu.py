"""The radix sort behind kmerDist's stage order and genDist's chunks, at the
sizes where its form changes: one block (2 and 8 items a thread), and passes
over tiles, with survivors at the edges of both.

Pairs of one read set in number around 2,048, 8,192 and 4,096-item tiles go
through genDist with a threshold that keeps them all, so each chunk is a
stable sort of distances with many ties; the oracle sorts the same way.
"""
import numpy as np
import pytest

import crispy_gb300 as cg
import oracle
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 31, 33, 2047, 2048, 2049, 8191, 8192, 8193, 12288, 12289, 40001])
def test_chunk_sort_sizes(engine, m):
    reads = synth.make_read_set(synth.ReadSetSpec(300, 6, 120, "uniform", 60, 100, 6, 700))
    buf, offs, lens = synth.pack_reads(reads)
    rng = np.random.default_rng(m)
    pairs = np.stack([rng.integers(0, len(reads), m), rng.integers(0, len(reads), m)], 1).astype(np.int32)
    d, _, _, _ = oracle.gen_all(buf, offs, lens, pairs, 10)
    want = oracle.gen_chunks(pairs, d, 1.0)
    engine.gen_prepare(buf, offs, lens)
    for _ in range(3):     # plain, captured and replayed launches
        got = engine.gen_run(pairs, 10, 1.0, cg.MODE_BATCHED)
        assert len(got) == len(want)
        for (ci, p, x), (wi, wp, wx) in zip(got, want):
            assert ci == wi and np.array_equal(p, wp)
            assert np.array_equal(x.view(np.uint32), wx.view(np.uint32))


@pytest.mark.parametrize("n", [60, 66, 129, 180, 400])
def test_stage_sort_sizes(engine, n):
    # every pair survives a cut of 1: n (n - 1) / 2 stage keys around 2,048 and
    # 8,192, and above
    reads = synth.make_read_set(synth.ReadSetSpec(n + 20, 5, 120, "uniform", 60, 100, 6, 710 + n))[:n]
    buf, offs, lens = synth.pack_reads(reads)
    op, od = oracle.kmer_all(buf, offs, lens, 6, 1.0)
    for k_mode in (cg.MODE_BATCHED, cg.MODE_STAGED):
        engine.kmer_prepare(buf, offs, lens, 6)
        cnt = engine.kmer_run(1.0, k_mode, True)
        pairs, d = engine.kmer_fetch(cnt, True)
        assert np.array_equal(pairs, op)
        assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
