"""Server slots that run jobs of different read lengths and K at the same time:
kernels whose shared memory depends on both are launched from several threads
at once.  No job may fail, and each result is the lone job's."""
import numpy as np
import pytest

import crispy_gb300 as cg
from crispy_gb300 import synth

pytestmark = pytest.mark.gpu


def _same(r1, r2):
    (k1, c1), (k2, c2) = r1, r2
    assert k1 == k2 and len(c1) == len(c2)
    for (i1, p1, d1), (i2, p2, d2) in zip(c1, c2):
        assert i1 == i2 and np.array_equal(p1, p2)
        assert np.array_equal(d1.view(np.uint32), d2.view(np.uint32))


def test_lengths_and_k_at_once(monkeypatch):
    monkeypatch.setenv("CRISPY_SERVE_COHORT", "0")       # every job by itself
    jobs = []
    for length in (100, 250, 400, 700):
        for k in (5, 6, 7):
            spec = synth.ReadSetSpec(140, 6, length + 20, "uniform", length - 15, length, k, 50 * length + k)
            jobs.append((synth.pack_reads(synth.make_read_set(spec)), k))
    with cg.Server(0, 0, 1) as srv:
        want = []
        for (buf, offs, lens), k in jobs:
            jid = srv.submit(buf, offs, lens, k=k, band=10)
            assert srv.wait(jid) == cg.JOB_DONE
            want.append(srv.result(jid))
    rng = np.random.default_rng(3)
    with cg.Server(0, 0, 4) as srv:
        for _ in range(4):
            order = rng.integers(0, len(jobs), 150)
            ids = [srv.submit(*jobs[q][0], k=jobs[q][1], band=10) for q in order]
            for q, jid in zip(order, ids):
                assert srv.wait(jid) == cg.JOB_DONE
                _same(srv.result(jid), want[q])
