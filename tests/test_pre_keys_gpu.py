"""The 128-bit sort keys of preprocess: reads that differ only in bytes the
keys map to ranges, before, at and behind the 28th, beside reads that share
long prefixes and whole duplicates; tile and merge edges.  The order must be
(length, bytes, record), each run of equal reads merged into its last."""
import numpy as np
import pytest

import crispy_gb300 as cg

pytestmark = pytest.mark.gpu

_BYTES = b"ACGTNacgtn*-.BDEFHIJKMORSUVWXYZ@[_bdefh~"


def _check(engine, tmp_path, reads):
    path = str(tmp_path / "raw.fa")
    with open(path, "wb") as f:
        for i, s in enumerate(reads):
            f.write(b">r%d\n%b\n" % (i, s))
    raw = cg.RawReads(path)
    assert [raw.seq(i) for i in range(raw.n)] == reads
    index, freq, _ = engine.preprocess(raw)
    order = sorted(range(len(reads)), key=lambda i: (len(reads[i]), reads[i], i))
    want, count = [], []
    for q, i in enumerate(order):
        if q and reads[order[q - 1]] == reads[i]:
            want[-1], count[-1] = i, count[-1] + 1
        else:
            want.append(i)
            count.append(1)
    assert index.tolist() == want and freq.tolist() == count
    raw.close()


@pytest.mark.parametrize("n", [2, 50, 1023, 1024, 1025, 2049, 5000])
def test_key_classes_and_prefixes(engine, tmp_path, n):
    rng = np.random.default_rng(n)
    base = rng.choice(np.frombuffer(b"ACGT", np.uint8), 60)
    reads = []
    for _ in range(n):
        s = base[:int(rng.integers(26, 60))].copy()
        for p in rng.integers(0, len(s) - 1, int(rng.integers(0, 3))):
            s[p] = _BYTES[int(rng.integers(0, len(_BYTES)))]
        s[-1] = b"ACGT"[int(rng.integers(0, 4))]      # the parser trims other endings
        reads.append(s.tobytes())
    _check(engine, tmp_path, reads)


@pytest.mark.parametrize("copies", [3, 40, 700])
def test_copies(engine, tmp_path, copies):
    # groups of equal keys small enough to settle one by one, and too large
    rng = np.random.default_rng(copies)
    base = rng.choice(np.frombuffer(b"ACGT", np.uint8), 80)
    reads = []
    for k in range(max(2, 9000 // copies)):
        s = base.copy()
        s[28 + k % 50] = b"ACGT"[int(rng.integers(0, 4))]
        s[int(rng.integers(0, 80))] = b"ACGT"[int(rng.integers(0, 4))]
        reads += [s.tobytes()] * copies
    reads = [reads[i] for i in rng.permutation(len(reads))]
    _check(engine, tmp_path, reads)


def test_short_reads_and_one_length(engine, tmp_path):
    rng = np.random.default_rng(9)
    reads = [rng.choice(np.frombuffer(b"ACGT", np.uint8), int(rng.integers(1, 5))).tobytes() for _ in range(1500)]
    reads += [rng.choice(np.frombuffer(b"AC", np.uint8), 28).tobytes() for _ in range(600)]
    _check(engine, tmp_path, reads)
