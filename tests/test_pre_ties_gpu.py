"""preprocess on sets whose sort keys (length, first 28 bytes) tie in groups
larger than the group-by-group settling takes: the sort has to start again
from the reads themselves, and every kernel before that decision must see a
valid order."""
import numpy as np
import pytest

import crispy_gb300 as cg

pytestmark = pytest.mark.gpu


def _run(eng, tmp_path, reads):
    path = str(tmp_path / "raw.fa")
    with open(path, "wb") as f:
        for i, s in enumerate(reads):
            f.write(b">r%d\n%b\n" % (i, s))
    raw = cg.RawReads(path)
    index, freq, _ = eng.preprocess(raw)
    raw.close()
    order = sorted(range(len(reads)), key=lambda i: (len(reads[i]), reads[i], i))
    want, count = [], []
    for q, i in enumerate(order):
        if q and reads[order[q - 1]] == reads[i]:
            want[-1], count[-1] = i, count[-1] + 1
        else:
            want.append(i)
            count.append(1)
    assert index.tolist() == want and freq.tolist() == count


def _reads(n, kind):
    rng = np.random.default_rng(n)
    base = rng.choice(np.frombuffer(b"ACGT", np.uint8), 60)
    if kind == "alike":
        return [base.tobytes()] * n
    out = []     # one key, told apart only behind the 28th byte
    for _ in range(n):
        s = base.copy()
        s[28 + int(rng.integers(0, 31))] = b"ACGT"[int(rng.integers(0, 4))]
        s[28 + int(rng.integers(0, 31))] = b"ACGTN"[int(rng.integers(0, 5))]
        out.append(s.tobytes())
    return out


# one tile of 1,024: its groups' work, n * n, passes 256 n + 4,096 from n = 272
@pytest.mark.parametrize("kind", ["alike", "behind"])
@pytest.mark.parametrize("n", [2, 271, 272, 300, 1023, 1024, 1025])
def test_one_group_of_ties(tmp_path, n, kind):
    reads = _reads(n, kind)
    eng = cg.Engine(0)          # nothing in its buffers yet
    try:
        _run(eng, tmp_path, reads)
        # buffers that held a larger set's order
        rng = np.random.default_rng(1)
        _run(eng, tmp_path, [rng.choice(np.frombuffer(b"ACGT", np.uint8), 40).tobytes() for _ in range(3000)])
        _run(eng, tmp_path, reads)
    finally:
        eng.close()


def test_ties_apart_in_every_tile(tmp_path):
    # 1,024 heads of 28 bases in turn, 4,200 times, each time with other tails:
    # no tile of 1,024 holds two equal keys, so the estimate sees no tie, but
    # every group is larger than those the settling knows the bounds of
    kinds, copies = 1024, 4200
    rng = np.random.default_rng(2)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    heads = np.unique(rng.integers(0, 4, (2 * kinds, 28)), axis=0)[:kinds]      # in order
    turn = rng.permutation(kinds)
    n = kinds * copies
    tails = rng.integers(0, 4, (n, 4))
    rows = np.empty((n, 35), np.uint8)
    rows[:, :2] = np.frombuffer(b">\n", np.uint8)
    rows[:, 2:30] = acgt[heads[np.tile(turn, copies)]]
    rows[:, 30:34] = acgt[tails]
    rows[:, 34] = 10
    path = str(tmp_path / "raw.fa")
    rows.tofile(path)
    raw = cg.RawReads(path)
    assert raw.n == n
    eng = cg.Engine(0)
    try:
        index, freq, _ = eng.preprocess(raw)
    finally:
        eng.close()
        raw.close()
    code = np.tile(turn, copies) * 256 + tails @ np.array([64, 16, 4, 1])       # order of the bytes
    last = np.zeros(kinds * 256, np.int64)
    last[code] = np.arange(n)
    count = np.bincount(code, minlength=kinds * 256)
    assert np.array_equal(index, last[count > 0])
    assert np.array_equal(freq, count[count > 0])


# most reads tie in their keys: a shared head, with and without a byte among
# its first 16 that only has a range, reads that end before, at and behind the
# 16th and 28th byte, one length, one read in many copies
@pytest.mark.parametrize("n", [700, 1024, 6000])
@pytest.mark.parametrize("kind", ["head", "range early", "range late", "short", "copies"])
def test_sets_of_many_ties(tmp_path, n, kind):
    rng = np.random.default_rng(n)
    head = rng.choice(np.frombuffer(b"ACGT", np.uint8), 40)
    if kind == "range early":
        head[3] = ord("R")
    if kind == "range late":
        head[20] = ord("K")
    lo, hi = (12, 33) if kind == "short" else (60, 64)
    reads = []
    for _ in range(n):
        tail = rng.choice(np.frombuffer(b"ACGTN", np.uint8), hi - 40 if hi > 40 else 1)
        s = np.concatenate([head, tail])[:int(rng.integers(lo, hi))].copy()
        if kind.startswith("range"):        # told apart behind the range byte, before and after the 16th
            s[int(rng.choice([5, 14, 25]))] = b"ACGT"[int(rng.integers(0, 4))]
        if kind == "short":
            s[int(rng.integers(0, len(s)))] = b"ACGT"[int(rng.integers(0, 4))]
        s[-1] = b"ACGT"[int(rng.integers(0, 4))]
        reads.append(s.tobytes())
    if kind == "copies":
        reads = [reads[int(rng.integers(0, 5))] if i % 3 else reads[i] for i in range(n)]
    eng = cg.Engine(0)
    try:
        _run(eng, tmp_path, reads)
    finally:
        eng.close()
