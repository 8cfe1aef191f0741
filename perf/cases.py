"""Performance cases: the work a user of crispy_gb300 has it do.

Every case goes through the package's public classes (Engine, Server,
RawReads) from host buffers to host results, as the drop-in programs do: the
reads of a job are uploaded, the k-mer structures built, both stages run and
their results fetched, in every pass.  A program that runs job after job keeps
one Engine (one Server), so the cases share one per process.

Read sets follow the package's own workload definition (crispy_gb300/synth.py:
OTU centroids around one root, reads with 0-3 % substitutions and
homopolymer-length indels, duplicates removed, ordered by (length, bytes) as
the preprocess step orders its output), drawn on the GPU from the seed.

Kinds:
    job    kmerDist -> genDist on one read set in one process (crispyDist)
    kmer   kmerDist alone with its pairs and distances fetched (kmerDist -d)
    gen    genDist alone on a given pair list (genDist -b B)
    align  per-pair alignment results (score, mismatches, length) of a few pairs
    serve  a burst of small jobs through the continuous-batching server
    pre    preprocess: filters and duplicate merge of raw reads
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import crispy_gb300 as cg

# codes 0..3 in ASCII order
_ASCII = (65, 67, 71, 84)
_WINDOW = 589824

# 16S-like read lengths: (root length, distribution, a, b); "normal" has mean a
# and deviation b, "uniform" runs from a to b
_LENGTHS = {
    "v250": (260, "normal", 250, 15),       # one hypervariable region, trimmed
    "v250w": (260, "normal", 250, 30),      # the same, less evenly trimmed
    "r300_500": (520, "uniform", 300, 500),  # ragged pyrosequencing reads
    "r1200_1600": (1650, "uniform", 1200, 1600),  # near full-length genes
    "r1800_2048": (2100, "uniform", 1800, 2048),  # up to the length limit
}


def _job(name, n, cents, lengths, k, band):
    return {"name": name, "kind": "job", "n": n, "cents": cents, "lengths": lengths, "k": k, "band": band}


def listed():
    return [
        # a handful of pairs checked by hand: the smallest call, all latency
        {"name": "align_200", "kind": "align", "n": 128, "cents": 4, "lengths": "v250", "pairs": 200, "band": 10},
        # a pilot sample of one region (the benchmark's small_1k set)
        _job("job_1k", 1000, 40, "v250", 6, 10),
        # an ordinary sample (plain_20k)
        _job("job_20k", 20000, 400, "v250", 6, 10),
        # a large sample of ragged reads, the benchmark's headline (uneven_100k)
        _job("job_100k", 100000, 1500, "r300_500", 6, 10),
        # the largest: a whole sequencing run at k = 8 (stress_500k)
        _job("job_500k_k8", 500000, 5000, "v250w", 8, 5),
        # kmerDist alone on near full-length genes
        {"name": "kmer_8k_long", "kind": "kmer", "n": 8000, "cents": 200, "lengths": "r1200_1600", "k": 6,
         "thr": -1.0},
        # kmerDist alone at another k, an odd number of ragged reads
        {"name": "kmer_30k_k7", "kind": "kmer", "n": 30001, "cents": 500, "lengths": "r300_500", "k": 7,
         "thr": -1.0},
        # kmerDist with a user's loose cut (-t 0.3): many pairs survive
        {"name": "kmer_6k_loose", "kind": "kmer", "n": 6000, "cents": 120, "lengths": "v250", "k": 5, "thr": 0.3},
        # genDist at its default band of 2: wide bands
        {"name": "gen_band2", "kind": "gen", "n": 5000, "cents": 100, "lengths": "v250", "pairs": 60000, "band": 2},
        # genDist near the length limit: the 32-bit kernel
        {"name": "gen_long", "kind": "gen", "n": 1500, "cents": 30, "lengths": "r1800_2048", "pairs": 12000,
         "band": 10},
        # many users' small samples arriving together
        {"name": "serve_32", "kind": "serve", "jobs": 32, "n": 600, "cents": 24, "lengths": "v250", "k": 6,
         "band": 10},
        # the step before: a raw file's reads, one in three a duplicate
        {"name": "pre_60k", "kind": "pre", "n": 60000, "cents": 1000, "lengths": "v250", "dups": 0.33},
    ]


def _loose(k, thr):
    return thr >= 0.2 or k <= 4


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "kmer", "kmer", "gen", "gen", "align", "serve", "pre"])
    if kind == "align":
        return {"kind": kind, "n": rng.randint(20, 400), "cents": rng.randint(2, 6),
                "lengths": rng.choice(["v250", "v250w", "r300_500", "r1200_1600"]), "pairs": _log_int(rng, 20, 3000),
                "band": rng.choice([2, 3, 5, 10])}
    if kind == "gen":
        lengths = rng.choice(["v250", "v250w", "r300_500", "r1200_1600", "r1800_2048"])
        top = 20000 if lengths.startswith("r1") else 150000
        return {"kind": kind, "n": _log_int(rng, 300, 8000), "cents": rng.randint(10, 150), "lengths": lengths,
                "pairs": _log_int(rng, 500, top), "band": rng.choice([2, 3, 5, 10] if top > 20000 else [5, 10])}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(6, 40), "n": _log_int(rng, 200, 2000), "cents": rng.randint(8, 40),
                "lengths": rng.choice(["v250", "v250w", "r300_500"]), "k": rng.choice([6, 6, 7]),
                "band": rng.choice([5, 10])}
    if kind == "pre":
        return {"kind": kind, "n": _log_int(rng, 1000, 100000), "cents": rng.randint(20, 1500),
                "lengths": rng.choice(["v250", "v250w", "r300_500"]), "dups": rng.choice([0.1, 0.33, 0.6])}
    lengths = rng.choice(["v250", "v250w", "r300_500", "r300_500", "r1200_1600"])
    n = _log_int(rng, 400, 12000 if lengths == "r1200_1600" else 110000)
    cents = max(4, int(n * rng.uniform(0.01, 0.04)))
    if kind == "job":
        k = rng.choice([5, 6, 6, 6, 7, 8])
        band = rng.choice([5, 10, 10]) if n > 20000 else rng.choice([3, 5, 10, 10])
        return {"kind": kind, "n": n, "cents": cents, "lengths": lengths, "k": k, "band": band}
    k = rng.choice([4, 5, 6, 6, 7, 8])
    thr = rng.choice([-1.0, -1.0, 0.1, 0.2, 0.3])
    if _loose(k, thr):        # many pairs survive: smaller sets
        n = max(400, min(n // 10, 6000))
        cents = max(4, n // 50)
    return {"kind": kind, "n": n, "cents": cents, "lengths": lengths, "k": k, "thr": thr}


# ---------------------------------------------------------------------------
# Read sets
# ---------------------------------------------------------------------------

def _raw_reads(case, seed, dups=0.0):
    """(codes [n, width] uint8 on the GPU, lengths, centroid of each read), as
    a sequencer gives them: in no order, duplicates among them."""
    root_len, dist, a, b = _LENGTHS[case["lengths"]]
    n, cents, k = case["n"], case["cents"], case.get("k", 6)
    dev = torch.device("cuda")
    g = torch.Generator(dev).manual_seed(int(seed))

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=dev)

    def substitute(seqs, rate):
        hit = rand(*seqs.shape) < rate[:, None]
        shift = torch.randint(1, 4, seqs.shape, generator=g, device=dev, dtype=torch.uint8)
        return torch.where(hit, (seqs + shift) % 4, seqs)

    root = torch.randint(0, 4, (1, root_len), generator=g, device=dev, dtype=torch.uint8)
    centroids = substitute(root.expand(cents, -1), 0.03 + 0.12 * rand(cents))
    pick = torch.randint(0, cents, (n,), generator=g, device=dev)
    reads = substitute(centroids[pick], 0.03 * rand(n))
    u = rand(n, root_len)
    reps = torch.where(u < 0.0025, 0, torch.where(u < 0.005, 2, 1))
    row_len = reps.sum(1)
    flat = torch.repeat_interleave(reads.reshape(-1), reps.reshape(-1))
    if dist == "normal":
        want = torch.round(a + b * torch.randn(n, generator=g, device=dev))
    else:
        want = torch.randint(a, b + 1, (n,), generator=g, device=dev)
    length = torch.minimum(want.long().clamp(k + 1, 2048), row_len)
    start = torch.cumsum(row_len, 0) - row_len
    col = torch.arange(int(length.max()), device=dev)
    at = (start[:, None] + col).clamp_(max=flat.numel() - 1)
    codes = flat[at]
    codes[col >= length[:, None]] = 4
    if dups:
        same = torch.randint(0, n, (n,), generator=g, device=dev)
        src = torch.where(rand(n) < dups, same, torch.arange(n, device=dev))
        codes, length, pick = codes[src], length[src], pick[src]
    return codes, length, pick


def _ordered(codes, length, pick):
    """Sorted by (length, bytes) with duplicates removed."""
    n, width = codes.shape
    words = []
    for c in range(0, width, 21):
        part = codes[:, c:c + 21].long()
        w = torch.zeros(n, dtype=torch.long, device=codes.device)
        for j in range(part.shape[1]):
            w = w * 8 + part[:, j]
        words.append(w)
    order = torch.arange(n, device=codes.device)
    for w in reversed(words):
        order = order[torch.sort(w[order], stable=True).indices]
    order = order[torch.sort(length[order], stable=True).indices]
    differs = length[order][1:] != length[order][:-1]
    for w in words:
        differs |= w[order][1:] != w[order][:-1]
    order = order[torch.cat([torch.ones(1, dtype=torch.bool, device=codes.device), differs])]
    return codes[order], length[order], pick[order]


def _packed(codes, length):
    """Host buffers: bases back to back, offsets, lengths."""
    table = torch.tensor(_ASCII + (0,), dtype=torch.uint8, device=codes.device)
    buf = table[codes.long()][codes < 4].cpu().numpy()
    lens = length.to(torch.int32).cpu().numpy()
    offs = np.zeros(len(lens), np.int64)
    np.cumsum(lens[:-1], out=offs[1:])
    return buf, offs, lens


def _read_set(case, seed):
    return _ordered(*_raw_reads(case, seed))


def _pairs(case, seed, pick):
    """Pairs (row < col) of reads of the same OTU, in row order, as kmerDist
    leaves them for genDist."""
    g = torch.Generator(pick.device).manual_seed(int(seed) + 7919)
    m, n = case["pairs"], pick.numel()
    by = torch.sort(pick, stable=True).indices
    place = torch.empty_like(by)
    place[by] = torch.arange(n, device=pick.device)
    size = torch.bincount(pick)
    first = torch.cumsum(size, 0) - size
    a = torch.randint(0, n, (m,), generator=g, device=pick.device)
    own = size[pick[a]]
    step = 1 + (torch.rand(m, generator=g, device=pick.device) * (own - 1).clamp(min=1)).long()
    b = by[first[pick[a]] + (place[a] - first[pick[a]] + step) % own]
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    order = torch.sort(lo * n + hi).indices
    return torch.stack([lo, hi], 1)[order].to(torch.int32).cpu().numpy()


# ---------------------------------------------------------------------------
# What a program has in hand, and one pass
# ---------------------------------------------------------------------------

_KEPT = {}


def _room(case):
    """Results a program of this kind makes room for."""
    if case["kind"] in ("gen", "align"):
        return case["pairs"]
    n = case["n"]
    if case["kind"] == "pre":
        return n
    every = n * (n - 1) // 2
    if _loose(case["k"], case.get("thr", -1.0)):
        return every
    return case.get("jobs", 1) * min(every, 20000 + 20 * n + int(2 * n * n / case["cents"]))


class _Results:
    """The program's own result arrays, one pass's results after the other's
    in the same place; what lies behind a pass's results is zero."""

    def __init__(self, room):
        self.pairs = np.zeros((room, 2), np.int32)
        self.dists = np.zeros(room, np.float32)
        self.sizes = np.zeros(64, np.int64)
        self.used = 0

    def take(self, parts):
        at = 0
        self.sizes[:] = 0
        for c, (p, d) in enumerate(parts):
            m = len(p)
            if at + m > len(self.pairs) or c >= len(self.sizes):
                raise RuntimeError("more results than there is room for")
            self.pairs[at:at + m] = p
            self.dists[at:at + m] = d
            self.sizes[c] = m
            at += m
        if at < self.used:
            self.pairs[at:self.used] = 0
            self.dists[at:self.used] = 0
        self.used = at
        return self


def _engine():
    if "engine" not in _KEPT:
        _KEPT["engine"] = cg.Engine(0)
    return _KEPT["engine"]


def _server():
    if "server" not in _KEPT:
        _KEPT["server"] = cg.Server(0, 0, 4)
    return _KEPT["server"]


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind not in ("align", "pre"):
        state["results"] = _Results(_room(case))
    if kind == "serve":
        state["server"] = _server()
        state["sets"] = [_packed(*_read_set(case, seed * 64 + j)[:2]) for j in range(case["jobs"])]
        return state
    state["engine"] = _engine()
    if kind == "pre":
        codes, length, _ = _raw_reads(case, seed, case["dups"])
        buf, offs, lens = _packed(codes, length)
        data = buf.tobytes()
        with tempfile.TemporaryDirectory() as d:
            path = os.path.join(d, "raw.fa")
            with open(path, "wb") as f:
                f.write(b"".join(b">r%d\n%b\n" % (i, data[o:o + l])
                                 for i, (o, l) in enumerate(zip(offs.tolist(), lens.tolist()))))
            state["raw"] = cg.RawReads(path)
        return state
    codes, length, pick = _read_set(case, seed)
    state["reads"] = _packed(codes, length)
    n = len(state["reads"][2])
    if kind in ("gen", "align"):
        state["pair_list"] = _pairs(case, seed, pick)
    state["thr_k"] = cg.default_threshold(n, case.get("thr", -1.0), 0)
    state["thr_g"] = cg.default_threshold(n, -1.0, 1)
    return state


def run(state):
    kind = state["kind"]
    if kind == "serve":
        srv, counts, parts = state["server"], [], []
        ids = [srv.submit(*s, state["k"], state["band"]) for s in state["sets"]]
        for job in ids:
            srv.wait(job)
            kmer_pairs, chunks = srv.result(job)
            counts.append([kmer_pairs, sum(len(d) for _, _, d in chunks)])
            parts += [(p, d) for _, p, d in chunks]
        got = state["results"].take(parts)
        return {"counts": np.array(counts, np.int64), "pairs": got.pairs, "dists": got.dists}
    eng = state["engine"]
    if kind == "pre":
        index, freq, stats = eng.preprocess(state["raw"])
        out = np.zeros((2, state["n"]), np.int32)
        out[0, :len(index)], out[1, :len(freq)] = index, freq
        return {"index": out[0], "freq": out[1], "kept": stats["kept"], "merges": stats["merges"]}
    buf, offs, lens = state["reads"]
    if kind == "align":
        eng.gen_prepare(buf, offs, lens)
        dist, score, ml, al = eng.gen_align(state["pair_list"], state["band"], cg.MODE_BATCHED)
        return {"dist": dist, "score": score, "ml": ml, "al": al}
    if kind == "kmer":
        eng.kmer_prepare(buf, offs, lens, state["k"])
        count = eng.kmer_run(state["thr_k"], cg.MODE_BATCHED, True)
        got = state["results"].take([eng.kmer_fetch(count, True)])
        return {"kmer_pairs": count, "pairs": got.pairs, "dists": got.dists}
    if kind == "job":
        eng.kmer_prepare(buf, offs, lens, state["k"])
        count = eng.kmer_run(state["thr_k"], cg.MODE_BATCHED, False)
        eng.gen_prepare_from_kmer()
        chunks = eng.gen_run_from_kmer(state["band"], state["thr_g"], cg.MODE_BATCHED)
    else:
        count = len(state["pair_list"])
        eng.gen_prepare(buf, offs, lens)
        chunks = eng.gen_run(state["pair_list"], state["band"], state["thr_g"], cg.MODE_BATCHED)
    got = state["results"].take([(p, d) for _, p, d in chunks])
    return {"kmer_pairs": count, "chunks": got.sizes, "pairs": got.pairs, "dists": got.dists}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _mean_length(case):
    _, dist, a, b = _LENGTHS[case["lengths"]]
    return a if dist == "normal" else (a + b) / 2


def _band_cells(length, band):
    half = length if band <= 1 else length / band
    return length * min(length, 2 * half + 1)


def work(case):
    """Bytes: reads in, results out.  Operations: every pair of reads decided
    once (kmerDist), ten integer operations per band cell of the pairs that
    are aligned (genDist: symbol compare, three candidates, maximum and path)."""
    kind, length = case["kind"], _mean_length(case)
    if kind == "pre":
        return {"bytes": case["n"] * (length + 13.0) + case["n"] * 8.0, "flops": case["n"] * length}
    if kind in ("gen", "align"):
        m = case["pairs"]
        return {"bytes": case["n"] * (length + 12.0) + m * (8.0 + 16.0),
                "flops": 10.0 * m * _band_cells(length, case["band"])}
    jobs, n = case.get("jobs", 1), case["n"]
    decided = n * (n - 1) / 2
    # about a fifth of the pairs within an OTU pass the default cut
    kept = 0.2 * n * n / (2 * case["cents"])
    cells = kept * _band_cells(length, case["band"]) if kind != "kmer" else 0.0
    return {"bytes": jobs * (n * (length + 12.0) + kept * 12.0), "flops": jobs * (decided + 10.0 * cells)}


# ---------------------------------------------------------------------------
# The same results in plain torch, distances in 64 bits
# ---------------------------------------------------------------------------

def _keep(d32, thr):
    """dist < thr or |dist - thr| < 1e-5 (single-precision difference)."""
    t = torch.tensor(thr, dtype=torch.float32, device=d32.device)
    return (d32 < t) | ((d32 - t).abs().double() < 1e-5)


def _threshold(n, user, num):
    if 0.0 <= user <= 1.0:
        return float(np.float32(user))
    v = num / math.log2(n) if n > 500 else num / math.log10(n)
    return float(np.float32(min(v, 1.0)))


def _kmer_pairs(codes, length, k, thr):
    """All pairs within the k-mer cut in the reference's stage order:
    (pairs [m, 2], distances in 64 bits)."""
    n, width = codes.shape
    dev = codes.device
    two_bit = torch.tensor([0, 3, 1, 2, 0], device=dev)[codes.long()]
    tuples = (length - k + 1).clamp(min=0)
    counts = torch.zeros(n, 4 ** k, dtype=torch.int16, device=dev)
    one = torch.ones(n, 1, dtype=torch.int16, device=dev)
    code = torch.zeros(n, width - k + 1, dtype=torch.long, device=dev)
    for j in range(k):
        code = code * 4 + two_bit[:, j:width - k + 1 + j]
    for p in range(code.shape[1]):
        counts.scatter_add_(1, code[:, p:p + 1], one * (p < tuples[:, None]).to(torch.int16))
    levels = []
    for t in range(1, int(counts.max()) + 1):
        hit = counts >= t
        used = hit.any(0)
        levels.append(hit[:, used].half())
    x = torch.cat(levels, 1)
    del levels, counts
    found = []
    step = 2048
    for r in range(0, n, step):
        m = x[r:r + step] @ x[r:].T          # sums up to 2,048: whole in half precision
        low = torch.minimum(tuples[r:r + step, None], tuples[None, r:])
        d32 = 1.0 - m.float() / low.float()
        row = torch.arange(r, min(n, r + step), device=dev)
        ok = _keep(d32, thr) & (row[:, None] < torch.arange(r, n, device=dev)[None, :])
        at = ok.nonzero()
        found.append((at[:, 0] + r, at[:, 1] + r, m[at[:, 0], at[:, 1]].double(), low[at[:, 0], at[:, 1]].double()))
    row, col, m, low = (torch.cat(v) for v in zip(*found))
    dim = min(1536, int(4 * 8.0 ** (math.floor(math.log10(n)) - 1)))
    stages = (n + dim - 1) // dim
    stage = (row // dim) * stages + col // dim
    order = torch.sort((stage * n + row) * n + col).indices
    return torch.stack([row, col], 1)[order], (1.0 - m / low)[order]


def _align(codes, length, pairs, band):
    """Banded alignment of every pair by anti-diagonals: (score, mismatches
    and gap columns, alignment length).  Cell (i, j) of a pair is held at
    q = (i - j + half) / 2 of its anti-diagonal i + j."""
    dev = codes.device
    out = []
    at = 0
    l1, l2 = length[pairs[:, 0]], length[pairs[:, 1]]
    limit = torch.maximum(l1, l2) if band <= 1 else (l1 + l2) // (2 * band)
    half = int(limit.max()) + 1 if len(pairs) else 1
    step = max(1, 120_000_000 // (half + 1))
    q = torch.arange(half + 1, device=dev, dtype=torch.int32)[None, :]
    far = -1000000
    while at < len(pairs):
        s1, s2 = codes[pairs[at:at + step, 0]], codes[pairs[at:at + step, 1]]
        a1, a2 = l1[at:at + step, None].int(), l2[at:at + step, None].int()
        lim = limit[at:at + step, None].int()
        p, width = s1.shape
        zero = torch.zeros(p, half + 1, dtype=torch.int32, device=dev)
        # score, path code (1 diagonal, 2 left, 4 up), mismatches, length
        two = one = (zero, zero, zero, zero)
        best = [torch.full((p, 1), far, dtype=torch.int32, device=dev) for _ in range(2)]
        kept = [torch.zeros(p, 2, dtype=torch.int32, device=dev) for _ in range(2)]
        for s in range(0, int((a1 + a2).max()) + 1):
            odd = (s + half) & 1
            d = 2 * q - half + odd
            i, j = (s + d) // 2, (s - d) // 2

            def shift(v, by):     # neighbour with i - j changed by `by` on the diagonal before
                if odd:
                    return v if by < 0 else torch.nn.functional.pad(v[:, 1:], (0, 1))
                return torch.nn.functional.pad(v[:, :-1], (1, 0)) if by < 0 else v

            if s < 2:
                two, one = one, (zero, zero, zero, zero + s)
                continue
            up, left = [shift(v, 1) for v in one], [shift(v, -1) for v in one]
            hit = (torch.gather(s2, 1, (i - 1).clamp(0, width - 1).long().expand(p, -1))
                   == torch.gather(s1, 1, (j - 1).clamp(0, width - 1).long().expand(p, -1))).int()
            c_diag = two[0] + hit * 9 - 4
            c_up = torch.where((d + 1 <= lim) & (d + 1 >= -lim), up[0] - 10 * (up[1] & 1) - (up[1] >> 2), far)
            c_left = torch.where((d - 1 <= lim) & (d - 1 >= -lim),
                                 left[0] - 10 * (left[1] & 1) - ((left[1] >> 1) & 1), far)
            m = torch.maximum(c_diag, torch.maximum(c_up, c_left))
            on_diag, on_up = m == c_diag, m == c_up
            code = torch.where(on_diag, 1, torch.where(on_up, 4, 2))
            ml = torch.where(on_diag, two[2] + 1 - hit, torch.where(on_up, up[2], left[2]) + 1)
            al = torch.where(on_diag, two[3], torch.where(on_up, up[3], left[3])) + 1
            border = (i == 0) | (j == 0)
            cur = (torch.where(border, 0, m), torch.where(border, 0, code), torch.where(border, 0, ml),
                   torch.where(border, s, al))
            inside = (d <= lim) & (d >= -lim) & (i >= 1) & (j >= 1) & (i <= a2) & (j <= a1)
            for e, last in enumerate((inside & (i == a2), inside & (j == a1))):
                any_, idx = last.any(1, keepdim=True), last.int().argmax(1, keepdim=True)
                value = torch.gather(cur[0], 1, idx)
                take = any_ & (value >= best[e])
                best[e] = torch.where(take, value, best[e])
                kept[e] = torch.where(take, torch.cat([torch.gather(cur[2], 1, idx), torch.gather(cur[3], 1, idx)], 1),
                                      kept[e])
            two, one = one, cur
        col = best[0] > best[1]
        out.append(torch.cat([torch.where(col, best[0], best[1]), torch.where(col, kept[0], kept[1])], 1))
        at += step
    return torch.cat(out) if out else torch.zeros(0, 3, dtype=torch.int32, device=dev)


def _gen_dists(codes, length, pairs, band, thr):
    """Distances of the pairs within the genetic cut, chunk by chunk in the
    reference's order, in 64 bits."""
    r = _align(codes, length, pairs, band)
    d64 = r[:, 1].double() / r[:, 2].double()
    keep = _keep(r[:, 1].float() / r[:, 2].float(), thr)
    chunks, pending, held = [], [], 0
    for w in range(0, len(pairs), _WINDOW):
        part = d64[w:w + _WINDOW][keep[w:w + _WINDOW]]
        pending.append(part)
        held += len(part)
        if held >= _WINDOW:
            chunks.append(torch.cat(pending))
            pending, held = [], 0
    if held:
        chunks.append(torch.cat(pending))
    return [torch.sort(c).values for c in chunks]


def _filled(case, parts):
    """The distances in the program's result array, zero behind them."""
    out = torch.zeros(_room(case), dtype=torch.float64, device="cuda")
    at = 0
    for d in parts:
        out[at:at + len(d)] = d
        at += len(d)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "pre" or case.get("k") == 8:
        # whole numbers only; at k = 8 the count table of every read is too large
        return None
    if kind == "serve":
        parts = []
        for j in range(case["jobs"]):
            codes, length, _ = _read_set(case, seed * 64 + j)
            n = len(length)
            pairs, _ = _kmer_pairs(codes, length, case["k"], _threshold(n, -1.0, 2))
            parts += _gen_dists(codes, length, pairs, case["band"], _threshold(n, -1.0, 1))
        return {"counts": None, "pairs": None, "dists": _filled(case, parts)}
    codes, length, pick = _read_set(case, seed)
    n = len(length)
    if kind == "align":
        pairs = torch.from_numpy(_pairs(case, seed, pick)).long().to(codes.device)
        r = _align(codes, length, pairs, case["band"])
        return {"dist": r[:, 1].double() / r[:, 2].double(), "score": None, "ml": None, "al": None}
    if kind == "kmer":
        _, d64 = _kmer_pairs(codes, length, case["k"], _threshold(n, case["thr"], 2))
        return {"kmer_pairs": None, "pairs": None, "dists": _filled(case, [d64])}
    if kind == "gen":
        pairs = torch.from_numpy(_pairs(case, seed, pick)).long().to(codes.device)
    else:
        pairs, _ = _kmer_pairs(codes, length, case["k"], _threshold(n, -1.0, 2))
    parts = _gen_dists(codes, length, pairs, case["band"], _threshold(n, -1.0, 1))
    return {"kmer_pairs": None, "chunks": None, "pairs": None, "dists": _filled(case, parts)}
