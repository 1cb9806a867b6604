"""The work a user of the BPMax fill has it do, as cases that can be timed and compared.

Every case goes through the public entry points of ``bpmax_b200`` on host sequences, as a program that
folds strand pairs calls them: scores and windows of one pair, whole tables in both layouts, uneven batches, one call
per pair, and gradients with respect to the scoring weights. A state holds an engine (the handle such a
program keeps) with its weights set, and the sequences.
"""
import numpy as np
import torch

from bpmax_b200 import Engine, workloads as W
from bpmax_b200.api import score_noalloc

WEIGHTS = ("integer", "reference", "real")


def listed():
    return [
        # a short probe against a short target, one call at a time: the smallest ordinary call
        {"name": "score_37x23", "kind": "score", "m": 37, "n": 23, "weights": "real"},
        # the same call where no device memory may be allocated (another framework's pool)
        {"name": "noalloc_64x32", "kind": "noalloc", "m": 64, "n": 32, "weights": "real"},
        # the plain single pair, whole table and score, in the compact layout
        {"name": "table_128x32", "kind": "compact", "m": 128, "n": 32, "weights": "integer"},
        # the reference program's own fill call: its layout (32-wide tiles) and weights, pinned output
        {"name": "fill_128x64", "kind": "reference", "m": 128, "n": 64, "n_tile": 32, "weights": "reference"},
        # the "windows" cases: the score, and the optimum of strand 1 against every window of strand 2 (the
        # inner table of the last outer cell). An odd pair a little over one tile of strand 2, non-integer weights
        {"name": "score_90x130", "kind": "windows", "m": 90, "n": 130, "weights": "real"},
        # the single large pair: long strand 1, strand 2 of one tile
        {"name": "score_1024x64", "kind": "windows", "m": 1024, "n": 64, "weights": "integer"},
        # the balanced pair, GC-rich
        {"name": "score_256x256", "kind": "windows", "m": 256, "n": 256, "weights": "integer", "gc_rich": True},
        # short strand 1, long strand 2: the two smaller whole-fill shapes published for the reference
        {"name": "score_16x750", "kind": "windows", "m": 16, "n": 750, "weights": "integer"},
        {"name": "score_32x1024", "kind": "windows", "m": 32, "n": 1024, "weights": "integer"},
        # a screen: 512 uneven pairs in one call
        {"name": "batch_512", "kind": "batch", "pairs": 512, "m": 200, "n": 64, "weights": "integer"},
        # the same kind of pairs when they arrive one by one, every pair of another shape
        {"name": "each_24", "kind": "each", "pairs": 24, "m": 200, "n": 64, "weights": "integer"},
        # fitting the weights: scores and exact usage counts of a batch
        {"name": "grad_16x256x64", "kind": "grad", "pairs": 16, "m": 256, "n": 64, "weights": "real"},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["score", "windows", "noalloc", "compact", "reference", "long", "tiled", "wide", "batch", "each", "grad"])
    c = {"kind": kind, "weights": rng.choice(WEIGHTS)}
    if kind == "score":
        c.update(m=_log(rng, 12, 256), n=rng.randint(8, 64), weights="real")
    elif kind == "noalloc":
        c.update(m=rng.randint(8, 110), n=rng.randint(8, 64), weights="real")
    elif kind == "windows":
        c.update(m=_log(rng, 12, 256), n=rng.randint(8, 64))
    elif kind == "compact":
        c.update(m=_log(rng, 12, 128), n=rng.randint(8, 64))
    elif kind == "reference":
        c.update(m=_log(rng, 12, 128), n=rng.randint(17, 64), n_tile=rng.choice([8, 12, 16]))
    elif kind == "long":
        c.update(kind="windows", m=_log(rng, 257, 900), n=rng.randint(25, 64))
    elif kind == "tiled":
        c.update(kind="windows", m=_log(rng, 24, 200), n=_log(rng, 65, 256), gc_rich=rng.random() < 0.5)
    elif kind == "wide":
        c.update(kind="windows", m=rng.randint(4, 24), n=_log(rng, 321, 900))
    elif kind == "batch":
        c.update(pairs=_log(rng, 16, 384), m=rng.randint(60, 200), n=rng.randint(24, 64))
    elif kind == "each":
        c.update(pairs=rng.randint(4, 24), m=rng.randint(40, 200), n=rng.randint(24, 64))
    else:
        c.update(pairs=rng.randint(2, 16), m=rng.randint(40, 256), n=rng.randint(16, 64))
    return c


def _weights(case, seed):
    if case["weights"] == "real":
        return W.random_weights(seed + 1000)
    return (W.INTEGER_WEIGHTS if case["weights"] == "integer" else W.REFERENCE_WEIGHTS).copy()


def _shapes(case):
    """Strand lengths of every pair. Those of an uneven batch belong to the case: another seed gives
    other sequences of the same lengths."""
    if case["kind"] in ("batch", "each"):
        rng = np.random.default_rng(4)
        return [(int(rng.integers(16, case["m"] + 1)), int(rng.integers(8, case["n"] + 1))) for _ in range(case["pairs"])]
    return [(case["m"], case["n"])] * case.get("pairs", 1)


def _pairs(case, seed):
    rng = np.random.default_rng(seed)
    probs = W.GC_RICH if case.get("gc_rich") else None
    return [(W.random_sequence(m, rng, probs), W.random_sequence(n, rng, probs)) for m, n in _shapes(case)]


def prepare(case, seed):
    s = {"kind": case["kind"], "pairs": _pairs(case, seed), "weights": _weights(case, seed)}
    if case["kind"] != "noalloc":
        s["engine"] = Engine(0)
        s["engine"].set_weights(s["weights"])
    if case["kind"] == "reference":
        s["n_tile"] = case["n_tile"]
        n = Engine.reference_size(case["m"], case["n"], case["n_tile"])
        s["pinned"] = torch.zeros(n, dtype=torch.float32, pin_memory=True)
        s["out"] = s["pinned"].numpy()
    return s


def run(state):
    kind, pairs = state["kind"], state["pairs"]
    if kind == "noalloc":
        return score_noalloc(*pairs[0], state["weights"])
    eng = state["engine"]
    if kind == "score":
        return eng.score(*pairs[0])
    if kind == "windows":
        m, n = len(pairs[0][0]), len(pairs[0][1])
        return eng.score(*pairs[0]), eng.read_cells(0, 0, 1, m - 1, m, n)
    if kind == "compact":
        return eng.fill_compact(*pairs[0])
    if kind == "reference":
        return eng.fill(*pairs[0], state["n_tile"], out=state["out"])
    if kind == "batch":
        return eng.score_batch(pairs)
    if kind == "each":
        return eng.score_each(pairs)
    return eng.grad_batch(pairs)


def work(case):
    shapes = _shapes(case)
    terms = sum(W.terms(m, n)["total"] for m, n in shapes)
    out = 4 * len(shapes) * (13 if case["kind"] == "grad" else 1)
    if case["kind"] == "windows":
        out += 4 * case["n"] ** 2
    if case["kind"] == "compact":
        out += 4 * (case["m"] * (case["m"] + 1) // 2) * case["n"] ** 2
    if case["kind"] == "reference":  # the outer cells i1 <= j1 of the layout
        m = case["m"]
        out += 4 * Engine.reference_size(m, case["n"], case["n_tile"]) * (m + 1) // (2 * m)
    return {"bytes": 4 * sum(m + n for m, n in shapes) + out, "flops": 2 * terms}


# ---- the same values in 64 bits, from the recurrence alone -------------------------------------------

_TYPES = {(0, 3): 0, (3, 0): 1, (2, 1): 2, (1, 2): 3, (2, 3): 4, (3, 2): 5}  # AU UA GC CG GU UG


def _pair_scores(a, b, w6):
    t = np.zeros((5, 5))
    for (x, y), k in _TYPES.items():
        t[x, y] = w6[k]
    return t[np.ix_(a, b)]


def _strand(s, w6):
    """Single-strand table: 0 up to a span of 3, -inf below the diagonal."""
    n = len(s)
    pr = _pair_scores(s, s, w6)
    T = np.full((n, n), -np.inf)
    for d in range(n):
        for i in range(n - d):
            j = i + d
            T[i, j] = 0.0 if d <= 3 else max(T[i + 1, j - 1] + pr[i, j], (T[i, i:j] + T[i + 1:j + 1, j]).max())
    return T


def _table(seq1, seq2, w12):
    """F[i1, j1, i2, j2] over the reversed strand 2 in float64 (-inf outside both triangles)."""
    s1, s2 = np.asarray(seq1), np.asarray(seq2)[::-1]
    w = np.asarray(w12, dtype=np.float64)
    M, N, dev, inf = len(s1), len(s2), "cuda", float("inf")

    def on(x):
        return torch.from_numpy(np.ascontiguousarray(x)).to(dev)

    S1, S2 = on(_strand(s1, w[:6])), on(_strand(s2, w[:6]))
    pair1, pair2 = on(_pair_scores(s1, s1, w[:6])), on(_pair_scores(s2, s2, w[:6]))
    inter = on(_pair_scores(s1, s2, w[6:]))
    F = torch.full((M, M, N, N), -inf, dtype=torch.float64, device=dev)
    for d in range(M):
        i = torch.arange(M - d, device=dev)
        acc = S1[i, i + d][:, None, None] + S2
        if d >= 4:
            acc = torch.maximum(acc, F[i + 1, i + d - 1] + pair1[i, i + d][:, None, None])
        for w0 in range(0, d, max(1, 2 ** 26 // (len(i) * N * N))):  # k1 = i1 + split, some splits at a time
            sp = torch.arange(w0, min(d, w0 + max(1, 2 ** 26 // (len(i) * N * N))), device=dev)[None, :]
            A, B = F[i[:, None], i[:, None] + sp], F[i[:, None] + sp + 1, (i + d)[:, None]]
            a1, b1 = S1[i[:, None], i[:, None] + sp], S1[i[:, None] + sp + 1, (i + d)[:, None]]
            acc = torch.maximum(acc, (B + a1[:, :, None, None]).amax(1))
            acc = torch.maximum(acc, (A + b1[:, :, None, None]).amax(1))
            for k in range(N - 1):
                r = (A[:, :, :k + 1, k, None] + B[:, :, k + 1, None, k + 1:]).amax(1)
                acc[:, :k + 1, k + 1:] = torch.maximum(acc[:, :k + 1, k + 1:], r)
        if d == 0:
            acc.diagonal(0, 1, 2).copy_(inter)
        for e in range(N):
            v = acc.diagonal(e, 1, 2)
            if e >= 4:
                v.copy_(torch.maximum(v, acc.diagonal(e - 2, 1, 2)[:, 1:-1] + pair2.diagonal(e)))
            if e + 1 < N:  # every open entry takes its two terms that read diagonal e
                D = v.clone()
                r1, r2 = D[:, :-1, None] + S2[e + 1:], S2[:, :N - e - 1] + D[:, None, 1:]
                acc[:, :N - e - 1] = torch.maximum(acc[:, :N - e - 1], r1)
                acc[:, :, e + 1:] = torch.maximum(acc[:, :, e + 1:], r2)
        F[i, i + d] = acc
    return F


def exact(case, seed):
    shapes = _shapes(case)
    if sum(m * n for m, n in shapes) > 130_000 or sum(W.terms(m, n)["total"] for m, n in shapes) > 2.5e11:
        return None
    if max(m * m * n * n for m, n in shapes) > 5e8:
        return None
    w = _weights(case, seed)
    scores = []
    for s1, s2 in _pairs(case, seed):
        F = _table(s1, s2, w)
        scores.append(F[0, len(s1) - 1, 0, len(s2) - 1].item())
    if case["kind"] in ("batch", "each"):
        return np.array(scores)
    if case["kind"] == "grad":  # usage counts are whole numbers of one optimum: no rounding to compare
        return np.array(scores), None
    if case["kind"] == "compact":
        i, j = np.triu_indices(case["m"])
        T = F[torch.from_numpy(i).cuda(), torch.from_numpy(j).cuda()]
        return torch.where(torch.isinf(T), float(np.finfo(np.float32).min), T), scores[0]
    if case["kind"] == "windows":
        T = F[0, case["m"] - 1][None, None]
        return scores[0], torch.where(torch.isinf(T), float(np.finfo(np.float32).min), T)
    if case["kind"] == "reference":  # the table's layout is the reference's: the score alone
        return None, scores[0]
    return scores[0]
