"""The measured workloads: what a search, a campaign or a learned ruin has
this engine do, each as ONE call sequence through the public entry points.

A case is a dict of plain values.  ``kind`` picks the sequence:

* ``search``: the state of a search on one cell (``GpuBackend``): the code
  recounted, its deficit, the gain map with its maximum, histogram and either
  the extraction a lazy greedy refreshes its heap from (``extract`` words at
  most) or the values at sampled candidates, the loss map read at the
  incumbents;
* ``queries``: exact per-candidate answers on one state: one large call of
  each coverage role, the small calls of a polish, single-word updates;
* ``lns``: ruin-and-repair rounds: losses, a ruin of the weakest incumbents,
  the device repair, the peel's check, one swap evaluation a round;
* ``batch``: a campaign's tick (``BatchEngine``): every cell's cnt, gain and
  loss in one launch, its scalars, one batched greedy for every cell;
* ``design``: the same state of a search on a covering design C(v,k,t);
* ``scorer``: the ruin scorer's logits for a round's incumbents and one
  gradient over a slice of the move log.

The ABI holds one cell per process, so the backend of a cell is opened once
and shared by every state on it; each pass starts from its own code.
Results are integers throughout (exact by construction, so there is nothing
to compare in 64 bits), except the scorer's, which ``exact`` restates.
"""
import math
from math import comb, prod

import numpy as np

from coldcore_b200.batch import BatchEngine
from coldcore_b200.gpu import GpuBackend
from coldcore_b200.incidence import GpuCoveringDesignBackend
from coldcore_b200.mlp import N_HID, N_IN, N_PARAMS, GpuMlp
from coldcore_b200.patterns import ball_size, wide_table


def listed():
    return [
        # the smallest call a user makes: a cell that a notebook or a unit
        # test searches, where launches and latency are everything
        {"name": "search K_3(8,2)", "kind": "search", "problem": "hamming",
         "axes": "3^8", "R": 2, "mu": 1, "words": 30, "extract": 4096},
        # a mixed-radix (football-pool like) cell covered twice: odd
        # strides, no power-of-two axis order, mu = 2 predicates
        {"name": "search 2^6 3^6 4^3 mu2", "kind": "search",
         "problem": "hamming", "axes": "2^6 3^6 4^3", "R": 2, "mu": 2,
         "words": 15000, "extract": 1 << 14},
        # a large ternary cell: the ordinary record-hunting size
        {"name": "search K_3(16,4)", "kind": "search", "problem": "hamming",
         "axes": "3^16", "R": 4, "mu": 1, "words": 1155, "extract": 1 << 15},
        # the largest single cell: the headline transform
        {"name": "search K_2(26,3)", "kind": "search", "problem": "hamming",
         "axes": "2^26", "R": 3, "mu": 1, "words": 20830,
         "extract": 1 << 15},
        # the Lee metric, about 60% covered
        {"name": "search Lee 7^8", "kind": "search", "problem": "lee",
         "axes": "7^8", "R": 4, "mu": 1, "words": 1460,
         "extract": 1 << 14},
        # king domination on a torus, two axes far above 16, at 3% density:
        # re-scored samples instead of a heap
        {"name": "search king 2048^2", "kind": "search",
         "problem": "torus_linf", "axes": "2048^2", "R": 1, "mu": 1,
         "words": 125829, "extract": 0},
        # per-candidate queries, 10^5 of them and the small calls around
        {"name": "queries K_3(16,4)", "kind": "queries",
         "problem": "hamming", "axes": "3^16", "R": 4, "mu": 1,
         "words": 1155, "cands": 100000, "updates": 64},
        # the LNS cell: four rounds of ruin and repair near a cover
        {"name": "lns K_3(14,3)", "kind": "lns", "problem": "hamming",
         "axes": "3^14", "R": 3, "mu": 1, "words": 6000, "rounds": 4,
         "ruin": 64},
        # a campaign of uneven cells, 10^3 to 10^7 words
        {"name": "batch 64 mixed", "kind": "batch", "cells": 64,
         "shapes": 7, "lo": 3.0, "hi": 7.0, "add": 16},
        # a campaign of small cells only: launches and tails dominate
        {"name": "batch 256 small", "kind": "batch", "cells": 256,
         "shapes": 11, "lo": 3.0, "hi": 5.0, "add": 16},
        # a covering design at its largest here: 5.9 M blocks, 70 of the
        # 27,405 four-subsets in each
        {"name": "design C(30,8,4)", "kind": "design", "v": 30, "k": 8,
         "t": 4, "mu": 1, "words": 900, "extract": 1 << 15},
        # the learned ruin's scorer: a K_3(14,3) round scored, and a slice
        # of the 10^5-move log in the backward direction
        {"name": "scorer 6104 / 20000", "kind": "scorer", "score": 6104,
         "train": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 5 + ["torus", "queries", "lns", "batch",
                                        "design", "scorer"])
    if kind == "torus":
        problem = rng.choice(["torus_linf", "grid_linf"])
        a, b = _log(rng, 40, 2048), _log(rng, 40, 2048)
        if rng.random() < 0.25:
            axes = [_log(rng, 17, 100) for _ in range(3)]
        else:
            axes = [a, b]
        size = prod(axes)
        return {"kind": "search", "problem": problem, "axes": _axes_text(axes),
                "R": rng.choice([1, 1, 2]), "mu": rng.choice([1, 1, 2]),
                "words": max(1, int(0.03 * size)), "extract": 0}
    if kind in ("search", "queries", "lns"):
        problem = "lee" if rng.random() < 0.25 else "hamming"
        q = rng.randint(2, 7)
        # the largest spaces are the binary and ternary ones
        top = 2.0 ** 24 if kind == "search" and q <= 3 else 4e6
        size = math.exp(rng.uniform(math.log(1e3), math.log(top)))
        if rng.random() < 0.3:
            axes = []
            while prod(axes) < size / 2 and len(axes) < 22:
                axes.append(rng.randint(2, 5))
            axes.sort()
        else:
            axes = [q] * max(3, round(math.log(size) / math.log(q)))
        R = rng.randint(1, min(4, len(axes)))
        mu = rng.choice([1, 1, 1, 2])
        ball = ball_size(axes, R, problem)
        frac = rng.uniform(0.3, 0.8)
        words = max(1, int(-math.log(1 - frac) * prod(axes) / ball * mu))
        case = {"kind": kind, "problem": problem, "axes": _axes_text(axes),
                "R": R, "mu": mu, "words": min(words, 60000)}
        if kind == "search":
            case["extract"] = rng.choice([4096, 1 << 14, 1 << 15])
        elif kind == "queries":
            case["cands"] = _log(rng, 64, 100000)
            case["updates"] = _log(rng, 1, 64)
        else:
            case["words"] = min(3 * words, 20000)
            case["rounds"] = rng.randint(1, 4)
            case["ruin"] = _log(rng, 8, 64)
        return case
    if kind == "batch":
        return {"kind": "batch", "cells": _log(rng, 4, 64),
                "shapes": rng.randint(0, 10 ** 6), "lo": 3.0,
                "hi": rng.uniform(4.0, 6.0), "add": _log(rng, 4, 16)}
    if kind == "design":
        k = rng.randint(4, 8)
        t = rng.randint(2, min(4, k - 1))
        v = rng.randint(k + 3, 28)
        return {"kind": "design", "v": v, "k": k, "t": t,
                "mu": rng.choice([1, 1, 2]),
                "words": max(2, comb(v, t) // (2 * comb(k, t))),
                "extract": 1 << 14}
    return {"kind": "scorer", "score": _log(rng, 64, 8192),
            "train": _log(rng, 64, 20000)}


# ---------------------------------------------------------------- the cells
def _axes_text(axes):
    """[2, 2, 3] -> "2^2 3^1": runs of equal axes in order."""
    out, i = [], 0
    while i < len(axes):
        j = i
        while j < len(axes) and axes[j] == axes[i]:
            j += 1
        out.append("%d^%d" % (axes[i], j - i))
        i = j
    return " ".join(out)


def _axes(text):
    return [int(a) for run in text.split()
            for a in [run.split("^")[0]] * int(run.split("^")[1])]


_OPEN = {"cell": None, "design": None}
_HANDLE = {}


def _shared(slot, key, make):
    """The one open backend of a library, reopened when the cell changes."""
    if _OPEN[slot] != key:
        if slot in _HANDLE:
            _HANDLE.pop(slot).close()
        _OPEN[slot] = None
        _HANDLE[slot] = make()
        _OPEN[slot] = key
    return _HANDLE[slot]


def _cell(case):
    axes = _axes(case["axes"])
    key = (case["problem"], tuple(axes), case["R"], case["mu"])
    return _shared("cell", key, lambda: GpuBackend(
        axes, case["R"], case["problem"], mu=case["mu"]))


def _design(case):
    key = (case["v"], case["k"], case["t"], case["mu"])
    return _shared("design", key, lambda: GpuCoveringDesignBackend(
        case["v"], case["k"], case["t"], mu=case["mu"]))


class _Batch:
    """A built batch that gives its memory back with its last reference."""

    def __init__(self, cells):
        self.engine = BatchEngine()
        for problem, axes, R, code in cells:
            self.engine.add(problem, axes, R, code)
        self.engine.build()
        for i, (problem, axes, R, _code) in enumerate(cells):
            self.engine.set_table(i, _table(problem, axes, R))

    def __del__(self):
        self.engine.close()


_TABLES = {}


def _table(problem, axes, R):
    """A cell's support table, enumerated once a program."""
    key = (problem, tuple(axes), R)
    if key not in _TABLES:
        if len(_TABLES) > 512:
            _TABLES.clear()
        _TABLES[key] = wide_table(axes, R, problem)
    return _TABLES[key]


def _code(rng, size, words):
    """``words`` distinct random words, sorted (never a permutation of the
    whole space: the large ones have 67 M words)."""
    got = np.unique(rng.integers(0, size, size=min(2 * size, words + words
                                                   // 8 + 16)))
    return np.sort(rng.permutation(got)[:words]).astype(np.int64)


def _shapes(case):
    """The batch's cells without their codes: q in 2..6, sizes log-uniform,
    R in 1..4, four fifths Hamming; the shapes follow ``shapes`` alone."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["cells"]):
        q = int(rng.integers(2, 7))
        n = max(1, round(rng.uniform(case["lo"], case["hi"]) * math.log(10)
                         / math.log(q)))
        R = min(int(rng.integers(1, 5)), n)
        problem = "hamming" if rng.random() < 0.8 else "lee"
        out.append((problem, (q,) * n, R))
    return out


_BALLS = {}


def _ball(problem, axes, R):
    key = (problem, tuple(axes), R)
    if key not in _BALLS:
        _BALLS[key] = ball_size(axes, R, problem)
    return _BALLS[key]


# ------------------------------------------------------------- preparation
def prepare(case, seed):
    rng = np.random.default_rng([seed, len(case)])
    kind = case["kind"]
    if kind == "scorer":
        mlp = GpuMlp(seed=0)
        p, X, T = _scorer_inputs(case, seed)
        mlp.set_params(p)
        return {"case": case, "mlp": mlp, "score": X[:case["score"]],
                "X": X[case["score"]:], "T": T}
    if kind == "batch":
        cells = []
        for problem, axes, R in _shapes(case):
            size = prod(axes)
            M = max(1, min(size, int(math.log(2.0) * size
                                     / _ball(problem, axes, R))))
            cells.append((problem, axes, R, _code(rng, size, M)))
        return {"case": case, "batch": _Batch(cells),
                "add": [case["add"]] * len(cells)}
    if kind == "design":
        b = _design(case)
        return {"case": case,
                "code": _code(rng, b.n_cand, min(case["words"],
                                                 b.n_cand // 2))}
    b = _cell(case)
    size = b.space.size
    code = _code(rng, size, min(case["words"], size // 2))
    state = {"case": case, "code": code}
    if kind == "search":
        state["cands"] = rng.integers(0, size, size=4096)
    elif kind == "queries":
        state["cands"] = rng.integers(0, size, size=case["cands"])
        fresh = np.setdiff1d(rng.integers(0, size,
                                          size=2 * case["updates"]), code)
        state["fresh"] = rng.permutation(fresh)[:case["updates"]]
    else:
        state["swap"] = rng.integers(0, size, size=64)
    return state


def _scorer_inputs(case, seed):
    """Random weights at their usual scale, features in [0, 1] like the
    ruin's (fractions of balls and ranks), and 0 / 1 labels."""
    rng = np.random.default_rng(seed)
    n = case["score"] + case["train"]
    X = rng.random((n, N_IN)).astype(np.float32)
    T = (rng.random(case["train"]) < 0.2).astype(np.float32)
    parts = [rng.normal(0, math.sqrt(2 / N_IN), N_IN * N_HID),
             rng.normal(0, 0.05, N_HID),
             rng.normal(0, math.sqrt(2 / N_HID), N_HID * N_HID),
             rng.normal(0, 0.05, N_HID),
             rng.normal(0, math.sqrt(1 / N_HID), N_HID),
             rng.normal(0, 0.05, 1)]
    return np.concatenate(parts).astype(np.float32), X, T


# ------------------------------------------------------------------ passes
def run(state):
    return _PASS[state["case"]["kind"]](state)


def _filled(a, n, dtype=np.int64):
    """``a`` at the start of an array of n, the rest -1."""
    out = np.full(n, -1, dtype=dtype)
    out[:len(a)] = a
    return out


def _refresh(b, cap):
    """A lazy greedy's heap refresh from the current gain map: the smallest
    threshold whose entries fit, its entries in index order."""
    mx = b.map_max()
    hist = b.map_hist(1024, max(1, mx))
    tail = np.cumsum(hist[::-1], dtype=np.int64)[::-1]
    fits = np.flatnonzero(tail <= cap)
    idx = val = np.zeros(0, dtype=np.int64)
    found = 0
    if mx >= 1 and len(fits):
        # bin i holds the values v with (v - 1) * 1024 // mx == i
        thr = -(-int(fits[0]) * mx // 1024) + 1
        if thr <= mx:
            idx, val, found = b.map_extract(thr, cap=cap)
            order = np.argsort(idx)
            idx, val = idx[order], val[order]
    return {"max": mx, "hist": hist, "found": found,
            "idx": _filled(idx, cap), "val": _filled(val, cap, np.int32)}


def _search(state):
    case = state["case"]
    b = _cell(case)
    b.recount(state["code"])
    out = {"deficit": b.uncovered()}
    b.gain_map()
    if case["extract"]:
        out["gain"] = _refresh(b, case["extract"])
    else:
        mx = b.map_max()
        out["gain"] = {"max": mx, "hist": b.map_hist(1024, max(1, mx)),
                       "at": b.map_read_at(state["cands"])}
    b.loss_map()
    out["loss"] = b.map_read_at(state["code"])
    return out


def _queries(state):
    b = _cell(state["case"])
    cands, code, fresh = state["cands"], state["code"], state["fresh"]
    b.recount(code)
    out = [b.ball_gather(cands, 0), b.ball_gather(cands, 1)]
    # a polish: single words in, the best few candidates re-scored
    for i, w in enumerate(fresh.tolist()):
        b.ball_update([w], +1)
        if i % 8 == 7:
            out.append(b.ball_gather(cands[i:i + 64], 0))
    out.append(b.uncovered())
    return out


def _lns(state):
    case = state["case"]
    b = _cell(case)
    code = state["code"]
    b.recount(code)
    out = [b.uncovered()]
    for r in range(case["rounds"]):
        b.loss_map()
        loss = b.map_read_at(code)
        k = min(case["ruin"] * (r + 1), len(code) - 1)
        pick = np.argsort(loss, kind="stable")[:k]
        b.ball_update(code[pick], -1)
        code = np.delete(code, pick)
        out += [_filled(loss, len(state["code"]), np.int32), b.uncovered()]
        placed, deficit = b.greedy_fill_device(k)
        code = np.sort(np.concatenate([code, placed]))
        out += [_filled(placed, k), deficit]
        out.append(_filled(b.ball_gather(code[:256], 1), 256, np.int32))
        out += list(b.swap_eval(code[:8], state["swap"]))
    return out


def _batch(state):
    e = state["batch"].engine
    e.run()
    scalars = e.scalars()
    got = e.greedy(np.arange(len(state["add"])), state["add"])
    return {"scalars": scalars,
            "placed": np.stack([_filled(p, n) for (p, _d), n
                                in zip(got, state["add"])]),
            "deficit": np.array([d for _p, d in got])}


def _design_pass(state):
    b = _design(state["case"])
    b.recount(state["code"])
    out = {"deficit": b.uncovered(), "cnt": b.read_cnt()}
    b.gain_map()
    out["gain"] = _refresh(b, state["case"]["extract"])
    b.loss_map()
    out["loss"] = b.map_read_at(state["code"])
    return out


def _scorer(state):
    return {"logits": state["mlp"].predict(state["score"]),
            "grad": state["mlp"].grad(state["X"], state["T"])}


_PASS = {"search": _search, "queries": _queries, "lns": _lns,
         "batch": _batch, "design": _design_pass, "scorer": _scorer}


# ------------------------------------------------------------- what it costs
def _field_bytes(space, words):
    """A state of one cell: the code read, cnt (2 bytes a word), the gain
    and loss maps (4 bytes a word each) written."""
    return 8 * words + 10 * space


def work(case):
    kind = case["kind"]
    if kind == "scorer":
        # forward 2 flops a weight, backward twice that
        mul = N_IN * N_HID + N_HID * N_HID + N_HID
        rows = case["score"] + case["train"]
        return {"bytes": 4 * (rows * (N_IN + 1) + 2 * N_PARAMS),
                "flops": 2 * mul * (rows + 2 * case["train"])}
    if kind == "batch":
        total = 0
        for problem, axes, R in _shapes(case):
            size = prod(axes)
            total += _field_bytes(size, 0.7 * size
                                  / _ball(problem, axes, R))
        return {"bytes": total, "flops": 0}
    if kind == "design":
        # cnt over the universe, both fields over the candidates
        cand, univ = comb(case["v"], case["k"]), comb(case["v"], case["t"])
        return {"bytes": 8 * case["words"] + 4 * univ + 8 * cand, "flops": 0}
    space = prod(_axes(case["axes"]))
    if kind == "search":
        return {"bytes": _field_bytes(space, case["words"]), "flops": 0}
    if kind == "queries":
        return {"bytes": 8 * case["words"] + 2 * space
                + 2 * 12 * case["cands"], "flops": 0}
    # a loss and a gain map a round
    return {"bytes": 8 * case["words"] + 2 * space
            + case["rounds"] * 8 * space, "flops": 0}


# -------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The scorer in float64: logits of the ReLU net, and the gradient of
    the mean binary cross-entropy with logits."""
    if case["kind"] != "scorer":
        return None                       # integers: compared as they are
    p, X, T = (a.astype(np.float64) for a in _scorer_inputs(case, seed))
    at = np.cumsum([N_IN * N_HID, N_HID, N_HID * N_HID, N_HID, N_HID])
    W1, b1, W2, b2, w3, b3 = np.split(p, at)
    W1, W2 = W1.reshape(N_IN, N_HID), W2.reshape(N_HID, N_HID)

    def forward(x):
        h1 = np.maximum(x @ W1 + b1, 0)
        h2 = np.maximum(h1 @ W2 + b2, 0)
        return h1, h2, h2 @ w3 + b3

    logits = forward(X[:case["score"]])[2]
    x = X[case["score"]:]
    h1, h2, y = forward(x)
    dy = (1 / (1 + np.exp(-y)) - T) / len(T)
    d2 = np.where(h2 > 0, dy[:, None] * w3, 0)
    d1 = np.where(h1 > 0, d2 @ W2.T, 0)
    grad = [x.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ dy, [dy.sum()]]
    return {"logits": logits,
            "grad": np.concatenate([np.ravel(g) for g in grad])}
