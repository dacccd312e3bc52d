"""Workloads of the swap-search engine, for timing and for comparing outputs.

Each case is one call, or the few calls that belong together, that a program
using the engine makes through the Python binding: deltas of rows and pairs,
the delta table, the schedules (serial, batched), permutation sets, annealing
chains, subset re-assignment, loading a pair with its greedy start, and the
learned proposer's scoring and gradients.

Graph pairs come from the package's generator: the two density models of its
configurations (1: Pareto out-degrees, about 20 edges a vertex; 3: joint
power law, 80 edges a vertex; 2: the full-scale pair, n = 18,524 with 3 M
edges and a greedy-similarity start).  A pair of one size is generated once in
a process; every seed relabels the vertices of both sides by its own random
permutations, so graphs, mapping and rows all differ from seed to seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_HERE = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_HERE, "brain-match_b200", "python"))

import bmb200 as bm  # noqa: E402

FULL_N, FULL_M = 18524, 3_000_000


def listed():
    full = {"n": FULL_N, "edges": FULL_M}
    return [
        # the smallest call: one row on the small pair, as an interactive or serial caller asks for it
        {"name": "row_small", "kind": "rows", "n": 2000, "edges": 40_000, "rows": 1},
        # one step of a throughput search: 57 rows x 18,523 partners (2^20 candidates), heavy and light rows mixed
        {"name": "rows_step", "kind": "rows", **full, "rows": 57},
        # a million arbitrary candidate pairs (random partners from elsewhere, checked exactly)
        {"name": "pairs_1m", "kind": "pairs", **full, "pairs": 1 << 20},
        # every pair's delta and the 1,024 best swaps of it
        {"name": "table", "kind": "table", **full, "topk": 1024},
        # the whole batched search from the greedy start to its local optimum
        {"name": "climb", "kind": "climb", **full, "sweeps": -1},
        # the reference's serial first-improvement loop on the small pair: many dependent small launches
        {"name": "serial", "kind": "serial", "n": 2000, "edges": 40_000, "accepts": 400},
        # permutation sets: 4,096 random 8-sets, all 40,320 permutations of each
        {"name": "sets8", "kind": "sets", **full, "k": 8, "sets": 4096},
        # batched annealing chains on pairs of uneven size
        {"name": "anneal", "kind": "anneal", "n": 2709, "n_last": 8192, "pairs": 4, "chains": 64, "steps": 100_000},
        # optimal re-assignment of random independent subsets of up to 4,096 members
        {"name": "assign", "kind": "assign", **full, "members": 4096, "iterations": 3},
        # what every program does first: load both graphs, make the greedy matching, set it, score it
        {"name": "start", "kind": "start", **full},
        # the learned proposer's scores of whole rows (tensor cores)
        {"name": "score_rows", "kind": "score", **full, "rows": 1184},
        # the learned proposer's training direction: loss and gradients of a minibatch
        {"name": "train", "kind": "train", "n": 2000, "edges": 40_000, "records": 8192},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    n = _log_uniform(rng, 500, FULL_N)
    edges = n * _log_uniform(rng, 20, min(160, n // 8))
    c = {"kind": rng.choice(["rows", "rows", "pairs", "table", "climb", "serial", "sets", "anneal", "assign", "start",
                             "score", "train"]), "n": n, "edges": edges}
    kind = c["kind"]
    if kind == "rows":
        c["rows"] = _log_uniform(rng, 1, 1000)
    elif kind == "pairs":
        c["pairs"] = _log_uniform(rng, 1, 1 << 20)
    elif kind == "table":
        c["topk"] = _log_uniform(rng, 1, 4096)
    elif kind == "climb":
        c["sweeps"] = rng.randint(1, 6)
    elif kind == "serial":
        c["n"] = min(n, 4000)
        c["edges"] = c["n"] * max(20, min(80, edges // n))
        c["accepts"] = _log_uniform(rng, 10, 400)
    elif kind == "sets":
        c["k"] = rng.randint(2, 8)
        c["sets"] = _log_uniform(rng, 16, 4096 if c["k"] == 8 else 65536)
    elif kind == "anneal":
        c = {"kind": kind, "n": min(n, 6000), "n_last": min(8192, n + _log_uniform(rng, 10, 2000)),
             "pairs": rng.randint(1, 4), "chains": _log_uniform(rng, 4, 96), "steps": _log_uniform(rng, 1000, 100_000)}
        c["n_last"] = max(c["n_last"], c["n"])
    elif kind == "assign":
        c["members"] = _log_uniform(rng, 8, 4096)
        c["iterations"] = rng.randint(1, 3)
    elif kind == "score":
        c["rows"] = _log_uniform(rng, 1, 1184)
    elif kind == "train":
        c["records"] = _log_uniform(rng, 64, 65536)
    return c


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=24)
def _base(n, edges):
    """(A, B, initial mapping) of one size: the configuration nearest to it."""
    if (n, edges) == (FULL_N, FULL_M):
        A, B, _, init = bm.gen_pair(2)
    elif edges <= 40 * n:
        A, B, _, init = bm.gen_pair(1, n=n, m_target=edges, max_degree=max(4, n // 4))
    else:
        A, B, _, init = bm.gen_pair(3, n=n, m_target=edges, max_degree=max(16, min(8000, n // 2)))
    return A, B, init


def _pair(n, edges, rng):
    """The base pair with both sides' vertices relabelled by rng's permutations."""
    A, B, init = _base(n, edges)
    pa = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    pb = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    pi = np.zeros(n + 1, np.int32)
    pi[pa] = pb[init]
    pi[0] = 0
    return (bm.Graph(n, pa[A.src], pa[A.dst], A.w), bm.Graph(n, pb[B.src], pb[B.dst], B.w), pi)


def _rows(A, count, rng):
    """`count` distinct rows spread over the weighted-degree ordering, as the
    ordering-driven schedules meet them."""
    wdeg = np.bincount(A.src, A.w, A.n + 1)[1:] + np.bincount(A.dst, A.w, A.n + 1)[1:]
    order = (np.argsort(-wdeg, kind="stable") + 1).astype(np.int32)
    start = int(rng.integers(0, A.n))
    return np.ascontiguousarray(np.roll(order, -start)[:min(count, A.n)])


def _glorot(rng):
    def u(fan_in, fan_out, size):
        lim = math.sqrt(6.0 / (fan_in + fan_out))
        return rng.uniform(-lim, lim, size)
    w = np.concatenate([u(24, 128, 24 * 128), rng.uniform(-0.1, 0.1, 128), u(128, 128, 128 * 128),
                        rng.uniform(-0.1, 0.1, 128), u(128, 1, 128), [0.05]])
    return w.astype(np.float32)


def _records(k, rng):
    """Feature rows as pairs of the power-law graphs have them (logs of
    degrees and weights, adjacency bits) and targets sign(d) log1p(|d|) / 8."""
    x = np.abs(rng.normal(4.0, 1.5, (k, 24)))
    x[:, 16:20] = np.abs(rng.normal(0.0, 1.0, (k, 4)))
    x[:, 20:22] = rng.random((k, 2)) < 0.03
    x[:, 22] = np.abs(rng.normal(0.0, 1.5, k))
    d = rng.normal(-100, 400, k)
    return x.astype(np.float32), (np.sign(d) * np.log1p(np.abs(d)) / 8).astype(np.float32)


class _State:
    """What the user's program holds: the engine with its inputs."""

    def __init__(self, case):
        self.case = case
        self.eng = None

    def __del__(self):
        if self.eng is not None:
            self.eng.close()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State(case)
    kind = case["kind"]
    s.eng = bm.Engine(0)
    if kind == "anneal":
        s.batch = bm.Batch(s.eng)
        inits = []
        for i in range(case["pairs"]):
            n = case["n"] + (case["n_last"] - case["n"]) * i // max(1, case["pairs"] - 1)
            A, B, pi = _pair(n, 80 * n, rng)
            s.batch.add_pair(A, B)
            inits.append(pi)
        s.chain_pair = (np.arange(case["chains"]) % case["pairs"]).astype(np.int32)
        s.keys = rng.integers(1, 1 << 62, case["chains"]).astype(np.uint64)
        s.inits = [inits[p] for p in s.chain_pair]
        return s
    s.A, s.B, s.pi = _pair(case["n"], case["edges"], rng)
    if kind == "start":
        return s
    s.eng.set_graphs(s.A, s.B)
    s.eng.set_mapping(s.pi)
    n = case["n"]
    if kind == "rows":
        s.rows = _rows(s.A, case["rows"], rng)
    elif kind in ("climb", "serial"):
        s.rows = _rows(s.A, n, rng)
    elif kind == "pairs":
        s.pairs = rng.integers(1, n + 1, (case["pairs"], 2)).astype(np.int32)
    elif kind == "table":
        s.ld = (n + 1 + 3) & ~3
        s.table = torch.zeros((n + 1, s.ld), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
    elif kind == "sets":
        k, count = case["k"], case["sets"]
        base = rng.integers(0, n, count)
        step = np.sort(rng.random((count, k - 1)), axis=1) * (n - k)  # distinct members: increasing offsets
        off = np.concatenate([np.zeros((count, 1), np.int64), step.astype(np.int64) + np.arange(1, k)], axis=1)
        s.sets = ((base[:, None] + off) % n + 1).astype(np.int32)
    elif kind == "score":
        s.mlp = bm.Mlp(s.eng, seed=1)
        s.mlp.set_params(_glorot(rng))
        s.rows = torch.from_numpy(_rows(s.A, case["rows"], rng)).cuda()
        s.scores = torch.zeros((s.rows.numel(), n), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
    elif kind == "train":
        s.mlp = bm.Mlp(s.eng, seed=1)
        s.mlp.set_params(_glorot(rng))
        s.x, s.y = _records(case["records"], rng)
    return s


# -------------------------------------------------------------------- passes

def _row_results(r):
    return {name: r[name].copy() for name in r.dtype.names}


def run(s):
    c, e = s.case, s.eng
    kind = c["kind"]
    if kind == "rows":
        return _row_results(e.rows_best(s.rows))
    if kind == "pairs":
        return e.delta_pairs(s.pairs)
    if kind == "table":
        e.delta_table_dev(s.table.data_ptr(), s.ld)
        pairs, deltas = e.table_topk(s.table.data_ptr(), s.ld, c["topk"])
        return {"table": s.table, "pairs": pairs, "deltas": deltas}
    if kind == "climb":
        e.set_mapping(s.pi)
        prog, _ = e.search_batched(s.rows, max_sweeps=c["sweeps"])
        return {"pi": e.get_mapping(), "score": prog.score, "accepts": prog.accepts}
    if kind == "serial":
        e.set_mapping(s.pi)
        prog, _ = e.sweep_parity(s.rows, max_accepts=c["accepts"])
        return {"pi": e.get_mapping(), "score": prog.score, "accepts": prog.accepts}
    if kind == "sets":
        best, perm = e.kset_eval(c["k"], s.sets)
        return {"best": best, "perm": perm}
    if kind == "anneal":
        pis, scores, accepts, _ = s.batch.sa_run(s.chain_pair, s.keys, s.inits, c["steps"], t0=5.0, t_end=0.01,
                                                 candidates=8)
        return {"pi": np.concatenate(pis), "scores": scores, "accepts": accepts}
    if kind == "assign":
        e.set_mapping(s.pi)
        prog, _ = e.search_hungarian(k=c["members"], seed=5, iterations=c["iterations"])
        return {"pi": e.get_mapping(), "score": prog.score, "moved": prog.accepts}
    if kind == "start":
        e.set_graphs(s.A, s.B)
        pi = e.greedy_match(s.A, s.B)
        e.set_mapping(pi)
        return {"pi": pi, "score": e.score(), "overlap": e.overlap()}
    if kind == "score":
        s.mlp.score_rows_dev(s.rows.data_ptr(), s.rows.numel(), s.scores.data_ptr())
        s.mlp.status()
        return s.scores
    if kind == "train":
        g, loss = s.mlp.gradients(s.x, s.y)
        return {"grads": g, "loss": np.float32(loss)}
    raise ValueError(kind)


# ---------------------------------------------------------------- necessity

def work(case):
    """Bytes and operations a pass cannot do without: every list that it has
    to look at once, from memory once, and every output once; two operations
    (minimum and sum) for each list entry that meets a candidate."""
    kind = case["kind"]
    if kind == "anneal":
        n = (case["n"] + case["n_last"]) / 2
        graphs = case["pairs"] * 4 * 80 * n * 4
        return {"bytes": graphs + 8 * case["chains"] * n, "flops": 2.0 * case["chains"] * case["steps"] * 4 * 80}
    n, m = case["n"], case["edges"]
    lists = 4 * 4.0 * m  # out- and in-lists of both graphs, 4 bytes an entry
    deg = m / n
    hop2 = 4 * deg * deg  # second-hop entries of an average row, without the hubs' share
    if kind == "rows":
        r = min(case["rows"], n)
        return {"bytes": min(lists, 4 * r * hop2) + r * 36, "flops": 2 * r * hop2}
    if kind == "pairs":
        k = case["pairs"]
        return {"bytes": min(lists, 4 * k * 4 * deg) + 16 * k, "flops": 2 * k * 4 * deg * 2}
    if kind == "table":
        return {"bytes": lists + 4.0 * n * n, "flops": 2 * n * hop2}
    if kind in ("climb", "serial"):
        sweeps = (max(1, case["sweeps"]) if case["sweeps"] > 0 else 10) if kind == "climb" else 1
        return {"bytes": lists + 12 * n, "flops": 2 * sweeps * n * hop2}
    if kind == "sets":
        k, s = case["k"], case["sets"]
        return {"bytes": min(lists, 16 * s * k * deg) + s * (8 * k + 8),
                "flops": s * (2.0 * math.factorial(k) + 4 * k * k * deg)}
    if kind == "assign":
        k = min(case["members"], 1569)
        return {"bytes": case["iterations"] * (lists / 2 + 4.0 * k * k) + 12 * n, "flops": case["iterations"] * 2.0 * k * hop2}
    if kind == "start":
        return {"bytes": 2 * 12.0 * m + lists + 12 * n, "flops": 2 * n * hop2 / 2 + 7.0 * n * n}
    if kind == "score":
        r = min(case["rows"], n)
        return {"bytes": 4.0 * r * n + 48 * n, "flops": 2.0 * r * n * (24 * 128 + 128 * 128 + 128)}
    if kind == "train":
        k = case["records"]
        return {"bytes": 100.0 * k + 8 * 19713, "flops": 3 * 2.0 * k * (24 * 128 + 128 * 128 + 128)}
    raise ValueError(kind)


# -------------------------------------------------------------- exact values

def _mlp64(w):
    o, parts = 0, []
    for shape in ((24, 128), (128,), (128, 128), (128,), (128,), (1,)):
        k = int(np.prod(shape))
        parts.append(torch.from_numpy(w[o:o + k].astype(np.float64).reshape(shape)))
        o += k
    return parts


def _vertex_table64(A, B, pi):
    """Per-vertex quantities of the pair features, in 64 bits: (n+1) x 9."""
    n = A.n
    keys = B.src.astype(np.int64) * (n + 1) + B.dst
    order = np.argsort(keys, kind="stable")
    keys, bw = keys[order], B.w[order].astype(np.int64)
    want = pi[A.src].astype(np.int64) * (n + 1) + pi[A.dst]
    at = np.minimum(np.searchsorted(keys, want), len(keys) - 1)
    w_b = np.where(keys[at] == want, bw[at], 0)
    ov = np.minimum(A.w, w_b)

    def per(v, weights=None):
        return np.bincount(v, weights, n + 1)

    s = per(A.src, ov) + per(A.dst, ov)
    wout, win = per(A.src, A.w), per(A.dst, A.w)
    miss = per(A.src, w_b == 0) + per(A.dst, w_b == 0)
    t = np.stack([per(A.src), per(A.dst), wout, win, s, np.maximum(wout + win - s, 0), miss, per(B.src)[pi],
                  per(B.dst)[pi]], 1)
    t = np.log1p(t)
    t[0] = 0
    return t, keys


def exact(case, seed):
    """64-bit values of the floating-point outputs.  The other cases return
    whole numbers, which admit no error and so need no value here."""
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "train":
        _pair(case["n"], case["edges"], rng)
        w = _glorot(rng)
        x, y = _records(case["records"], rng)
        params = [p.requires_grad_(True) for p in _mlp64(w)]
        w1, b1, w2, b2, w3, b3 = params
        xd, yd = torch.from_numpy(x).double(), torch.from_numpy(y).double()
        h = torch.relu(torch.relu(xd @ w1 + b1) @ w2 + b2)
        loss = ((h @ w3 + b3 - yd) ** 2).mean()
        loss.backward()
        return {"grads": torch.cat([p.grad.reshape(-1) for p in params]), "loss": loss.detach()}
    if kind == "score":
        A, B, pi = _pair(case["n"], case["edges"], rng)
        n = A.n
        w1, b1, w2, b2, w3, b3 = [p.to(dev) for p in _mlp64(_glorot(rng))]
        rows = _rows(A, case["rows"], rng)
        if dev == "cpu" and rows.size * n > 2_000_000:
            return None
        table, keys = _vertex_table64(A, B, pi)
        t = torch.from_numpy(table[1:]).to(dev)
        keys = torch.from_numpy(keys).to(dev)
        img = torch.from_numpy(pi[1:].astype(np.int64)).to(dev)
        out = torch.empty((rows.size, n), dtype=torch.float64, device=dev)

        def present(want):
            at = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
            return (keys[at] == want).double()

        for i, u in enumerate(rows.tolist()):
            a, b = t[u - 1], t
            fu = img[u - 1]
            x = torch.empty((n, 24), dtype=torch.float64, device=dev)
            x[:, 0:7], x[:, 7] = a[0:7], a[7] + a[8]
            x[:, 8:15], x[:, 15] = b[:, 0:7], b[:, 7] + b[:, 8]
            x[:, 16], x[:, 17] = (a[0] - b[:, 7]).abs(), (a[1] - b[:, 8]).abs()
            x[:, 18], x[:, 19] = (b[:, 0] - a[7]).abs(), (b[:, 1] - a[8]).abs()
            x[:, 20], x[:, 21] = present(fu * (n + 1) + img), present(img * (n + 1) + fu)
            x[:, 22], x[:, 23] = (a[4] - b[:, 4]).abs(), a[5] + b[:, 5]
            h = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2)
            out[i] = h @ w3 + b3
            out[i, u - 1] = -math.inf
        return out
    return None
