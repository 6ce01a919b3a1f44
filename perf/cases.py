"""The workloads this engine is measured on: whole calls of the public Python entry points.

A case is a dict: `op` names the call, `kind`, `n`, `m` (and `gamma`, `dmax`, `abc`) the seeded
graph generator's setting, `k` the pattern size. The seed of `prepare` draws the graph, so
another seed is another graph of the same shape. Sizes are those of the benchmark
configurations (Erdos-Renyi 2,000 / 10,000; Chung-Lu 18,700 / 198,000; R-MAT of about 100,000
vertices / 1.08M edges and of about 321,000 / 1.05M; batches of Chung-Lu graphs) and of the
tests (R-MAT 2,000 / 8,000).
"""
from __future__ import annotations

import math
import tempfile
from itertools import combinations, permutations

import numpy as np
import torch

import dumato_b200 as dm
from dumato_b200 import workloads

ER, CHUNG_LU, RMAT = dm.GEN_ER, dm.GEN_CHUNG_LU, dm.GEN_RMAT
CAP = 12_000_000  # rows of a host-side enumeration that `exact` still does


def listed():
    cl18k = dict(kind=CHUNG_LU, n=18_700, m=198_000, gamma=2.1, dmax=500.0)
    rmat100k = dict(kind=RMAT, n=170_000, m=1_080_000)
    rmat317k = dict(kind=RMAT, n=1_400_000, m=1_050_000)
    rmat2k = dict(kind=RMAT, n=2_000, m=8_000)
    return [
        # the smallest call: triangles of a small sparse graph, all launch and call latency
        dict(name="clique3_er2k", op="clique", k=3, kind=ER, n=2_000, m=10_000),
        # the headline: every clique size 3..7 of a power-law graph in one launch
        dict(name="upto7_chunglu18k", op="upto", k=7, **cl18k),
        # one clique query on a large sparse skewed graph (few heavy roots, many empty ones)
        dict(name="clique7_rmat317k", op="clique", k=7, **rmat317k),
        # one clique query with wide roots (out-degrees up to about 170) and billions of cliques
        dict(name="clique6_rmat100k", op="clique", k=6, **rmat100k),
        # a pattern-aware query: 6-cliques missing one edge, on a small skewed graph
        dict(name="near6_rmat2k", op="near", k=6, **rmat2k),
        # 3-vertex motif census of a graph with hubs of degree 10,000
        dict(name="motif3_rmat100k", op="motif", k=3, **rmat100k),
        # 4-vertex motif census of a power-law graph (billions of subgraphs)
        dict(name="motif4_chunglu18k", op="motif", k=4, **cl18k),
        # 5-vertex motif census of a mid-size power-law graph
        dict(name="motif5_chunglu3k", op="motif", k=5, kind=CHUNG_LU, n=3_000, m=18_000, gamma=2.2, dmax=120.0),
        # 6-vertex motif census of a small sparse graph without hubs
        dict(name="motif6_er2k", op="motif", k=6, kind=ER, n=2_000, m=10_000),
        # a mining service's mix: many graphs of uneven size, one query each, one launch
        dict(name="batch24", op="batch", graphs=24, mix=4),
        # the reference's own flow: read an edgelist file, count one pattern, done
        dict(name="file4_rmat100k", op="file", k=4, **rmat100k),
        # train the work predictor on a subtree log (forward, backward, Adam), then count with it
        dict(name="learn5_chunglu18k", op="learn", k=5, epochs=4, batch=256, **cl18k),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, n_lo, n_hi, avg_hi, kinds=(ER, CHUNG_LU, RMAT), hub=25.0):
    kind = rng.choice(kinds)
    n = _log_int(rng, n_lo, n_hi)
    avg = min(rng.uniform(4.0, avg_hi), (n - 1) / 4.0)
    m = min(int(n * avg / 2), 1_080_000)
    c = dict(kind=kind, n=n, m=m)
    if kind == CHUNG_LU:
        c["gamma"] = round(rng.uniform(2.05, 2.5), 3)
        c["dmax"] = float(max(8, min(n - 1, int(hub * 2 * m / n))))
    return c


def _batch_cost(mix, graphs):
    """Rough work of a batch (its motif queries), to keep drawn batches below the listed one."""
    return sum(q["n"] * (4.4 * q["m"] / q["n"]) ** (q["k"] - 1)
               for q in workloads.batch_specs(mix, graphs) if q["query"] == "motif")


def _denser(c, avg):
    """The same with an average degree of at least `avg`, and hubs that make cliques likely."""
    c["m"] = max(c["m"], int(c["n"] * avg / 2))
    if c["kind"] == CHUNG_LU:
        c["gamma"] = min(c["gamma"], 2.2)
        c["dmax"] = float(min(c["n"] - 1, max(c["dmax"], 100.0)))
    return c


def draw(rng):
    op = rng.choice(["clique", "clique", "upto", "near", "motif3", "motif4", "motif5", "motif6", "batch", "file",
                     "learn"])
    if op == "clique":
        c = _draw_graph(rng, 200, 300_000, 22.0)
        # (graphs without dense cores hold hardly any larger clique)
        top = {ER: 3, CHUNG_LU: 4, RMAT: 7}[c["kind"]]
        return dict(op="clique", k=rng.randint(3, top), **_denser(c, 5.0))
    if op == "upto":
        return dict(op="upto", k=rng.randint(4, 8), **_denser(_draw_graph(rng, 200, 300_000, 22.0), 3.0))
    if op == "near":
        return dict(op="near", k=rng.randint(4, 7), **_denser(_draw_graph(rng, 200, 2_500, 8.0, (RMAT,)), 3.0))
    if op == "motif3":
        return dict(op="motif", k=3, **_draw_graph(rng, 200, 300_000, 22.0))
    if op == "motif4":
        return dict(op="motif", k=4, **_draw_graph(rng, 200, 19_000, 21.0, (ER, CHUNG_LU)))
    if op == "motif5":
        return dict(op="motif", k=5, **_draw_graph(rng, 100, 3_000, 12.0, (ER, CHUNG_LU), hub=10.0))
    if op == "motif6":
        return dict(op="motif", k=6, **_draw_graph(rng, 100, 2_000, 10.0, (ER, CHUNG_LU), hub=3.0))
    if op == "batch":
        graphs, limit = rng.randint(6, 20), _batch_cost(4, 24)
        mix = rng.randint(1, 9_999)
        while _batch_cost(mix, graphs) > limit:
            mix = rng.randint(1, 9_999)
        return dict(op="batch", graphs=graphs, mix=mix)
    if op == "file":
        return dict(op="file", k=rng.randint(3, 4), **_denser(_draw_graph(rng, 500, 100_000, 21.0, (CHUNG_LU, RMAT)), 6.0))
    return dict(op="learn", k=rng.randint(4, 6), epochs=rng.randint(2, 4), batch=rng.choice([100, 128, 256, 500]),
                **_draw_graph(rng, 1_000, 19_000, 21.0, (ER, CHUNG_LU)))


def _graph(case, seed):
    return dm.Graph.generate(case["kind"], case["n"], case["m"], seed=seed, gamma=case.get("gamma", 2.1),
                             dmax=case.get("dmax", 500.0))


def _batch_queries(case, seed):
    """The benchmark's batch distribution: `mix` fixes the sizes and queries, the seed draws the graphs."""
    dicts, out = {}, []
    for i, q in enumerate(workloads.batch_specs(case["mix"], case["graphs"])):
        g = dm.Graph.generate(CHUNG_LU, q["n"], q["m"], seed=seed * 1009 + i, gamma=q["gamma"], dmax=q["dmax"])
        if q["query"] == "clique":
            out.append(dm.Query(dm.QUERY_CLIQUE, q["k"], g))
        else:
            if q["k"] not in dicts:
                dicts[q["k"]] = dm.Dictionary.generate(q["k"])
            out.append(dm.Query(dm.QUERY_MOTIF, q["k"], g, dicts[q["k"]]))
    return out


def prepare(case, seed):
    op = case["op"]
    s = {"case": case, "seed": seed}
    if op == "batch":
        s["queries"] = _batch_queries(case, seed)
        s["batch"] = dm.Batch(s["queries"])
        return s
    g = _graph(case, seed)
    if op == "file":
        s["dir"] = tempfile.TemporaryDirectory(prefix="edges_")
        s["path"] = s["dir"].name + "/graph.edgelist"
        g.write_edgelist(s["path"])
        g.free()
        return s
    s["graph"] = g
    if op == "motif":
        s["dict"] = dm.Dictionary.generate(case["k"])
    if op == "learn":
        X, T, mask = dm.subtree_log(g, case["k"])
        s["X"] = np.ascontiguousarray(X[mask])
        s["T"] = np.ascontiguousarray(T[mask])
        s["init"] = _initial_weights(seed)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "clique":
        return dm.count_cliques(s["graph"], case["k"])[0]
    if op == "upto":
        counts, _ = dm.count_cliques_upto(s["graph"], case["k"])
        return [counts[k] for k in sorted(counts)]
    if op == "near":
        return dm.count_near_cliques(s["graph"], case["k"])[0]
    if op == "motif":
        return dm.count_motifs(s["graph"], case["k"], s["dict"])[0]
    if op == "batch":
        return s["batch"].run()[0]
    if op == "file":
        g, _ = dm.Graph.load_edgelist_device(s["path"])
        i = g.info()
        count = dm.count_cliques(g, case["k"])[0]
        g.free()
        return [i.n_vertices, i.n_edges, i.max_degree, count]
    # learn: a predictor from the given weights, trained and then used to schedule a count
    p = dm.Predictor(s["seed"])
    p.set_params(s["init"])
    p.train(s["X"], s["T"], epochs=case["epochs"], batch=case["batch"], lr=3e-3)
    count, _ = dm.count_cliques(s["graph"], case["k"], dm.Options(scheduler=dm.SCHED_LEARNED, predictor=p.handle))
    return {"weights": p.get_params(), "count": count}


def work(case):
    """Bytes: the graph's arrays read once (4 bytes per row start and per stored neighbour; cliques
    need each edge once, motifs both directions) and the results written. The counting itself
    is integer work that depends on the drawn graph, so `flops` holds the training's only."""
    op = case["op"]
    if op == "batch":
        # the mean of the batch's distribution: 2,525 vertices and 27,700 edges per graph
        return {"bytes": case["graphs"] * (4 * 2_525 + 6 * 27_700), "flops": 0}
    n, m = case["n"], case["m"]
    if op == "file":
        return {"bytes": 12 * m, "flops": 0}  # about 12 characters per line
    if op in ("clique", "upto"):
        return {"bytes": 4 * (n + m) + 8 * case["k"], "flops": 0}
    if op == "learn":
        rows = n // 2
        return {"bytes": 4 * (n + m) + 36 * rows, "flops": 6 * rows * case["epochs"] * (8 * 32 + 32 * 32 + 32)}
    return {"bytes": 4 * (n + 2 * m) + 8, "flops": 0}


def tolerance(case):
    if case["op"] == "learn":
        # FP32 Adam steps whose gradient sums are taken in any order: mostly 3e-7 from `exact`, but 3e-4
        # was measured where a unit's input passes so close to zero that rounding decides its ReLU in
        # some step. The count stays exact.
        return {"rel": 2e-3, "max": 0.1}
    return "exact"


# ---- the same results in plain numpy and torch, 64 bits ----


class _Host:
    """A graph on the host: CSR, and its edges oriented by (degree, id) as sorted keys."""

    def __init__(self, u, v, n):
        self.n = n
        self.u, self.v = u.astype(np.int64), v.astype(np.int64)
        self.deg = np.bincount(np.concatenate([u, v]), minlength=n).astype(np.int64)
        order = np.lexsort((np.arange(n), self.deg))
        rank = np.empty(n, np.int64)
        rank[order] = np.arange(n)
        a, b = rank[self.u], rank[self.v]
        a, b = np.minimum(a, b), np.maximum(a, b)
        o = np.lexsort((b, a))
        self.rank, self.order = rank, order
        self.src, self.dst = a[o], b[o]
        self.key = self.src * n + self.dst
        self.row = np.searchsorted(self.src, np.arange(n + 1))

    def has(self, a, b):
        k = a * self.n + b
        i = np.searchsorted(self.key, k)
        i[i == self.key.size] = 0
        return self.key[i] == k if self.key.size else np.zeros(k.size, bool)

    def cliques(self, k):
        """Counts of every clique size up to k and the k-cliques (ranks); None above CAP rows."""
        C = np.stack([self.src, self.dst], 1)
        counts = {2: C.shape[0]}
        for s in range(3, k + 1):
            last = C[:, -1]
            d = self.row[last + 1] - self.row[last]
            total = int(d.sum())
            if total > CAP:
                return counts, None
            rep = np.repeat(np.arange(C.shape[0]), d)
            pos = np.arange(total) - np.repeat(np.cumsum(d) - d, d) + np.repeat(self.row[last], d)
            x = self.dst[pos]
            ok = np.ones(total, bool)
            for j in range(s - 2):
                idx = np.flatnonzero(ok)
                ok[idx] = self.has(C[rep[idx], j], x[idx])
            C = np.concatenate([C[rep[ok]], x[ok][:, None]], 1)
            counts[s] = C.shape[0]
        return counts, C

    def dense(self):
        A = torch.zeros((self.n, self.n), dtype=torch.float32, device="cuda")
        u, v = torch.from_numpy(self.u).cuda(), torch.from_numpy(self.v).cuda()
        A[u, v] = 1.0
        A[v, u] = 1.0
        return A


def _host(g):
    u, v = g.edges()
    return _Host(u, v, g.info().n_vertices)


def _classes(k):
    """Class order of the k-vertex dictionary: ascending largest adjacency code."""
    pairs = list(combinations(range(k), 2))
    codes = {}

    def code(edges):
        best = 0
        for p in permutations(range(k)):
            c = 0
            for a, b in pairs:
                c = (c << 1) | ((min(p[a], p[b]), max(p[a], p[b])) in edges)
            best = max(best, c)
        return best

    for bits in range(1, 1 << len(pairs)):
        e = {pairs[i] for i in range(len(pairs)) if bits >> i & 1}
        codes[code(e)] = e
    return {c: i for i, c in enumerate(sorted(codes))}, code


def _motif3(h):
    counts, t = h.cliques(3)
    if t is None:
        return None
    wedges = int((h.deg * (h.deg - 1) // 2).sum()) - 3 * counts[3]
    return np.array([0, wedges, counts[3]], np.int64)


def _motif4(h):
    if h.n > 20_000:
        return None
    counts, t3 = h.cliques(4)
    if t3 is None:
        return None
    tri = h.cliques(3)[1]
    d = h.deg
    k4 = counts[4]
    # triangles per edge and per vertex
    te = np.zeros(h.key.size, np.int64)
    for a, b in ((0, 1), (0, 2), (1, 2)):
        np.add.at(te, np.searchsorted(h.key, tri[:, a] * h.n + tri[:, b]), 1)
    tv = np.bincount(h.order[tri.reshape(-1)], minlength=h.n)
    du, dv = d[h.order[h.src]], d[h.order[h.dst]]
    A = h.dense()
    torch.backends.cuda.matmul.allow_tf32 = False
    c4 = 0
    for r in range(0, h.n, 4096):
        cod = (A[r:r + 4096] @ A).round().double()
        cod[torch.arange(cod.shape[0]), torch.arange(r, r + cod.shape[0])] = 0
        c4 += int((cod * (cod - 1) / 2).sum().item())
    c4 //= 4
    # subgraph copies (not induced)
    star = int((d * (d - 1) * (d - 2) // 6).sum())
    path = int(((du - 1) * (dv - 1)).sum()) - 3 * counts[3]
    paw = int((tv * (d - 2)).sum())
    dia = int((te * (te - 1) // 2).sum())
    # induced
    dia_i = dia - 6 * k4
    c4_i = c4 - dia_i - 3 * k4
    paw_i = paw - 4 * dia_i - 12 * k4
    path_i = path - 2 * paw_i - 4 * c4_i - 6 * dia_i - 12 * k4
    star_i = star - paw_i - 2 * dia_i - 4 * k4
    ids, code = _classes(4)
    out = np.zeros(len(ids), np.int64)
    E = {"star": [(0, 1), (0, 2), (0, 3)], "path": [(0, 1), (1, 2), (2, 3)],
         "paw": [(0, 1), (0, 2), (1, 2), (2, 3)], "c4": [(0, 1), (1, 2), (2, 3), (0, 3)],
         "dia": [(0, 1), (0, 2), (1, 2), (1, 3), (2, 3)], "k4": list(combinations(range(4), 2))}
    for name, value in (("star", star_i), ("path", path_i), ("paw", paw_i), ("c4", c4_i), ("dia", dia_i), ("k4", k4)):
        out[ids[code(set(E[name]))]] = value
    return out


def _clique(h, k):
    counts, C = h.cliques(k)
    return None if C is None else counts[k]


def _near(h, k):
    c = k - 2
    C = h.cliques(c)[1] if c > 2 else np.stack([h.src, h.dst], 1)
    if C is None or C.shape[0] * h.n > 4e9 or h.n > 20_000:
        return None
    A = h.dense()
    C = torch.from_numpy(h.order[C]).cuda()
    total = 0
    step = max(1, int(2e8 // h.n))
    for r in range(0, C.shape[0], step):
        rows = C[r:r + step]
        common = A[rows[:, 0]]
        for j in range(1, c):
            common = common * A[rows[:, j]]
        t = common.sum(1).double()
        total += int((t * (t - 1) / 2).sum().item())
    return total


def _initial_weights(seed):
    rng = np.random.default_rng(seed)
    a1, a2 = math.sqrt(6 / 8), math.sqrt(6 / 32)
    return np.concatenate([rng.uniform(-a1, a1, 256), np.full(32, 0.01), rng.uniform(-a2, a2, 1024),
                           np.full(32, 0.01), rng.uniform(-a2, a2, 32) * 0.5, [0.0]]).astype(np.float32)


def _mix(x):
    M = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & M
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M
    return x ^ (x >> 31)


def _train(X, T, init, seed, epochs, batch, lr=3e-3):
    """Adam over shuffled minibatches in float64, in the engine's minibatch order (a Fisher-Yates
    shuffle of the previous epoch's order, drawn from a splitmix64 chain)."""
    X, T = X.astype(np.float64), T.astype(np.float64)
    p = init.astype(np.float64)
    at = np.cumsum([256, 32, 1024, 32, 32])
    m, v = np.zeros_like(p), np.zeros_like(p)
    idx = list(range(X.shape[0]))
    s, step = seed ^ 0x5DEECE66D, 0
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    for _ in range(epochs):
        for i in range(len(idx) - 1, 0, -1):
            s = _mix(s)
            j = s % (i + 1)
            idx[i], idx[j] = idx[j], idx[i]
        order = np.array(idx)
        for off in range(0, len(idx), batch):
            q = order[off:off + batch]
            x, t = X[q], T[q]
            W1, c1, W2, c2, W3, c3 = np.split(p, at)
            W1, W2 = W1.reshape(32, 8), W2.reshape(32, 32)
            h1 = np.maximum(x @ W1.T + c1, 0)
            h2 = np.maximum(h1 @ W2.T + c2, 0)
            dy = 2 * (h2 @ W3 + c3[0] - t) / len(q)
            d2 = np.outer(dy, W3) * (h2 > 0)
            d1 = (d2 @ W2) * (h1 > 0)
            g = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dy, [dy.sum()]])
            step += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p - lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + 1e-8)
    return p


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        out = []
        for q in _batch_queries(case, seed):
            h = _host(q.graph)
            if q.kind == dm.QUERY_CLIQUE:
                out.append(_clique(h, q.k))
            else:
                out.append({3: _motif3, 4: _motif4}.get(q.k, lambda _: None)(h))
        return out
    if op == "learn":
        s = prepare(case, seed)
        if s["X"].shape[0] * case["epochs"] > 400_000:
            return None
        return {"weights": _train(s["X"], s["T"], s["init"], seed, case["epochs"], case["batch"]),
                "count": _clique(_host(s["graph"]), case["k"])}
    g = _graph(case, seed)
    h = _host(g)
    k = case["k"]
    if op == "clique":
        return _clique(h, k)
    if op == "upto":
        counts, C = h.cliques(k)
        return None if C is None else [counts[j] for j in range(3, k + 1)]
    if op == "near":
        return _near(h, k)
    if op == "motif":
        return {3: _motif3, 4: _motif4}.get(k, lambda _: None)(h)
    return [h.n, int(h.u.size), int(h.deg.max()), _clique(h, k)]
