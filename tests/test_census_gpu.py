"""Whole-graph census of 3- and 4-vertex motifs (GPU) against the oracle's closed forms and
against the enumerating kernel (an explicit vwarp keeps the enumeration), at the sizes where its
parts change: the warp hash table (at most 512 two-paths), the block counters, several counter
windows, 32-bit counters, and graphs without a complete clique index. Exact counts."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def complete(n):
    return np.triu_indices(n, 1)


def star(leaves, extra=0):
    rng = np.random.default_rng(leaves)
    s, t = np.zeros(leaves, np.int64), np.arange(1, leaves + 1)
    return np.concatenate([s, rng.integers(1, leaves + 1, extra)]), np.concatenate([t, rng.integers(1, leaves + 1, extra)])


def bipartite(a, b):
    s, t = np.meshgrid(np.arange(a), a + np.arange(b), indexing="ij")
    return s.ravel(), t.ravel()


def random_graph(n, m, seed, hubs=0, core=0):
    rng = np.random.default_rng(seed)
    s, t = [rng.integers(0, n, m)], [rng.integers(0, n, m)]
    for h in range(hubs):
        s.append(np.full(n // 3, h))
        t.append(rng.integers(0, n, n // 3))
    if core:
        u, v = np.triu_indices(core, 1)
        ids = rng.permutation(n)[:core]
        s.append(ids[u])
        t.append(ids[v])
    return np.concatenate(s), np.concatenate(t)


GRAPHS = {
    "edge": lambda: (np.array([0]), np.array([1])),
    "loop_only": lambda: (np.array([3]), np.array([3])),
    "path": lambda: (np.arange(40), np.arange(1, 41)),
    "star511": lambda: star(511, 30),
    "star600": lambda: star(600, 200),
    "k33": lambda: complete(33),
    "k129": lambda: complete(129),
    "k257": lambda: complete(257),      # out-degree 256: the widest index rows
    "k258": lambda: complete(258),      # out-degree 257: enumerated
    "k3_700": lambda: bipartite(3, 700),
    "k30_40": lambda: bipartite(30, 40),
    "hubs": lambda: random_graph(1500, 6000, 3, hubs=4, core=30),
    "ragged": lambda: random_graph(4099, 20011, 5, hubs=1),
}


def types4(dm, orc, hist, d):
    q2c, _ = d.tables()
    out = {}
    for c, t in enumerate(orc.class_types4(q2c, d.n_classes)):
        if t is None:
            assert int(hist[c]) == 0
        else:
            out[t] = out.get(t, 0) + int(hist[c])
    return out


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_census_vs_closed_form_and_enumeration(dm, orc, gpu, name):
    g = dm.Graph.from_edges(*GRAPHS[name]())
    og = orc.OracleGraph.from_pairs(*g.edges()) if g.info().n_edges else None
    for k in (3, 4):
        d = dm.Dictionary.generate(k)
        got, st = dm.count_motifs(g, k, d)
        if k == 3 or name not in ("k257", "k258"):
            enumerated, _ = dm.count_motifs(g, k, d, dm.Options(vwarp=32))
            assert np.array_equal(got, enumerated), (name, k)
        if og is not None and k == 4:
            assert types4(dm, orc, got, d) == orc.graphlet4(og), name
        again, _ = dm.count_motifs(g, k, d, dm.Options(threads=512))
        assert np.array_equal(got, again)


@pytest.mark.parametrize("n,m,hub", [(230_000, 500_000, 0), (230_000, 500_000, 9_000), (80_000, 150_000, 70_000)])
def test_census_counter_windows(dm, orc, gpu, n, m, hub):
    """No vertex for the block counters; a hub whose counters take several windows (16 bits); a degree of
    65,536 or more (32-bit counters, two windows)."""
    rng = np.random.default_rng(n)
    s, t = rng.integers(0, n, m), rng.integers(0, n, m)
    if hub:
        s, t = np.concatenate([s, np.full(hub, 5)]), np.concatenate([t, 6 + np.arange(hub)])
    g = dm.Graph.from_edges(s, t)
    if hub:
        assert (g.info().max_degree >= 65_536) == (hub >= 65_536)
    d = dm.Dictionary.generate(4)
    got, _ = dm.count_motifs(g, 4, d)
    assert types4(dm, orc, got, d) == orc.graphlet4(orc.OracleGraph.from_pairs(*g.edges()))


def test_census_after_other_calls_and_reupload(dm, gpu):
    """The census shares a graph's device copy with the clique calls: any order, and again after the
    device copy was released."""
    g = dm.Graph.from_edges(*GRAPHS["hubs"]())
    d = dm.Dictionary.generate(4)
    first, _ = dm.count_motifs(g, 4, d)
    k4, _ = dm.count_cliques(g, 4)
    near, _ = dm.count_near_cliques(g, 5)
    for _ in range(2):
        g.release_device()
        assert dm.count_near_cliques(g, 5)[0] == near
        assert np.array_equal(dm.count_motifs(g, 4, d)[0], first)
        assert dm.count_cliques(g, 4)[0] == k4
    _, code = d.tables()
    assert int(first[int(np.where(code == 63)[0][0])]) == k4


@pytest.mark.parametrize("k", [3, 4, 5])
def test_table_that_ignores_isomorphism(dm, orc, gpu, tmp_path, k):
    """A hand-made table whose classes split an isomorphism type is looked up code by code, in the
    enumeration's order, exactly as the oracle does."""
    nq = 1 << (k * (k - 1) // 2 - 1)
    q2c = np.random.default_rng(k).integers(0, 7, nq).astype(np.int32)
    p = tmp_path / f"{k}.csv"
    p.write_text(f"#quick,cg_local\n{nq}\n" + "".join(f"{q},{c}\n" for q, c in enumerate(q2c)) +
                 "#cg_local,cg_global\n7\n" + "".join(f"{c},{c}\n" for c in range(7)))
    d = dm.Dictionary.load_csv(p)
    g = dm.Graph.from_edges(*random_graph(150, 500, 2, core=9))
    og = orc.OracleGraph.from_pairs(*g.edges())
    want = orc.motifs(og, k, q2c, 7)
    for w in (0, 8, 32):
        got, _ = dm.count_motifs(g, k, d, dm.Options(vwarp=w))
        assert np.array_equal(got, want), w
