"""5- and 6-cliques of roots with more than 64 out-neighbours (rows of two to four words, counted in
plain loops) on the GPU against the oracle and the other counting paths, with out-degrees on
both sides of every row width, donated ranges, shards and subtree logs. Exact counts."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def two_sides(dm, a, b, p, seed):
    """Complete between sides of a and b vertices, sparse inside them: out-degrees up to about
    max(a, b) without many cliques."""
    rng = np.random.default_rng(seed)
    s, t = np.meshgrid(np.arange(a), a + np.arange(b), indexing="ij")
    src, dst = [s.ravel()], [t.ravel()]
    for lo, n in ((0, a), (a, b)):
        u, v = np.triu_indices(n, 1)
        keep = rng.random(u.size) < p
        src.append(lo + u[keep])
        dst.append(lo + v[keep])
    ids = rng.permutation(a + b)
    return dm.Graph.from_edges(ids[np.concatenate(src)], ids[np.concatenate(dst)])


@pytest.mark.parametrize("a,b,p", [(62, 70, 0.1), (66, 64, 0.15), (120, 128, 0.08), (127, 140, 0.06), (180, 192, 0.05),
                                   (193, 200, 0.05), (240, 250, 0.02)])
def test_wide_roots_vs_oracle(dm, orc, gpu, a, b, p):
    g = two_sides(dm, a, b, p, seed=a)
    assert 64 < g.info().max_out_degree <= 256
    og = orc.OracleGraph.from_pairs(*g.edges())
    for k in (5, 6):
        want, _ = orc.clique_dag_bytes(og, k)
        per = np.zeros(g.info().n_vertices, np.uint64)
        for opts in (None, dm.Options(mode=dm.MODE_REBUILD), dm.Options(staging=dm.STAGE_LOADS),
                     dm.Options(test_flags=dm.TEST_EAGER_DONATION), dm.Options(threads=256),
                     dm.Options(subtree_counts=per), dm.Options(threshold=100)):
            assert dm.count_cliques(g, k, opts)[0] == want, (k, opts)
        assert int(per.sum()) == want
        assert sum(dm.count_cliques(g, k, dm.Options(rank=r, world_size=3))[0] for r in range(3)) == want


@pytest.mark.parametrize("n", [67, 70])
def test_complete_graphs(dm, gpu, n):
    from math import comb

    g = dm.Graph.from_edges(*np.triu_indices(n, 1))
    for k in (5, 6):
        assert dm.count_cliques(g, k)[0] == comb(n, k)


@pytest.mark.parametrize("n,p", [(1500, 0.1), (300, 0.5)])
def test_light_and_heavy_sets_vs_oracle(dm, orc, gpu, n, p):
    """Wide roots whose sets are mostly empty (an item on every lane, and no ranges handed out for
    tasks of some microseconds: a donation per root at most, where ranges split to the last made
    more than two) and ones whose sets hold many members. Exact counts."""
    rng = np.random.default_rng(n)
    u, v = np.triu_indices(n, 1)
    keep = rng.random(u.size) < p
    g = dm.Graph.from_edges(u[keep], v[keep])
    assert 64 < g.info().max_out_degree <= 256
    og = orc.OracleGraph.from_pairs(*g.edges())
    for k in (5, 6):
        want, _ = orc.clique_dag_bytes(og, k)
        assert dm.count_cliques(g, k, dm.Options(test_flags=dm.TEST_EAGER_DONATION))[0] == want
        for _ in range(3):
            got, st = dm.count_cliques(g, k)
            assert got == want
            if p < 0.2:
                assert st.donations < n, st.donations
