"""The motif kernel's bulk count of the last two vertices (GPU) against the enumerating oracle:
extension sets below, at and above a group's width, rows longer than the group, dense cores
(joined pairs), donated ranges in the middle of a set, shards and subtree logs. Exact counts."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(dm, kind):
    rng = np.random.default_rng(17)
    if kind == "clique":
        u, v = np.triu_indices(13, 1)
    elif kind == "wheel":      # a hub whose rows are longer than a group, and a rim
        u = np.concatenate([np.zeros(45, int), np.arange(1, 45)])
        v = np.concatenate([np.arange(1, 46), np.arange(2, 46)])
    elif kind == "star33":
        u, v = np.zeros(33, int), np.arange(1, 34)
    else:                      # sparse with a dense core, ids shuffled
        a, b = np.triu_indices(8, 1)
        ids = rng.permutation(90)
        u = np.concatenate([rng.integers(0, 90, 130), ids[a]])
        v = np.concatenate([rng.integers(0, 90, 130), ids[b]])
    return dm.Graph.from_edges(u, v)


@pytest.mark.parametrize("vwarp", [8, 16, 32])
@pytest.mark.parametrize("k", [4, 5, 6, 7])
@pytest.mark.parametrize("kind", ["clique", "wheel", "star33", "core"])
def test_sweep_vs_oracle(dm, orc, gpu, kind, k, vwarp):
    if kind in ("wheel", "star33") and k == 7:
        pytest.skip("too many subgraphs for the oracle")
    g = graph(dm, kind)
    og = orc.OracleGraph.from_pairs(*g.edges())
    d = dm.Dictionary.generate(k)
    want = orc.motifs(og, k, d.tables()[0], d.n_classes)
    for flags in (0, dm.TEST_EAGER_DONATION):
        per = np.zeros(g.info().n_vertices, np.uint64)
        got, _ = dm.count_motifs(g, k, d, dm.Options(vwarp=vwarp, test_flags=flags, subtree_counts=per))
        assert np.array_equal(got, want), flags
        assert int(per.sum()) == int(want.sum())
    parts = [dm.count_motifs(g, k, d, dm.Options(vwarp=vwarp, rank=r, world_size=3))[0] for r in range(3)]
    assert np.array_equal(sum(parts), want)


@pytest.mark.parametrize("q", [4, 5, 6, 9])
def test_near_cliques_of_wide_universes(dm, orc, gpu, q):
    """Edges with more than 256 common neighbours, and rows beyond a warp's shared memory."""
    rng = np.random.default_rng(q)
    a, b = np.triu_indices(24, 1)
    core = [(int(x), int(y)) for x, y in zip(a, b) if rng.random() < 0.8]
    outer = [(24 + i, int(c)) for i in range(400) for c in rng.choice(24, 9, replace=False)]
    s, t = np.array(core + outer).T
    g = dm.Graph.from_edges(s, t)
    og = orc.OracleGraph.from_pairs(*g.edges())
    want = orc.near_cliques(og, q)
    assert dm.count_near_cliques(g, q)[0] == want
    assert sum(dm.count_near_cliques(g, q, dm.Options(rank=r, world_size=3))[0] for r in range(3)) == want
    assert dm.count_near_cliques(g, q, dm.Options(threads=256))[0] == want


@pytest.mark.parametrize("vwarp,blades", [(8, 20), (16, 20), (32, 130)])
def test_seven_vertices_of_a_windmill(dm, gpu, vwarp, blades):
    """k = 7 sets of up to 2 blades - 4 members, more than 255 (where the 16-bit pair counters are left
    out) or fewer, with joined pairs: triangles sharing one vertex. A connected 7-subgraph is the
    centre and six rim vertices with j of the rim edges: C(b, j) C(b - j, 6 - 2j) 2^(6 - 2j) of them."""
    from math import comb

    rim = 1 + np.arange(2 * blades)
    u = np.concatenate([np.zeros(2 * blades, int), rim[::2]])
    v = np.concatenate([rim, rim[1::2]])
    g = dm.Graph.from_edges(u, v)
    d = dm.Dictionary.generate(7)
    got, _ = dm.count_motifs(g, 7, d, dm.Options(vwarp=vwarp))
    want = [comb(blades, j) * comb(blades - j, 6 - 2 * j) * 2 ** (6 - 2 * j) for j in range(4)]
    assert sorted(int(x) for x in got if x) == sorted(want)


@pytest.mark.parametrize("k,vwarp", [(6, 8), (6, 32), (7, 32), (7, 8)])
def test_tables_with_a_class_per_code(dm, orc, gpu, tmp_path, k, vwarp):
    """Hand-made tables of 16,384 classes (k = 6), and of 30,000 (k = 7), whose block counters leave no
    shared memory for the bitmaps, or none for themselves: looked up code by code as the oracle does."""
    nq = 1 << (k * (k - 1) // 2 - 1)
    nc = min(nq, 30_000)
    q2c = (np.arange(nq) % nc).astype(np.int32)
    p = tmp_path / f"{k}.csv"
    p.write_text(f"#quick,cg_local\n{nq}\n" + "".join(f"{q},{c}\n" for q, c in enumerate(q2c)) +
                 f"#cg_local,cg_global\n{nc}\n" + "".join(f"{c},{c}\n" for c in range(nc)))
    d = dm.Dictionary.load_csv(p)
    g = graph(dm, "core")
    want = orc.motifs(orc.OracleGraph.from_pairs(*g.edges()), k, q2c, nc)
    assert np.array_equal(dm.count_motifs(g, k, d, dm.Options(vwarp=vwarp))[0], want)
