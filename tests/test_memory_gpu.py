"""Calls on a device with little memory left: buffers that the library keeps for later are given back
when an allocation finds no room, launches shrink to the workspace that fits, and an error leaves
nothing behind for the next call."""
from __future__ import annotations

from contextlib import contextmanager

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextmanager
def little_memory(leave):
    """All of the device's free memory but `leave` bytes, held by another owner."""
    import torch

    torch.cuda.synchronize()
    held = []
    for piece in (1 << 33, 1 << 30, 1 << 26):
        while torch.cuda.mem_get_info()[0] >= leave + piece:
            held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def drop_kept(dm):
    """Has the library give back what it keeps: a batch that asks for 8 GB where there is no room."""
    g = dm.Graph.generate(dm.GEN_ER, 1_000_000, 1000, seed=1)
    d = dm.Dictionary.generate(5)

    def drop():
        with little_memory(300 << 20):
            dm.Batch([dm.Query(dm.QUERY_MOTIF, 5, g, d, vwarp=8)]).close()

    return drop


def dense(dm, n, p, seed=1):
    rng = np.random.default_rng(seed)
    u, v = np.triu_indices(n, 1)
    keep = rng.random(u.size) < p
    return dm.Graph.from_edges(u[keep], v[keep])


def test_pooled_buffers_are_given_back(dm, gpu, tmp_path):
    """A file's temporaries stay with the library (up to 4 GB); a call that needs more than is left
    beside them takes their place and runs at its full size."""
    import torch

    g = dm.Graph.generate(dm.GEN_ER, 1_000_000, 1_100_000, seed=2)
    d = dm.Dictionary.generate(5)
    big = dm.Graph.generate(dm.GEN_ER, 1_000_000, 16_000_000, seed=1)
    path = tmp_path / "big.edgelist"
    big.write_edgelist(path)
    big.free()
    before = torch.cuda.mem_get_info()[0]
    h, _ = dm.Graph.load_edgelist_device(path)
    h.free()
    assert before - torch.cuda.mem_get_info()[0] > 2.2e9
    with little_memory(400 << 20):
        got, st = dm.count_motifs(g, 5, d)
    g.release_device()
    want, full = dm.count_motifs(g, 5, d)
    assert st.grid == full.grid and np.array_equal(got, want)


def test_motif_launch_shrinks_to_the_memory_left(dm, gpu, drop_kept):
    """1.8 GB of bitmaps for all warps at 32 lanes (four times that at 8), 900 MB left."""
    g = dm.Graph.generate(dm.GEN_ER, 1_000_000, 1_100_000, seed=2)
    for k in (5, 6):
        d = dm.Dictionary.generate(k)
        want, full = dm.count_motifs(g, k, d)
        for vwarp in (32, 8):
            g.release_device()
            drop_kept()
            with little_memory(900 << 20):
                got, st = dm.count_motifs(g, k, d, dm.Options(vwarp=vwarp))
            assert st.grid < full.grid and np.array_equal(got, want), (k, vwarp)


def test_batch_shrinks_to_the_memory_left(dm, gpu, drop_kept):
    d = dm.Dictionary.generate(5)
    g = dm.Graph.generate(dm.GEN_ER, 1_000_000, 1_100_000, seed=3)
    h = dense(dm, 300, 0.2)
    queries = [dm.Query(dm.QUERY_MOTIF, 5, g, d), dm.Query(dm.QUERY_CLIQUE, 5, h)]
    b = dm.Batch(queries)
    want, full = b.run()
    b.close()
    drop_kept()
    with little_memory(900 << 20):
        b = dm.Batch(queries)
        got, st = b.run()
        b.close()
    assert st.grid < full.grid
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]


def test_near_cliques_shrink_to_the_memory_left(dm, gpu, drop_kept):
    """600 MB of rows for all warps on a complete graph of 700 vertices."""
    from math import comb

    g = dense(dm, 700, 1.1)
    want = comb(700, 3) * comb(697, 2)
    drop_kept()
    with little_memory(300 << 20):
        got, st = dm.count_near_cliques(g, 5)
    assert got == want


def test_failed_allocation_leaves_no_error_behind(dm, orc, gpu, drop_kept):
    g = dense(dm, 200, 0.2)
    huge = dm.Graph.generate(dm.GEN_ER, 50_000_000, 1000, seed=1)
    drop_kept()
    want = orc.clique_dag_bytes(orc.OracleGraph.from_pairs(*g.edges()), 4)[0]
    assert dm.count_cliques(g, 4)[0] == want
    with little_memory(200 << 20):
        for _ in range(2):
            with pytest.raises(dm.DMError) as e:
                dm.count_cliques(huge, 4)
            assert e.value.status in (-4, -6)
            assert dm.count_cliques(g, 4)[0] == want
