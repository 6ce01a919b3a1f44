"""Edgelist ingest on the GPU against the host reader: the same graph (CSR, orientation,
counts, statistics) and the same format errors."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _same_graph(dm, a, b):
    ia, ib = a.info(), b.info()
    for f in ("n_vertices", "n_edges", "max_degree", "max_out_degree", "n_self_loops", "n_input_pairs"):
        assert getattr(ia, f) == getattr(ib, f), f
    oa, xa = a.csr()
    ob, xb = b.csr()
    assert np.array_equal(oa, ob) and np.array_equal(xa, xb)
    ua, va = a.edges()
    ub, vb = b.edges()
    assert np.array_equal(ua, ub) and np.array_equal(va, vb)


@pytest.mark.parametrize("name", ["test", "citeseer"])
def test_device_ingest_reference_files(dm, gpu, name):
    path = GOLDEN / f"{name}.edgelist"
    g, ms = dm.Graph.load_edgelist_device(path)
    assert ms > 0
    _same_graph(dm, g, dm.Graph.load_edgelist(path))


@pytest.mark.parametrize("name", ["er2k", "chunglu18k", "rmat100k"])
def test_device_ingest_workloads(dm, orc, gpu, tmp_path, name):
    from dumato_b200 import workloads

    src = workloads.make(name, 1)
    path = tmp_path / f"{name}.edgelist"
    src.write_edgelist(path)
    g, _ = dm.Graph.load_edgelist_device(path)
    h = dm.Graph.load_edgelist(path)
    _same_graph(dm, g, h)
    for k in (3, 4):  # the orientation drives the clique engine
        assert dm.count_cliques(g, k)[0] == dm.count_cliques(h, k)[0]


def test_device_ingest_separators_comments_duplicates(dm, gpu, tmp_path):
    text = ("# a comment line\n0 1\r\n1 0\n2,3\n3 3\n% another comment\n4 2 # trailing comment 9 9\n"
            "1\t2\n\n0 1\n7 5\n")
    path = tmp_path / "mixed.edgelist"
    path.write_text(text)
    g, _ = dm.Graph.load_edgelist_device(path)
    h = dm.Graph.load_edgelist(path)
    _same_graph(dm, g, h)
    info = g.info()
    assert (info.n_vertices, info.n_edges, info.n_self_loops, info.n_input_pairs) == (8, 5, 1, 8)


@pytest.mark.parametrize("text", ["0 1\n2 -3\n", "0 1\n2 x\n", "0 1 2\n", "0 4294967296\n"])
def test_device_ingest_format_errors(dm, gpu, tmp_path, text):
    path = tmp_path / "bad.edgelist"
    path.write_text(text)
    with pytest.raises(dm.DMError) as host_err:
        dm.Graph.load_edgelist(path)
    with pytest.raises(dm.DMError) as dev_err:
        dm.Graph.load_edgelist_device(path)
    assert dev_err.value.status == host_err.value.status == -3


def test_device_ingest_empty_file(dm, gpu, tmp_path):
    path = tmp_path / "empty.edgelist"
    path.write_text("")
    g, _ = dm.Graph.load_edgelist_device(path)
    assert g.info().n_vertices == 0 and g.info().n_edges == 0


@pytest.mark.parametrize("size", [(4 << 20) - 1, 4 << 20, (4 << 20) + 1, (8 << 20) + 3])
def test_device_ingest_staging_edges(dm, gpu, tmp_path, size):
    """Files that end just before, at and after a 4 MiB staging piece, with a token across it."""
    rng = np.random.default_rng(size)
    head = "\n".join(f"{a} {b}" for a, b in rng.integers(0, 70_000, (30_000, 2))) + "\n"
    cut = min(size - 40, (4 << 20) - 3)
    text = head + " " * (cut - len(head)) + "123456 654321\n"  # straddles the first piece's end
    text += "9 10\n" * max(0, (size - len(text)) // 5)
    text += "\n" * (size - len(text))
    assert len(text) == size
    path = tmp_path / "edge.edgelist"
    path.write_text(text)
    g, _ = dm.Graph.load_edgelist_device(path)
    h = dm.Graph.load_edgelist(path)
    _same_graph(dm, g, h)
    for _ in range(2):  # staged first upload, then the page-locked one
        assert dm.count_cliques(g, 3)[0] == dm.count_cliques(h, 3)[0]
        g.release_device()


SLOW_READS = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <unistd.h>
static FILE* sought;
size_t fread(void* p, size_t s, size_t n, FILE* f) {
  static size_t (*real)(void*, size_t, size_t, FILE*);
  if (!real) real = (size_t(*)(void*, size_t, size_t, FILE*))dlsym(RTLD_NEXT, "fread");
  if (s * n >= 1 << 20) usleep(150000);
  return real(p, s, n, f);
}
size_t __fread_chk(void* p, size_t room, size_t s, size_t n, FILE* f) { return fread(p, s, n, f); }
int fseek(FILE* f, long o, int w) {
  static int (*real)(FILE*, long, int);
  if (!real) real = (int (*)(FILE*, long, int))dlsym(RTLD_NEXT, "fseek");
  sought = f;
  return real(f, o, w);
}
int fclose(FILE* f) {
  static int (*real)(FILE*);
  if (!real) real = (int (*)(FILE*))dlsym(RTLD_NEXT, "fclose");
  if (f == sought) sought = NULL;
  return real(f);
}
int setvbuf(FILE* f, char* b, int m, size_t n) {
  static int (*real)(FILE*, char*, int, size_t);
  if (!real) real = (int (*)(FILE*, char*, int, size_t))dlsym(RTLD_NEXT, "setvbuf");
  if (f == sought) fputs("late setvbuf\n", stderr);
  return real(f, b, m, n);
}
"""


def test_device_ms_leaves_out_the_reads(dm, gpu, tmp_path):
    """On a disk that takes 150 ms for each of the file's four pieces the call takes 0.6 s, device_ms
    does not; and the stream's buffering is chosen before its first use."""
    import os
    import subprocess
    import sys

    from conftest import ROOT

    shim, path = tmp_path / "slow.so", tmp_path / "slow.edgelist"
    (tmp_path / "slow.c").write_text(SLOW_READS)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(shim), str(tmp_path / "slow.c"), "-ldl"], check=True)
    rng = np.random.default_rng(4)
    np.savetxt(path, rng.integers(100_000, 999_999, (1_000_000, 2)), fmt="%d")
    assert 3 << 22 < path.stat().st_size < 4 << 22
    code = ("import sys, time, dumato_b200 as dm\n"
            "for _ in range(3):\n"
            "    t = time.perf_counter()\n"
            "    g, ms = dm.Graph.load_edgelist_device(sys.argv[1])\n"
            "    print(g.info().n_edges, ms, 1e3 * (time.perf_counter() - t))\n")
    res = subprocess.run([sys.executable, "-c", code, str(path)], cwd=ROOT, capture_output=True, text=True,
                         timeout=120, env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert res.returncode == 0, res.stderr
    assert "late setvbuf" not in res.stderr
    edges, device_ms, total_ms = map(float, res.stdout.splitlines()[-1].split())
    assert edges > 990_000
    assert total_ms >= 600 and 0 < device_ms < 150
