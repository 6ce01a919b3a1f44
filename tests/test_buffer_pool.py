"""The pool of freed device buffers (dumato_b200/csrc/buf_pool.hpp) against a fake device, on the CPU."""
from __future__ import annotations

import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent / "pool" / "pool_selftest.cpp"


def test_pool_logic(tmp_path):
    exe = tmp_path / "pool_selftest"
    res = subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-o", str(exe), str(SRC)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and "pool ok" in res.stdout, res.stdout
