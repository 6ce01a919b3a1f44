"""Thread-to-rank maps of the in-list kernels (census.cu), restated from their source, at the largest
graphs that the entry points take: every rank below 2^31 has its eight threads."""
from __future__ import annotations

import re
from pathlib import Path

SRC = Path(__file__).resolve().parents[1] / "dumato_b200" / "csrc" / "census.cu"


def test_in_list_ranks_beyond_32_bit_thread_numbers():
    text = SRC.read_text()
    maps = re.findall(r"const int r = (.*) >> 3\), l = threadIdx.x & 7;", text)
    assert len(maps) == 2
    for expr in maps:
        wide = "256ll" in expr  # a 64-bit product; unsigned 32-bit otherwise
        for rank in (0, 1, (1 << 29) - 1, 1 << 29, (1 << 31) - 2):
            for lane in (0, 7):
                thread = 8 * rank + lane
                block, t = divmod(thread, 256)
                product = block * 256 + t
                assert (product if wide else product % (1 << 32)) >> 3 == rank, expr
