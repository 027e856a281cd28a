"""Sizes of the dedup tables: powers of two with room for every item, up to the largest batch."""
import subprocess

from bonxai_gb300 import build as B
from conftest import ROOT


def test_table_sizes(tmp_path):
    exe = tmp_path / "dedup_entries"
    subprocess.run([B.nvcc(), *B.NVCC_FLAGS, *B.ARCH, "-o", str(exe),
                    str(ROOT / "tests" / "cpp" / "dedup_entries_main.cu")],
                   check=True, capture_output=True)
    steps = [13, 16, 17, 29, 30]
    sizes = [0, 1, 4, 5, (1 << 31) - 2] + [(1 << s) + d for s in steps for d in (-1, 0, 1)]
    out = subprocess.run([str(exe), *map(str, sizes)], check=True, capture_output=True,
                         text=True, timeout=60).stdout.split()
    for n, p in zip(sizes, map(int, out)):
        assert p & (p - 1) == 0 and n < p <= 1 << 31
        if n:
            assert p >= min(2 * n, 1 << 31)
    assert len(out) == len(sizes)
