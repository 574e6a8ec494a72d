"""Shared memory of a warp of the LU pass: the n x n matrix, and only where the pass is
asked for its explicit inverse, room for the part of that which C does not hold (host
code, compiled here)."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
DEPTHS = (2, 10, 30, 45, 64)

PROGRAM = """
#include <cstdio>
#include "pix_args.cuh"
int main() {
    for (int n : {%s})
        for (int wx : {1, 23})
            printf("%%d %%d %%zu %%zu\\n", n, wx, dpl::make_layout(n, wx, true).bytes,
                   dpl::make_layout(n, wx, true, true).bytes);
}
"""


def _up(x, a):
    return -(-x // a) * a


def test_lu_pass(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("needs nvcc")
    src = tmp_path / "layout.cu"
    src.write_text(PROGRAM % ", ".join(map(str, DEPTHS)))
    exe = tmp_path / "layout"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    str(ROOT / "dolphin_gb300" / "csrc"), "-o", str(exe), str(src)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for line in filter(None, lines):
        n, wx, got, probing = map(int, line.split())
        tri = n * (n + 1) // 2
        parts = [8 * tri, 4 * n * (n | 1), 8 * max(wx * ((n + 1) & ~1) + 32, tri, n * n), 8 * 64, 4 * 64, 4 * 128]
        assert got == _up(sum(_up(p, 16) for p in parts), 128), (n, wx)
        # the inverse, n x (n | 1), lies over C's end
        assert probing == _up(sum(_up(p, 16) for p in [8 * (n * (n | 1) - tri)] + parts), 128), (n, wx)
