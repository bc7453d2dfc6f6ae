"""Grids whose stencil copy's cell indices do not fit in 32 bits get none (no GPU): the leaf table takes up
to 2^30 cells, and the copy has one cell more along each axis, more than twice as many for thin grids."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

CASES = [(1, 1, 1), (8, 8, 8), (63, 63, 63), (1024, 1024, 1024), (1, 1, 1 << 28), (2, 2, 1 << 28), (1, 4, 1 << 28), (1 << 28, 4, 1),
         (4, 1 << 28, 1), (1, 1, (1 << 29) - 1), (1, 1, (1 << 29) - 2), (1, 1, 1 << 29), (1289, 1289, 646), (32767, 32767, 1),
         (32767, 32766, 1)]


def test_cells_fit_in_32_bits(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    from rtc8_gb300 import build

    src = tmp_path / "cells.cpp"
    calls = "\n".join(f'  std::printf("%lld\\n", (long long)vpt::stencil_cells({a}, {b}, {c}));' for a, b, c in CASES)
    src.write_text(f'#include "{ROOT}/rtc8_gb300/csrc/vpt_ctx.h"\n#include <cstdio>\nint main() {{\n{calls}\n}}\n')
    exe = tmp_path / "cells"
    include = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run([cxx, "-std=c++17", "-w", "-I", str(include), str(src), "-o", str(exe)], check=True)
    got = [int(x) for x in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]
    for (a, b, c), cells in zip(CASES, got):
        want = (a + 1) * (b + 1) * (c + 1)
        assert cells == (want if want < 1 << 31 else 0), (a, b, c)
    assert 0 in got and any(a * b * c <= 1 << 30 and cells == 0 for (a, b, c), cells in zip(CASES, got))
