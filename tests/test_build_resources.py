"""Registers of the kernels whose speed rests on several CTAs per SM, from the
compiler's report of the build (``delta_b200/csrc/_build``). An SM has 65536
registers; a block of 256 threads takes 256 times its count, rounded up to 8."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

BUILD = Path(__file__).resolve().parents[1] / "delta_b200" / "csrc" / "_build"


def _registers(unit: str) -> dict[str, int]:
    path = BUILD / f"{unit}.ptxas.txt"
    if not path.exists():
        pytest.skip(f"no compiler report of {unit} (make -C delta_b200/csrc)")
    out = {}
    for name, regs in re.findall(r"Compiling entry function '(\S+)'.*?Used (\d+) registers", path.read_text(), re.S):
        out[name] = int(regs)
    return out


def _ctas(regs: int, threads: int = 256) -> int:
    return 65536 // (threads * ((regs + 7) // 8 * 8))


@pytest.mark.parametrize("kernel,ctas", [
    ("k_rows_fwdILi0E", 4), ("k_rows_invILi0E", 4), ("k_colsILi0E", 4),  # radix-2 lines: blocks of 8 to 64, 1024
    ("k_colsILi128E", 3), ("k_colsILi256E", 2),                          # blocks of 128 and 256
])
def test_line_transforms_leave_room_for_several_ctas(kernel, ctas):
    regs = [r for name, r in _registers("k_fft").items() if kernel in name]
    assert regs, f"{kernel}: not in the build"
    assert all(_ctas(r) >= ctas for r in regs), (kernel, regs)
