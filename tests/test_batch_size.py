"""The batch's table memory holds what the kernels hand out of it (CPU: the sizes are host code)."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_table_memory_holds_every_piece(tmp_path):
    exe = tmp_path / "batch_size_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "hash-join-optimizer_gb300" / "csrc"),
                    str(ROOT / "tests" / "batch_size_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
