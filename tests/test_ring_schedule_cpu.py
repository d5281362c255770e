"""The ring kernel's step blocks, walked on the CPU (ring_schedule_check.cpp)
and compared with the direct sum over terms: runs, tables, row signs, folds and
block cuts, both precisions and every tile shape."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tencirpauli_b200", "csrc")


def test_ring_blocks_reproduce_the_direct_sum(tmp_path) -> None:
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "ring_schedule_check")
    subprocess.run(
        [gxx, "-std=c++17", "-O2", "-I/usr/local/cuda/include", os.path.join(HERE, "ring_schedule_check.cpp"),
         os.path.join(CSRC, "tcp_plan.cpp"), "-o", exe, "-ldl"],
        check=True,
    )
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout[-2000:]
