"""Index bounds of the sector rank tables (u1_rank_check.cpp), on the CPU."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_pair_lookups_stay_inside_the_rank_tables(tmp_path) -> None:
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "u1_rank_check")
    subprocess.run([gxx, "-std=c++17", "-O2", os.path.join(HERE, "u1_rank_check.cpp"), "-o", exe], check=True)
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout[-2000:]
