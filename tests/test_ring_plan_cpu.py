"""Properties of the ring schedules (ring_plan_check.cpp) on the CPU: building
one takes work linear in the number of terms, whatever the length of a run, and
the complex64 sums are folded in time across the steps of a schedule."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tencirpauli_b200", "csrc")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("ring") / "ring_plan_check")
    subprocess.run(
        [gxx, "-std=c++17", "-O2", "-I/usr/local/cuda/include", os.path.join(HERE, "ring_plan_check.cpp"),
         os.path.join(CSRC, "tcp_plan.cpp"), "-o", exe, "-ldl"],
        check=True,
    )
    return exe


@pytest.mark.parametrize("check", ["work", "folds"])
def test_ring_plans(checker: str, check: str) -> None:
    proc = subprocess.run([checker, check], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout[-2000:]
