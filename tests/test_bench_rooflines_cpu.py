"""bench.py's shared-memory line counts only the schedule that runs."""

from __future__ import annotations

import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench_rooflines", os.path.join(ROOT, "bench.py"))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def test_shared_memory_rate_is_given_for_complex128_alone() -> None:
    bench = _bench()
    line = bench._smem_roofline("c128", 20, 300, 100, 2.0, 40e12)
    nbytes = 2**20 * 400 * 16
    assert line["bytes_per_launch"] == nbytes
    assert abs(line["achieved"] - nbytes / 2e-3 / 1e12) < 1e-9 and abs(line["frac"] - nbytes / 2e-3 / 40e12) < 1e-12
    line = bench._smem_roofline("c64", 20, 300, 100, 2.0, 40e12)
    assert line["achieved"] is None and line["frac"] is None and line["peak"] == 40.0


def test_sector_line_names_the_kernel_that_runs() -> None:
    bench = _bench()
    for lattice in ("4x6", "4x7"):
        assert bench._profile_instructions("k_u1_pairs", f"j1j2_{lattice}_half_c128")
