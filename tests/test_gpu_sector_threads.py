"""Sector plans of different table sizes applied from several threads at once:
every launch gets the shared memory it asks for."""

from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, U1Sector  # noqa: E402


def _exchange(n: int, complex_constant: bool) -> PauliOperator:
    """X X + Y Y on a ring of n sites; X Y - Y X beside it makes the constants complex."""
    rows, coeffs = [], []
    for a in range(n):
        b = (a + 1) % n
        for letters, w in (((1, 1), 0.5), ((2, 2), 0.5), ((1, 2), 0.25), ((2, 1), -0.25)):
            if letters[0] != letters[1] and not complex_constant:
                continue
            row = np.zeros(n, dtype=np.uint8)
            row[a], row[b] = letters
            rows.append(row)
            coeffs.append(w)
    return PauliOperator.from_code_arrays(np.asarray(rows), np.asarray(coeffs, dtype=np.complex128))


# the pair kernel and the general one
@pytest.mark.parametrize("complex_constant", [False, True])
def test_plans_of_two_sizes_from_four_threads(complex_constant: bool) -> None:
    work = []
    for n, k in ((6, 3), (24, 2), (6, 2), (24, 3)):
        plan = _exchange(n, complex_constant).restrict_charge(U1Sector(n, k)).mvp_plan()
        x = torch.randn(plan.dimension, dtype=torch.complex128, device="cuda")
        expect = torch.empty_like(x)
        plan.apply_device(x, expect)
        work.append((plan, x, expect, torch.empty_like(x)))
    torch.cuda.synchronize()
    errors = []

    def loop(plan, x, y) -> None:
        try:
            stream = torch.cuda.Stream()
            for _ in range(3000):
                plan.apply_device(x, y, stream=stream)
            stream.synchronize()
        except Exception as error:  # noqa: BLE001 - reported below
            errors.append(error)

    threads = [threading.Thread(target=loop, args=(plan, x, y)) for plan, x, _, y in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for _, _, expect, y in work:
        assert torch.equal(y, expect)
