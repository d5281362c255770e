"""An infinite entry of a complex64 state makes the rows it reaches infinite, not
NaN, where nothing else is added to them after it."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, U1Sector  # noqa: E402


@pytest.mark.parametrize("n", [2, 5, 16, 26])
def test_one_pair_of_a_sector(n: int) -> None:
    """One exchange term: its row has one live pair, and dead padding follows."""
    codes = np.zeros((2, n), dtype=np.uint8)
    codes[0, [0, n - 1]] = 1
    codes[1, [0, n - 1]] = 2
    op = PauliOperator.from_code_arrays(codes, np.array([0.75, 0.75], dtype=np.complex128))
    plan = op.restrict_charge(U1Sector(n, 1)).mvp_plan()
    x = torch.full((n,), 0.25 + 0.5j, dtype=torch.complex64, device="cuda")
    x[0] = complex(float("inf"), 0.5)  # the state with the last qubit's particle
    y = torch.empty_like(x)
    plan.apply_device(x, y)
    expect = torch.zeros_like(x)
    expect[0] = 1.5 * (0.25 + 0.5j)
    expect[n - 1] = complex(float("inf"), 0.75)
    assert torch.equal(torch.view_as_real(y), torch.view_as_real(expect))


@pytest.mark.parametrize("n", [1, 3, 8, 11])
@pytest.mark.parametrize("overflow", [False, True])
def test_one_term_of_a_small_state(n: int, overflow: bool) -> None:
    """2.5 X on the last qubit: every thread that adds something adds one product."""
    codes = np.zeros((1, n), dtype=np.uint8)
    codes[0, n - 1] = 1
    plan = PauliOperator.from_code_arrays(codes, np.array([2.5], dtype=np.complex128)).native_mvp_plan()
    x = torch.full((1 << n,), 0.25 + 0.5j, dtype=torch.complex64, device="cuda")
    x[0] = 3e38 if overflow else float("inf")
    y = torch.empty_like(x)
    plan.apply_device(x, y)
    assert float(y[1].real) == float("inf")
    expect = torch.full_like(x, 2.5 * (0.25 + 0.5j))
    assert torch.equal(y[0], expect[0]) and torch.equal(y[2:], expect[2:])
