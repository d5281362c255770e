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


def _flips(n: int, words: int, seed: int) -> PauliOperator:
    """Words of X and I with positive weights: no sum mixes signs, and every word
    is a run of its own."""
    rng = np.random.default_rng(seed)
    codes = np.unique(rng.integers(0, 2, size=(4 * words, n)).astype(np.uint8), axis=0)
    codes = codes[rng.permutation(len(codes))[:words]]
    return PauliOperator.from_code_arrays(codes, rng.uniform(0.5, 2.0, size=len(codes)).astype(np.complex128))


# no fold before the last, several; 8 and 16 rows per thread
@pytest.mark.parametrize("n,words,nrhs", [(12, 7, 1), (12, 60, 1), (13, 7, 80), (13, 40, 80), (20, 60, 1)])
def test_many_runs(n: int, words: int, nrhs: int) -> None:
    plan = _flips(n, words, seed=n).native_mvp_plan()
    x = torch.full((nrhs, 1 << n), 0.25 + 0.5j, dtype=torch.complex64, device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    plan.apply_device(x, y)
    where = (1 << n) // 3
    x[:, where] = complex(float("inf"), 0.5)
    unit = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    unit[where] = 1.0
    reached = torch.empty_like(unit)
    plan.apply_device(unit, reached)
    plan.apply_device(x, z)
    hit = reached.real > 0
    assert int(hit.sum()) == words
    assert bool(torch.all(z[:, hit].real == float("inf")))
    assert torch.equal(z[:, hit].imag, y[:, hit].imag)
    assert torch.equal(z[:, ~hit], y[:, ~hit])


@pytest.mark.parametrize("n", [12, 14, 20])
def test_overflow(n: int) -> None:
    plan = _flips(n, 40, seed=n).native_mvp_plan()
    x = torch.full((1 << n,), 3e38, dtype=torch.complex64, device="cuda")
    y = torch.empty_like(x)
    plan.apply_device(x, y)
    assert bool(torch.all(y.real == float("inf")))


@pytest.mark.parametrize("n", [12, 13])
def test_transverse_field_chain(n: int) -> None:
    """Fewer groups than a fold takes, more runs: n flips and a diagonal."""
    codes = np.zeros((2 * n, n), dtype=np.uint8)
    for q in range(n):
        codes[q, q] = 1
        codes[n + q, [q, (q + 1) % n]] = 3
    op = PauliOperator.from_code_arrays(codes, np.full(2 * n, 1.0, dtype=np.complex128))
    x = torch.full((1 << n,), 0.25 + 0.5j, dtype=torch.complex64, device="cuda")
    x[0] = complex(float("inf"), 0.5)
    y = torch.empty_like(x)
    op.native_mvp_plan().apply_device(x, y)
    flipped = torch.tensor([1 << q for q in range(n)], device="cuda")
    assert bool(torch.all(y[flipped].real == float("inf"))) and float(y[0].real) == float("inf")
    y[flipped] = 0
    y[0] = 0
    assert bool(torch.all(torch.isfinite(torch.view_as_real(y))))
