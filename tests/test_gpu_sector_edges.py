"""The pair kernel in sectors of 25 to 32 qubits whose rows have dead pairs with
sources far outside the sector: no particles, one, all but one, all."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, U1Sector  # noqa: E402


def _exchange(n: int, seed: int) -> PauliOperator:
    """X X + Y Y on every pair, every second one with a Z string, and levels."""
    rng = np.random.default_rng(seed)
    rows, coeffs = [], []
    for a in range(n):
        for b in range(a + 1, n):
            w = rng.normal()
            for letter in (1, 2):
                row = np.zeros(n, dtype=np.uint8)
                if (a + b) % 2:
                    row[a + 1 : b] = 3
                row[a] = row[b] = letter
                rows.append(row)
                coeffs.append(w)
        row = np.zeros(n, dtype=np.uint8)
        row[a] = 3
        rows.append(row)
        coeffs.append(rng.normal())
    return PauliOperator.from_code_arrays(np.asarray(rows), np.asarray(coeffs, dtype=np.complex128))


# FP64: each row adds up to 32 products; FP32: compensated sums of rounded products
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-12), ("complex64", 2e-6)])
@pytest.mark.parametrize("n", [25, 26, 27, 28, 29, 30, 31, 32])
def test_nearly_empty_and_nearly_full_sectors(n: int, dtype: str, tol: float) -> None:
    op = _exchange(n, seed=n)
    for k in (0, 1, n - 1, n):
        plan = op.restrict_charge(U1Sector(n, k)).mvp_plan()
        rng = np.random.default_rng(k)
        x = (rng.normal(size=plan.dimension) + 1j * rng.normal(size=plan.dimension)).astype(dtype)
        xd = torch.from_numpy(x).cuda()
        yd = torch.full_like(xd, float("nan"))
        plan.apply_device(xd, yd)
        ref = oracle.u1_apply(n, k, op.x_words, op.z_words, op.coefficients, x.astype(np.complex128))
        assert np.linalg.norm(yd.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
