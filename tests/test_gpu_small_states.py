"""States below one ring tile: every size, few and many terms per row thread,
more terms than one shared-memory stage, blocks of vectors, accumulation."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, workloads  # noqa: E402


def _operator(n: int, words: int, seed: int) -> PauliOperator:
    rng = np.random.default_rng(seed)
    codes = rng.integers(0, 4, size=(words, n)).astype(np.uint8)
    return PauliOperator.from_code_arrays(codes, rng.normal(size=words) + 1j * rng.normal(size=words))


# dense random words: up to 4^n terms, so 5 qubits and more exceed one stage
@pytest.mark.parametrize("n,words", [(1, 1), (1, 4), (2, 9), (3, 63), (4, 64), (5, 65), (6, 1500), (7, 512), (8, 513), (9, 40), (10, 2000), (11, 63), (11, 700)])
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-12), ("complex64", 2e-6)])
def test_small_states_match_the_oracle(n: int, words: int, dtype: str, tol: float) -> None:
    op = _operator(n, words, seed=n * 7 + words)
    plan = op.native_mvp_plan()
    xm, zm, wp = oracle.matrix_terms(n, op.x_words, op.z_words, op.coefficients)
    x = workloads.random_state_device(n, seed=1, dtype=getattr(torch, dtype), nrhs=3)
    y0 = workloads.random_state_device(n, seed=2, dtype=getattr(torch, dtype), nrhs=3)
    y, z = torch.full_like(x, float("nan")), y0.clone()
    plan.apply_device(x, y)
    plan.apply_device(x, z, accumulate=True)
    one = torch.full_like(x[2], float("nan"))
    plan.apply_device(x[2].clone(), one)
    assert torch.equal(one, y[2])
    for v in range(3):
        ref = oracle.apply_term_direct(n, xm, zm, wp, x[v].cpu().numpy().astype(np.complex128))
        scale = np.linalg.norm(ref)
        assert np.linalg.norm(y[v].cpu().numpy() - ref) <= tol * scale
        assert np.linalg.norm(z[v].cpu().numpy() - ref - y0[v].cpu().numpy()) <= tol * (scale + 1.0)


def test_empty_operator_writes_zeros() -> None:
    plan = PauliOperator.empty(6).native_mvp_plan()
    x = workloads.random_state_device(6, seed=1, dtype=torch.complex64)
    y = torch.full_like(x, float("nan"))
    plan.apply_device(x, y)
    assert not torch.any(y)
