"""The ring kernel's tile shapes at the edges of their ranges: complex64 blocks
that take the 8192-row tiles (16 rows per thread, Kahan sums in tensor memory)
and the largest that do not, vectors per launch, accumulation, the chunked host
apply -- against the oracle, or the FP64 kernel where the oracle is too slow."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, mapping, workloads  # noqa: E402

# FP32 products of FP32-rounded weights with compensated sums: rounding of the
# inputs, of D and of each product, about 2^-23 each in the norm.
C64_NORM_RTOL = 2e-6
FP64_NORM_RTOL = 1e-12


def _operator(n: int, seed: int) -> PauliOperator:
    """Complex weights, groups of many terms, and the dense diagonal."""
    rng = np.random.default_rng(seed)
    codes, coeffs = workloads.random_k_local(n=n, words=120, seed=seed)
    diag, dcoef = workloads.heisenberg_2d_open(n, seed)
    m = min(n, 6)
    hc, hw = mapping.jordan_wigner_integrals(*mapping.chemistry_integrals(m, seed=seed))
    chem = np.zeros((hc.shape[0], n), dtype=np.uint8)
    chem[:, n - m :] = hc  # on the row bits inside a tile
    return PauliOperator.from_code_arrays(
        np.concatenate([codes, diag, chem]),
        np.concatenate([coeffs * np.exp(1j * rng.uniform(0, 6, size=len(coeffs))), dcoef, hw]),
    )


def _relative(got: np.ndarray, ref: np.ndarray) -> float:
    return float(np.linalg.norm(got - ref) / np.linalg.norm(ref))


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n,nrhs", [(12, 1), (12, 150), (13, 1), (13, 74), (13, 75), (14, 37), (14, 38), (16, 3), (20, 1)])
def test_shapes_match_the_oracle(n: int, nrhs: int, dtype: str) -> None:
    op = _operator(n, seed=n + nrhs)
    plan = op.native_mvp_plan()
    xm, zm, wp = oracle.matrix_terms(n, op.x_words, op.z_words, op.coefficients)
    x = workloads.random_state_device(n, seed=nrhs, dtype=getattr(torch, dtype), nrhs=nrhs)
    y0 = workloads.random_state_device(n, seed=nrhs + 1, dtype=getattr(torch, dtype), nrhs=nrhs)
    y, z = torch.full_like(x, float("nan")), y0.clone()
    plan.apply_device(x, y)
    plan.apply_device(x, z, accumulate=True)
    torch.cuda.synchronize()
    plan._native_plan.device_status()
    tol = C64_NORM_RTOL if dtype == "complex64" else FP64_NORM_RTOL
    for v in {0, nrhs // 2, nrhs - 1}:
        ref = oracle.apply_term_direct(n, xm, zm, wp, x[v].cpu().numpy().astype(np.complex128))
        assert _relative(y[v].cpu().numpy(), ref) <= tol
        assert _relative(z[v].cpu().numpy(), ref + y0[v].cpu().numpy()) <= tol


def test_host_apply_in_parts_matches_the_device_apply() -> None:
    n = 25  # the smallest state that goes in by parts
    op = _operator(n, seed=3)
    plan = op.native_mvp_plan()
    x = workloads.random_state_device(n, seed=5, dtype=torch.complex64)
    y = torch.empty_like(x)
    plan.apply_device(x, y)
    got = plan._native_plan.apply_c64(x.cpu().numpy())
    assert _relative(got, y.cpu().numpy()) <= C64_NORM_RTOL


def test_unaligned_output_of_a_complex64_block() -> None:
    n = 20
    op = _operator(n, seed=9)
    plan = op.native_mvp_plan()
    x = workloads.random_state_device(n, seed=5, dtype=torch.complex64)
    y = torch.empty_like(x)
    plan.apply_device(x, y)
    shifted = torch.empty(x.numel() + 1, dtype=x.dtype, device="cuda")[1:]  # 8 bytes off a 16-byte boundary
    plan.apply_device(x, shifted)
    assert _relative(shifted.cpu().numpy(), y.cpu().numpy()) <= C64_NORM_RTOL
