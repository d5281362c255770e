"""The two-row complex64 combine and the pair kernel of the U(1) sectors (real
exchange and hopping constants) at the edges of their ranges: every class of
pairs (low half, high half, across, with and without a sign string), two- and
three-level ranks, sectors of a single state, and operators next to the rule
that must keep the general kernel."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import PauliOperator, U1Sector, solver_ops  # noqa: E402

FP64_NORM_RTOL = 1e-12
C64_NORM_RTOL = 2e-6  # FP32 products, compensated sums


def _hopping(n: int, seed: int, complex_hop: bool = False, four_body: bool = False, diagonal: bool = True) -> PauliOperator:
    rng = np.random.default_rng(seed)
    rows, coeffs = [], []

    def add(letters, weight):
        row = np.zeros(n, dtype=np.uint8)
        for q, letter in letters.items():
            row[q] = letter
        rows.append(row)
        coeffs.append(weight)

    pairs = {(0, n - 1), (0, 1), (n - 2, n - 1)} | {tuple(sorted(rng.choice(n, 2, replace=False).tolist())) for _ in range(2 * n)}
    for k, (a, b) in enumerate(sorted(p for p in pairs if p[0] != p[1])):
        h = complex(rng.normal(), rng.normal() if complex_hop and k == 0 else 0.0)
        string = {q: 3 for q in range(a + 1, b)} if k % 2 else {}
        for letter in (1, 2):
            add({**string, a: letter, b: letter}, h)
    if four_body:  # (XX + YY)(XX + YY) on sites 0 .. 3
        for letters in ((1, 1, 1, 1), (1, 1, 2, 2), (2, 2, 1, 1), (2, 2, 2, 2)):
            add(dict(zip((0, 1, 2, 3), letters)), 0.3)
    if diagonal:
        for q in range(n):
            add({q: 3}, rng.normal())
    return PauliOperator.from_code_arrays(np.asarray(rows), np.asarray(coeffs))


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n,k", [(2, 1), (3, 1), (5, 5), (6, 0), (8, 4), (11, 3), (16, 8), (23, 2), (24, 3), (25, 2), (31, 2), (32, 2)])
def test_pairs_match_the_oracle(n: int, k: int, dtype: str) -> None:
    op = _hopping(n, seed=n * 40 + k, diagonal=n % 2 == 0)
    plan = op.restrict_charge(U1Sector(n, k)).mvp_plan()
    rng = np.random.default_rng(n)
    x = (rng.normal(size=(3, plan.dimension)) + 1j * rng.normal(size=(3, plan.dimension))).astype(dtype)
    xd = torch.from_numpy(x).cuda()
    yd = torch.full_like(xd, float("nan"))
    plan.apply_device(xd, yd)
    for v in range(3):
        ref = oracle.u1_apply(n, k, op.x_words, op.z_words, op.coefficients, x[v].astype(np.complex128))
        err = np.linalg.norm(yd[v].cpu().numpy() - ref)
        assert err <= (FP64_NORM_RTOL if dtype == "complex128" else C64_NORM_RTOL) * max(np.linalg.norm(ref), 1e-30)


@pytest.mark.parametrize("kind", [{"complex_hop": True}, {"four_body": True}])
def test_operators_beside_the_rule(kind) -> None:
    n, k = 10, 4
    op = _hopping(n, 7, **kind)
    plan = op.restrict_charge(U1Sector(n, k)).mvp_plan()
    rng = np.random.default_rng(1)
    x = rng.normal(size=plan.dimension) + 1j * rng.normal(size=plan.dimension)
    ref = oracle.u1_apply(n, k, op.x_words, op.z_words, op.coefficients, x)
    assert np.linalg.norm(plan.apply(x) - ref) <= FP64_NORM_RTOL * np.linalg.norm(ref)


@pytest.mark.parametrize("p,k", [(1, 1), (7, 3), (8, 4), (9, 5), (40, 4), (33, 32)])
@pytest.mark.parametrize("n,offset", [(2, 0), (510, 0), (1031, 0), (4098, 0), (4098, 1)])
def test_complex64_combine(p: int, k: int, n: int, offset: int) -> None:
    """Even lengths take the two-row kernel; odd ones, and blocks 8 bytes off a
    16-byte boundary, the one-row kernel."""
    rng = np.random.default_rng(p * k + n)

    def block(rows):
        a = (rng.normal(size=(rows, n)) + 1j * rng.normal(size=(rows, n))).astype(np.complex64)
        t = torch.empty(rows * n + offset, dtype=torch.complex64, device="cuda")[offset:]
        return a, t.copy_(torch.from_numpy(a.reshape(-1))).view(rows, n)

    (a, A), (o, out) = block(p), block(k)
    S = rng.normal(size=(p, k)) + 1j * rng.normal(size=(p, k))
    for beta in (0.0, 0.5):
        _, fresh = o, out.copy_(torch.from_numpy(o))
        solver_ops.combine(A, torch.from_numpy(S), fresh, alpha=-1.5, beta=beta)
        expect = -1.5 * (S.T @ a.astype(np.complex128)) + beta * o
        # FP64 arithmetic, one rounding to FP32 per component
        assert np.abs(fresh.cpu().numpy() - expect).max() <= 2.0**-23 * np.abs(expect).max()
