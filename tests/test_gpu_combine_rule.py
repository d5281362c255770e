"""complex64 combines on both sides of the rule between one and two rows per
thread: whole and nearly empty last rounds of blocks, few and many outputs."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import solver_ops  # noqa: E402


# rb rows (pairs) per block: 128 for 8 outputs, 32 for 20 and 32
@pytest.mark.parametrize("k,rb", [(8, 128), (20, 32), (32, 32)])
@pytest.mark.parametrize("blocks", [1, 137, 138, 148, 149, 275, 276, 1184, 1185, 1776, 1777])
def test_both_kernels_give_the_same_bits(k: int, rb: int, blocks: int) -> None:
    n = 2 * rb * blocks
    gen = torch.Generator(device="cuda")
    gen.manual_seed(blocks)
    A = torch.randn(6, n, dtype=torch.complex64, device="cuda", generator=gen)
    S = torch.from_numpy(np.random.default_rng(k).normal(size=(6, k)) * (1 + 0.5j)).cuda()
    out = torch.empty(k, n, dtype=torch.complex64, device="cuda")
    solver_ops.combine(A, S, out)
    odd = torch.empty(k, n + 1, dtype=torch.complex64, device="cuda")  # an odd length: one row per thread
    solver_ops.combine(torch.cat([A, A[:, :1]], dim=1), S, odd)
    assert torch.equal(out, odd[:, :n])
    expect = S.T @ A.to(torch.complex128)
    assert float((out - expect).abs().max()) <= 2.0**-23 * float(expect.abs().max())
