"""The alignment objective's sums by one block per set and by a cluster per set:
many small sets, few large ones, and both sides of the rule between them."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import solver_ops  # noqa: E402


@pytest.mark.parametrize(
    "sizes",
    [[48], [49], [2 * 48 * 2, 1], [2 * 48 * 2, 2], [255, 256, 257] * 20, [1 + 7 * k for k in range(300)], [5000] * 40],
    ids=["1x48", "1x49", "2x96.5", "2x97", "60 sets", "300 sets", "40x5000"],
)
def test_sums_of_blocks_and_clusters(sizes) -> None:
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    c = rng.normal(scale=0.5, size=n).astype(np.float32)
    den = rng.uniform(0.5, 3.0, size=n).astype(np.float32)
    alpha, gamma = (rng.normal(size=n) + 1j * rng.normal(size=n) for _ in range(2))
    gamma = gamma / np.sqrt(4.0 * n)
    a = rng.uniform(0.5, 2.0, size=n)
    E = rng.uniform(1.0, 2.0, size=len(sizes)) * np.asarray(sizes)
    seg = np.repeat(np.arange(len(sizes)), sizes)
    begin = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    loss, dc = solver_ops.alignment_grad(
        *[torch.from_numpy(v).cuda() for v in (c, den, alpha, a, gamma, E, seg.astype(np.int64), begin)], 4.0)
    ref, dref = mo.alignment_loss_and_dc(c, den, alpha, a, gamma, E, seg, len(sizes))
    assert abs(loss - ref) <= 1e-10 * max(1.0, abs(ref))
    # the bound of the cancelling terms, each summed in FP64 and rounded to FP32
    np.testing.assert_allclose(dc.cpu().numpy(), dref, rtol=1e-6, atol=1e-13 * n)
