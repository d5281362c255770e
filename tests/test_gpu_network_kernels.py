"""The network kernels at the edges of their work splits: residual counts that
do not fill a thread's rows, sample counts around the chunks, rows that 16-byte
loads cannot address, training sets smaller than a cluster's threads."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("CUDA device required", allow_module_level=True)

from tencirpauli_b200 import solver_ops  # noqa: E402

# FP32 network with activations good to about 1e-7 each: 33 of them through two
# layers of weights below 1 in size stay within 1e-5 of the FP64 network.
NETWORK_ATOL = 1e-5


def _params(seed: int) -> np.ndarray:
    return np.random.default_rng(seed).normal(scale=0.3, size=mo.NPARAM).astype(np.float32)


def _shifted(a: np.ndarray):
    """The same rows, 4 bytes off a 16-byte boundary."""
    t = torch.empty(a.size + 1, dtype=torch.float32, device="cuda")[1:]
    t.copy_(torch.from_numpy(a.reshape(-1)))
    return t.view(a.shape)


@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 511, 513, 1023, 4097])
@pytest.mark.parametrize("aligned", [True, False])
def test_forward_counts(count: int, aligned: bool) -> None:
    X = np.random.default_rng(count).normal(size=(count, mo.IN)).astype(np.float32)
    p = _params(1)
    dev = torch.from_numpy(X).cuda() if aligned else _shifted(X)
    c = solver_ops.mlp_forward(dev, torch.from_numpy(p).cuda()).cpu().numpy()
    ref = np.asarray(mo.forward(p.astype(np.float64), X.astype(np.float64))[0]).reshape(-1)
    np.testing.assert_allclose(c, ref, rtol=0, atol=NETWORK_ATOL)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_every_residual_of_a_block_is_corrected_as_alone(k: int, dtype: str) -> None:
    n = 777
    rng = np.random.default_rng(k)
    feat = rng.uniform(0.5, 20.0, size=(n, 8)).astype(np.float32)
    R = (rng.normal(size=(k, n)) + 1j * rng.normal(size=(k, n))).astype(dtype)
    diag = torch.from_numpy(feat[:, 0].astype(np.complex128)).cuda()
    theta = torch.from_numpy(-3.0 - np.arange(k, dtype=np.float64)).cuda()
    p = torch.from_numpy(_params(2)).cuda()
    Rd = torch.from_numpy(R).cuda()
    out = torch.full_like(Rd, float("nan"))
    solver_ops.mlp_precondition(Rd, torch.from_numpy(feat).cuda(), diag, theta, p, 2.5, out)
    shifted = torch.full_like(Rd, float("nan"))
    solver_ops.mlp_precondition(Rd, _shifted(feat), diag, theta, p, 2.5, shifted)
    assert torch.equal(out, shifted)
    for j in range(k):
        one = torch.full_like(Rd[j : j + 1], float("nan"))
        solver_ops.mlp_precondition(Rd[j : j + 1].contiguous(), torch.from_numpy(feat).cuda(), diag, theta[j : j + 1], p, 2.5, one)
        assert torch.equal(out[j], one[0])
        expect = mo.mlp_correction(_params(2).astype(np.float64), feat.astype(np.float64), R[j].astype(np.complex128), float(theta[j]), 2.5)
        np.testing.assert_allclose(out[j].cpu().numpy(), expect, rtol=1e-4, atol=1e-6 * np.abs(expect).max())


@pytest.mark.parametrize("count", [1, 127, 128, 129, 300, 128 * 296 + 5])
@pytest.mark.parametrize("aligned", [True, False])
def test_gradient_counts(count: int, aligned: bool) -> None:
    rng = np.random.default_rng(count)
    X = rng.normal(size=(count, mo.IN)).astype(np.float32)
    den = rng.uniform(0.5, 3.0, size=count).astype(np.float32)
    a, e2 = (rng.uniform(0.1, 2.0, size=count).astype(np.float32) for _ in range(2))
    b = rng.normal(size=count).astype(np.float32)
    wt = np.full(count, 1.0 / count, dtype=np.float32)
    p = _params(3)
    trainer = solver_ops.MLPTrainer(torch.from_numpy(p.copy()).cuda())
    dev = [torch.from_numpy(v).cuda() for v in (den, a, b, e2, wt)]
    trainer.step(torch.from_numpy(X).cuda() if aligned else _shifted(X), *dev, lr=0.0)
    loss, grad = mo.loss_and_grad(p.astype(np.float64), X.astype(np.float64), den.astype(np.float64), a, b, e2, wt)
    # FP32 sums of `count` terms of one size, at most 2^-23 each in a tree
    np.testing.assert_allclose(trainer.grad.cpu().numpy(), grad, rtol=1e-4, atol=1e-5 * np.abs(grad).max())
    assert abs(trainer.loss.item() - loss) <= 1e-5 * abs(loss)


@pytest.mark.parametrize("sizes", [[1], [1, 31, 4097], [512 * 8, 512 * 8 + 1, 3]])
def test_alignment_set_sizes(sizes) -> None:
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
    # dL/dc is the difference of two terms below 1 in size, each summed in FP64
    # and then rounded to FP32; for a set of one state they cancel exactly
    np.testing.assert_allclose(dc.cpu().numpy(), dref, rtol=1e-6, atol=1e-13 * n)
