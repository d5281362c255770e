"""The work whose speed this repository is judged by: one case per way a
program uses the framework, each through the public entry points.

``listed()`` names the cases, ``draw()`` gives more of the same ranges,
``prepare()`` builds what a program holds before the call, ``run()`` is one
pass, ``work()`` counts the bytes and operations a pass cannot do without and
``exact()`` gives the same outputs from plain torch in 64 bits.

Kinds:

* ``mvp``      y = H x on device tensors (``NativeMVPPlan.apply_device``);
* ``batch``    many lattices x a block of right-hand sides (``BatchedMVP``);
* ``sector``   y = H x inside a fixed-particle-number sector;
* ``host``     y = H x on ordinary NumPy arrays (``NativeMVPPlan.apply_into``);
* ``davidson`` the vector work of one eigensolver iteration: projected matrix,
  residual block and its Gram matrix;
* ``precond``  the learned correction of a block of residuals;
* ``train``    one training step of the preconditioner network.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from tencirpauli_b200 import PauliOperator, U1Sector, mapping, precond, solver_ops, workloads
from tencirpauli_b200.batch import BatchedMVP

CLAMP = 4.0  # default clamp of the learned correction
EPS = 1e-8   # default floor of |H_ii - theta|


def listed():
    return [
        # smallest call: a 10-qubit lattice inside a host-side loop; launch bound
        {"name": "mvp_c128_lattice10", "kind": "mvp", "model": "lattice", "n": 10, "dtype": "c128", "nrhs": 1},
        # the plain 20-qubit periodic Heisenberg chain, one state
        {"name": "mvp_c128_chain20", "kind": "mvp", "model": "chain", "n": 20, "dtype": "c128", "nrhs": 1},
        # the headline workload: 2,000 random 2..4-local words on 28 qubits
        {"name": "mvp_c128_random28", "kind": "mvp", "model": "random", "n": 28, "words": 2000, "dtype": "c128",
         "nrhs": 1},
        # the same generator in the FP32-with-compensation mode
        {"name": "mvp_c64_random26", "kind": "mvp", "model": "random", "n": 26, "words": 2000, "dtype": "c64",
         "nrhs": 1},
        # the MVP of a Davidson block on the periodic 4 x 6 J1-J2 lattice
        {"name": "mvp_c64_j1j2_24_block4", "kind": "mvp", "model": "j1j2", "n": 24, "lx": 4, "j2": 0.5,
         "dtype": "c64", "nrhs": 4},
        # Jordan-Wigner chemistry-like operator: tens of thousands of words
        {"name": "mvp_c128_chemistry20", "kind": "mvp", "model": "chemistry", "n": 20, "dtype": "c128", "nrhs": 1},
        # lattices of uneven size, 8 right-hand sides each, one call
        {"name": "batch_c64_lattices16to22", "kind": "batch", "members": 12, "nmin": 16, "nmax": 22, "nrhs": 8,
         "dtype": "c64"},
        # half filling of the periodic 4 x 6 J1-J2 lattice
        {"name": "sector_c128_j1j2_24", "kind": "sector", "model": "j1j2", "n": 24, "lx": 4, "j2": 0.5, "k": 12,
         "dtype": "c128", "nrhs": 1},
        # a NumPy caller: 64 MiB in, 64 MiB out, ordinary memory
        {"name": "host_c128_chain22", "kind": "host", "model": "chain", "n": 22},
        # Rayleigh-Ritz and residual of a 40-vector complex64 basis, block of 4
        {"name": "davidson_c64_basis40", "kind": "davidson", "n": 1 << 22, "basis": 40, "block": 4, "dtype": "c64"},
        # learned correction of 4 residuals in the FP64 phase
        {"name": "precond_c128_block4", "kind": "precond", "n": 1 << 22, "block": 4, "dtype": "c128"},
        # one gradient of the default (alignment) training objective: forward, loss
        # and dL/dc, back-propagation over the states of 24 4 x 4 lattice sets
        {"name": "train_alignment_24sets", "kind": "train", "objective": "alignment", "sets": 24, "size": 1 << 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mvp"] * 6 + ["batch", "sector", "sector", "host", "davidson", "precond", "train"])
    dtype = rng.choice(["c128", "c64"])
    if kind in ("mvp", "host"):
        model = rng.choice(["lattice", "chain", "random", "random", "j1j2", "chemistry"])
        case = {"kind": kind, "model": model}
        if model == "random":
            case["n"] = rng.randint(8, 25 if kind == "host" else 27)
            case["words"] = _log_int(rng, 20, 2000)
        elif model == "j1j2":
            case["lx"] = rng.choice([3, 4, 5])
            case["n"] = case["lx"] * rng.randint(2, 24 // case["lx"])
            case["j2"] = round(rng.uniform(0.0, 0.6), 3)
        elif model == "chemistry":
            case["n"] = rng.randint(8, 19)
        else:
            case["n"] = rng.randint(6, 25)
        if kind == "mvp":
            case["dtype"] = dtype
            case["nrhs"] = rng.choice([1, 1, 1, 2, 3, 4]) if case["n"] <= 24 else 1
        return case
    if kind == "batch":
        nmin = rng.randint(12, 17)
        return {"kind": kind, "members": rng.randint(3, 24), "nmin": nmin, "nmax": nmin + rng.randint(0, 5),
                "nrhs": rng.choice([1, 2, 3, 4, 8]), "dtype": dtype}
    if kind == "sector":
        model = rng.choice(["j1j2", "chain", "hopping"])
        case = {"kind": kind, "model": model, "dtype": dtype, "nrhs": rng.choice([1, 1, 2, 4])}
        if model == "j1j2":
            case["lx"] = rng.choice([3, 4])
            case["n"] = case["lx"] * rng.randint(3, 24 // case["lx"])
            case["j2"] = round(rng.uniform(0.0, 0.6), 3)
        else:
            case["n"] = rng.randint(10, 24)
        case["k"] = rng.randint(max(1, case["n"] // 4), case["n"] - max(1, case["n"] // 4))
        return case
    if kind == "davidson":
        return {"kind": kind, "n": _log_int(rng, 1 << 14, 1 << 22), "basis": rng.randint(4, 64),
                "block": rng.randint(1, 6), "dtype": dtype}
    if kind == "precond":
        return {"kind": kind, "n": _log_int(rng, 1 << 14, 1 << 23), "block": rng.randint(1, 6), "dtype": dtype}
    if rng.random() < 0.5:
        return {"kind": kind, "objective": "l2", "samples": _log_int(rng, 1 << 12, 1 << 21)}
    return {"kind": kind, "objective": "alignment", "sets": rng.randint(1, 32), "size": _log_int(rng, 1 << 10, 1 << 16)}


# ------------------------------- inputs --------------------------------------
def _terms(case, seed):
    """Term rows (codes, coefficients) of the case's Hamiltonian."""
    n, model = case["n"], case["model"]
    if model == "lattice":
        return workloads.heisenberg_2d_open(n, seed)
    if model == "chain":
        return workloads.heisenberg_chain(n, field=0.5)
    if model == "j1j2":
        return workloads.j1j2_periodic(case["lx"], n // case["lx"], 1.0, case["j2"])
    if model == "random":
        return workloads.random_k_local(n=n, words=case["words"], seed=seed)
    if model == "hopping":
        return _hopping(n, seed)
    return mapping.jordan_wigner_integrals(*mapping.chemistry_integrals(n, seed=seed))


def _hopping(n, seed):
    """Jordan-Wigner hopping between 3n random pairs of modes (X Z..Z X +
    Y Z..Z Y), density-density couplings on the same pairs and random levels."""
    rng = np.random.default_rng(seed)
    rows, coeffs = [], []
    for _ in range(3 * n):
        p, q = sorted(int(v) for v in rng.choice(n, size=2, replace=False))
        t, v = rng.normal(size=2)
        for letter in (1, 2):
            row = np.zeros(n, dtype=np.uint8)
            row[p + 1 : q] = 3
            row[p] = row[q] = letter
            rows.append(row)
            coeffs.append(0.5 * t)
        row = np.zeros(n, dtype=np.uint8)
        row[p] = row[q] = 3
        rows.append(row)
        coeffs.append(0.25 * v)
    for p in range(n):
        row = np.zeros(n, dtype=np.uint8)
        row[p] = 3
        rows.append(row)
        coeffs.append(rng.normal())
    return np.asarray(rows, dtype=np.uint8), np.asarray(coeffs, dtype=np.complex128)


def _dtype(case):
    return torch.complex128 if case.get("dtype", "c128") == "c128" else torch.complex64


def _state(length, seed, dtype, nrhs=1):
    """I.i.d. normal, normalised; (length,) or (nrhs, length)."""
    x = workloads.random_state_device(0, seed=seed, dtype=dtype, nrhs=nrhs, length=length)
    return x[0].clone() if nrhs == 1 else x


def _lattices(case, seed):
    # the sizes belong to the case, the couplings to the seed
    sizes = np.random.default_rng(case["members"]).integers(case["nmin"], case["nmax"] + 1, size=case["members"])
    sizes[0], sizes[-1] = case["nmax"], case["nmin"]
    return [(int(n), *workloads.heisenberg_2d_open(int(n), seed + 1 + i)) for i, n in enumerate(sizes)]


def _normal(gen, shape, dtype):
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    return torch.complex(torch.randn(shape, generator=gen, device="cuda", dtype=real),
                         torch.randn(shape, generator=gen, device="cuda", dtype=real))


def _davidson_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, m, k, dtype = case["n"], case["basis"], case["block"], _dtype(case)
    scale = 1.0 / math.sqrt(2.0 * n)
    V = _normal(gen, (m, n), dtype).mul_(scale)
    W = _normal(gen, (m, n), dtype).mul_(scale)
    S = _normal(gen, (m, k), torch.complex128) / math.sqrt(2.0 * m)
    theta = torch.randn(k, generator=gen, device="cuda", dtype=torch.float64)
    return V, W, S, theta


def _params(seed):
    params = precond.init_params(seed)
    rng = np.random.default_rng(seed + 1)
    params[-17:] = rng.normal(scale=0.3, size=17)  # a trained network's output layer is not zero
    return torch.from_numpy(params).cuda()


def _precond_inputs(case, seed):
    """Residuals, per-state features and diagonal of a spin lattice's size and spread."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, k = case["n"], case["block"]
    R = _normal(gen, (k, n), _dtype(case)).mul_(1e-5 / math.sqrt(n))
    diag = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) * 6.0
    count = torch.randint(20, 60, (n,), generator=gen, device="cuda").to(torch.float32)
    noise = torch.randn((n, 2), generator=gen, device="cuda")
    feat = torch.zeros((n, solver_ops.TCP_FEATURES), dtype=torch.float32, device="cuda")
    feat[:, 0] = diag.to(torch.float32)
    feat[:, 1] = feat[:, 0] * 0.9 + noise[:, 0]
    feat[:, 2] = feat[:, 1] - 4.0 - noise[:, 1].abs()
    feat[:, 3] = 1.5 * count
    feat[:, 4] = 2.5 * count
    feat[:, 5] = count
    feat[:, 6] = torch.rand(n, generator=gen, device="cuda") - 0.5
    theta = -45.0 + 0.7 * torch.arange(k, device="cuda", dtype=torch.float64)
    return R, feat, torch.complex(diag, torch.zeros_like(diag)), theta, _params(seed), 11.0


def _train_inputs(case, seed):
    """Network inputs and what the objective needs beside them, then the parameters."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["objective"] == "l2":
        n = case["samples"]
    else:
        n = case["sets"] * case["size"]
    X = torch.randn((n, solver_ops.TCP_MLP_IN), generator=gen, device="cuda") * 0.7
    den = 0.5 + 3.0 * torch.rand(n, generator=gen, device="cuda")
    if case["objective"] == "l2":
        r = torch.randn(n, generator=gen, device="cuda")
        e = -r / den * (1.0 + 0.3 * torch.randn(n, generator=gen, device="cuda"))
        wt = torch.full((n,), 1.0 / n, device="cuda")
        return X, den, r * r, e * r, e * e, wt, _params(seed)
    r = _normal(gen, (n,), torch.complex128)
    e = -r / den * torch.exp(0.5 * X[:, 0].to(torch.float64)) + 0.3 * _normal(gen, (n,), torch.complex128)
    u = _normal(gen, (n,), torch.complex128) / math.sqrt(2.0 * case["size"])
    E = (e.real**2 + e.imag**2).view(case["sets"], case["size"]).sum(1)
    seg = torch.arange(case["sets"], device="cuda").repeat_interleave(case["size"])
    begin = torch.arange(case["sets"] + 1, device="cuda") * case["size"]
    return X, den, torch.conj(e) * r, r.real**2 + r.imag**2, torch.conj(u) * r, E, seg, begin, _params(seed)


# ------------------------------ the measured path ----------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mvp":
        plan = PauliOperator.from_code_arrays(*_terms(case, seed)).native_mvp_plan()
        x = _state(1 << case["n"], seed, _dtype(case), case["nrhs"])
        return {"kind": kind, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "batch":
        plans, xs = [], []
        for i, (n, codes, coeffs) in enumerate(_lattices(case, seed)):
            plans.append(PauliOperator.from_code_arrays(codes, coeffs).native_mvp_plan())
            xs.append(workloads.random_state_device(0, seed=seed + i, dtype=_dtype(case), nrhs=case["nrhs"], length=1 << n))
        batch = BatchedMVP(plans, case["nrhs"], "complex128" if case["dtype"] == "c128" else "complex64")
        return {"kind": kind, "batch": batch, "xs": xs, "ys": [torch.empty_like(x) for x in xs]}
    if kind == "sector":
        op = PauliOperator.from_code_arrays(*_terms(case, seed))
        plan = op.restrict_charge(U1Sector(case["n"], case["k"])).mvp_plan()
        x = _state(math.comb(case["n"], case["k"]), seed, _dtype(case), case["nrhs"])
        return {"kind": kind, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "host":
        plan = PauliOperator.from_code_arrays(*_terms(case, seed)).native_mvp_plan()
        x = _state(1 << case["n"], seed, torch.complex128).cpu().numpy()
        return {"kind": kind, "plan": plan, "x": x, "y": np.zeros_like(x)}
    if kind == "davidson":
        V, W, S, theta = _davidson_inputs(case, seed)
        Sv = -S * theta.to(torch.complex128)
        return {"kind": kind, "V": V, "W": W, "S": S, "Sv": Sv, "R": torch.empty_like(V[: case["block"]]),
                "block": case["block"]}
    if kind == "precond":
        R, feat, diag, theta, params, scale = _precond_inputs(case, seed)
        return {"kind": kind, "args": (R, feat, diag, theta, params, scale), "out": torch.empty_like(R)}
    *data, params = _train_inputs(case, seed)
    data = [t.resolve_conj().contiguous() for t in data]
    state = {"kind": kind, "objective": case["objective"], "data": data, "params": params}
    if case["objective"] == "alignment":
        X, den, alpha, a, gamma, E, seg, begin = data
        state["sets"] = precond.AlignmentSets(X, den, alpha, a, gamma, E, seg, case["sets"], begin)
    return state


def run(state):
    kind = state["kind"]
    if kind in ("mvp", "sector"):
        state["plan"].apply_device(state["x"], state["y"])
        return state["y"]
    if kind == "batch":
        state["batch"].apply(state["xs"], state["ys"])
        return state["ys"]
    if kind == "host":
        state["plan"].apply_into(state["x"], state["y"])
        return state["y"]
    if kind == "davidson":
        V, W, R = state["V"], state["W"], state["R"]
        G = solver_ops.gram(V, W[-state["block"]:])  # new columns of the projected matrix
        solver_ops.combine(V, state["Sv"], R)        # R = W S - V S diag(theta)
        solver_ops.combine(W, state["S"], R, beta=1.0)
        return {"projected": G, "residual": R, "norms": solver_ops.gram(R, R)}
    if kind == "precond":
        return solver_ops.mlp_precondition(*state["args"], state["out"])
    trainer = solver_ops.MLPTrainer(state["params"].clone())
    if state["objective"] == "l2":
        trainer.step(*state["data"], 3e-3)
        return {"params": trainer.params, "m": trainer.m, "v": trainer.v, "grad": trainer.grad, "loss": trainer.loss}
    sets = state["sets"]
    c = solver_ops.mlp_forward(sets.X, trainer.params)
    loss, dc = precond.alignment_loss_and_dc(c, sets, CLAMP)
    # the gradient alone: this objective does not change with the output bias, so
    # Adam would divide that parameter's rounding noise by itself
    trainer.backward_step(sets.X, dc, 0.0)
    return {"grad": trainer.grad, "loss": loss, "c": c, "dc": dc}


# ------------------------------ what a pass needs ----------------------------
def _mvp_work(n, length, codes, nrhs, elem):
    """x read once and y written once; per amplitude every term's signed weight
    is added once and every distinct flip pattern takes one multiply-add."""
    flips = ((codes == 1) | (codes == 2)).astype(np.uint8)
    groups = np.unique(flips, axis=0).shape[0] if codes.shape[0] else 0
    words = np.unique(codes, axis=0).shape[0] if codes.shape[0] else 0
    return 2.0 * length * elem * nrhs, float(length) * nrhs * (2 * words + 8 * groups)


def work(case):
    kind = case["kind"]
    elem = 16 if case.get("dtype", "c128") == "c128" else 8
    if kind in ("mvp", "host"):
        nbytes, flops = _mvp_work(case["n"], 1 << case["n"], _terms(case, 0)[0], case.get("nrhs", 1), elem)
    elif kind == "sector":
        nbytes, flops = _mvp_work(case["n"], math.comb(case["n"], case["k"]), _terms(case, 0)[0], case["nrhs"], elem)
    elif kind == "batch":
        parts = [_mvp_work(n, 1 << n, codes, case["nrhs"], elem) for n, codes, _ in _lattices(case, 0)]
        nbytes, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "davidson":
        n, m, k = case["n"], case["basis"], case["block"]
        nbytes = float(elem) * n * (2 * m + k)
        flops = 8.0 * n * (3 * m * k + k * k)
    elif kind == "precond":
        n, k = case["n"], case["block"]
        nbytes = n * (2.0 * elem * k + 32 + 16)
        flops = 2.0 * n * k * (8 * 16 + 16 * 16 + 16)
    else:
        if case["objective"] == "l2":
            n, nbytes = case["samples"], case["samples"] * (8 + 5) * 4.0
        else:  # inputs, den, alpha, a, gamma and the set index in; c and dL/dc out
            n = case["sets"] * case["size"]
            nbytes = n * (32.0 + 4 + 16 + 8 + 16 + 8 + 4 + 4)
        flops = n * 6.0 * (8 * 16 + 16 * 16 + 16)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------ 64-bit results -------------------------------
def _dense_apply(n, codes, coeffs, x):
    """sum_k c_k P_k x for x of shape (..., 2^n), complex128, term by term.
    Qubit 0 is the most significant index bit."""
    rows, inverse = np.unique(codes, axis=0, return_inverse=True)
    weights = np.zeros(rows.shape[0], dtype=np.complex128)
    np.add.at(weights, inverse.reshape(-1), np.asarray(coeffs, dtype=np.complex128))
    ny = (rows == 2).sum(axis=1) % 4
    weights = weights * np.array([1.0, 1.0j, -1.0, -1.0j])[ny]
    flips = (rows == 1) | (rows == 2)
    signs = (rows == 2) | (rows == 3)
    order = np.lexsort(flips.T[::-1])
    lead = x.numel() >> n
    xr = torch.view_as_real(x.to(torch.complex128).contiguous())
    acc = [torch.zeros_like(xr), None]  # real weights, imaginary weights

    def shape_of(qubits):
        shape, prev = [lead], -1
        for q in qubits:
            shape += [1 << (q - prev - 1), 2]
            prev = q
        return shape + [1 << (n - 1 - prev), 2]

    last, xf = None, None
    for t in order:
        if weights[t] == 0:
            continue
        key = flips[t].tobytes()
        if key != last:
            last = key
            fq = np.flatnonzero(flips[t])
            xf = xr.view(shape_of(fq)).flip([2 + 2 * i for i in range(len(fq))]).contiguous() if len(fq) else xr
        zq = np.flatnonzero(signs[t])
        # (P x)[r] = w (-1)^{z.(r ^ m)} x[r ^ m]: the flipped qubits add a constant sign
        flip = -1.0 if int((flips[t] & signs[t]).sum()) & 1 else 1.0
        shape = shape_of(zq)
        sign = torch.ones([1] * len(shape), dtype=torch.float64, device=x.device)
        for i in range(len(zq)):
            s = [1] * len(shape)
            s[2 + 2 * i] = 2
            sign = sign * torch.tensor([1.0, -1.0], dtype=torch.float64, device=x.device).view(s)
        for part, w in ((0, weights[t].real), (1, weights[t].imag)):
            if w != 0.0:
                if acc[part] is None:
                    acc[part] = torch.zeros_like(xr)
                acc[part].view(shape).addcmul_(xf.view(shape), sign, value=float(w) * flip)
    y = torch.view_as_complex(acc[0])
    if acc[1] is not None:
        y = y + 1j * torch.view_as_complex(acc[1])
    return y.view(x.shape)


def _network(params, X):
    """(c, h1, h2) of the 8-16-16-1 tanh network for rows of X, in FP64."""
    p = params.to(torch.float64)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [128, 16, 256, 16, 16, 1])
    h1 = torch.tanh(X @ w1.view(16, 8).T + b1)
    h2 = torch.tanh(h1 @ w2.view(16, 16).T + b2)
    return h2 @ w3 + b3, h1, h2


def _exact_precond(case, seed):
    R, feat, diag, theta, params, scale = _precond_inputs(case, seed)
    f = feat.to(torch.float64)
    out = torch.empty(R.shape, dtype=torch.complex128, device=R.device)
    for j in range(R.shape[0]):
        th = theta[j]
        d = f[:, 0] - th
        den = torch.where(d.abs() < EPS, torch.where(d < 0, -EPS, EPS), d)
        ratio = f[:, 4] / (den.abs() * torch.clamp((f[:, 1] - th).abs(), min=EPS))
        X = torch.stack([d / scale, (f[:, 1] - th) / scale, (f[:, 2] - th) / scale, f[:, 3] / scale,
                         f[:, 4] / scale**2, f[:, 5] * 0.05, f[:, 6], ratio / (1.0 + ratio)], dim=1)
        c = torch.clamp(_network(params, X)[0], -CLAMP, CLAMP)
        d = diag.real - th
        den = torch.where(d.abs() < EPS, torch.where(d < 0, -EPS, EPS), d)
        out[j] = (-torch.exp(c) / den) * R[j].to(torch.complex128)
    return out


def _exact_train(case, seed):
    *data, params = _train_inputs(case, seed)
    params = params.to(torch.float64)
    p = params.clone().requires_grad_(True)
    if case["objective"] == "l2":
        X, den, a, b, e2, wt = [t.to(torch.float64) for t in data]
        c = _network(p, X)[0]
        g = -torch.exp(c) / den
        loss = (wt * (g * g * a - 2.0 * g * b + e2)).sum()
        loss.backward()
    else:
        X, den, alpha, a, gamma, E = data[:6]
        c = _network(p, X.to(torch.float64))[0]
        g = -torch.exp(torch.clamp(c, -CLAMP, CLAMP)) / den.to(torch.float64)
        shape = (case["sets"], case["size"])
        A = [(g * v).view(shape).sum(1) for v in (alpha.real, alpha.imag)]
        C = [(g * v).view(shape).sum(1) for v in (gamma.real, gamma.imag)]
        D = (g * g * a).view(shape).sum(1) - C[0] ** 2 - C[1] ** 2
        loss = (1.0 - (A[0] ** 2 + A[1] ** 2) / (E * D)).mean()
        c.retain_grad()
        loss.backward()
    grad = p.grad
    if case["objective"] == "alignment":
        return {"grad": grad, "loss": float(loss.detach()), "c": c.detach(), "dc": c.grad}
    # first Adam step: the bias-corrected moments are the gradient and its square
    new = params - 3e-3 * grad / (grad.abs() + 1e-8)
    return {"params": new, "m": 0.1 * grad, "v": 0.001 * grad * grad, "grad": grad, "loss": loss.detach().reshape(1)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mvp", "host"):
        codes, coeffs = _terms(case, seed)
        dtype = torch.complex128 if kind == "host" else _dtype(case)
        x = _state(1 << case["n"], seed, dtype, case.get("nrhs", 1))
        return _dense_apply(case["n"], codes, coeffs, x)
    if kind == "batch":
        ys = []
        for i, (n, codes, coeffs) in enumerate(_lattices(case, seed)):
            x = workloads.random_state_device(0, seed=seed + i, dtype=_dtype(case), nrhs=case["nrhs"], length=1 << n)
            ys.append(_dense_apply(n, codes, coeffs, x))
        return ys
    if kind == "sector":
        codes, coeffs = _terms(case, seed)
        n = case["n"]
        x = _state(math.comb(n, case["k"]), seed, _dtype(case), case["nrhs"])
        idx = torch.arange(1 << n, device="cuda")
        ones = sum((idx >> b) & 1 for b in range(n))
        basis = torch.nonzero(ones == case["k"]).flatten()
        full = torch.zeros((*x.shape[:-1], 1 << n), dtype=torch.complex128, device="cuda")
        full[..., basis] = x.to(torch.complex128)
        return _dense_apply(n, codes, coeffs, full)[..., basis].contiguous()
    if kind == "davidson":
        V, W, S, theta = _davidson_inputs(case, seed)
        k, m = case["block"], case["basis"]
        R = torch.zeros((k, case["n"]), dtype=torch.complex128, device="cuda")
        G = torch.empty((m, k), dtype=torch.complex128, device="cuda")
        new = W[-k:].to(torch.complex128)
        for i in range(m):
            v, w = V[i].to(torch.complex128), W[i].to(torch.complex128)
            G[i] = new @ v.conj()
            R += S[i][:, None] * w - (S[i] * theta)[:, None] * v
        return {"projected": G, "residual": R, "norms": R.conj() @ R.T}
    if kind == "precond":
        return _exact_precond(case, seed)
    return _exact_train(case, seed)
