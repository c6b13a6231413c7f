"""The calls a user of this framework makes, as cases to be timed and compared.

A case is one evaluation ``(F, dF/du)`` of an ensemble problem (what every
optimiser iteration calls), its F-only form (line searches), a batched
evaluation of uneven problems, or a short optimiser run, each through the
package's public handles with host controls in and host results out.  Sizes
are those of ``workloads.py``, the tests and ``bench.py``.

``exact`` restates the same quantities in complex128 torch: ``matrix_exp`` for
the propagators and the block-triangular exponential for the Frechet
derivative.

Gradients of the mixed-precision path are handed on as float32: that path
computes them in FP32 (its documented bar is 1e-4 relative) and only stores
them in FP64 buffers.  Its F stays float64, and the FP64 path's outputs all do.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pg = load_package()
from pulsar_gb300 import workloads as W  # noqa: E402


def listed():
    return [
        # the smallest call: the quickstart's single qubit, latency and launches only
        dict(name="qubit_eval_fp64", kind="qubit", slices=100, members=1, precision="fp64", grad="ref_grape", want_grad=True),
        # the quickstart's whole optimiser call: twenty gradient-ascent iterations
        dict(name="qubit_grape_fp64", kind="ascent", slices=100, members=1, precision="fp64", grad="ref_grape", iterations=20),
        # one long pulse on two qubits, no ensemble: nothing to spread over the chip but the slices
        dict(name="long_pulse_d4_mixed", kind="uneven", d=4, slices=2000, members=1, controls=4, target="gate",
             precision="mixed", grad="exact", fidelity="square", want_grad=True),
        # an MR state-transfer ensemble with a dimension that is no power of two, first-order MR gradient
        dict(name="states_d6_mr_fp64", kind="uneven", d=6, slices=333, members=37, controls=3, target="states", pairs=2,
             precision="fp64", grad="ref_mr", fidelity="real", want_grad=True),
        # an ordinary gate ensemble in the default precision
        dict(name="gate_d8_fp64", kind="uneven", d=8, slices=500, members=32, controls=4, target="gate",
             precision="fp64", grad="exact", fidelity="square", want_grad=True),
        # the broadband four-spin ensemble at full size in the default precision
        dict(name="spin4_gate_fp64", kind="spin4", slices=1000, offsets=21, scales=11, target="gate", precision="fp64",
             grad="exact", want_grad=True),
        # two-qubit Lindblad gates in the default precision
        dict(name="lindblad2q_fp64", kind="lindblad", qubits=2, slices=500, members=32, precision="fp64", grad="exact", want_grad=True),
        # the same broadband ensemble, mixed precision: the benchmark's own step
        dict(name="spin4_gate_mixed", kind="spin4", slices=1000, offsets=21, scales=11, target="gate", precision="mixed",
             grad="exact", want_grad=True),
        # a line-search trial point of it: F alone
        dict(name="spin4_value_mixed", kind="spin4", slices=1000, offsets=21, scales=11, target="gate", precision="mixed",
             grad="exact", want_grad=False),
        # a large d = 32 gate ensemble, the class that dominates uneven batches
        dict(name="gate_d32_mixed", kind="uneven", d=32, slices=500, members=64, controls=4, target="gate",
             precision="mixed", grad="exact", fidelity="square", want_grad=True),
        # three-qubit Lindblad gates (superoperators of 64 x 64)
        dict(name="lindblad3q_mixed", kind="lindblad", qubits=3, slices=500, members=32, precision="mixed", grad="exact", want_grad=True),
        # many uneven problems evaluated together, as one graph
        dict(name="batch24_mixed", kind="batch", problems=24, shapes=4, max_slices=400, max_members=32, precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["uneven"] * 5 + ["spin4", "lindblad", "qubit", "ascent", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    if kind in ("qubit", "ascent"):
        case = dict(kind=kind, slices=_log_int(rng, 20, 2000), members=1, precision="fp64", grad="ref_grape")
        case.update(dict(iterations=rng.randint(3, 20)) if kind == "ascent" else dict(want_grad=rng.random() < 0.8))
        return case
    if kind == "spin4":
        return dict(kind=kind, slices=_log_int(rng, 30, 1000), offsets=rng.randint(1, 21), scales=rng.randint(1, 11),
                    target=rng.choice(["gate", "states"]), precision=precision, grad=rng.choice(["exact", "exact", "ref_mr"]),
                    want_grad=rng.random() < 0.8)
    if kind == "lindblad":
        qubits = rng.choice([1, 2, 2, 3])
        most = 16000 if precision == "mixed" or qubits < 3 else 2000
        slices = _log_int(rng, 20, 500)
        return dict(kind=kind, qubits=qubits, slices=slices, members=_log_int(rng, 1, min(32, most // slices)),
                    precision=precision, grad="exact", want_grad=True)
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 32), shapes=rng.randint(0, 1 << 20), max_slices=_log_int(rng, 60, 400),
                    max_members=_log_int(rng, 2, 32), precision="mixed")
    d = rng.choice([2, 3, 4, 6, 8, 9, 12, 16, 16, 20, 32])
    padded = 1 << (d - 1).bit_length()
    units = int((2.0e9 if precision == "mixed" else 9.0e8) / padded ** 3)
    slices = min(_log_int(rng, 30, 2000), units)
    target = rng.choice(["gate", "gate", "states"])
    case = dict(kind=kind, d=d, slices=slices, members=_log_int(rng, 1, max(1, min(128, units // slices))),
                controls=rng.randint(2, 6), target=target, precision=precision,
                grad=rng.choice(["exact", "exact", "ref_mr", "ref_grape"]), fidelity=rng.choice(["square", "real"]),
                want_grad=rng.random() < 0.8)
    if target == "states":
        case["pairs"] = rng.randint(1, 4)
    return case


def _uneven(rng, d, slices, members, controls):
    """``workloads.uneven_problem`` with its number of controls given."""
    spec, u0 = W.uneven_problem(rng, d=d, n_t=slices, n_members=members)
    sigma = 2 * np.pi * 1e6
    a = rng.normal(0.0, sigma, (controls, d, d)) + 1j * rng.normal(0.0, sigma, (controls, d, d))
    spec.controls = (a + a.conj().transpose(0, 2, 1)) / 2
    return spec, rng.uniform(-1, 1, (controls, slices))


def _unit_vectors(rng, n, d):
    v = rng.standard_normal((n, d)) + 1j * rng.standard_normal((n, d))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _specs(case, seed):
    """[(Spec, u0)] of a case: one, or one per problem of a batch."""
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("qubit", "ascent"):
        spec, _ = W.single_qubit_transfer(seed=seed, explicit_init=True)
        n_t = case["slices"]
        spec.dt = np.full(n_t, np.pi / n_t)
        return [(spec, rng.uniform(-0.5, 0.5, (2, n_t)))]
    if kind == "spin4":
        make = W.spin4_ensemble if case["target"] == "gate" else W.spin4_state_transfer
        return [make(seed=seed, n_t=case["slices"], n_off=case["offsets"], n_b1=case["scales"])]
    if kind == "lindblad":
        return [W.lindblad_gate(seed=seed, n_qubits=case["qubits"], n_t=case["slices"], n_draws=case["members"],
                                duration=2e-6 * case["slices"] / 500)]
    if kind == "batch":
        shapes = np.random.default_rng(case["shapes"])
        out = []
        for _ in range(case["problems"]):
            d = int(shapes.choice([2, 4, 8, 16, 32]))
            n_t = int(round(math.exp(shapes.uniform(math.log(50), math.log(case["max_slices"])))))
            nm = int(round(math.exp(shapes.uniform(0.0, math.log(case["max_members"])))))
            out.append(_uneven(rng, d, n_t, nm, int(shapes.integers(2, 7))))
        return out
    spec, u0 = _uneven(rng, case["d"], case["slices"], case["members"], case["controls"])
    spec.fidelity = case["fidelity"]
    if case["target"] == "states":
        spec.target, spec.target_op = "states", None
        spec.states_init = _unit_vectors(rng, case["pairs"], case["d"])
        spec.states_target = _unit_vectors(rng, case["pairs"], case["d"])
    return [(spec, u0)]


def prepare(case, seed):
    grad, precision = case.get("grad", "exact"), case["precision"]
    items = [(pg.Problem(**spec.problem_kwargs(grad, precision)), u0) for spec, u0 in _specs(case, seed)]
    state = dict(case=case, problems=[p for p, _ in items], u=[u for _, u in items])
    if case["kind"] == "batch":
        state["batch"] = pg.Batch(state["problems"], n_streams=8)
    return state


def run(state):
    case = state["case"]
    as_computed = np.float32 if case["precision"] == "mixed" else np.float64
    if case["kind"] == "batch":
        batch = state["batch"]
        for i, u in enumerate(state["u"]):
            batch.set_controls(i, u)
        F = batch.eval()
        return {"F": F, "G": [batch.get_controls(i)[1].astype(as_computed) for i in range(len(F))]}
    problem, u = state["problems"][0], state["u"][0]
    if case["kind"] == "ascent":
        # a small fixed step: every run does all its iterations and stays far from the stop rules
        r = problem.optimize(u, "grape", max_iter=case["iterations"], convergence_tol=1e-300, gradient_norm_tol=1e-300,
                             step_size=0.01, max_step_size=0.1)
        return {"controls": r.controls, "F": np.float64(r.fidelity), "F_history": np.array(r.fidelity_history),
                "G_norms": np.array(r.gradient_norm_history)}
    F, G = problem.eval(u, want_grad=case["want_grad"])
    F = np.float64(F)
    return {"F": F, "G": G.astype(as_computed)} if case["want_grad"] else {"F": F}


def work(case):
    """Per member and slice, in complex D x D products of 8 D^3 operations: the
    exponential by its cheapest polynomial (3), the forward chain (1) and, with
    a gradient, the backward chain (2) and one Frechet derivative (3 products
    for each of the exponential's); state targets move vectors in place of
    matrices in both chains, and first-order gradients take no derivative."""
    flops = bytes_ = 0.0
    if case["kind"] == "batch":
        shapes = np.random.default_rng(case["shapes"])
        sizes = []
        for _ in range(case["problems"]):
            d = int(shapes.choice([2, 4, 8, 16, 32]))
            n_t = int(round(math.exp(shapes.uniform(math.log(50), math.log(case["max_slices"])))))
            nm = int(round(math.exp(shapes.uniform(0.0, math.log(case["max_members"])))))
            sizes.append((d, n_t, nm, int(shapes.integers(2, 7)), "gate", 0, "exact", True, 1))
    else:
        kind = case["kind"]
        d = {"qubit": 2, "ascent": 2, "spin4": 16}.get(kind) or (4 ** case["qubits"] if kind == "lindblad" else case["d"])
        nm = case["offsets"] * case["scales"] if kind == "spin4" else case["members"]
        n_c = 2 * case["qubits"] if kind == "lindblad" else case.get("controls", 2)
        target = "states" if kind in ("qubit", "ascent") else case.get("target", "gate")
        sizes = [(d, case["slices"], nm, n_c, target, case.get("pairs", 2 if kind == "spin4" else 1), case["grad"],
                  case.get("want_grad", True), case.get("iterations", 1))]
    for d, n_t, nm, n_c, target, pairs, grad, want_grad, passes in sizes:
        product = 8.0 * d ** 3
        chain = product if target == "gate" else 8.0 * pairs * d * d
        per_unit = 3 * product + chain
        if want_grad:
            per_unit += (2 if target == "gate" else 1) * chain + 8.0 * n_c * d * d
            if grad == "exact":
                per_unit += 9 * product
        flops += passes * nm * n_t * per_unit
        bytes_ += 16.0 * d * d * (n_c + 2) + 8.0 * n_t * (1 + 2 * n_c) + 32.0 * nm
    return {"bytes": bytes_, "flops": flops}


def _c(x, device):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device=device)


def _exact_eval(spec, u, grad, want_grad, device):
    di, sc, of, w = spec.members()
    nm, n_t, n_c, D = spec.n_members, spec.n_t, spec.n_c, spec.D
    factor = -1j if spec.generator == "hermitian" else 1.0
    drifts, ctrls = _c(spec.drifts, device), _c(spec.controls, device)
    offset = _c(spec.offset_op, device) if spec.offset_op is not None else torch.zeros(D, D, dtype=torch.complex128, device=device)
    scale, off, weight, dt = (torch.as_tensor(np.asarray(v, float), device=device) for v in (sc, of, w, spec.dt))
    H0 = drifts[torch.as_tensor(np.asarray(di), device=device, dtype=torch.int64)] + off[:, None, None] * offset
    Hc = torch.einsum("jk,jab->kab", torch.as_tensor(u, dtype=torch.complex128, device=device), ctrls)
    A = factor * dt[None, :, None, None] * (H0[:, None] + scale[:, None, None, None] * Hc[None])
    flat = A.reshape(-1, D, D)
    per = max(1, int(2.5e8 / (D * D * 16)))
    U = torch.cat([torch.linalg.matrix_exp(flat[i:i + per]) for i in range(0, len(flat), per)]).reshape(nm, n_t, D, D)
    chain_grad = spec.target == "gate" or want_grad
    eye = torch.eye(D, dtype=torch.complex128, device=device).expand(nm, D, D)
    X = eye if spec.target == "gate" else _c(spec.states_init, device).T.expand(nm, D, -1)
    before = torch.empty((nm, n_t) + X.shape[1:], dtype=torch.complex128, device=device) if chain_grad else None
    for k in range(n_t):
        if before is not None:
            before[:, k] = X
        X = U[:, k] @ X
    if spec.target == "gate":
        T = _c(spec.target_op, device)
        z = torch.einsum("ab,mab->m", T.conj(), X)[:, None] / D
    else:
        T = _c(spec.states_target, device).T
        z = torch.einsum("as,mas->ms", T.conj(), X)
    if spec.fidelity == "square":
        f, kappa = z.abs() ** 2, 2 * z.conj()
    else:
        f, kappa = z.real, torch.ones_like(z)
    F = float((weight[:, None] * f).sum())
    if not want_grad:
        return np.float64(F), None
    kappa = kappa * weight[:, None]
    if spec.target == "gate":
        cost = (kappa / D)[:, :, None] * T.conj().T       # Lambda: dF = Re Tr(Lambda dU_total)
    else:
        cost = kappa[:, :, None] * T.conj().T             # rows kappa_s <t_s|
    M = torch.empty((nm, n_t, D, D), dtype=torch.complex128, device=device)
    for k in range(n_t - 1, -1, -1):
        if grad == "ref_grape":
            cost = cost @ U[:, k]
        M[:, k] = before[:, k] @ cost
        if grad != "ref_grape":
            cost = cost @ U[:, k]
    del before, U
    if grad == "exact":
        flat_m = M.reshape(-1, D, D)
        per = max(1, per // 16)
        for i in range(0, len(flat), per):
            a = flat[i:i + per]
            block = torch.zeros(len(a), 2 * D, 2 * D, dtype=torch.complex128, device=device)
            block[:, :D, :D], block[:, D:, D:], block[:, :D, D:] = a, a, flat_m[i:i + per]
            flat_m[i:i + per] = torch.linalg.matrix_exp(block)[:, :D, D:]
        M = flat_m.reshape(nm, n_t, D, D)
    G = torch.zeros(n_c, n_t, dtype=torch.float64, device=device)
    for j in range(n_c):
        t = torch.einsum("mkab,ba->mk", M, ctrls[j]) * factor
        G[j] = (t.real * scale[:, None]).sum(0) * dt
    return np.float64(F), G.cpu().numpy()


def exact(case, seed):
    if case["kind"] == "ascent":
        return None  # an optimiser's whole trajectory: held to the bound of its type
    device = "cuda" if torch.cuda.is_available() else "cpu"
    out = [_exact_eval(spec, u, case.get("grad", "exact"), case.get("want_grad", True), device) for spec, u in _specs(case, seed)]
    if case["kind"] == "batch":
        return {"F": np.array([F for F, _ in out]), "G": [G for _, G in out]}
    return {"F": out[0][0], "G": out[0][1]} if case["want_grad"] else {"F": out[0][0]}
