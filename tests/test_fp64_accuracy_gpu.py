"""Rounding of the FP64 path against long double, and norms along long pulses.

The first test holds gate gradients to the error of the same evaluation in
doubles on the host (scipy's exponential, complex128 products), pooled over a
few short pulses: there propagators lie near the identity, where doubles keep
the small entries that the controls read to 53 bits of themselves and a block
format needs its spare bits.  Pools of three or four pulses scatter, hence half
as much again.
"""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


def _dag(x):
    return np.swapaxes(x.conj(), -1, -2)


def _expm_long(A):
    """exp(A) for norms below 1: the Taylor sum of A / 16, squared four times."""
    B = A / np.longdouble(16)
    E = np.eye(len(A), dtype=A.dtype) + B
    T = B
    for k in range(2, 20):
        T = T @ B / np.longdouble(k)
        E = E + T
    for _ in range(4):
        E = E @ E
    return E


def _frechet(A, N, real):
    """L_exp(A, M) from N = M exp(A): sum of commutators ad_A^n(N) / (n + 1)!."""
    X, T, f = N, N, real(1)
    for n in range(1, 26):
        T = A @ T - T @ A
        f = f / (n + 1)
        X = X + f * T
    return X


def _gradient(spec, u, mode, real, cplx, kappa=None):
    """dF/du of the spec's one member (square fidelity; kappa = 1: the real part) in the given types, the
    overlaps times their weight, and sum |dG/d overlap|^2."""
    c = cplx(-1j) if spec.generator == "hermitian" else cplx(1)
    ctrls = [np.asarray(x).astype(cplx) for x in spec.controls]
    di, sc, of, w = spec.members()
    sc, w = real(sc[0]), real(w[0])
    H = np.asarray(spec.drifts)[int(di[0])].astype(cplx)
    if spec.offset_op is not None:
        H = H + real(of[0]) * np.asarray(spec.offset_op).astype(cplx)
    A = [c * real(spec.dt[k]) * (H + sum(sc * real(u[j, k]) * ctrls[j] for j in range(len(ctrls)))) for k in range(len(spec.dt))]
    U = [sla.expm(a) if cplx is np.complex128 else _expm_long(a) for a in A]
    D = len(A[0])
    gate = spec.target == "gate"
    P = [np.eye(D, dtype=cplx) if gate else np.asarray(spec.states_init).astype(cplx).T]
    for x in U:
        P.append(x @ P[-1])
    T = np.asarray(spec.target_op if gate else np.asarray(spec.states_target).T).astype(cplx)
    z = np.array([np.trace(_dag(T) @ P[-1]) / D]) if gate else (T.conj() * P[-1]).sum(0)
    G, g = np.zeros(u.shape, real), real(0)
    for s in range(len(z)):
        lam = w / D * _dag(T) if gate else w * _dag(T[:, s:s + 1])
        for k in range(len(U) - 1, -1, -1):
            X = P[k] if gate else P[k][:, s:s + 1]
            after, lam = lam, lam @ U[k]
            X = _frechet(A[k], X @ lam, real) if mode == "exact" else X @ after
            for j in range(len(ctrls)):
                d = 2 * c * real(spec.dt[k]) * sc * (X.T * ctrls[j]).sum()
                G[j, k] += (np.conj(z[s]) * d if kappa is None else kappa * d / 2).real
                g += abs(d) ** 2
    return G, z * w, float(g)


def _rms(x):
    return float(np.sqrt((np.abs(x) ** 2).sum()))


def _pulses(kind):
    from pulsar_gb300 import workloads as W
    if kind == "lindblad":
        return [W.lindblad_gate(seed=n, n_qubits=2, n_t=n, n_draws=1, duration=2e-6 * n / 500) for n in (21, 33, 45, 60)]
    if kind == "uneven":
        return [W.uneven_problem(np.random.default_rng(d), d=d, n_t=30, n_members=1) for d in (5, 8, 20)]
    return [W.spin4_ensemble(seed=n, n_t=n, n_off=1, n_b1=1) for n in (30, 37, 46, 56)]


@pytest.mark.parametrize("mode", ["exact", "ref_mr"])
@pytest.mark.parametrize("kind", ["lindblad", "uneven", "spin4"])
def test_gate_gradient_of_short_pulses(pg, kind, mode):
    device, host = [], []
    for spec, u in _pulses(kind):
        G = _gradient(spec, u, mode, np.longdouble, np.clongdouble)[0]
        p = pg.Problem(**spec.problem_kwargs(mode, "fp64"))
        _, Gd = p.eval(u)
        p.close()
        device.append(_rms(Gd - G) / _rms(G))
        host.append(_rms(_gradient(spec, u, mode, np.float64, np.complex128)[0] - G) / _rms(G))
    print(f"{kind} {mode}: device", device, "doubles", host)
    assert _rms(device) <= 1.5 * _rms(host)


@pytest.mark.parametrize("n_t", [30, 56])
@pytest.mark.parametrize("mode", ["exact", "ref_mr"])
def test_basis_state_transfer(pg, n_t, mode):
    """Four-spin transfers between basis states, whose overlaps start at 1e-4.  A
    step rounds a vector's parts to 2^-60 of its norm and meets propagators
    rounded to 2^-59, about 2^-61 rms each, independently; four times their sum
    over 2 n_t steps, through the overlaps (dG / dz) and through the vectors
    themselves."""
    from pulsar_gb300 import workloads as W
    spec, u = W.spin4_state_transfer(seed=n_t, n_t=n_t, n_off=1, n_b1=1)
    G, zw, g = _gradient(spec, u, mode, np.longdouble, np.clongdouble)
    p = pg.Problem(**spec.problem_kwargs(mode, "fp64"))
    _, Gd = p.eval(u)
    p.close()
    norms = sum(np.linalg.norm(x, 2) ** 2 for x in np.asarray(spec.controls))
    reach = np.sqrt((np.asarray(spec.dt) ** 2).sum() * norms) * 2 * _rms(zw)
    tol = 4 * 2.0 ** -61 * np.sqrt(2 * n_t) * (reach + np.sqrt(g)) + 2.0 ** -52 * _rms(G)
    err = _rms(Gd - G)
    print(f"{n_t} slices {mode}: device error {err / _rms(G):.1e} of |G|, bar {tol / _rms(G):.1e}")
    assert err <= tol


@pytest.mark.parametrize("precision,D,n_t", [("fp64", 2, 1500), ("fp64", 6, 1500), ("fp64", 8, 1500), ("fp64", 16, 1500),
                                             ("fp64", 32, 600), ("mixed", 16, 1500), ("mixed", 32, 600)])
def test_norm_along_long_pulses(pg, precision, D, n_t):
    """F = |<t|psi>|^2 with t the normalised final state is the norm squared (a
    wrong direction enters squared).  Each slice's entries are rounded once, by
    2^-54 of themselves (doubles) or 2^-48 (df), independently of the slice
    before, so the norm wanders by about that times sqrt(n_t); a part that is
    the same every time would grow with n_t.  Four times that."""
    from pulsar_gb300 import workloads as W
    unit = 2.0 ** -54 if precision == "fp64" else 2.0 ** -48
    for seed in range(3):
        spec, u = W.uneven_problem(np.random.default_rng(seed), d=D, n_t=n_t, n_members=1)
        H = spec.drifts[0] + spec.member_offset[0] * spec.offset_op
        psi = np.eye(D, dtype=complex)[0]
        t = psi
        for k in range(n_t):
            t = sla.expm(-1j * spec.dt[k] * (H + spec.member_scale[0] * np.tensordot(u[:, k], spec.controls, 1))) @ t
        kw = spec.problem_kwargs("ref_mr", precision)
        kw.pop("target_op")
        kw.update(target="states", states_init=psi[None], states_target=(t / np.linalg.norm(t))[None], fidelity="square")
        p = pg.Problem(**kw)
        F, _ = p.eval(u, want_grad=False)
        p.close()
        print(f"{precision} d = {D}: {(F - 1) / n_t:.1e} a slice")
        assert abs(F - 1) <= 4 * unit * np.sqrt(n_t) + 2.0 ** -51


@pytest.mark.parametrize("D", [8, 16, 32])
@pytest.mark.parametrize("mode", ["exact", "ref_mr"])
def test_trace_of_equal_entries(pg, D, mode):
    """Every product of the trace Tr(X C) at its largest and of one sign (a
    control of equal entries, states spread evenly, entries just below a power of
    two): the integer sums hold it.  FP64's bar against the oracle."""
    from oracle import members as mb
    psi = np.full((1, D), D ** -0.5, complex)
    kw = dict(drifts=np.zeros((1, D, D)), controls=np.full((2, D, D), 0.999), dt=np.full(3, 1e-3 / D), target="states",
              fidelity="real", states_init=psi, states_target=1j * psi, member_weight=np.array([0.74]))
    u = np.array([[0.3, -0.2, 0.1], [0.1, 0.2, 0.3]])
    Fo, Go = mb.eval_problem(mb.Problem(n_members=1, **kw), u, mode)
    p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
    F, G = p.eval(u)
    p.close()
    assert abs(F - Fo) <= 1e-10 and np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()


@pytest.mark.parametrize("D", [2, 4, 8, 16, 20, 32])
def test_state_sums_of_equal_entries(pg, D):
    """A state chain's first step with every product at its largest and of one
    sign: a propagator I + k (1 - i) J, J all ones, on a vector of equal entries
    (1 + i) just below a power of two.  Against the closed form; the exponential
    of norm 9 costs seven squarings, 2^7 (D + 40) 2^-53 relative."""
    k = 100.0
    J = np.ones((D, D))
    a = np.log(1 + D * k * (1 - 1j)) / D
    v = np.full((1, D), 0.999 * (1 + 1j))
    kw = dict(drifts=a * J[None], controls=0 * J[None], dt=np.ones(1), generator="liouvillian", target="states",
              fidelity="square", states_init=v, states_target=v)
    p = pg.Problem(grad_mode="ref_mr", precision="fp64", **kw)
    F, G, st = p.eval(np.zeros((1, 1)), stats=True)
    F1, _ = p.eval(np.zeros((1, 1)), want_grad=False)
    p.close()
    z = np.vdot(v, v + k * (1 - 1j) * (J @ v.T).T)
    assert F1 == F and abs(F / abs(z) ** 2 - 1) <= 2 * 2.0 ** 7 * (D + 40) * 2.0 ** -53


@pytest.mark.parametrize("n_qubits,n_t", [(1, 30), (1, 167), (2, 28), (2, 99)])
def test_dissipative_basis_states(pg, n_qubits, n_t):
    """First-order gradients of Lindblad pulses between basis states, vectors
    with one large part, as FP64's small components are: a step rounds each part
    to about 2^-59 of the vector's sum and the propagators' parts to 2^-59; rms
    2^-60.5, four times their sum over 2 n_t steps, through the vectors (real
    overlaps: dG / dz is the gradient itself)."""
    from pulsar_gb300 import workloads as W
    spec, u = W.lindblad_gate(seed=n_t, n_qubits=n_qubits, n_t=n_t, n_draws=1, duration=2e-6 * n_t / 500)
    D, d = 4 ** n_qubits, 2 ** n_qubits
    e = np.eye(D, dtype=complex)
    spec.target, spec.target_op, spec.fidelity = "states", None, "real"
    spec.states_init, spec.states_target = e[:1], e[D - 1:] if n_qubits == 1 else e[d + 1:d + 2]
    G = _gradient(spec, u, "ref_mr", np.longdouble, np.clongdouble, kappa=1)[0]
    p = pg.Problem(**spec.problem_kwargs("ref_mr", "fp64"))
    _, Gd = p.eval(u)
    p.close()
    norms = sum(np.linalg.norm(x, 2) ** 2 for x in np.asarray(spec.controls))
    w = spec.members()[3][0]
    tol = 4 * 2.0 ** -60.5 * np.sqrt(2 * n_t) * np.sqrt((np.asarray(spec.dt) ** 2).sum() * norms) * w + 2.0 ** -52 * _rms(G)
    err = _rms(Gd - G)
    print(f"{n_qubits} qubits, {n_t} slices: device error {err / _rms(G):.1e} of |G|, bar {tol / _rms(G):.1e}")
    assert err <= tol
