"""Routes of the padded dimensions 8 to 64 that a size alone does not reach: the
D = 64 mixed kernels through their own evaluation, slices of large norm beside
small ones, evaluation graphs after every setter, the teams in use."""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


def _dag(x):
    return np.swapaxes(x.conj(), -1, -2)


def _herm(rng, n, D):
    x = rng.normal(size=(n, D, D)) + 1j * rng.normal(size=(n, D, D))
    return x + _dag(x)


def _shift(D, k, phase):
    return phase * np.roll(np.eye(D), k, axis=0)


@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D", [33, 64])
@pytest.mark.parametrize("nrm", [0.0, 1e-9, 3e-5, 0.003, 0.03, 0.1, 0.17, 0.4, 0.8, 1.6, 7.0, 60.0])
def test_mixed_expm_64_through_its_evaluation(pg, gen, D, nrm):
    """The sliced exponential (block sizes 2 to 4, four to seven levels,
    squarings) read through F = Re Tr(T'U) / D with shifts T, the mean of D
    entries of U.  An entry is held to 2^-53 of 1 and stored as a df pair (2^-48
    of itself), and squarings double the error: a mean of D stays within 4
    2^-48 2^s.  The CUDA-core team within the same bar."""
    rng = np.random.default_rng(D + int(1e3 * nrm))
    H = _herm(rng, 4, D)
    if gen == "liouvillian":  # dissipative, not normal: the propagator stays bounded
        H = H * 1j
        H[0] += -0.2 * np.eye(D) + 0.05 * np.triu(rng.normal(size=(D, D)), 1)
    u = rng.normal(size=(3, 1))
    A = H[0] + np.tensordot(u[:, 0], H[1:], 1)
    dt = nrm / np.abs(A).sum(0).max()
    E = sla.expm((-1j if gen == "hermitian" else 1.0) * dt * A)
    s = max(0, int(np.ceil(np.log2(max(nrm, 1e-300) / 0.1))))
    bar = 4 * 2.0 ** (s - 48) * max(1.0, np.abs(E).max())
    for k, phase in ((0, 1), (0, 1j), (1, 1), (D // 2, 1j)):
        T = _shift(D, k, phase)
        p = pg.Problem(H[:1], H[1:], np.array([dt]), generator=gen, target="gate", target_op=T, fidelity="real",
                       precision="mixed", grad_mode="exact")
        assert p.teams[0] == 1
        F, _ = p.eval(u, want_grad=False)
        F1, G1 = p.eval(u)
        p.set_teams(256, 0)
        Fc, Gc = p.eval(u)
        p.close()
        Fo = (np.trace(T.conj().T @ E) / D).real
        assert F1 == F
        assert abs(F - Fo) <= bar and abs(Fc - Fo) <= bar
        # the gradient of the same kernel on either propagators: FP32 class
        assert np.abs(G1 - Gc).max() <= 1e-5 * max(np.abs(Gc).max(), 1e-30)


@pytest.mark.parametrize("n_t", [1, 4, 6, 9])
def test_mixed_generators_64_of_many_members(pg, n_t):
    """Members enough for the prologue that assembles four slices of a member at
    a time, with a short last group: every member's fidelity against its
    propagators, the bar above for each slice; F-only and CUDA-core teams too."""
    rng = np.random.default_rng(n_t)
    n_m, D = 320, 36
    X = _herm(rng, 4, D)
    u = rng.normal(size=(2, n_t))
    sc, of = rng.uniform(0.9, 1.1, n_m), rng.uniform(-0.1, 0.1, n_m)
    dt = rng.uniform(0.5, 1.0, n_t) * 0.02
    T = _shift(D, 1, 1j)
    p = pg.Problem(X[:1], X[1:3], dt, offset_op=X[3], member_scale=sc, member_offset=of, target="gate", target_op=T,
                   fidelity="real", precision="mixed", grad_mode="exact")
    F, G = p.eval(u)
    f = p.member_fidelities()
    F1, _ = p.eval(u, want_grad=False)
    p.set_teams(256, 0)
    Fc, Gc = p.eval(u)
    p.close()
    bar = n_t * 4 * 2.0 ** (4 - 48)  # norms up to 1.6
    assert F1 == F and abs(F - f.mean()) <= 2.0 ** -48 and abs(F - Fc) <= bar
    assert np.abs(G - Gc).max() <= 1e-5 * np.abs(Gc).max()
    for m in (0, 1, 151, 152, 303, 304, n_m - 1):
        E = np.eye(D)
        for k in range(n_t):
            E = sla.expm(-1j * dt[k] * (X[0] + of[m] * X[3] + sc[m] * np.tensordot(u[:, k], X[1:3], 1))) @ E
        assert abs(f[m] - (np.trace(T.conj().T @ E) / D).real) <= bar


@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("D,n_t,n_m", [(7, 9, 2), (16, 33, 1), (12, 40, 3), (32, 12, 1), (20, 7, 2)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_slice_of_large_norm(pg, precision, target, D, n_t, n_m):
    """One slice beyond the exact gradient's series among small ones: on the
    FP64 path that slice alone takes the derivative kernel, on the mixed path the
    whole evaluation the CUDA-core gradient.  Against the oracle with the paths'
    bars; where the mixed path falls back, the bits of that team's own run."""
    from oracle import members as mb
    rng = np.random.default_rng(D * n_t)
    X = _herm(rng, 3, D)
    u = rng.normal(size=(2, n_t))
    nrm = np.array([np.linalg.norm(X[0] + np.tensordot(u[:, k], X[1:], 1), 2) for k in range(n_t)])
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    to = dict(target_op=Q) if target == "gate" else dict(states_init=Q[:2], states_target=Q[2:4])
    team = 32 if D <= 16 else 128
    for big in (None, 0, n_t // 2, n_t - 1, "all"):
        dt = 0.1 / nrm
        if big == "all":
            dt = 9.0 / nrm
        elif big is not None:
            dt[big] = 9.0 / nrm[big]
        kw = dict(drifts=X[:1], controls=X[1:], dt=dt, member_scale=rng.uniform(0.95, 1.05, n_m), target=target, **to)
        Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, "exact")
        p = pg.Problem(grad_mode="exact", precision=precision, **kw)
        F, G = p.eval(u)
        scale = np.abs(Go).max()
        if precision == "fp64":
            assert abs(F - Fo) <= 1e-10 and np.abs(G - Go).max() <= 1e-8 * scale
        else:
            assert abs(F - Fo) <= 1e-8 and np.abs(G - Go).max() <= 1e-4 * scale
            if D > 8:
                p.set_teams(0, team)
                F1, G1 = p.eval(u)
                assert F1 == F
                if big is None:  # two FP32-class evaluations of 15 products of D terms
                    assert np.abs(G - G1).max() <= 15 * np.sqrt(D) * 2.0 ** -23 * scale
                else:
                    assert np.array_equal(G, G1)
        p.close()


def _setters(pg, precision, target, D, n_t, X, rng):
    """(name, what to call on a problem) in the order they are applied."""
    R = _herm(rng, 2, D)
    out = [("penalties", lambda p: p.set_penalties([("energy", 0.01), ("NS", 0.02)])),
           ("one penalty", lambda p: p.set_penalties([("SNS", 0.5, -0.2, 0.2)])),
           ("no penalty", lambda p: p.set_penalties([])),
           ("drifts", lambda p: p.set_drifts(X[3][None])),
           ("ramp", lambda p: p.set_drift_ramp(R[:1], [0, -1], np.linspace(0, 1, n_t))),
           ("two ramps", lambda p: p.set_drift_ramp(R, [1, 0], np.linspace(1, 0, n_t))),
           ("drifts again", lambda p: p.set_drifts(X[0][None])),
           ("no ramp", lambda p: p.set_drift_ramp(np.zeros((0, D, D)), [], []))]
    if precision == "fp64" and target == "states":
        rho = R @ _dag(R) / D
        out += [("tracking", lambda p: p.set_tracking([1, n_t], [0.5, 0.5], rho)),
                ("other tracking", lambda p: p.set_tracking([2], [1.0], rho[:1])),
                ("no tracking", lambda p: p.set_tracking([], [], []))]
    if precision == "mixed" and D >= 16:
        big = 256 if D > 32 else 128
        out += [("teams", lambda p: p.set_teams(big, 0)), ("default teams", lambda p: p.set_teams(0, 0))]
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("D,n_t", [(2, 40), (5, 20), (16, 12), (40, 3)])
def test_setters_after_the_evaluation_graph(pg, precision, target, D, n_t):
    """Six evaluations of each kind after every setter (the graph is captured at
    the third) against a fresh problem set up the same way, bit for bit; stage
    timing on and off around an existing graph."""
    if precision == "fp64" and D > 32:
        n_t = 2
    rng = np.random.default_rng(D + n_t)
    X = _herm(rng, 4, D)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    kw = dict(dt=np.full(n_t, 0.1 / D), member_scale=np.array([0.9, 1.1]), target=target, precision=precision,
              grad_mode="exact", fidelity="square")
    kw.update(dict(target_op=Q) if target == "gate" else dict(states_init=Q[:1], states_target=Q[1:2]))
    us = rng.normal(size=(6, 2, n_t))
    p = pg.Problem(X[:1], X[1:3], **kw)
    done = []

    def check(name):
        q = pg.Problem(X[:1], X[1:3], **kw)
        for _, f in done:
            f(q)
        for u in us:
            for want_grad in (True, False):
                F, G = p.eval(u, want_grad=want_grad)
                if u is us[0] or u is us[5]:
                    Fq, Gq = q.eval(u, want_grad=want_grad)
                    assert F == Fq and (not want_grad or np.array_equal(G, Gq)), name
        q.close()

    check("new")
    p.ctx.set_stage_timing(True)
    check("stage timing")
    p.ctx.stage_times()
    p.ctx.set_stage_timing(False)
    check("no stage timing")
    for name, f in _setters(pg, precision, target, D, n_t, X, rng):
        f(p)
        done.append((name, f))
        check(name)
    p.close()


def test_batch_after_set_drifts(pg):
    """A batch's graph reads drifts that were replaced after its capture."""
    rng = np.random.default_rng(3)
    probs, us = [], []
    for D in (2, 4, 16):
        X = _herm(rng, 4, D)
        mk = lambda H, X=X, D=D: pg.Problem(H[None], X[1:3], np.full(9, 0.1 / D), target="gate", target_op=np.eye(D),
                                            precision="mixed", grad_mode="exact")
        probs.append((mk(X[0]), mk(X[3]), X[3]))
        us.append(rng.normal(size=(2, 9)))
    b = pg.Batch([p for p, _, _ in probs], n_streams=2)
    for i, u in enumerate(us):
        b.set_controls(i, u)
    first = b.eval()
    for p, _, H in probs:
        p.set_drifts(H[None])
    F = b.eval()
    for i, (p, q, _) in enumerate(probs):
        Fq, Gq = q.eval(us[i])
        assert F[i] == Fq != first[i] and np.array_equal(b.get_controls(i)[1], Gq)
    b.close()
    for p, q, _ in probs:
        p.close()
        q.close()


@pytest.mark.parametrize("D,core", [(16, (128, 32)), (32, (256, 128)), (64, (256, 512))])
def test_teams_in_use(pg, D, core):
    """`teams` names the kernels that run: the tensor-core value only where its
    kernels take the problem, whatever was set, and again once they do."""
    rng = np.random.default_rng(D)
    few, many = 2, 30
    X = _herm(rng, many + 2, D)
    dt = np.full(3, 0.05 / D)
    gate = dict(target="gate", target_op=np.eye(D))
    states = dict(target="states", states_init=np.eye(D)[:1], states_target=np.eye(D)[1:2])

    def teams(n_c, mode, to, teams=None, ramp=False):
        p = pg.Problem(X[:1], X[1:1 + n_c], dt, precision="mixed", grad_mode=mode, **to)
        if teams:
            p.set_teams(*teams)
        if ramp:
            p.set_drift_ramp(X[-1:], [0], np.ones(3))
        t = p.teams
        p.close()
        return t

    assert teams(few, "exact", gate) == (1, 1)
    series = (1, 1) if D < 64 else (1, core[1])
    assert teams(few, "exact", states) == series
    assert teams(few, "ref_mr", gate) == (1, core[1])
    if D < 64:
        assert teams(many, "exact", gate) == core
        for to in (gate, states):
            assert teams(few, "ref_mr", to, (1, 1)) == (1, core[1])
            assert teams(many, "exact", to, (1, 1)) == core
        assert teams(few, "exact", gate, (core[0], 0)) == core  # the series needs the tensor-core expm
        assert teams(few, "exact", gate, (0, core[1])) == (1, core[1])
        most = 23 if D == 16 else 6  # with a ramp one generator term too many
        assert teams(most, "exact", gate) == (1, 1)
        assert teams(most, "exact", gate, ramp=True) == core
