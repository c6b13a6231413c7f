"""Evaluation graphs after every setter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dag(x):
    return np.swapaxes(x.conj(), -1, -2)


def _herm(rng, n, D):
    x = rng.normal(size=(n, D, D)) + 1j * rng.normal(size=(n, D, D))
    return x + _dag(x)


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
