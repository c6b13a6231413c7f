"""Block fixed-point kernels of the FP64 path (csrc/pgx_fx.cuh) against scipy
and the numpy oracle.

Tolerances.  A propagator's elements are at most 1 in modulus for Hermitian
generators; every product keeps its absolute error near 2^-57 and s squarings
double it each time, so 2^s (D + 2 degree) 2^-53 bounds U with a wide margin
for the double rounding of the output and the oracle's own rounding.
"""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


def _problem(pg, D, nrm, gen, n_c, rng, precision="fp64"):
    H = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
    C = rng.normal(size=(n_c, D, D)) + 1j * rng.normal(size=(n_c, D, D))
    if gen == "hermitian":
        H, C = H + H.conj().T, C + C.conj().transpose(0, 2, 1)
    else:  # dissipative, not normal: the propagator stays bounded
        H = H - H.conj().T - 0.2 * np.eye(D) + 0.05 * np.triu(H, 1)
        C = C - C.conj().transpose(0, 2, 1)
    u = rng.normal(size=(n_c, 1))
    A = H + np.tensordot(u[:, 0], C, 1)
    dt = nrm / np.abs(A).sum(0).max()
    p = pg.Problem(H[None], C, np.array([dt]), generator=gen, target="gate", target_op=np.eye(D), precision=precision)
    return p, u, (-1j if gen == "hermitian" else 1.0) * A * dt


@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D", [5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("nrm,n_c", [(0.0, 1), (1e-9, 2), (0.0016, 2), (0.07, 3), (0.5, 23), (1.6, 22), (0.3, 7), (60.0, 6)])
def test_propagator(pg, gen, D, nrm, n_c):
    """Every degree, squarings, padding, one term to the last that fits (and one
    more, which takes the general kernel)."""
    p, u, A = _problem(pg, D, nrm, gen, n_c, np.random.default_rng(D * 100 + n_c))
    U = p.total_propagator(u)
    p.close()
    s = max(0, int(np.ceil(np.log2(max(nrm, 1e-300) / 1.5))))
    E = sla.expm(A)
    assert np.abs(U - E).max() <= 2.0 ** s * (D + 40) * 2.0 ** -53 * max(1.0, np.abs(E).max())


@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D", [33, 64])
@pytest.mark.parametrize("nrm", [0.0, 1e-9, 3e-5, 0.003, 0.03, 0.1, 0.17, 0.4, 0.8, 1.6, 7.0, 60.0])
def test_mixed_propagator_64(pg, gen, D, nrm):
    """The sliced tensor-core exponential with every block size and number of
    levels.  Each product keeps its entries to about 2^-53 of 1 (2^-48 allows
    for the double-float inputs and output), and squarings double the error."""
    p, u, A = _problem(pg, D, nrm, gen, 3, np.random.default_rng(D), precision="mixed")
    U = p.total_propagator(u)
    p.close()
    s = max(0, int(np.ceil(np.log2(max(nrm, 1e-300) / 0.1))))
    E = sla.expm(A)
    assert np.abs(U - E).max() <= 2.0 ** s * (D + 40) * 2.0 ** -48 * max(1.0, np.abs(E).max())


@pytest.mark.parametrize("n_t", [1, 4, 6])
def test_mixed_generators_64_by_groups(pg, n_t):
    """Members enough for the prologue that assembles four slices at a time
    (with a short last group) against each member alone (one at a time); bar
    as above, per slice."""
    rng = np.random.default_rng(n_t)
    n_m, D = 320, 36
    X = rng.normal(size=(4, D, D)) + 1j * rng.normal(size=(4, D, D))
    X = X + X.conj().transpose(0, 2, 1)
    u = rng.normal(size=(2, n_t))
    sc, of = rng.uniform(0.9, 1.1, n_m), rng.uniform(-0.1, 0.1, n_m)
    kw = dict(dt=rng.uniform(0.5, 1.0, n_t) * 0.02, target="gate", target_op=np.eye(D), precision="mixed")
    p = pg.Problem(X[:1], X[1:3], offset_op=X[3], member_scale=sc, member_offset=of, **kw)
    U = [p.total_propagator(u, member=m) for m in (0, n_m - 1)]
    p.close()
    for m, V in zip((0, n_m - 1), U):
        p = pg.Problem(X[:1], X[1:3], offset_op=X[3], member_scale=sc[m:m + 1], member_offset=of[m:m + 1], **kw)
        W = p.total_propagator(u)
        p.close()
        E = np.eye(D)
        for k in range(n_t):
            E = sla.expm(-1j * kw["dt"][k] * (X[0] + of[m] * X[3] + sc[m] * np.tensordot(u[:, k], X[1:3], 1))) @ E
        for A in (V, W):
            assert np.abs(A - E).max() <= n_t * 8 * (D + 40) * 2.0 ** -48


def test_propagator_not_finite(pg):
    """A generator that overflows gives NaN, not a finite matrix."""
    D = 16
    H = np.eye(D) * 1e300
    p = pg.Problem(H[None], np.stack([np.eye(D)]) * 1e300, np.array([1.0]), target="gate", target_op=np.eye(D))
    U = p.total_propagator(np.full((1, 1), 1e10))
    p.close()
    assert np.isnan(U).any()


@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D,n_t,n_m", [(7, 1, 1), (8, 13, 3), (9, 2, 2), (16, 13, 3), (19, 3, 1), (32, 5, 2)])
@pytest.mark.parametrize("nrm", [0.03, 0.4, 3.0, 9.0])
def test_exact_gradient(pg, target, gen, D, n_t, n_m, nrm):
    """(F, G) of slices with few and many Horner steps and squarings, members of
    different scale and offset, against the oracle.  FP64's own bars: |dF| <=
    1e-10 and 1e-8 of the largest gradient entry; the sums of n_t D-term
    products stay well inside both."""
    from oracle import members as mb
    rng = np.random.default_rng(D + n_t)
    n_c = 3
    H = rng.normal(size=(2, D, D)) + 1j * rng.normal(size=(2, D, D))
    C = rng.normal(size=(n_c, D, D)) + 1j * rng.normal(size=(n_c, D, D))
    O = rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D))
    dag = lambda x: np.swapaxes(x.conj(), -1, -2)  # noqa: E731
    if gen == "hermitian":
        H, C, O = H + dag(H), C + dag(C), O + dag(O)
    else:
        H = H - dag(H) - 0.2 * np.eye(D) + 0.05 * np.triu(H, 1)
        C, O = C - dag(C), O - dag(O)
    u = rng.normal(size=(n_c, n_t))
    dt = nrm / np.abs(H[0] + np.tensordot(u[:, 0], C, 1)).sum(0).max() * rng.uniform(0.1, 1.0, n_t)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    kw = dict(drifts=H, controls=C, dt=dt, generator=gen, offset_op=O, member_drift=np.arange(n_m) % 2,
              member_scale=rng.uniform(0.9, 1.1, n_m), member_offset=rng.uniform(-0.1, 0.1, n_m), target=target,
              fidelity="square")
    kw.update(dict(target_op=Q) if target == "gate" else dict(states_init=Q[:2], states_target=Q[2:4]))
    Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, "exact")
    p = pg.Problem(grad_mode="exact", precision="fp64", **kw)
    F, G = p.eval(u)
    p.close()
    assert abs(F - Fo) <= 1e-10
    assert np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()


@pytest.mark.parametrize("mode", ["exact", "ref_mr", "ref_grape"])
@pytest.mark.parametrize("D,n_t,n_m", [(2, 1, 1), (2, 67, 1), (3, 2, 2), (3, 8, 3), (4, 301, 2), (4, 41, 200), (2, 5, 5000),
                                       (5, 1, 2), (8, 7, 1), (8, 301, 2), (11, 2, 1), (16, 67, 1), (16, 41, 200),
                                       (32, 2, 1), (25, 23, 2)])
def test_gate_chain_blocks(pg, mode, D, n_t, n_m):
    """Gate chains in one block, in blocks with a short last one, of one slice,
    and of many members, in every gradient mode; F-only gives the same F.  Bars
    as above."""
    from oracle import members as mb
    rng = np.random.default_rng(7 * D + n_t)
    dag = lambda x: np.swapaxes(x.conj(), -1, -2)  # noqa: E731
    X = rng.normal(size=(3, D, D)) + 1j * rng.normal(size=(3, D, D))
    X = X + dag(X)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    u = rng.normal(size=(2, n_t))
    kw = dict(drifts=X[:1], controls=X[1:], dt=np.full(n_t, 0.3 / (D + 4)), member_scale=rng.uniform(0.9, 1.1, n_m),
              target="gate", fidelity="square", target_op=Q)
    Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, mode) if n_t * n_m < 2000 else (None, None)
    p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
    F, G = p.eval(u)
    F1, _ = p.eval(u, want_grad=False)
    Ut = p.total_propagator(u, member=n_m - 1)
    F2, G2 = p.eval(u)
    p.close()
    assert F1 == F and F2 == F and np.array_equal(G, G2)
    assert np.abs(dag(Ut) @ Ut - np.eye(D)).max() <= n_t * (D + 40) * 2.0 ** -53
    if Fo is None:  # many members: mean over two of them against the oracle
        kw["member_scale"] = kw["member_scale"][[0, n_m - 1]]
        Fo, Go = mb.eval_problem(mb.Problem(n_members=2, **kw), u, mode)
        p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
        F, G = p.eval(u)
        p.close()
    assert abs(F - Fo) <= 1e-10
    assert np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()


@pytest.mark.parametrize("mode", ["exact", "ref_mr", "ref_grape"])
@pytest.mark.parametrize("D,n_t,n_m,n_p", [(2, 1, 1, 1), (2, 300, 2, 8), (3, 2, 3, 2), (4, 17, 1, 3), (7, 9, 2, 1),
                                           (8, 40, 2, 8), (13, 3, 1, 5), (16, 21, 2, 8),
                                           (20, 9, 2, 8), (32, 6, 1, 3)])
def test_state_chains(pg, mode, D, n_t, n_m, n_p):
    """State chains of one slice to many, one to eight pairs (the fewest slices
    in flight), pairs of very different norms, a dissipative generator.  FP64's
    bars; a vector's own exponent keeps the small pair's overlap to the same
    relative error."""
    from oracle import members as mb
    rng = np.random.default_rng(11 * D + n_t)
    X = rng.normal(size=(3, D, D)) + 1j * rng.normal(size=(3, D, D))
    X = X - np.swapaxes(X.conj(), -1, -2)
    X[0] -= 0.05 * np.eye(D)
    V = rng.normal(size=(2, n_p, D)) + 1j * rng.normal(size=(2, n_p, D))
    V /= np.linalg.norm(V, axis=2, keepdims=True)
    if n_p > 1:
        V[:, -1] *= 1e-6
    kw = dict(drifts=X[:1], controls=X[1:], dt=np.full(n_t, 0.2 / (D + 4)), generator="liouvillian",
              member_scale=rng.uniform(0.9, 1.1, n_m), target="states", fidelity="square", states_init=V[0],
              states_target=V[1])
    u = rng.normal(size=(2, n_t))
    Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, mode)
    p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
    F, G = p.eval(u)
    F1, _ = p.eval(u, want_grad=False)
    p.close()
    assert F1 == F
    assert abs(F - Fo) <= 1e-10
    assert np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()
    if n_p > 1:  # the small pair alone
        kw.update(states_init=V[0, -1:], states_target=V[1, -1:])
        Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, mode)
        p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
        F, G = p.eval(u)
        p.close()
        assert abs(F - Fo) <= 1e-10 * abs(Fo)
        assert np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()


@pytest.mark.parametrize("D,n_t,n_p", [(2, 64, 1), (2, 129, 2), (4, 33, 8), (8, 8, 3), (8, 9, 8), (16, 5, 8), (12, 2, 1),
                                       (32, 7, 8), (17, 1, 2)])
def test_state_chains_hermitian(pg, D, n_t, n_p):
    """Unitary state chains at the edges of a chunk of slices (one, exactly
    full, one over), both gradient forms against the oracle."""
    from oracle import members as mb
    rng = np.random.default_rng(13 * D + n_t)
    X = rng.normal(size=(3, D, D)) + 1j * rng.normal(size=(3, D, D))
    X = X + np.swapaxes(X.conj(), -1, -2)
    V = rng.normal(size=(2, n_p, D)) + 1j * rng.normal(size=(2, n_p, D))
    V /= np.linalg.norm(V, axis=2, keepdims=True)
    kw = dict(drifts=X[:1], controls=X[1:], dt=np.full(n_t, 0.3 / (D + 4)), member_scale=np.array([0.9, 1.0, 1.1]),
              target="states", fidelity="square", states_init=V[0], states_target=V[1])
    u = rng.normal(size=(2, n_t))
    for mode in ("exact", "ref_grape"):
        Fo, Go = mb.eval_problem(mb.Problem(n_members=3, **kw), u, mode)
        p = pg.Problem(grad_mode=mode, precision="fp64", **kw)
        F, G = p.eval(u)
        F1, _ = p.eval(u, want_grad=False)
        p.close()
        assert F1 == F
        assert abs(F - Fo) <= 1e-10
        assert np.abs(G - Go).max() <= 1e-8 * np.abs(Go).max()


@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D,n_t,n_m,n_c", [(16, 1, 1, 1), (9, 30, 3, 23), (16, 37, 2, 3), (32, 3, 2, 6), (21, 26, 1, 2), (32, 9, 1, 7)])
@pytest.mark.parametrize("nrm", [0.02, 0.7, 4.0])
def test_mixed_series_gradient(pg, target, gen, D, n_t, n_m, n_c, nrm):
    """The mixed path at D = 16 and 32: the series gradient, the CUDA-core one
    that takes over for norms above 1 (nrm = 4), more controls than the
    generator's shared memory holds; against the oracle with the mixed path's
    bars (|dF| <= 1e-8, gradient 1e-4), and the CUDA-core team's own gradient
    within FP32's rounding of it."""
    from oracle import members as mb
    rng = np.random.default_rng(D + n_t + n_c)
    dag = lambda x: np.swapaxes(x.conj(), -1, -2)  # noqa: E731
    X = rng.normal(size=(1 + n_c, D, D)) + 1j * rng.normal(size=(1 + n_c, D, D))
    X = X + dag(X) if gen == "hermitian" else X - dag(X)
    if gen == "liouvillian":
        X[0] -= 0.1 * np.eye(D)
    u = rng.normal(size=(n_c, n_t))
    dt = nrm / np.abs(X[0] + np.tensordot(u[:, 0], X[1:], 1)).sum(0).max() * rng.uniform(0.1, 1.0, n_t)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    kw = dict(drifts=X[:1], controls=X[1:], dt=dt, generator=gen, member_scale=rng.uniform(0.9, 1.1, n_m), target=target)
    kw.update(dict(target_op=Q) if target == "gate" else dict(states_init=Q[:2], states_target=Q[2:4]))
    Fo, Go = mb.eval_problem(mb.Problem(n_members=n_m, **kw), u, "exact")
    p = pg.Problem(grad_mode="exact", precision="mixed", **kw)
    F, G = p.eval(u)
    p.set_teams(grad=128)
    F1, G1 = p.eval(u)
    p.close()
    scale = np.abs(Go).max()
    assert F1 == F and abs(F - Fo) <= 1e-8
    assert np.abs(G - Go).max() <= 1e-4 * scale and np.abs(G1 - Go).max() <= 1e-4 * scale


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("D,n_t", [(2, 40), (4, 300), (16, 12)])
def test_repeated_evaluations(pg, precision, target, D, n_t):
    """Evaluations enqueued directly and replayed as a graph give the same bits,
    with and without the gradient, and setters take effect in between."""
    rng = np.random.default_rng(D + n_t)
    X = rng.normal(size=(4, D, D)) + 1j * rng.normal(size=(4, D, D))
    X = X + X.conj().transpose(0, 2, 1)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    kw = dict(dt=np.full(n_t, 0.1 / D), target=target, precision=precision, grad_mode="exact", fidelity="square")
    kw.update(dict(target_op=Q) if target == "gate" else dict(states_init=Q[:1], states_target=Q[1:2]))

    def fresh(drift, u, want_grad):
        p = pg.Problem(drift[None], X[1:3], **kw)
        r = p.eval(u, want_grad=want_grad)
        p.close()
        return r

    us = rng.normal(size=(7, 2, n_t))
    p = pg.Problem(X[:1], X[1:3], **kw)
    for drift in (X[0], X[3]):
        p.set_drifts(drift[None])
        for u in us:
            for want_grad in (True, False):
                F, G = p.eval(u, want_grad=want_grad)
                Fo, Go = fresh(drift, u, want_grad)
                assert F == Fo and (not want_grad or np.array_equal(G, Go))
    p.close()


@pytest.mark.parametrize("target", ["gate", "states"])
@pytest.mark.parametrize("D,n_c", [(16, 2), (16, 26), (32, 9)])
def test_teams_carry_over(pg, target, D, n_c):
    """The teams of an exact gate problem are accepted by every problem of its
    dimension: first order, states, more terms than the tensor cores take."""
    rng = np.random.default_rng(D + n_c)
    X = rng.normal(size=(n_c + 1, D, D)) + 1j * rng.normal(size=(n_c + 1, D, D))
    X = X + X.conj().transpose(0, 2, 1)
    dt = np.full(3, 0.05 / D)
    p = pg.Problem(X[:1], X[1:3], dt, target="gate", target_op=np.eye(D), grad_mode="exact", precision="mixed")
    teams = p.teams
    p.close()
    to = dict(target_op=np.eye(D)) if target == "gate" else dict(states_init=np.eye(D)[:1], states_target=np.eye(D)[1:2])
    u = rng.normal(size=(n_c, 3))
    p = pg.Problem(X[:1], X[1:], dt, target=target, grad_mode="ref_mr", precision="mixed", **to)
    F, G = p.eval(u)
    p.set_teams(*teams)
    F1, G1 = p.eval(u)
    p.close()
    assert F1 == F and np.array_equal(G, G1)


@pytest.mark.parametrize("n_m,n_t", [(1, 1), (7, 11), (8, 16), (9, 17), (300, 33)])
def test_member_sums(pg, n_m, n_t):
    """F and G of an ensemble against the weighted sums of its members, each
    evaluated alone: sums of n_m terms, n_m 2^-52 of their absolute sum."""
    rng = np.random.default_rng(n_m)
    X = rng.normal(size=(3, 2, 2)) + 1j * rng.normal(size=(3, 2, 2))
    X = X + X.conj().transpose(0, 2, 1)
    sc, wt = rng.uniform(0.9, 1.1, n_m), rng.uniform(0.1, 1.0, n_m)
    wt /= wt.sum()
    u = rng.normal(size=(2, n_t))
    kw = dict(dt=np.full(n_t, 0.1), target="gate", target_op=np.eye(2), grad_mode="ref_mr", precision="fp64")
    p = pg.Problem(X[:1], X[1:], member_scale=sc, member_weight=wt, **kw)
    F, G = p.eval(u)
    F1, _ = p.eval(u, want_grad=False)
    p.close()
    Fs, Gs = [], []
    for m in range(n_m):
        p = pg.Problem(X[:1], X[1:], member_scale=sc[m:m + 1], member_weight=wt[m:m + 1], **kw)
        f, g = p.eval(u)
        p.close()
        Fs.append(f)
        Gs.append(g)
    assert F1 == F
    assert abs(F - sum(Fs)) <= (n_m + 8) * 2.0 ** -52 * np.abs(Fs).sum()
    assert (np.abs(G - sum(Gs)) <= (n_m + 8) * 2.0 ** -52 * np.abs(Gs).sum(0)).all()


@pytest.mark.parametrize("mode", ["exact", "ref_grape"])
@pytest.mark.parametrize("D,n_t,n_m", [(2, 128, 1), (2, 3001, 2), (4, 145, 2), (3, 600, 1), (8, 129, 1), (7, 1000, 3),
                                       (8, 4000, 1)])
def test_mixed_many_blocks(pg, mode, D, n_t, n_m):
    """Mixed gate chains of 16 blocks (the fewest that the eight-warp combine
    takes) to many, full and short last runs, against the FP64 path.  The mixed
    path's bars: |dF| 1e-9, gradient 2e-5 of its norm."""
    rng = np.random.default_rng(n_t)
    X = rng.normal(size=(3, D, D)) + 1j * rng.normal(size=(3, D, D))
    X = X + X.conj().transpose(0, 2, 1)
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    u = rng.normal(size=(2, n_t))
    kw = dict(dt=np.full(n_t, 0.5 / D), member_scale=rng.uniform(0.9, 1.1, n_m), target="gate", target_op=Q,
              fidelity="square", grad_mode=mode)
    out = []
    for precision in ("fp64", "mixed"):
        p = pg.Problem(X[:1], X[1:], precision=precision, **kw)
        F, G = p.eval(u)
        F1, _ = p.eval(u, want_grad=False)
        p.close()
        assert F1 == F
        out.append((F, G))
    assert abs(out[0][0] - out[1][0]) <= 1e-9
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 2e-5 * np.linalg.norm(out[0][1])


@pytest.mark.parametrize("D,n_t,n_m", [(9, 16, 1), (16, 64, 1), (16, 50, 40), (20, 33, 2), (32, 64, 1), (32, 24, 30)])
def test_mixed_prefixes_of_unequal_slices(pg, D, n_t, n_m):
    """In-block prefixes of the mixed path whose neighbouring slices differ by
    2^16 in scale, so a slice read with its neighbour's exponent is off by that
    factor.  The oracle with the mixed path's bars; the same bits every time."""
    from oracle import members as mb
    rng = np.random.default_rng(D * n_t)
    X = rng.normal(size=(3, D, D)) + 1j * rng.normal(size=(3, D, D))
    X = (X - np.swapaxes(X.conj(), -1, -2)) / D
    X[2] = np.eye(D)
    u = rng.normal(size=(2, n_t))
    u[1] = 8 * np.log(2.0) * (1 - 2 * (np.arange(n_t) % 2))
    if n_t % 2:
        u[1, -1] = 0.0
    Q, _ = np.linalg.qr(rng.normal(size=(D, D)) + 1j * rng.normal(size=(D, D)))
    kw = dict(drifts=X[:1], controls=X[1:], dt=np.ones(n_t), generator="liouvillian", target="gate", target_op=Q,
              fidelity="square", offset_op=X[0], member_offset=rng.uniform(-0.1, 0.1, n_m))
    few = dict(kw, member_offset=kw["member_offset"][:2])
    p = pg.Problem(grad_mode="exact", precision="mixed", **few)
    F, G = p.eval(u)
    p.close()
    Fo, Go = mb.eval_problem(mb.Problem(n_members=len(few["member_offset"]), **few), u, "exact")
    assert abs(F - Fo) <= 1e-8
    assert np.abs(G - Go).max() <= 1e-4 * np.abs(Go).max()
    p = pg.Problem(grad_mode="exact", precision="mixed", **kw)
    F, G = p.eval(u)
    for _ in range(20):
        F1, G1 = p.eval(u)
        assert F1 == F and np.array_equal(G1, G)
    p.close()
