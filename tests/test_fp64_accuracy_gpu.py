"""Norms of the FP64 and mixed paths' states along long pulses."""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


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
