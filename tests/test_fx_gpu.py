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


def _problem(pg, D, nrm, gen, n_c, rng):
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
    p = pg.Problem(H[None], C, np.array([dt]), generator=gen, target="gate", target_op=np.eye(D), precision="fp64")
    return p, u, (-1j if gen == "hermitian" else 1.0) * A * dt


@pytest.mark.parametrize("gen", ["hermitian", "liouvillian"])
@pytest.mark.parametrize("D", [5, 8, 9, 16])
@pytest.mark.parametrize("nrm,n_c", [(0.0, 1), (1e-9, 2), (0.0016, 2), (0.07, 3), (0.5, 23), (1.6, 22), (60.0, 3)])
def test_propagator(pg, gen, D, nrm, n_c):
    """Every degree, squarings, padding, one term to the last that fits (and one
    more, which takes the general kernel)."""
    p, u, A = _problem(pg, D, nrm, gen, n_c, np.random.default_rng(D * 100 + n_c))
    U = p.total_propagator(u)
    p.close()
    s = max(0, int(np.ceil(np.log2(max(nrm, 1e-300) / 1.5))))
    E = sla.expm(A)
    assert np.abs(U - E).max() <= 2.0 ** s * (D + 40) * 2.0 ** -53 * max(1.0, np.abs(E).max())


def test_propagator_not_finite(pg):
    """A generator that overflows gives NaN, not a finite matrix."""
    D = 16
    H = np.eye(D) * 1e300
    p = pg.Problem(H[None], np.stack([np.eye(D)]) * 1e300, np.array([1.0]), target="gate", target_op=np.eye(D))
    U = p.total_propagator(np.full((1, 1), 1e10))
    p.close()
    assert np.isnan(U).any()
