"""Rows of Gamma1 and columns of Gamma2 to their own size, on the bidiagonal route.

Gamma1 = U / Lambda0 and Gamma2 = V^H / Lambda2: where a Lambda is small, so is the row of U or
V, and an error that is small against 1 only would be divided by it.  The residuals of
Theta V = U sigma and Theta^H U = V sigma are taken row by row, relative to the row of Theta,
with Theta formed in extended precision.  Bound: sums of n products to eps, errors of the
vectors of a few eps that add up at random: 32 sqrt(n) eps.  The values are accurate to eps of
the largest by the route's definition (2 eps sigma + eps ||Theta|| of the bisection, as much of
the bidiagonalisation): 4 eps sigma_0 / sigma_i of a column, at most that of the smallest kept.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


def _graded(rng, chi, d, spans, r0, r2):
    """A bond close to canonical form whose Lambdas span `spans`, r0 and r2 of the outer ones kept."""
    lam = [s ** (np.arange(chi) / (chi - 1)) for s in spans]
    lam[0][r0:] = 0.0
    lam[2][r2:] = 0.0
    lam = [x / np.linalg.norm(x) for x in lam]
    w0, w2 = np.where(lam[0] > 0, lam[0], 1.0), np.where(lam[2] > 0, lam[2], 1.0)
    shape = (chi, d, chi)
    a = lam[0][:, None, None] * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    b = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * lam[2]
    a = np.linalg.qr(a.reshape(chi * d, chi))[0].reshape(shape)
    b = np.linalg.qr(b.reshape(chi, d * chi).conj().T)[0].conj().T.reshape(shape)
    gam = [np.asfortranarray(a * (lam[0] > 0)[:, None, None] / w0[:, None, None]),
           np.asfortranarray(b * (lam[2] > 0) / w2)]
    h = rng.standard_normal((d * d, d * d))
    w, v = np.linalg.eigh(h + h.T)
    return gam, lam, (v * np.exp(-0.05j * w)) @ v.conj().T


@pytest.mark.parametrize("chi,d,r0,r2", [(40, 2, 40, 40), (33, 3, 33, 29), (33, 3, 25, 33), (64, 4, 64, 64)])
@pytest.mark.parametrize("spans", [(1e-2, 1e-2, 1e-2), (1e-4, 1e-2, 1e-8), (1e-8, 1e-8, 1e-8), (1e-12, 1e-2, 1e-12)])
@pytest.mark.parametrize("svd_mode", [0, 3])
def test_row_residuals(pkg, chi, d, r0, r2, spans, svd_mode):
    rng = np.random.default_rng(chi * d)
    gam, lam, gate = _graded(rng, chi, d, spans, r0, r2)
    with pkg.Chain(2, d, chi, svd_mode=svd_mode) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, gate)
        g1, g2, l1 = c.get_gamma(1), c.get_gamma(2), c.get_lambda(2)
        assert c.stats()["bidiag_updates"] == 1
    ext = [x.astype(np.longdouble) for x in lam]
    th = (gam[0] * ext[0][:, None, None] * ext[1]).reshape(chi * d, chi) @ (gam[1] * ext[2]).reshape(chi, d * chi)
    th = np.einsum("pq,aqb->apb", gate.astype(np.clongdouble), th.reshape(chi, d * d, chi)).reshape(chi * d, d * chi)
    u = (g1 * lam[0][:, None, None]).reshape(chi * d, chi)
    v = (g2 * lam[2]).reshape(chi, d * chi).conj().T
    keep = l1 > 0
    # the factor between sigma and Lambda1, from the largest value
    scale = np.linalg.norm((th @ v[:, :1]).astype(complex)) / l1[0]
    rows = np.sqrt(np.sum(np.abs(th) ** 2, axis=1))
    cols = np.sqrt(np.sum(np.abs(th) ** 2, axis=0))
    left = (th @ v - u * (l1 * scale))[:, keep]
    right = (th.conj().T @ u - v * (l1 * scale))[:, keep]
    orth = 32 * np.sqrt(chi * d) * EPS
    bound = orth + 4 * EPS * l1[0] / np.min(l1[keep])
    assert np.max(np.sqrt(np.sum(np.abs(left) ** 2, axis=1))[rows > 0] / rows[rows > 0]) <= bound
    assert np.max(np.sqrt(np.sum(np.abs(right) ** 2, axis=1))[cols > 0] / cols[cols > 0]) <= bound
    assert np.max(np.abs(u[:, keep].conj().T @ u[:, keep] - np.eye(keep.sum()))) <= orth
    assert np.max(np.abs(v[:, keep].conj().T @ v[:, keep] - np.eye(keep.sum()))) <= orth
