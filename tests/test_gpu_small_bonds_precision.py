"""Saturated bonds below 64 columns keep the precision of the Jacobi sweeps (default route).

A Schmidt value of 1e-6 of the largest is accurate to its own size, and so is a row of Gamma
whose Lambda is as small: a bidiagonal SVD gives both to eps of the largest only, and the
division by the small Lambda leaves 1e-10.  The oracle is a one-sided Jacobi SVD in extended
precision.  Bound: the QR route's error is n eps times the condition of Theta with rows and
columns scaled to one another's size, up to some 1e2 here: 100 n eps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


def _jacobi(x):
    """Columns of x made orthogonal (clongdouble), in descending order of their norms."""
    x = x.astype(np.clongdouble)
    n = x.shape[1]
    for _ in range(40):
        worst = 0.0
        for i in range(n - 1):
            for j in range(i + 1, n):
                a, b = np.sum(np.abs(x[:, i]) ** 2), np.sum(np.abs(x[:, j]) ** 2)
                g = np.sum(np.conj(x[:, i]) * x[:, j])
                if abs(g) == 0 or abs(g) <= 1e-18 * np.sqrt(a * b):
                    continue
                worst = max(worst, float(abs(g) / np.sqrt(a * b)))
                z = (b - a) / (2 * abs(g))
                t = (1 if z >= 0 else -1) / (abs(z) + np.sqrt(1 + z * z))
                c = 1 / np.sqrt(1 + t * t)
                s = c * t * g / abs(g)
                x[:, i], x[:, j] = c * x[:, i] - np.conj(s) * x[:, j], s * x[:, i] + c * x[:, j]
        if worst < 1e-17:
            break
    order = np.argsort(-np.sqrt(np.sum(np.abs(x) ** 2, axis=0)).astype(float))
    return x[:, order]


@pytest.mark.parametrize("chi,d", [(16, 2), (7, 3)])
@pytest.mark.parametrize("spans", [(1e-2, 1e-2, 1e-2), (1e-6, 1e-6, 1e-6), (1e-8, 1e-8, 1e-8), (1e-6, 1e-2, 1e-6)])
def test_values_and_rows(pkg, chi, d, spans):
    rng = np.random.default_rng(chi)
    lam = [s ** (np.arange(chi) / (chi - 1)) for s in spans]
    lam = [x / np.linalg.norm(x) for x in lam]
    # isometries over the graded rows and columns, so that the state is close to canonical
    shape = (chi, d, chi)
    a = lam[0][:, None, None] * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    b = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * lam[2]
    a = np.linalg.qr(a.reshape(chi * d, chi))[0].reshape(shape)
    b = np.linalg.qr(b.reshape(chi, d * chi).conj().T)[0].conj().T.reshape(shape)
    gam = [np.asfortranarray(a / lam[0][:, None, None]), np.asfortranarray(b / lam[2])]
    h = rng.standard_normal((d * d, d * d))
    w, v = np.linalg.eigh(h + h.T)
    gate = (v * np.exp(-0.05j * w)) @ v.conj().T
    with pkg.Chain(2, d, chi) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, gate)
        g1, l1 = c.get_gamma(1), c.get_lambda(2)
    ext = [x.astype(np.longdouble) for x in lam]
    th = np.einsum("aig,g,gjb->aijb", gam[0].astype(np.clongdouble) * ext[0][:, None, None], ext[1],
                   gam[1].astype(np.clongdouble) * ext[2]).reshape(chi, d * d, chi)
    th = np.einsum("pq,aqb->apb", gate.astype(np.clongdouble), th).reshape(chi * d, d * chi)
    x = _jacobi(th)[:, :chi]
    s = np.sqrt(np.sum(np.abs(x) ** 2, axis=0))
    norm = np.sqrt(np.sum(s * s))
    bound = 100 * chi * d * EPS
    assert np.max(np.abs(l1 / (s / norm) - 1)) <= bound
    x = (x / norm).reshape(chi, d, chi) / ext[0][:, None, None]  # Gamma1 Lambda1
    want = np.einsum("aig,big->ab", x, x.conj())
    got = np.einsum("aig,big->ab", g1 * l1, (g1 * l1).conj())
    size = np.sqrt(np.outer(np.diag(want).real, np.diag(want).real))
    assert np.max(np.abs(got - want) / size) <= bound
