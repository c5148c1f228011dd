"""Multiplets among the singular values, on the bidiagonal route.

A chain with a non-abelian symmetry has multiplets of Schmidt values.  Inverse iteration gives
their vectors as combinations of the multiplet's, the left and the right ones in one solve;
each set is then re-orthogonalised by itself, which keeps the pairs only as far as the
raw vectors are independent.  Theta rebuilt from the update shows both.

Bound: a vector of a multiplet is a combination of values that lie within the solves' shift of
one another, 64 eps of the largest, and the rounding of the re-orthogonalisation grows with
the condition of the raw vectors, at most some 1e3: 1024 eps of Theta's norm.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


def _unitary(rng, n):
    return np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]


def _rebuilt(pkg, theta, svd_mode=3):
    """Theta from one update (d = 1, unit Lambdas), and Theta, both of norm 1."""
    n = theta.shape[0]
    gam = [np.asfortranarray(theta[:, None, :]), np.asfortranarray(np.eye(n, dtype=complex)[:, None, :])]
    lam = [np.full(n, n**-0.5) for _ in range(3)]
    lam[1] = np.ones(n)
    with pkg.Chain(2, 1, n, svd_mode=svd_mode) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, np.eye(1, dtype=complex))
        l1, g1, g2 = c.get_lambda(2), c.get_gamma(1)[:, 0, :], c.get_gamma(2)[:, 0, :]
    back = (g1 * lam[0][:, None] * l1) @ (g2 * lam[2])
    return back / np.linalg.norm(back), theta / np.linalg.norm(theta)


def _multiplets(n, size, span):
    k = np.arange(n)
    return span ** ((k // size) * size / n)


@pytest.mark.parametrize("n", [33, 64, 128, 257])
@pytest.mark.parametrize("size,span", [(2, 1e-2), (3, 1e-5), (4, 1e-8), (16, 1e-8), (21, 0.05)])
def test_multiplets(pkg, n, size, span):
    rng = np.random.default_rng(n * size)
    back, want = _rebuilt(pkg, (_unitary(rng, n) * _multiplets(n, size, span)) @ _unitary(rng, n).conj().T)
    assert np.linalg.norm(back - want) <= 1024 * EPS


@pytest.mark.parametrize("n", [64, 128, 256, 512])
@pytest.mark.parametrize("svd_mode", [3, 5])
def test_equal_values(pkg, n, svd_mode):
    rng = np.random.default_rng(n)
    back, want = _rebuilt(pkg, _unitary(rng, n), svd_mode)
    assert np.linalg.norm(back - want) <= 1024 * EPS


@pytest.mark.parametrize("n", [64, 200])
def test_one_cluster_among_graded_values(pkg, n):
    rng = np.random.default_rng(n)
    s = np.exp(-3.0 * np.arange(n) / n)
    s[n // 4 : n // 4 + 21] = s[n // 4]
    back, want = _rebuilt(pkg, (_unitary(rng, n) * s) @ _unitary(rng, n).conj().T)
    assert np.linalg.norm(back - want) <= 1024 * EPS
