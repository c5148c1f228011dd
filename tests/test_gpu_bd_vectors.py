"""Singular vectors of the bidiagonal route where the values are close together.

Inverse iteration gives no orthogonality inside a cluster: it all comes from the
re-orthogonalisation (bdorth.cu).  One bond with d = 1 and unit Lambdas, so that Theta is
a chosen U diag(s) V^H; sizes around the panels of eight vectors and the 32-row groups.
Bounds: the vectors orthonormal to 1e-12 (16 n eps at n = 257).  Theta rebuilt to
10 n^2 eps of its norm: the members of a cluster are random combinations, whose condition
is about n, and the left and the right set are re-orthogonalised by themselves.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _unitary(rng, n):
    return np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]


def _values(kind, n):
    s = np.ones(n)
    if kind == "pairs":  # 1e-13 apart
        s = np.exp(-3.0 * (np.arange(n) // 2) / n) * (1.0 + 1e-13 * (np.arange(n) % 2))
    elif kind == "cluster":  # a block of equal values that crosses panels, graded ones around it
        s = np.exp(-3.0 * np.arange(n) / n)
        s[n // 4 : n // 4 + min(n // 2, 21)] = s[n // 4]
    return np.sort(s)[::-1]


@pytest.mark.parametrize("n", [7, 8, 9, 33, 64, 100, 257])
@pytest.mark.parametrize("kind", ["equal", "pairs", "cluster"])
@pytest.mark.parametrize("svd_mode", [3, 5])
def test_clusters(pkg, n, kind, svd_mode):
    if svd_mode == 5 and n < 64:
        pytest.skip("the double-float form bidiagonalises from 64 columns")
    rng = np.random.default_rng(n)
    s = _values(kind, n)
    theta = (_unitary(rng, n) * s) @ _unitary(rng, n).conj().T
    gam = [np.asfortranarray(theta[:, None, :]), np.asfortranarray(np.eye(n, dtype=complex)[:, None, :])]
    lam = [np.full(n, n**-0.5) for _ in range(3)]
    lam[1] = np.ones(n)
    with pkg.Chain(2, 1, n, svd_mode=svd_mode) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, np.eye(1, dtype=complex))
        l1, g1, g2 = c.get_lambda(2), c.get_gamma(1)[:, 0, :], c.get_gamma(2)[:, 0, :]
    u, v = g1 * lam[0][:, None], g2 * lam[2]
    assert np.max(np.abs(u.conj().T @ u - np.eye(n))) <= 1e-12
    assert np.max(np.abs(v @ v.conj().T - np.eye(n))) <= 1e-12
    ref = s / np.linalg.norm(s)
    assert np.max(np.abs(l1 / np.linalg.norm(l1) - ref)) <= 1e-12 * ref[0]
    want = theta / np.linalg.norm(theta)
    back = (u * l1) @ v
    assert np.linalg.norm(back / np.linalg.norm(back) - want) <= 10 * n * n * 2.2e-16


@pytest.mark.parametrize("sizes", [(170, 128, 96, 33), (300, 256, 129, 64), (40, 170, 7, 2), (520, 300, 40, 256)])
def test_one_batch_of_several_sizes(pkg, sizes):
    """Three bonds of different Theta in one batch: the launch is sized by the largest."""
    rng = np.random.default_rng(sum(sizes))
    chi = max(sizes)
    gam = [np.asfortranarray(rng.standard_normal((chi, 1, chi)) + 1j * rng.standard_normal((chi, 1, chi)))
           for _ in range(6)]
    lam = [np.ones(chi) for _ in range(7)]
    for q, r in enumerate(sizes):  # Theta of bond 2 q + 1 is sizes[q] x sizes[q + 1]
        lam[2 * q] = np.where(np.arange(chi) < r, np.exp(-2.0 * np.arange(chi) / chi), 0.0)
        lam[2 * q] /= np.linalg.norm(lam[2 * q])
    with pkg.Chain(6, 1, chi, svd_mode=3) as c:
        c.set_state(gam, lam)
        c.apply_bonds([1, 3, 5], [np.eye(1, dtype=complex)] * 3)
        for b in range(3):
            l0, l2, l1 = lam[2 * b], lam[2 * b + 2], c.get_lambda(2 * b + 2)
            want = (l0[:, None] * gam[2 * b][:, 0, :]) @ (gam[2 * b + 1][:, 0, :] * l2)
            back = (l0[:, None] * c.get_gamma(2 * b + 1)[:, 0, :] * l1) @ (c.get_gamma(2 * b + 2)[:, 0, :] * l2)
            assert np.linalg.norm(back / np.linalg.norm(back) - want / np.linalg.norm(want)) <= 1e-12
