"""Small singular values beside large ones: what the fixed-point bidiagonalisation adds to them.

Theta = H S H^T / n with Hadamard matrices, rows and columns permuted and multiplied by powers of
i: its entries are exact, and so are its singular values.  Bound on the values below a
hundredth of the largest: the bisection's width, eps of the largest; four roundings per column
and entry of half a unit of 2^-61 in the scale of the matrix, a power of two up to twice its
norm F: 2^-61 F each, which add up at random over 4 n of them; twice that for the largest of n
errors.  (Products kept in units of 2^-58 give up to eight times as much.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


def _hadamard(n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    return h


@pytest.mark.parametrize("n", [128, 256, 512])
@pytest.mark.parametrize("kind", ["octaves", "two_groups"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_small_values(pkg, n, kind, seed):
    rng = np.random.default_rng(seed)
    k = np.arange(n)
    s = 2.0 ** (-(k % 16)) if kind == "octaves" else np.where(k < n // 4, 1.0, 2.0**-10) * (1 - (k % 64) * 2.0**-9)
    h, p, q = _hadamard(n), rng.permutation(n), rng.permutation(n)
    theta = (1j ** rng.integers(0, 4, n))[:, None] * ((h[p] * s) @ h[q].T / n) * 1j ** rng.integers(0, 4, n)
    gam = [np.asfortranarray(theta[:, None, :]), np.asfortranarray(np.eye(n, dtype=complex)[:, None, :])]
    with pkg.Chain(2, 1, n, svd_mode=3) as c:
        c.set_state(gam, [np.ones(n)] * 3)
        c.two_site_op(1, np.eye(1, dtype=complex))
        l1 = c.get_lambda(2)
    want = np.sort(s)[::-1]
    norm = np.sqrt(np.sum(want**2))
    err = np.abs(l1.astype(np.longdouble) * norm - want)[want < 0.01]
    assert np.max(err) <= EPS + 2 * np.sqrt(4 * n) * 2.0**-61 * norm * 2


@pytest.mark.parametrize("n,value", [(64, 1.0), (64, 1.0 - 2.0**-30), (200, 0.5 + 2.0**-40)])
def test_one_dominant_row(pkg, n, value):
    """A norm at a power of two in a single row: the panel's vectors are at their largest."""
    rng = np.random.default_rng(n)
    theta = 1e-6 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    theta[0] = 0.0
    theta[0, 1:] = rng.standard_normal(n - 1)
    theta *= value / np.linalg.norm(theta)
    gam = [np.asfortranarray(theta[:, None, :]), np.asfortranarray(np.eye(n, dtype=complex)[:, None, :])]
    with pkg.Chain(2, 1, n, svd_mode=3) as c:
        c.set_state(gam, [np.ones(n)] * 3)
        c.two_site_op(1, np.eye(1, dtype=complex))
        l1, g1, g2 = c.get_lambda(2), c.get_gamma(1)[:, 0, :], c.get_gamma(2)[:, 0, :]
    back = (g1 * l1) @ g2
    assert np.linalg.norm(back / np.linalg.norm(back) - theta / np.linalg.norm(theta)) <= 1e-14
