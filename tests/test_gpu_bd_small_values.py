"""Values near the rounding of the largest, on the bidiagonal route.

Values down to the guard (1e-15) are kept with their vectors.  Each value and its negative are
eigenvalues of the matrix that inverse iteration works on; where a shift is not small
against the value, left and right vectors of different values come out together, and Theta
rebuilt from the update is off by the size of these values.

Bound, with the largest value as the unit: 2 eps for each of the n values (the bisection's
width and the counts' rounding), which add up to 2 sqrt(n) eps in norm; 16 eps for the
bidiagonalisation and the larger values; a value below the guard, 4.5 eps, is dropped, at most
n / 4 of them here: 2.25 sqrt(n) eps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


@pytest.mark.parametrize("n", [128, 256, 400])
@pytest.mark.parametrize("kind", ["graded", "half"])
def test_theta_from_small_values(pkg, n, kind):
    rng = np.random.default_rng(n)
    k = np.arange(n)
    if kind == "graded":
        s = 10.0 ** (-15.0 * k / (n - 1))
    else:  # half of the values between 1e-13 and 2e-15 of the largest
        s = np.where(k < n // 2, np.exp(-2.0 * k / n), 10.0 ** (-13.0 - 1.7 * (k - n // 2) / n * 2))
    u, v = (np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0] for _ in range(2))
    theta = (u * s) @ v.conj().T
    gam = [np.asfortranarray(theta[:, None, :]), np.asfortranarray(np.eye(n, dtype=complex)[:, None, :])]
    lam = [np.full(n, n**-0.5) for _ in range(3)]
    lam[1] = np.ones(n)
    with pkg.Chain(2, 1, n, svd_mode=3) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, np.eye(1, dtype=complex))
        l1, g1, g2 = c.get_lambda(2), c.get_gamma(1)[:, 0, :], c.get_gamma(2)[:, 0, :]
    back = (g1 * lam[0][:, None] * l1) @ (g2 * lam[2])
    want = theta / np.linalg.norm(theta)
    assert np.linalg.norm(back - want) <= (4.25 * n**0.5 + 16.0) * EPS
