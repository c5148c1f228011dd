"""Saturated bonds below 64 columns (default route): every singular value is reported.

The route computes vectors for the chi kept values only; the values beyond them come from
the bisection alone.  Bound: 1e-13 of the largest value, 450 eps, as for the larger bonds.
The second case is a bond whose values span more than 1e-8, which keeps the Jacobi route.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,d", [(4, 2), (5, 3), (7, 2), (16, 2), (31, 2), (12, 5)])
@pytest.mark.parametrize("decay", [3.0, 25.0])
def test_all_values(pkg, chi, d, decay):
    rng = np.random.default_rng(100 * chi + d)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(2)]
    lam = [np.exp(-decay * np.arange(chi) / chi) for _ in range(3)]
    lam = [x / np.linalg.norm(x) for x in lam]
    q = np.linalg.qr(rng.standard_normal((d * d, d * d)) + 1j * rng.standard_normal((d * d, d * d)))[0]
    a = lam[0][:, None, None] * gam[0] * lam[1]
    th = np.einsum("aib,bjc->aijc", a, gam[1] * lam[2]).reshape(chi, d * d, chi)
    th = np.einsum("pq,aqc->apc", q, th).reshape(chi * d, d * chi)
    ref = np.linalg.svd(th / np.linalg.norm(th), compute_uv=False)
    with pkg.Chain(2, d, chi) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, q)
        s = np.asarray(c.singular_values(1))
        kept = c.get_lambda(2)
    assert len(s) == chi * d
    assert np.max(np.abs(s - ref)) <= 1e-13
    assert np.max(np.abs(kept - ref[:chi] / np.linalg.norm(ref[:chi]))) <= 1e-13
