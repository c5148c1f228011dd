"""The fixed-point bidiagonalisation (gebrd.cu) at the edges of its blocks.

One bond with d = 1, so that the compacted Theta is any r0 x r2 matrix: sizes around
the 8-column panels, the 8-row blocks dealt out to the CTAs, the 32-entry padding and
the split of the products.  Bound: the singular values of a backward-stable
bidiagonal SVD lie within a small multiple of eps ||Theta||_2 of LAPACK's; 1e-13 of the
largest is 450 eps, the bar of the other parity tests.  Vectors: the bond's tensor
rebuilt from the updated Gammas and Lambda (all values kept) must give Theta back to
1e-12 of its norm.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bond(rng, chi, r0, r2, decay):
    """Gammas and Lambdas whose Theta is r0 x r2, its columns and rows graded by `decay`."""
    gam = [np.asfortranarray(rng.standard_normal((chi, 1, chi)) + 1j * rng.standard_normal((chi, 1, chi)))
           for _ in range(2)]
    lam = [np.zeros(chi) for _ in range(3)]
    lam[0][:r0] = np.exp(-decay * np.arange(r0) / r0)
    lam[1][:] = 1.0
    lam[2][:r2] = np.exp(-decay * np.arange(r2) / r2)
    return gam, [l / np.linalg.norm(l) for l in lam]


@pytest.mark.parametrize("r0,r2", [(2, 2), (7, 3), (8, 8), (9, 8), (16, 17), (33, 31), (64, 64), (65, 129), (127, 128),
                                   (257, 255), (300, 40), (40, 300), (640, 513)])
@pytest.mark.parametrize("svd_mode", [3, 5])
@pytest.mark.parametrize("decay", [0.0, 12.0])
def test_values_and_vectors(pkg, r0, r2, svd_mode, decay):
    if svd_mode == 5 and min(r0, r2) < 64:
        pytest.skip("the double-float form bidiagonalises from 64 columns")
    rng = np.random.default_rng(1000 * r0 + r2)
    chi = max(r0, r2)
    gam, lam = _bond(rng, chi, r0, r2, decay)
    theta = (lam[0][:, None] * gam[0][:, 0, :] * lam[1]) @ (gam[1][:, 0, :] * lam[2])
    theta /= np.linalg.norm(theta)
    with pkg.Chain(2, 1, chi, svd_mode=svd_mode) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, np.eye(1, dtype=complex))
        s, l1 = c.singular_values(1), c.get_lambda(2)
        g1, g2 = c.get_gamma(1), c.get_gamma(2)
        if min(r0, r2) >= 64:
            assert c.stats()["bidiag_updates"] == 1
    ref = np.linalg.svd(theta, compute_uv=False)[: len(s)]
    assert np.max(np.abs(s[: len(ref)] - ref)) <= 1e-12 * ref[0]
    back = (lam[0][:, None] * g1[:, 0, :] * l1) @ (g2[:, 0, :] * lam[2])
    assert np.linalg.norm(back / np.linalg.norm(back) - theta) <= 1e-12


@pytest.mark.parametrize("scale", [1e-120, 1e-9, 1e9, 1e120])
def test_unnormalised_scales(pkg, scale):
    """Swapping decomposes the unnormalised Theta: the fixed-point unit follows its norm."""
    rng = np.random.default_rng(5)
    chi, d = 40, 2
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(2)]
    lam = [np.exp(-np.arange(chi) / 10.0) for _ in range(3)]
    gam[0] = np.asfortranarray(gam[0] * scale)
    th = (lam[0][:, None, None] * gam[0] * lam[1]).reshape(chi * d, chi) @ (gam[1] * lam[2]).reshape(chi, d * chi)
    sw = th.reshape(chi, d, d, chi).transpose(0, 2, 1, 3).reshape(chi * d, d * chi)
    with pkg.Chain(2, d, chi, svd_mode=3) as c:
        c.set_state(gam, lam)
        c.swapping(1)
        s = c.singular_values(1)
    ref = np.linalg.svd(sw, compute_uv=False)[: len(s)]
    assert np.max(np.abs(s[: len(ref)] - ref)) <= 1e-12 * ref[0]
