"""The QR + Jacobi route at the edges of its kernels' sizes and ranks.

One bond with d = 1 whose Theta is r0 x r2 of rank k: one warp's rows, a few more, wide and
tall, columns beyond the shared memory of the cluster (900) and a scratch beyond that of a
CTA (4200).  Bounds as for the other routes: singular values within 1e-13 of the
largest, Theta rebuilt to 1e-12 of its norm; the small values of a graded spectrum within
1e-6 of their own size (they are 1e-9 of the largest or more).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r0,r2,k", [(1, 1, 1), (2, 3, 2), (31, 33, 5), (64, 64, 64), (65, 40, 40), (170, 160, 36),
                                     (40, 300, 17), (300, 40, 40), (900, 880, 20), (4200, 24, 3)])
@pytest.mark.parametrize("scale", [1.0, 1e-100])
def test_rank_and_vectors(pkg, r0, r2, k, scale):
    if scale != 1.0 and r0 > 400:
        pytest.skip("one scale is enough for the large sizes")
    rng = np.random.default_rng(r0 + r2)
    chi = max(r0, r2)
    u = np.linalg.qr(rng.standard_normal((r0, k)) + 1j * rng.standard_normal((r0, k)))[0]
    v = np.linalg.qr(rng.standard_normal((r2, k)) + 1j * rng.standard_normal((r2, k)))[0].conj().T
    s = 10.0 ** (-9.0 * np.arange(k) / max(1, k - 1))
    gam = [np.zeros((chi, 1, chi), dtype=complex, order="F") for _ in range(2)]
    gam[0][:r0, 0, :k] = u * scale
    gam[1][:k, 0, :r2] = v
    lam = [np.zeros(chi) for _ in range(3)]
    lam[0][:r0] = r0**-0.5
    lam[1][:k] = s
    lam[2][:r2] = r2**-0.5
    with pkg.Chain(2, 1, chi, svd_mode=4) as c:
        c.set_state(gam, lam)
        c.two_site_op(1, np.eye(1, dtype=complex))
        sv, l1 = np.asarray(c.singular_values(1)), c.get_lambda(2)
        g1, g2 = c.get_gamma(1)[:r0, 0, :], c.get_gamma(2)[:, 0, :r2]
        assert c.stats()["bidiag_updates"] == 0
    ref = s / np.linalg.norm(s)
    assert np.max(np.abs(sv[:k] - ref)) <= 1e-13
    assert np.max(np.abs(sv[:k] / ref - 1.0)) <= 1e-6
    assert np.all(sv[k:] <= 1e-13)
    want = (u * s) @ v
    back = (g1 * l1) @ g2
    assert np.linalg.norm(back / np.linalg.norm(back) - want / np.linalg.norm(want)) <= 1e-12
