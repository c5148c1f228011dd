"""The observables' kernels at the edges of their tiles and splits: odd and even chains
(the overlap's two halves), local dimensions 1 to 8, bond dimensions around 16 and 32.
Sums of positive and mixed terms in FP64: 1e-12 of the largest entry."""
import numpy as np
import pytest

from oracle import observables as obs

pytestmark = pytest.mark.gpu


def _chain(rng, L, d, chi):
    gam = [np.asfortranarray((rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
                             / np.sqrt(d * chi)) for _ in range(L)]
    lam = [np.sort(rng.random(chi))[::-1] for _ in range(L + 1)]
    if chi > 4:
        lam[1][-2:] = 0.0
    return gam, [l / np.linalg.norm(l) * np.sqrt(chi) for l in lam]


@pytest.mark.parametrize("L,d,chi", [(2, 2, 1), (2, 1, 5), (3, 2, 15), (4, 3, 16), (5, 5, 17), (7, 4, 33), (3, 8, 31),
                                     (2, 6, 40), (6, 7, 12)])
def test_against_numpy(pkg, L, d, chi):
    rng = np.random.default_rng(100 * L + 10 * d + chi)
    gam, lam = _chain(rng, L, d, chi)
    oth, olam = _chain(rng, L, d, chi)
    with pkg.Chain(L, d, chi) as c, pkg.Chain(L, d, chi) as o:
        c.set_state(gam, lam)
        o.set_state(oth, olam)
        rho, ov = c.single_site_rho(), c.inner_product(o)
        rho2 = [c.two_site_rho(k) for k in range(1, L)]
    for s in range(L):
        ref = obs.single_site_rho(lam[s], gam[s], lam[s + 1])
        assert np.max(np.abs(rho[s] - ref)) <= 1e-12 * np.max(np.abs(ref))
    for k in range(L - 1):
        ref = obs.two_site_rho(lam[k], gam[k], lam[k + 1], gam[k + 1], lam[k + 2])
        assert np.max(np.abs(rho2[k] - ref)) <= 1e-12 * np.max(np.abs(ref))
    ref = obs.inner_product(gam, lam, oth, olam)
    norm = np.sqrt(abs(obs.inner_product(gam, lam, gam, lam)) * abs(obs.inner_product(oth, olam, oth, olam)))
    assert abs(ov - ref) <= 1e-12 * norm
