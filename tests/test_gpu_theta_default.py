"""Theta of the default form from digit planes (large products), at the edges of its tiles.

The two-site density matrix of a bond is quadratic in Theta: its entries are held to
1e-14 of its trace, FP64's own rounding of the few thousand terms of an entry (each
within eps of the factors) with a decade to spare.  Non-finite factors have zero digits,
so that they are reported apart.
"""
import numpy as np
import pytest

from oracle import observables as obs

pytestmark = pytest.mark.gpu


def _chain(chi, d, r0, r1, r2, decay, seed):
    rng = np.random.default_rng(seed)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(2)]
    lam = []
    for r in (r0, r1, r2):
        v = np.zeros(chi)
        v[:r] = np.exp(-decay * np.arange(r) / r)
        lam.append(v / np.linalg.norm(v))
    return gam, lam


@pytest.mark.parametrize("chi,d,r0,r1,r2", [(64, 4, 64, 64, 64), (64, 4, 33, 61, 64), (127, 2, 127, 100, 127),
                                            (128, 2, 65, 128, 128), (129, 2, 129, 129, 129), (100, 3, 100, 97, 43),
                                            (90, 5, 90, 90, 90)])
@pytest.mark.parametrize("decay", [0.0, 30.0])
def test_rho2(pkg, chi, d, r0, r1, r2, decay):
    assert d * r0 * d * r2 * r1 >= 1 << 20  # both sides of the switch at 2^21
    gam, lam = _chain(chi, d, r0, r1, r2, decay, chi + d)
    with pkg.Chain(2, d, chi) as c:
        c.set_state(gam, lam)
        rho = c.two_site_rho(1)
    ref = obs.two_site_rho(lam[0], gam[0], lam[1], gam[1], lam[2])
    assert np.max(np.abs(rho - ref)) <= 1e-14 * np.trace(ref).real


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_factors(pkg, bad):
    chi, d = 64, 4
    gam, lam = _chain(chi, d, chi, chi, chi, 3.0, 1)
    gam[0][3, 1, 5] = bad
    with pkg.Chain(2, d, chi) as c:
        c.set_state(gam, lam)
        assert np.isnan(c.two_site_rho(1)).any()
        with pytest.raises(pkg.TebdError) as e:
            c.two_site_op(1, np.eye(d * d, dtype=complex))
        assert e.value.code == 5  # TEBD_ERR_NONFINITE
        g, l = c.get_state()
        assert np.array_equal(l[1], lam[1])
