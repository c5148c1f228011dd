"""Two-site density matrices: a bond's sum split over the GPU where few bonds are asked for.

Single bonds of sizes around the split (two stages of 16 pairs of rows and columns per part)
and local dimensions that leave most of a CTA without entries.  FP64 sums in another order:
1e-13 of the trace.
"""
import numpy as np
import pytest

from oracle import observables as obs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,d", [(1, 2), (5, 1), (6, 3), (8, 2), (31, 3), (70, 2), (97, 1), (40, 8)])
def test_single_bonds(pkg, chi, d):
    rng = np.random.default_rng(chi + d)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(3)]
    lam = [np.sort(rng.random(chi))[::-1] + 0.1 for _ in range(4)]
    with pkg.Chain(3, d, chi) as c:
        c.set_state(gam, lam)
        for k in (1, 2):
            ref = obs.two_site_rho(lam[k - 1], gam[k - 1], lam[k], gam[k], lam[k + 1])
            assert np.max(np.abs(c.two_site_rho(k) - ref)) <= 1e-13 * np.trace(ref).real
