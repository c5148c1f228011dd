"""Swapping decomposes the unnormalised Theta on the bidiagonal route: far from 1, with columns far
below the norm.

A column of 1e-10 of a Theta of 1e-130 has a squared norm of 1e-280; the reflectors'
scalars are to be formed in the scale of the matrix.  Bound: 1e-12 of the largest value, as at
the ordinary scales.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-145, 1e-135, 1e-130, 1.0, 1e130, 1e145])
@pytest.mark.parametrize("decay", [1.5, 4.0])
def test_graded_columns_at_extreme_scales(pkg, scale, decay):
    rng = np.random.default_rng(7)
    chi, d = 40, 2
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(2)]
    lam = [np.exp(-np.arange(chi) / decay) for _ in range(3)]
    th = (lam[0][:, None, None] * gam[0] * lam[1]).reshape(chi * d, chi) @ (gam[1] * lam[2]).reshape(chi, d * chi)
    sw = th.reshape(chi, d, d, chi).transpose(0, 2, 1, 3).reshape(chi * d, d * chi)
    ref = np.linalg.svd(sw, compute_uv=False)
    with pkg.Chain(2, d, chi, svd_mode=3) as c:
        c.set_state([np.asfortranarray(gam[0] * scale), gam[1]], lam)
        c.swapping(1)
        s = np.asarray(c.singular_values(1)) / scale
    assert np.max(np.abs(s[: len(ref)] - ref[: len(s)])) <= 1e-12 * ref[0]
