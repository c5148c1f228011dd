"""A non-finite Theta on the bidiagonal route fails in less than the time of a finite one.

The error is found at the end of the batch; until then the kernels run on NaNs.  The
bidiagonalisation, the largest part of the time, returns at once, so that the whole must be
shorter, unless a later kernel takes a slow path (the rescaling of the inverse iteration
rewrote a whole vector at every step of every solve: 2.5 times a finite batch at 127
columns, in proportion to their number).  Sizes below the digit-plane Theta, whose digits of
a NaN are zeros.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,d", [(127, 1), (60, 2)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_time_of_the_error(pkg, chi, d, bad):
    rng = np.random.default_rng(1)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(2)]
    lam = [np.exp(-3.0 * np.arange(chi) / chi) for _ in range(3)]
    lam = [x / np.linalg.norm(x) for x in lam]
    broken = [gam[0].copy(order="F"), gam[1]]
    broken[0][3, d - 1, 5] = bad
    times = {}
    with pkg.Chain(2, d, chi, svd_mode=3) as c:
        for name, g in (("finite", gam), ("broken", broken)):
            times[name] = np.inf
            for _ in range(4):
                c.set_state(g, lam)
                c.sync()
                t0 = time.perf_counter()
                if name == "finite":
                    c.two_site_op(1, np.eye(d * d, dtype=complex))
                else:
                    with pytest.raises(pkg.TebdError) as e:
                        c.two_site_op(1, np.eye(d * d, dtype=complex))
                    assert e.value.code == 5  # TEBD_ERR_NONFINITE
                times[name] = min(times[name], time.perf_counter() - t0)
    assert times["broken"] < times["finite"]
