"""Observables of a chain of more sites than a grid has rows (65535)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_single_site_rho_of_a_long_chain(pkg):
    L, d = 70001, 2
    rng = np.random.default_rng(1)
    amp = rng.standard_normal((L, d)) + 1j * rng.standard_normal((L, d))
    amp /= np.linalg.norm(amp, axis=1)[:, None]
    gam = [np.asfortranarray(a.reshape(1, d, 1)) for a in amp]
    with pkg.Chain(L, d, 1, max_batch=2) as c:
        c.set_state(gam, [np.ones(1)] * (L + 1))
        rho = c.single_site_rho()
    want = amp[:, :, None] * amp[:, None, :].conj()
    assert np.max(np.abs(np.asarray(rho) - want)) <= 1e-15
