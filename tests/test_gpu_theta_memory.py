"""The default form on a GPU without room for the digit planes of a large Theta.

Their workspace is taken at the first large product.  Where the device memory is full it
must not fail: Theta is formed on the CUDA cores then.  Bound: both ways are FP64 class; 1e-13
of the largest Schmidt value, as between the other forms.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_full_memory(pkg):
    torch = pytest.importorskip("torch")
    L, d, chi = 8, 4, 256  # four bonds of 1024 x 1024: 100 MB of planes
    rng = np.random.default_rng(3)
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(L)]
    lam = [np.exp(-8.0 * np.arange(chi) / chi) for _ in range(L + 1)]
    lam = [x / np.linalg.norm(x) for x in lam]
    links, gates = list(range(1, L, 2)), [np.eye(d * d, dtype=complex)] * (L // 2)

    with pkg.Chain(L, d, chi) as a, pkg.Chain(L, d, chi) as b:
        for c in (a, b):
            c.set_state(gam, lam)
        a.apply_bonds(links, gates)  # loads the kernels, too
        hold, keep = [], 48 << 20
        try:
            for _ in range(4):
                free = torch.cuda.mem_get_info()[0]
                if free > keep + (2 << 20):
                    hold.append(torch.empty(free - keep, dtype=torch.uint8, device="cuda"))
            assert torch.cuda.mem_get_info()[0] < 90 << 20
            b.apply_bonds(links, gates)
        finally:
            hold.clear()
            torch.cuda.empty_cache()
        for k in links:
            x, y = a.get_lambda(k + 1), b.get_lambda(k + 1)
            assert np.max(np.abs(x - y)) <= 1e-13 * x[0]
