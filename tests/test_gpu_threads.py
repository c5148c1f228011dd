"""Two threads with chains of different sizes: neither's launches depend on what the other sets.

The limit of a kernel's dynamic shared memory belongs to the process.  Where a call set it to
its own need, a smaller call between another thread's setting and launch made that launch fail.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(workers):
    errors = []

    def run(work):
        try:
            work()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=(w,)) for w in workers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]


def test_gates_of_different_d(pkg):
    def work(d, n):
        rng = np.random.default_rng(d)
        gam = [np.asfortranarray(rng.standard_normal((2, d, 2)) + 1j * rng.standard_normal((2, d, 2))) for _ in range(2)]
        lam = [np.array([0.8, 0.6])] * 3
        gate = np.eye(d * d, dtype=complex)
        with pkg.Chain(2, d, 2) as c:
            c.set_state(gam, lam)
            for _ in range(n):
                c.two_site_op(1, gate)

    _together([lambda: work(8, 1500), lambda: work(2, 3000), lambda: work(3, 3000)])


def test_products_of_different_forms(pkg):
    torch = pytest.importorskip("torch")
    lib = pkg.load_library()
    n = 64
    a, b = (torch.randn((1, n, n), dtype=torch.complex128, device="cuda") for _ in range(2))

    def work(form):
        out = torch.zeros((1, n, n), dtype=torch.complex128, device="cuda")
        for _ in range(2000):
            rc = lib.tebd_zgemm_tc(1, n, n, n, a.data_ptr(), n * n, n, b.data_ptr(), n * n, n, out.data_ptr(), n * n, n,
                                   form, None)
            if rc:
                raise RuntimeError("form %d: %d" % (form, rc))

    _together([lambda: work(1), lambda: work(3)])
