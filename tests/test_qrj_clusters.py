"""Clusters of the QR route (qrj.cu): distributed shared memory only between running CTAs.

A CTA's shared memory may be accessed by the others of its cluster only after all of
them have started, which a cluster barrier guarantees.  The first test reads the sources: a
kernel that accesses another CTA's shared memory, itself or in a function that it calls, has
a cluster barrier before.  The second runs batches of more clusters than the GPU holds
at once, beside launches of one bond each: no sum of the route depends on the cluster's size,
so that both give the same bits.
"""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "opentebd-extended_gb300", "csrc")


def _bodies(text):
    """(header, body) of every brace block that follows a parameter list."""
    out = []
    for m in re.finditer(r"\)\s*(?:const\s*)?\{", text):
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        start = max(text.rfind(";", 0, m.start()), text.rfind("}", 0, m.start()), 0)
        out.append((text[start : m.start()], text[m.end() : i]))
    return out


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_a_barrier_before_remote_shared_memory(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    if "map_shared_rank" not in text:
        return
    names = {"map_shared_rank"}  # and the device functions that use it
    for header, body in _bodies(text):
        name = re.search(r"(\w+)\s*\([^()]*(?:\([^()]*\)[^()]*)*$", header)
        if "__device__" in header and name and "map_shared_rank" in body:
            names.add(name.group(1))
    kernels = [(h, b) for h, b in _bodies(text) if "__global__" in h]
    assert kernels
    for header, body in kernels:
        uses = [m.start() for m in re.finditer(r"\b(?:%s)\s*(?:<\w+>)?\s*\(" % "|".join(names), body)]
        if uses:
            first = body.find("cluster.sync()")
            assert 0 <= first < min(uses), header


@pytest.mark.gpu
@pytest.mark.parametrize("L,d,chi", [(400, 2, 17), (120, 3, 40), (40, 2, 80)])
def test_batches_and_single_bonds_alike(pkg, L, d, chi):
    rng = np.random.default_rng(L)
    rank = chi // 2  # unsaturated: the QR route
    gam = [np.asfortranarray(rng.standard_normal((chi, d, chi)) + 1j * rng.standard_normal((chi, d, chi)))
           for _ in range(L)]
    lam = [np.where(np.arange(chi) < rank, np.exp(-0.5 * np.arange(chi)), 0.0) for _ in range(L + 1)]
    lam = [x / np.linalg.norm(x) for x in lam]
    gate = np.linalg.qr(rng.standard_normal((d * d, d * d)) + 1j * rng.standard_normal((d * d, d * d)))[0]
    links = list(range(1, L, 2))
    with pkg.Chain(L, d, chi, svd_mode=4) as a, pkg.Chain(L, d, chi, svd_mode=4) as b:
        a.set_state(gam, lam)
        b.set_state(gam, lam)
        a.apply_bonds(links, [gate] * len(links))
        some = links[:: max(1, len(links) // 12)]
        for k in some:
            b.two_site_op(k, gate)
        for k in some:
            assert np.array_equal(a.get_lambda(k + 1), b.get_lambda(k + 1))
            assert np.array_equal(a.get_gamma(k), b.get_gamma(k))
            assert np.array_equal(a.get_gamma(k + 1), b.get_gamma(k + 1))
