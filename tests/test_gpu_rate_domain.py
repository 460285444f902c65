"""Quantum parameters outside the rates' domain create no event: the
differential rates take the power 2/3 of a quotient that is negative there."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip, dev, host, ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["sfp_photon_from_rejection_sampling", "sfp_pair_from_rejection_sampling"])
def test_no_event_outside_the_domain(fn):
    d = cuda_or_skip()
    from sfparticles_b200 import _lib
    from sfparticles_b200.qed import device_tables
    n = 200_000
    tab = device_tables.rs_table(d)
    counts = []
    for chi in (np.full(n, 2.0), -np.geomspace(1e-3, 1e3, n), np.full(n, np.nan), np.zeros(n)):
        ig, c = dev(np.full(n, 1e-3)), dev(chi)
        pruned, event, delta = dev(np.zeros(n, bool)), dev(np.zeros(n, bool)), dev(np.zeros(n))
        _lib.call(fn, ptr(ig), ptr(c), 2e-14, n, ptr(pruned), ptr(event), ptr(delta), ctypes.byref(tab), 7, 0, 0,
                  stream())
        counts.append(int(host(event).sum()))
    assert counts[0] > 0 and counts[1:] == [0, 0, 0]
