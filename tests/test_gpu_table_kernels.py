"""The group-parallel table kernels (csrc/sfp_tables.cu: a warp per rate, a block
of 21 warps per total) at the edges of their shapes, against the same
generator compiled for the host, one thread per row.

Tolerance 5e-12 relative: host and device differ by their exp and pow
(about 1e-15 per integrand value), which the extrapolation of the adaptive
quadrature carries to 1.2e-12 at most on the full tables."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip
from test_table_generator import D, DP, lib  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 2), (2, 33), (3, 34), (149, 5)])
def test_od_rows_match_the_host_build(lib, kind, rows, cols):  # noqa: F811
    cuda_or_skip()
    import torch
    from sfparticles_b200 import _lib
    from sfparticles_b200.qed import tables as T
    factor = T.photon_factor() if kind == 0 else T.pair_factor()
    chi = np.logspace(-2.9, 2.9, rows) if rows > 1 else np.array([0.3])
    delta = np.logspace(-6, 0, cols) if cols > 1 else np.array([1e-6])
    dev = torch.device("cuda")
    c, d = torch.as_tensor(chi, device=dev), torch.as_tensor(delta, device=dev)
    tot, first = (torch.empty(rows, dtype=torch.float64, device=dev) for _ in range(2))
    cum = torch.empty((rows, cols), dtype=torch.float64, device=dev)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.call("sfp_table_od", kind, factor, p(c), rows, p(d), cols, p(tot), p(cum), p(first), None)
    torch.cuda.synchronize()
    tot, cum, first = tot.cpu().numpy(), cum.cpu().numpy(), first.cpu().numpy()
    for r in sorted({0, 1, rows // 2, rows - 1} & set(range(rows))):
        t, row = D(), np.zeros(cols)
        lib.od_row(kind, factor, chi[r], delta.ctypes.data_as(DP), cols, ctypes.byref(t), row.ctypes.data_as(DP))
        for got, want in ((tot[r:r + 1], np.array([t.value])), (first[r:r + 1], row[:1]), (cum[r], row)):
            big = np.abs(want) > 1e-250
            assert np.all(np.abs(got[~big]) <= 1e-250)
            if big.any():
                assert np.max(np.abs(got[big] - want[big]) / np.abs(want[big])) < 5e-12, (r, got, want)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 600])
def test_rs_points_match_the_host_build(lib, n):  # noqa: F811
    cuda_or_skip()
    import torch
    from sfparticles_b200 import _lib
    z = np.linspace(0.0, 107.0, n) if n > 1 else np.array([2.0])
    dev = torch.device("cuda")
    zd = torch.as_tensor(z, device=dev)
    ia, da = torch.empty_like(zd), torch.empty_like(zd)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.call("sfp_table_rs", p(zd), n, p(ia), p(da), None)
    torch.cuda.synchronize()
    want_i, want_d = np.zeros(n), np.zeros(n)
    lib.rs_rows.argtypes = [DP, ctypes.c_long, DP, DP]
    lib.rs_rows(z.ctypes.data_as(DP), n, want_i.ctypes.data_as(DP), want_d.ctypes.data_as(DP))
    for got, want in ((ia.cpu().numpy(), want_i), (da.cpu().numpy(), want_d)):
        big = np.abs(want) > 1e-250
        assert np.max(np.abs(got[big] - want[big]) / np.abs(want[big])) < 5e-12
