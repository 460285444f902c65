"""Growth of a species' arrays in one allocation and one launch, against an
array at a time.  Copies and constant fills: the bytes are the same."""
import numpy as np
import pytest

import sfparticles_b200 as S
from sfparticles_b200 import _lib, particles

pytestmark = pytest.mark.gpu


def _grown(old, new, together, monkeypatch):
    monkeypatch.setattr(particles, "GROW_TOGETHER", 1 << 28 if together else 0)
    rng = np.random.default_rng(old)
    p = S.SpinParticles("electron", -1, 1, N=old, props=tuple(rng.normal(size=old) for _ in range(9)))
    p._to_gpu()
    p._d("event"), p._d("chi")
    if old:
        p._arr["event"].random_(0, 2)
    before = {k: v.cpu().numpy() for k, v in p._arr.items()}
    p._resize(new)
    assert p.buffer_size == new
    return before, {k: v.cpu().numpy() for k, v in p._arr.items()}, {k: v.data_ptr() for k, v in p._arr.items()}


@pytest.mark.parametrize("old,new", [(0, 1), (0, 300), (1, 1), (1, 2), (31, 257), (255, 256), (4097, 5000),
                                     (100001, 700003)])
def test_grown_arrays(old, new, monkeypatch):
    for together in (True, False):
        before, after, at = _grown(old, new, together, monkeypatch)
        for k, v in after.items():
            assert v.shape == (new,) and v.dtype == before[k].dtype
            assert np.array_equal(v[:old], before[k])
            assert np.all(v[old:] == (1 if k == "_to_be_pruned" else 0)), k
        if together:  # one block, each array on a 256-byte boundary of it
            assert len({a % 256 for a in at.values()}) == 1
    # more arrays than one launch takes
    import ctypes
    import torch
    n = 70
    src = torch.arange(n * 8, dtype=torch.float64, device="cuda").reshape(n, 8)
    dst = torch.full((n, 20), -1.0, dtype=torch.float64, device="cuda")
    jobs = (_lib.GrowArray * n)(*[_lib.GrowArray(src[i].data_ptr(), dst[i].data_ptr(), 8, 0) for i in range(n)])
    _lib.call("sfp_grow_arrays", jobs, n, 8, 20, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert torch.equal(dst[:, :8], src) and bool((dst[:, 8:] == 0).all())


def test_arrays_of_other_sizes_keep_to_the_general_path(monkeypatch):
    p = S.Particles("electron", -1, 1, N=10, props=tuple(np.arange(10.0) for _ in range(6)))
    p._to_gpu()
    p._arr["x"] = p._arr["x"].repeat(2)[::2]  # strided
    want = p._arr["x"].cpu().numpy()
    assert p._grow_together(10, 20) is False
    p._resize(20)
    assert np.array_equal(p._arr["x"].cpu().numpy()[:10], want) and p._arr["x"].shape == (20,)
