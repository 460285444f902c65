"""An empty species resized to nothing stays empty."""
import pytest

import sfparticles_b200 as S
from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu


def test_no_slots():
    cuda_or_skip()
    p = S.Particles("photon", 0, 0)
    p._to_gpu()
    p._resize(0)
    assert p.buffer_size == 0 and all(v.shape == (0,) for v in p._arr.values())
    p._resize(3)
    assert p._to_be_pruned.all() and p.x.shape == (3,)
