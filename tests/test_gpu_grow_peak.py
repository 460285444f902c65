"""A species too large to grow in one block grows an array at a time: beside
the grown species it needs the room of one array, not of a second species."""
import numpy as np
import pytest

import sfparticles_b200 as S
from gpu_helpers import cuda_or_skip
from sfparticles_b200 import particles

pytestmark = pytest.mark.gpu


def test_room_that_a_large_growth_takes():
    import torch
    cuda_or_skip()
    old, new = 5_000_000, 6_000_000
    p = S.Particles("electron", -1, 1, N=old, props=tuple(np.arange(old, dtype=float) for _ in range(6)))
    p._to_gpu()
    arrays = 6 * 8 + 1  # bytes a slot
    assert new * arrays > particles.GROW_TOGETHER
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    p._resize(new)
    # (an allocation is rounded up to 2 MiB at most)
    room = (new - old) * arrays + 8 * new + len(p._arr) * (2 << 20)
    assert torch.cuda.max_memory_allocated() - before <= room
    assert torch.cuda.memory_allocated() - before <= (new - old) * arrays + len(p._arr) * (2 << 20)
    assert np.array_equal(p.ux[:old], np.arange(old)) and not p.ux[old:].any()
