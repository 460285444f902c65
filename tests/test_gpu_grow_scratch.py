"""The scratch arrays of a grown species are freed without its state."""
import numpy as np
import pytest

import sfparticles_b200 as S
from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("old,new", [(100_000, 700_001), (1_000_000, 1_500_000)])
def test_dropped_scratch_frees_its_memory(old, new):
    import torch
    cuda_or_skip()
    p = S.Particles("electron", -1, 1, N=old, props=tuple(np.arange(old, dtype=float) for _ in range(6)))
    p._to_gpu()
    p._drop_scratch()
    for k in ("chi", "Ex", "Ey", "Ez", "Bx", "By", "Bz", "event"):
        p._d(k)
    p._resize(new)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    p._drop_scratch()
    assert before - torch.cuda.memory_allocated() >= new * (7 * 8 + 1)
    assert np.array_equal(p.ux[:old], np.arange(old)) and p._to_be_pruned[old:].all()
