"""The training kernel (csrc/sfp_mlp.cu, k_mlp_grad) at the edges of its
32-sample tiles and three-pipeline blocks, against the same gradient in
float64 through torch's autograd.

Tolerance: a float32 sum of N terms in any order is within N 2^-24 of the sum
of their magnitudes, and activations and derivatives carry a few 2^-24 of
their own; per parameter block the gradient of random features and targets
is no smaller than 1e-2 of that sum, so 2e-4 relative (2-norm) for N up to
5000, and 1e-5 for the loss, whose terms are positive."""
import numpy as np
import pytest

from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 95, 96, 97, 5000])
def test_gradient_at_tile_edges(n):
    cuda_or_skip()
    import torch
    from sfparticles_b200 import mlp
    g = torch.Generator(device="cuda").manual_seed(n)
    s = mlp.PhotonSampler(mlp.init_params(2))
    feat = 2 * torch.rand((n, 2), device="cuda", generator=g) - 1
    targ = 2.0 + torch.rand(n, device="cuda", generator=g)
    got, loss = s.grad(feat, targ)
    p = s.params.clone()
    for k, (o, shape) in mlp.OFFSETS.items():
        if k[0] == "W":
            m = int(np.prod(shape))
            p[o:o + m] = p[o:o + m].bfloat16().float()
    p = p.double().requires_grad_()
    w = {k: p[o:o + (int(np.prod(sh)) if sh else 1)].reshape(sh) for k, (o, sh) in mlp.OFFSETS.items()}
    h = feat.double()
    for k in range(3):
        h = torch.nn.functional.silu(h @ w[f"W{k}"].T + w[f"b{k}"])
    want = ((h @ w["W3"] + w["b3"] - targ.double()) ** 2).sum()
    want.backward()
    assert abs(loss - want.item()) <= 1e-5 * want.item()
    for k, (o, sh) in mlp.OFFSETS.items():
        m = int(np.prod(sh)) if sh else 1
        a, b = got[o:o + m].double(), p.grad[o:o + m]
        assert float((a - b).norm()) <= 2e-4 * float(b.norm()), k
