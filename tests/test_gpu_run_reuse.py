"""A run's bookkeeping block and stream are handed on to later runs
(csrc/sfp_capi.cu): results of runs that follow one another, of runs alive
together and of runs on several host threads equal those of a run alone,
bit for bit."""
import threading

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu


def _run(n, seed, steps, form="fp64"):
    import sfparticles_b200 as S
    from sfparticles_b200.fields import gaussian_laser_pulse
    r = np.random.default_rng(seed)
    ele = S.Particles("e", -1, 1, N=n, props=(r.normal(0, 4e-6, n), r.normal(0, 1e-6, n), r.normal(0, 1e-6, n),
                                             np.full(n, 2000.0), np.zeros(n), np.zeros(n)))
    pos, pho = S.Particles("p", 1, 1), S.Particles("g", 0, 0)
    ele.set_photon(pho)
    pos.set_photon(pho)
    pho.set_pair(ele, pos)
    sim = S.Simulation(ele, pos, pho, dt=2.7e-17, fields=gaussian_laser_pulse(150.0, 3e-6, 6e-6, direction=-1),
                       print_every=None, seed=seed, form=form)
    sim.start(steps)
    return [getattr(p, k).copy() for p in (ele, pos, pho) for k in ("x", "y", "ux", "uy")]


def _same(a, b):
    return all(x.shape == y.shape and np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_runs_one_after_another_and_on_threads(form):
    cuda_or_skip()
    sizes = [(40, 1), (3000, 2), (700, 3), (1, 4)]
    alone = [_run(n, seed, 70, form) for n, seed in sizes]
    for (n, seed), want in zip(sizes[::-1], alone[::-1]):
        assert _same(_run(n, seed, 70, form), want)
    got = [None] * len(sizes)

    def work(k):
        import torch
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(3):
                got[k] = _run(*sizes[k], 70, form)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, want in zip(got, alone):
        assert g is not None and _same(g, want)
