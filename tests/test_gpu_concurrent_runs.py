"""Two runs in three launches a step (more than 2^20 electrons) on two host
threads and streams: their launches compete for the SMs, so blocks of one
start late.  From no photons at all the tiles of a step's photon launch grow
most from step to step.  Each run equals the same run alone, bit for bit."""
import threading

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu

N, STEPS = (1 << 20) + 12345, 24


def _sim(seed, form):
    import sfparticles_b200 as S
    from sfparticles_b200.fields import gaussian_laser_pulse
    r = np.random.default_rng(seed)
    ele = S.Particles("e", -1, 1, N=N, props=(r.normal(0, 4e-6, N), r.normal(0, 1e-6, N), r.normal(0, 1e-6, N),
                                             np.full(N, 2000.0), np.zeros(N), np.zeros(N)))
    pos, pho = S.Particles("p", 1, 1), S.Particles("g", 0, 0)
    ele.set_photon(pho)
    pos.set_photon(pho)
    pho.set_pair(ele, pos)
    return S.Simulation(ele, pos, pho, dt=2.7e-17, fields=gaussian_laser_pulse(200.0, 3e-6, 6e-6, direction=-1),
                        print_every=None, seed=seed, form=form)


def _result(seed, form, steps=STEPS, at=None):
    sim = _sim(seed, form)
    sim.run_on_device(1)  # (the run is made: its steps start together with the other's)
    if at is not None:
        at.wait(60)
    sim.run_on_device(steps - 1)
    sim.finish()
    return [getattr(p, k) for p in sim.all_particles for k in ("x", "y", "z", "ux", "uy", "uz")]


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_two_runs_at_once_equal_each_alone(form):
    cuda_or_skip()
    import torch
    alone = [_result(seed, form) for seed in (1, 2)]
    assert all(a[12].size > 1 << 20 for a in alone)  # photons
    got, at = [None, None], threading.Barrier(2)

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[k] = _result(k + 1, form, at=at)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for have, want in zip(got, alone):
        assert have is not None and all(x.shape == y.shape and np.array_equal(x, y) for x, y in zip(have, want))
