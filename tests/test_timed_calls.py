"""time_step_kernel refuses calls of no steps, which would never end (host check, before any device is asked for)."""
import numpy as np
import pytest

import sfparticles_b200 as S
from sfparticles_b200.fields import gaussian_laser_pulse


def _sim():
    e = S.Particles("e", -1, 1, N=3, props=tuple(np.zeros(3) for _ in range(6)))
    return S.Simulation(e, dt=1e-17, fields=gaussian_laser_pulse(1.0, 2e-6, 5e-6), print_every=None, seed=1)


@pytest.mark.parametrize("per_call", [0, -1])
@pytest.mark.parametrize("make", [_sim, lambda: S.Ensemble([_sim(), _sim()])])
def test_calls_of_no_steps(make, per_call):
    with pytest.raises(ValueError, match="per_call"):
        make().time_step_kernel(4, per_call=per_call)
