"""The per-op engine draws events through _photon_event and _pair_event where
a program replaces them: on a subclass, on an object, or on the class."""
import numpy as np
import pytest

import sfparticles_b200 as S
from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu

N, STEPS = 3000, 12


class Silent(S.Particles):
    """Emits nothing."""
    calls = 0

    def _photon_event(self, dt):
        type(self).calls += 1
        event, delta = super()._photon_event(dt)
        assert event.shape == delta.shape == (self.buffer_size,)
        self._d("event").zero_()
        self._touch()
        return self.event, self.photon_delta


class Sterile(S.Particles):
    """Creates no pair."""
    calls = 0

    def _pair_event(self, dt):
        type(self).calls += 1
        event, delta = super()._pair_event(dt)
        self._d("event").zero_()
        self._touch()
        return self.event, self.pair_delta


def _run(electrons=S.Particles, photons=S.Particles, change=None):
    from sfparticles_b200.fields import gaussian_laser_pulse
    r = np.random.default_rng(3)
    ele = electrons("e", -1, 1, N=N, props=(r.normal(0, 2e-6, N), r.normal(0, 1e-6, N), r.normal(0, 1e-6, N),
                                           np.full(N, 3000.0), np.zeros(N), np.zeros(N)))
    pos, pho = S.Particles("p", 1, 1), photons("g", 0, 0)
    ele.set_photon(pho)
    pos.set_photon(pho)
    pho.set_pair(ele, pos)
    if change is not None:
        change(ele, pho)
    sim = S.Simulation(ele, pos, pho, dt=2.7e-17, fields=gaussian_laser_pulse(400.0, 3e-6, 6e-6, direction=-1),
                       print_every=None, seed=9, engine="ops")
    sim.start(STEPS)
    return ele.N_buffered, pos.N_buffered, pho.N_buffered


def test_replaced_event_methods_are_called(monkeypatch):
    cuda_or_skip()
    ele, pos, pho = _run()
    assert pho > 0
    Silent.calls = Sterile.calls = 0
    assert _run(electrons=Silent) == (N, 0, 0) and Silent.calls == STEPS
    no_pairs = _run(photons=Sterile)
    assert no_pairs[:2] == (N, 0) and no_pairs[2] > 0 and Sterile.calls == STEPS
    seen = []

    def on_object(e, g):
        e._photon_event = lambda dt: (seen.append("object"), S.Particles._photon_event(e, dt))[1]

    assert _run(change=on_object) == (ele, pos, pho) and seen == ["object"] * STEPS
    own = S.Particles._pair_event
    monkeypatch.setattr(S.Particles, "_pair_event", lambda self, dt: (seen.append("class"), own(self, dt))[1])
    assert _run() == (ele, pos, pho) and seen.count("class") == STEPS
