"""The kernel that runs several steps of a small population in one launch
(csrc/sfp_step.cuh, sfp_steps_body) against the step's separate launches
(sfp_run_steps_timed takes those): the same counts, flags and particles, at
populations below and above one tile per warp, across a stop for room, with
spin, both event methods and both samplers, for one instance and several; and
its barrier's time limit.

Tolerance 1e-9 of each array's largest value: the two round alike but for the
product of a child's momentum and its share (2^-53 relative), which 60
steps of a fifth of a radian's rotation each amplify by far less than 1e6."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu


def _species(n, seed, od, spin):
    import sfparticles_b200 as S
    from sfparticles_b200 import qed
    r = np.random.default_rng(seed)
    xyz = (r.normal(0, 3e-6, n), r.normal(0, 1e-6, n), r.normal(0, 1e-6, n))
    u = (np.full(n, 3000.0), r.normal(0, 1, n), r.normal(0, 1, n))
    qed.set_method("od" if od else "rs")
    try:
        if spin:
            ele = S.SpinParticles("e", -1, 1, N=n, props=(*xyz, *u, np.zeros(n), np.zeros(n), np.ones(n)))
        else:
            ele = S.Particles("e", -1, 1, N=n, props=(*xyz, *u))
        pos, pho = S.Particles("p", 1, 1), S.Particles("g", 0, 0)
        ele.set_photon(pho)
        pos.set_photon(pho)
        pho.set_pair(ele, pos)
    finally:
        qed.set_method("rs")
    return ele, pos, pho


def _sim(n, seed=3, form="fp64", od=False, spin=False, sampler="table", a0=400.0):
    import sfparticles_b200 as S
    from sfparticles_b200.fields import gaussian_laser_pulse
    f = gaussian_laser_pulse(a0, 3e-6, 6e-6, direction=-1)
    return S.Simulation(*_species(n, seed, od, spin), dt=2.7e-17, fields=f, print_every=None, seed=seed, form=form,
                        sampler=sampler)


def _arrays(sim):
    return [getattr(p, k)[:p.N_buffered].copy() for p in sim.all_particles
            for k in p.attrs if k in ("x", "y", "z", "ux", "uy", "uz", "sx", "sy", "sz", "tau", "_to_be_pruned")]


def _check(a, b):
    for x, y in zip(a, b):
        assert x.shape == y.shape
        if x.dtype == bool:
            assert np.array_equal(x, y)
        elif x.size:
            assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(x))


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("n,od,spin,sampler", [(1, False, False, "table"), (33, False, True, "table"),
                                               (20000, False, False, "table"), (150000, False, False, "table"),
                                               (500, True, True, "table"), (30000, True, False, "mlp")])
def test_one_launch_equals_separate_launches(form, n, od, spin, sampler):
    cuda_or_skip()
    steps = 60 if n < 100000 else 12
    one, sep = (_sim(n, form=form, od=od, spin=spin, sampler=sampler) for _ in range(2))
    before = one.kernel_launches
    one.run_on_device(steps)
    assert one.kernel_launches - before < 2 * steps  # not three launches per step, waits for room included
    sep.reserve(0)
    while sep.step < steps:
        sep.time_step_kernel(1)
    _check(_arrays(one), _arrays(sep))
    assert one.particle_steps == sep.particle_steps and one.t == sep.t
    one.finish()
    sep.finish()


def test_ensemble_of_small_runs():
    cuda_or_skip()
    import sfparticles_b200 as S
    ens = [S.Ensemble([_sim(n, seed=k, form="fp32", a0=a0) for k, (n, a0) in enumerate(((1, 300.0), (70, 500.0), (5000, 100.0)))])
           for _ in range(2)]
    ens[0].run_on_device(40)
    while ens[1].step < 40:
        ens[1].time_step_kernel(1)
    for u, v in zip(ens[0].sims, ens[1].sims):
        _check(_arrays(u), _arrays(v))
    for e in ens:
        e.finish()


def test_barrier_wait_runs_out_and_the_context_stays_usable():
    cuda_or_skip()
    from sfparticles_b200 import _lib
    sim = _sim(100)
    sim._begin()
    _lib.call("sfp_run_barrier_withheld", sim._run, None)
    st, nb = _lib.RunState(), (ctypes.c_int64 * 3)()
    _lib.call("sfp_run_read_state", sim._run, ctypes.byref(st), nb, None)
    assert st.error == 4 and st.step == 0
    with pytest.raises(_lib.SFPError, match="barrier"):
        sim.run_on_device(1)
    sim._pos_dirty = False
    sim._end()
    good = _sim(100)
    good.start(20)
    assert good.step == 20
