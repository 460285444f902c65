"""The store of hot photons that a call of several steps keeps
(csrc/sfp_step.cuh, sfp_hot_*) against the full photon kernel, which calls of
one step run: the same particles, bit for bit, with photons that are mostly
too soft, all hot (the store overflows and is given up), hot photons born
during the call, converted ones, flags set by the caller, a field without a
bound, and several instances."""
import numpy as np
import pytest

from gpu_helpers import cuda_or_skip

pytestmark = pytest.mark.gpu

N = 2_200_000  # the photon group's long-tile population starts at 2^21
STEPS = 9


def _sim(form, energy, seed=5, n_e=3000, field="gauss", n_ph=N):
    import sfparticles_b200 as S
    from sfparticles_b200.fields import focused_gaussian_laser_pulse, gaussian_laser_pulse
    r = np.random.default_rng(seed)
    pos = lambda n: (r.normal(0, 4e-6, n), r.normal(0, 1e-6, n), r.normal(0, 1e-6, n))  # noqa: E731
    g = energy(r, n_ph)
    a = r.normal(0, 0.2, n_ph)
    pho = S.Particles("g", 0, 0, N=n_ph, props=(*pos(n_ph), g * np.cos(a), g * np.sin(a), np.zeros(n_ph)))
    ele = S.Particles("e", -1, 1, N=n_e, props=(*pos(n_e), np.full(n_e, 3000.0), np.zeros(n_e), np.zeros(n_e)))
    p = S.Particles("p", 1, 1)
    ele.set_photon(pho)
    p.set_photon(pho)
    pho.set_pair(ele, p)
    if field == "gauss":
        f = gaussian_laser_pulse(250.0, 3e-6, 6e-6, direction=-1)
    else:
        f = focused_gaussian_laser_pulse(250.0, 3e-6, 6e-6, direction=-1)
    return S.Simulation(ele, p, pho, dt=2.7e-17, fields=f, print_every=None, seed=seed, form=form)


def _soft(r, n):
    return np.where(r.random(n) < 0.1, r.uniform(100, 2500, n), r.uniform(2, 40, n))


def _hard(r, n):
    return r.uniform(800, 2500, n)


def _arrays(sim):
    return [getattr(p, k)[:p.N_buffered].copy() for p in sim.all_particles
            for k in ("x", "y", "z", "ux", "uy", "uz", "_to_be_pruned")]


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("energy,field", [(_soft, "gauss"), (_hard, "gauss"), (_soft, "focused")])
def test_store_equals_the_full_kernel(form, energy, field):
    cuda_or_skip()
    one, many = (_sim(form, energy, field=field, n_ph=N if field == "gauss" else N) for _ in range(2))
    for _ in range(STEPS):
        one.run_on_device(1)
    many.run_on_device(STEPS)
    a, b = _arrays(one), _arrays(many)
    assert [x.shape for x in a] == [x.shape for x in b]
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert len(a[7]) > 0 or field != "gauss"  # pairs were created
    one.finish()
    many.finish()


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_flags_set_between_calls_count(form):
    cuda_or_skip()
    import torch
    sims = [_sim(form, _soft) for _ in range(2)]
    for k, s in enumerate(sims):
        for step in range(2):
            if k == 0:
                for _ in range(5):
                    s.run_on_device(1)
            else:
                s.run_on_device(5)
            if step == 0:  # the caller prunes every third photon
                s.all_particles[2]._sync_positions()
                s.all_particles[2]._d("_to_be_pruned")[0:N:3] = 1
                torch.cuda.synchronize()
    a, b = (_arrays(s) for s in sims)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    for s in sims:
        s.finish()


def test_several_instances():
    cuda_or_skip()
    import sfparticles_b200 as S
    ens = [S.Ensemble([_sim("fp32", _soft, seed=s, n_ph=n) for s, n in ((1, 1_400_000), (2, 900_000), (3, 257))])
           for _ in range(2)]
    for _ in range(STEPS):
        ens[0].run_on_device(1)
    ens[1].run_on_device(STEPS)
    for u, v in zip(ens[0].sims, ens[1].sims):
        for x, y in zip(_arrays(u), _arrays(v)):
            assert np.array_equal(x, y)
    for e in ens:
        e.finish()


# entries: 5/8, 3/8 and 1/4 of 8e6 photons, with 1/8 to grow into, take 228, 138 and 93 MB in the float32 form;
# the store may take half of the free memory
@pytest.mark.parametrize("free_mb,kept", [(2000, True), (360, True), (230, True), (120, False)])
def test_store_where_memory_is_short(free_mb, kept):
    import ctypes

    import torch

    from sfparticles_b200 import _lib
    cuda_or_skip()
    one, many = (_sim("fp32", _soft, n_ph=8_000_000) for _ in range(2))
    for s in (one, many):
        s.run_on_device(2)
        s.reserve(STEPS)
    for _ in range(STEPS):
        one.run_on_device(1)
    _lib.call("sfp_release_cached")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.mem_get_info()[0] - free_mb * 1_000_000
    filler = torch.empty(room, dtype=torch.uint8, device="cuda")
    many.run_on_device(STEPS)
    n = ctypes.c_int64()
    _lib.call("sfp_run_hot_photons", many._run, ctypes.byref(n))
    del filler
    torch.cuda.empty_cache()
    assert (n.value > 0) == kept
    for x, y in zip(_arrays(one), _arrays(many)):
        assert np.array_equal(x, y)
    one.finish()
    many.finish()
