"""The life of a run's store of hot photons: whether a call kept one, a store
that newborn photons fill in the middle of a call, a step that waits for room
while the store is live, memory that the species need more, memory that comes
free again, and fields whose photons are all hot.  Whatever becomes of the
store, the particles are those of single-step calls, bit for bit."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda_or_skip
from test_gpu_hot_photons import N, _arrays, _hard, _sim, _soft

pytestmark = pytest.mark.gpu


def _kept(sim):
    from sfparticles_b200 import _lib
    n = ctypes.c_int64(-1)
    _lib.call("sfp_run_hot_photons", sim._run, ctypes.byref(n))
    return n.value


def _launches(sim):
    from sfparticles_b200 import _lib
    n = ctypes.c_int64(-1)
    _lib.call("sfp_run_launches", sim._run, ctypes.byref(n))
    return n.value


def _same(a, b):
    a, b = _arrays(a), _arrays(b)
    assert [x.shape for x in a] == [x.shape for x in b]
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def _room(sim, slots):
    """Free slots for every species, without the halts of a run that begins with full buffers."""
    for p in sim.all_particles:
        p._to_gpu()
        p._resize(p.N_buffered + slots)


class _LeaveFree:
    """The device's memory taken but for `free` bytes."""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        import torch
        from sfparticles_b200 import _lib
        _lib.call("sfp_release_cached")
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - self.free, dtype=torch.uint8, device="cuda")

    def __exit__(self, *a):
        import torch
        self.block = None
        torch.cuda.empty_cache()


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("energy,field,kept", [(_soft, "gauss", True), (_hard, "gauss", False),
                                               (_soft, "focused", False)])
def test_a_store_that_was_given_up_is_reported_as_none(form, energy, field, kept):
    cuda_or_skip()
    sim = _sim(form, energy, field=field)
    _room(sim, 400_000)
    sim.run_on_device(6)
    n = _kept(sim)
    assert (n > 0) == kept
    if kept:  # one photon in ten is hot, and what the electrons emitted since
        assert 0.09 * N < n < 0.2 * N
    sim.finish()


HOT = 1_300_000  # the store has room for 5/8 N + 65536 = 1440536


def _nearly_full(r, n):
    return np.where(np.arange(n) < HOT, r.uniform(100, 2500, n), r.uniform(2, 40, n))


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_newborn_photons_fill_the_store_within_a_call(form):
    cuda_or_skip()
    steps = 40
    few, one, many = (_sim(form, _nearly_full, n_e=300_000) for _ in range(3))
    for s in (few, one, many):
        _room(s, 3_000_000)
    few.run_on_device(4)
    assert HOT <= _kept(few) <= 1_440_536  # a short call keeps it
    few.finish()
    for _ in range(steps):
        one.run_on_device(1)
    many.run_on_device(steps)
    assert _kept(many) == 0  # a long one does not
    _same(one, many)
    for s in (one, many):
        s.finish()


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("give_back", [False, True])
def test_a_step_waits_for_room_while_the_store_is_live(form, give_back, monkeypatch):
    cuda_or_skip()
    from sfparticles_b200 import _lib, simulation
    one, many = (_sim(form, _soft, n_e=100_000) for _ in range(2))
    _room(one, 3_000_000)
    _room(many, 30_000)
    waits, resolve = [], simulation.resolve_pending

    def resolved(run, species, update):
        waits.append(_kept(many))
        if give_back:  # the store's memory goes before the children are written
            _lib.call("sfp_release_stores", None)
            assert _kept(many) == 0
        resolve(run, species, update)

    for _ in range(24):
        one.run_on_device(1)
    monkeypatch.setattr(simulation, "resolve_pending", resolved)
    many.run_on_device(24)
    assert waits and waits[0] > 0  # steps ran through the store before the wait
    _same(one, many)
    for s in (one, many):
        s.finish()


@pytest.mark.parametrize("together", [False, True])
def test_a_growth_that_fits_only_without_the_store(together, monkeypatch):
    cuda_or_skip()
    from sfparticles_b200 import particles
    if together:
        monkeypatch.setattr(particles, "GROW_TOGETHER", 1 << 30)
    one, many = (_sim("fp32", _soft, n_ph=8_000_000) for _ in range(2))
    for s in (one, many):
        s.run_on_device(2)
        s.reserve(20)
    for _ in range(12):
        one.run_on_device(1)
    many.run_on_device(6)
    assert _kept(many) > 0  # about 228 MB
    pho = many.all_particles[2]
    # 65 bytes a slot; the store holds about 228 MB
    if together:  # the whole species anew
        slots = pho.buffer_size
        need = slots * 65
    else:  # what it grows by, and one array beside it
        slots = pho.buffer_size + 4_000_000
        need = (slots - pho.buffer_size) * 65 + slots * 8
    with _LeaveFree(need - 100_000_000):
        pho._resize(slots)
        many._update_run(many._run)
    many.run_on_device(6)
    _same(one, many)
    for s in (one, many):
        s.finish()


def test_a_spectrum_that_fits_only_without_the_store():
    import torch
    from sfparticles_b200.diagnostics import photon_spectrum_device
    cuda_or_skip()
    sim = _sim("fp32", _soft, n_ph=8_000_000)
    sim.run_on_device(2)
    sim.reserve(20)
    sim.run_on_device(6)
    assert _kept(sim) > 0  # about 228 MB
    pho = sim.all_particles[2]
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    want = photon_spectrum_device(pho)
    need = torch.cuda.max_memory_allocated() - before
    with _LeaveFree(need - 100_000_000):
        assert np.array_equal(photon_spectrum_device(pho), want)
    assert want.sum() > 0 and _kept(sim) == 0
    sim.finish()


def test_a_store_is_kept_again_once_there_is_memory():
    cuda_or_skip()
    sim = _sim("fp32", _soft, n_ph=8_000_000)
    sim.run_on_device(2)
    sim.reserve(30)
    with _LeaveFree(120_000_000):  # half of it is less than a store of 1/4 takes (93 MB)
        sim.run_on_device(5)
        assert _kept(sim) == 0
    sim.run_on_device(5)
    assert _kept(sim) > 0
    sim.finish()


def test_a_field_without_a_bound_takes_no_store():
    import torch
    cuda_or_skip()
    sim = _sim("fp32", _soft, field="focused")
    _room(sim, 400_000)
    sim.run_on_device(1)
    torch.cuda.synchronize()
    free, before = torch.cuda.mem_get_info()[0], _launches(sim)
    sim.run_on_device(6)
    assert torch.cuda.mem_get_info()[0] == free
    sim.run_on_device(6)
    # each call: the first step's bookkeeping, then three kernels a step; once in the run, the question for the bound
    assert _launches(sim) - before <= 2 * (1 + 3 * 6) + 1
    sim.finish()


def test_steps_beside_a_capture_on_another_thread():
    """A thread captures a graph in the global mode, in which no thread may make an unsafe call, while another steps
    a run that takes its store's memory: the capture stays whole."""
    import threading

    import torch
    cuda_or_skip()
    one, many = (_sim("fp32", _soft) for _ in range(2))
    for s in (one, many):
        _room(s, 400_000)
    for _ in range(7):
        one.run_on_device(1)
    many.run_on_device(1)
    from sfparticles_b200 import _lib
    x = torch.arange(1000, dtype=torch.float32, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    began, stepped, fault = threading.Event(), threading.Event(), []

    def capture():
        try:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
                y.copy_(x)
                began.set()
                stepped.wait(60)
                y.mul_(2)
            g.replay()
            torch.cuda.synchronize()
        except Exception as e:
            fault.append(e)
            began.set()

    t = threading.Thread(target=capture)
    t.start()
    began.wait(60)
    rc = _lib.load().sfp_run_steps(many._run, 6, 0, ctypes.c_void_p(0))
    stepped.set()
    t.join()
    assert rc == 0 and not fault
    assert torch.equal(y, 2 * x)
    many._pos_dirty = True
    nbuf, st = (ctypes.c_int64 * 3)(), _lib.RunState()
    many._sync_state(many._run, st, nbuf)
    assert not st.halted and _kept(many) > 0
    _same(one, many)
    for s in (one, many):
        s.finish()
