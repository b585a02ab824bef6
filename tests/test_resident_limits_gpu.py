"""Resident pair lists at their limits: more entries than the lists hold."""
import numpy as np
import pytest

from pacific_b200 import scenarios as S
from pacific_b200.abi import CUDA_ERROR, FP64, MIXED, PAIR_OVERFLOW, TIMEOUT, GrainsError

from helpers import make

pytestmark = pytest.mark.gpu


def failing_step(sim, n, dt):
    with pytest.raises(GrainsError) as err:
        sim.step(n, 0.0, dt)
        sim.synchronize()
    return err.value.code


def test_more_entries_than_32_bits_count(gpu_lib):
    """A million spheres piled into 12^3 cells, 580 a cell: some 2,900 partners
    each, more than 2^31 list entries in all.  The build has to find that they do
    not fit, whatever the sum is modulo 2^32."""
    rng = np.random.default_rng(1)
    n, r, edge = 1_000_000, 1.0e-3, 24.0e-3
    sc = S.small_box(8, seed=1)
    x = rng.uniform(0.0, edge, (n, 3))
    sc.particles = S._spheres(n, np.full(n, r), 2500.0, x, np.zeros((n, 3)), 1.0e-3)
    sc.obstacles = [[]]
    sc.domains = [dict(origin=(0.0,) * 3, size=(edge,) * 3, cell_size=2.0 * r, gravity=(0.0,) * 3)]
    hits = np.mean([np.sum(((x - x[k]) ** 2).sum(1) < (2.2 * r) ** 2) - 1 for k in range(50)])
    assert n * hits > 1.1 * 2.0 ** 31
    sim = make(gpu_lib, sc, MIXED)
    with pytest.raises(GrainsError) as err:
        sim.initialize_leapfrog(0.0, 1.0e-9)
    assert err.value.code & PAIR_OVERFLOW
    sim.reset_stats()
    code = failing_step(sim, 8, 1.0e-9)
    assert code & PAIR_OVERFLOW and not code & (TIMEOUT | CUDA_ERROR)
    sim.close()


def memories(sim):
    """Contact memory by (owner, other)"""
    m = sim.contact_memory(cap=64 * sim.n)
    values = np.concatenate([m["kdelta"], m["prev_normal"], m["spring_torque"]], axis=1)
    return {k: v for k, v in zip(zip(m["owner"].tolist(), m["other"].tolist()), values)}


def shrinking_lattice(precision):
    """A cubic lattice of overlapping spheres on the floor that shrinks by 1e-4 a
    step: an inner sphere has 26 neighbours in touch (the shells up to sqrt(3)
    spacings), and 6 more from the step on in which two spacings are less than a
    diameter."""
    side, r, dt = 20, 0.8e-3, 1.0e-7
    n, a = side ** 3, 1.00085 * r
    sc = S.small_box(n, seed=1, velocity_sigma=0.0)
    k = np.arange(n)
    ijk = np.stack([k % side, k // side % side, k // side ** 2], 1)
    x = a * ijk + np.random.default_rng(3).uniform(-1.0e-10, 1.0e-10, (n, 3))
    sc.particles = S._spheres(n, np.full(n, r), 2500.0, x + [5.0e-3, 5.0e-3, r - 1.0e-6],
                              -1.0e-4 / dt * (x - [9.0 * a, 10.0 * a, 0.0]), 0.5e-3)
    sc.laws = [[(p, q, S.HOOKE_MEMORY, [1.0e2, 0.9, -1.0, 0.5, 0.8e2, 0.0, 0.0, 0.0]) for p, q, _, _ in sc.laws[0]]]
    sc.domains[0]["gravity"] = (0.0, 0.0, 0.0)
    sc.dt = dt
    return sc


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_a_run_stands_still_where_its_lists_do_not_fit(gpu_lib, precision):
    """The lattice outgrows a list capacity of 28 in the middle of a run: the call
    ends in PAIR_OVERFLOW with the particles and the contact memory (of pairs and
    of the floor) as after the last step whose lists fitted, the state that the
    launched pipeline has after that step."""
    sc = shrinking_lattice(precision)
    sim = make(gpu_lib, sc, precision)
    sim.set_tuning(list_capacity=28)
    assert sim.launches_per_step() == 3
    sim.initialize_leapfrog(0.0, sc.dt)
    assert failing_step(sim, 25, sc.dt) == PAIR_OVERFLOW
    sim.reset_stats()
    at, memory = sim.download()["position"], memories(sim)
    sim.close()
    ref = make(gpu_lib, sc, precision)
    ref.set_tuning(list_capacity=52)  # more than twice the memory's 24: the launched pipeline
    assert ref.launches_per_step() > 3
    ref.initialize_leapfrog(0.0, sc.dt)
    steps, t = 0, 0.0
    while steps < 25:
        t = ref.step(1, t, sc.dt)
        steps += 1
        if np.array_equal(ref.download()["position"], at):
            break
    assert 4 < steps < 24
    want = memories(ref)
    ref.close()
    # the force evaluation that ended the call listed at most 28 contacts a sphere
    assert len(memory) > 0.8 * len(want) and set(memory) <= set(want)
    assert sum(other < 0 for _, other in memory) == sum(other < 0 for _, other in want) == 400
    for k in memory:
        assert np.array_equal(memory[k], want[k]), k


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_contacts_that_just_fit(gpu_lib, precision):
    """Every inner sphere of a lattice touches 32 others, the list capacity, and
    24 more miss it by 2e-5 of a diameter: too many for any skin, yet the contacts
    alone fit, so the call is accepted and its results are the launched
    pipeline's."""
    side, a = 20, 0.7e-3
    n, r = side ** 3, 0.5 * np.sqrt(5.0) * a * (1.0 - 2.0e-5)
    sc = shrinking_lattice(precision)
    k = np.arange(n)
    x = a * np.stack([k % side, k // side % side, k // side ** 2], 1) + 5.0e-3
    x += np.random.default_rng(4).uniform(-1.0e-10, 1.0e-10, (n, 3))
    sc.particles = S._spheres(n, np.full(n, r), 2500.0, x, np.zeros((n, 3)), 0.5e-3)
    sc.domains[0]["cell_size"] = 2.0 * r
    sc.obstacles = [[]]
    out = []
    for capacity in (32, 52):  # resident lists, the launched pipeline
        sim = make(gpu_lib, sc, precision)
        sim.set_tuning(list_capacity=capacity)
        assert (sim.launches_per_step() == 3) == (capacity == 32)
        sim.initialize_leapfrog(0.0, 1.0e-8)
        sim.step(9, 0.0, 1.0e-8)
        sim.synchronize()
        out.append((sim.download(), memories(sim), sim.stats()))
        sim.close()
    (a0, m0, s0), (a1, m1, s1) = out
    assert a0["coordination"].max() == 32 and s0["status"] == s1["status"] == 0
    for key in a0:
        assert np.array_equal(a0[key], a1[key]), key
    assert set(m0) == set(m1) and all(np.array_equal(m0[q], m1[q]) for q in m0)


@pytest.mark.parametrize("polls,skip", [(20000, 0), (20000, 3), (1, -1)])
def test_a_build_whose_waits_run_out(gpu_lib, polls, skip):
    """A block that leaves a rebuild before its first barrier, or waits of one
    poll: TIMEOUT comes back, the particles stand where the last step with
    complete lists left them, and the context runs on after a new upload."""
    sc = S.small_box(1000, seed=3, velocity_sigma=1.0, radius_range=(0.9, 1.1), spacing=2.3, jitter=0.02)
    sc.dt = 2.0e-6
    sim, ref = make(gpu_lib, sc, FP64), make(gpu_lib, sc, FP64)
    sim.set_barrier_test(polls=polls, skip_block=skip)
    sim.initialize_leapfrog(0.0, sc.dt)
    assert failing_step(sim, 400, sc.dt) & TIMEOUT
    sim.reset_stats()
    at = sim.download()["position"]
    ref.set_tuning(list_capacity=20)  # the launched pipeline
    ref.initialize_leapfrog(0.0, sc.dt)
    steps, t, found = 0, 0.0, False
    while steps < 399 and not found:
        t = ref.step(1, t, sc.dt)
        steps += 1
        found = np.array_equal(ref.download()["position"], at)
    # the first build of the run gives up, or one that particles have asked for
    assert found and (steps == 1 if skip < 0 else steps > 1)
    sim.set_barrier_test()
    sim.upload(sc.particles)
    sim.initialize_leapfrog(0.0, sc.dt)
    sim.step(steps + 20, 0.0, sc.dt)
    sim.synchronize()
    ref.step(20, t, sc.dt)
    a, b = sim.download(), ref.download()
    for key in a:
        assert np.array_equal(a[key], b[key]), key
    sim.close()
    ref.close()


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


class Filled:
    """Device memory taken until about `left` bytes are free"""

    def __init__(self, left):
        import torch
        torch.cuda.empty_cache()
        self.block = torch.empty(max(0, free_bytes() - left), dtype=torch.uint8, device="cuda")

    def release(self):
        import torch
        del self.block
        torch.cuda.empty_cache()


def sized(gpu_lib, sc):
    sim = make(gpu_lib, sc, FP64)
    sim.set_tuning(list_capacity=28)
    return sim


def run_out(sim, sc):
    sim.initialize_leapfrog(0.0, sc.dt)
    sim.step(20, 0.0, sc.dt)
    sim.synchronize()
    return sim.download()


def large_box():
    sc = S.small_box(60000, seed=9, velocity_sigma=0.2, spacing=2.03)
    sc.dt = 2.0e-6
    return sc


def test_without_room_for_the_lists_steps_are_launched(gpu_lib):
    """Device memory that holds the context but not the lists' buffer: the upload
    succeeds, the steps are launched, the bits are the same; an upload that finds
    room brings the lists back."""
    sc = large_box()
    free = free_bytes()
    sim = sized(gpu_lib, sc)
    assert sim.launches_per_step() == 3
    with_lists = free - free_bytes()
    want = run_out(sim, sc)
    sim.close()
    free = free_bytes()
    sim = sized(gpu_lib, S.small_box(60000, seed=9, spacing=2.03, radius_range=(0.2, 1.0)))  # radii apart: no lists
    assert sim.launches_per_step() > 3
    lists = with_lists - (free - free_bytes())
    assert lists > (64 << 20)
    # room for less than the lists' buffer
    full = Filled(lists // 2)
    try:
        sim.upload(sc.particles)
        assert sim.launches_per_step() > 3
        got = run_out(sim, sc)
    finally:
        full.release()
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    sim.upload(sc.particles)
    assert sim.launches_per_step() == 3
    got = run_out(sim, sc)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    sim.close()


def test_lists_give_their_room_to_other_allocations(gpu_lib):
    """An adjoint that fits only in the room of the resident lists: it gets it,
    and the context runs on without the lists, the same bits."""
    from pacific_b200.abi import Adjoint
    sc = large_box()
    sim = sized(gpu_lib, sc)
    want = run_out(sim, sc)
    sim.upload(sc.particles)
    none = np.zeros((sc.n, 3))

    def gradient():
        adj = Adjoint(sim, checkpoint_every=2)
        out = adj.forward(2, sc.dt)
        adj.backward(none, none, none)
        need = free - free_bytes()
        adj.close()
        return out, need
    free = 0
    gradient()  # the first one loads its kernels
    free = free_bytes()
    final, need = gradient()
    assert sim.launches_per_step() == 3 and need > (128 << 20)
    full = Filled(need - (24 << 20))
    try:
        again, _ = gradient()
        assert sim.launches_per_step() > 3
        got = run_out(sim, sc)
    finally:
        full.release()
    for k in final:
        assert np.array_equal(final[k], again[k]), k
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    sim.close()


def test_an_adjoint_whose_checkpoints_do_not_fit(gpu_lib):
    """A run too long for the device memory fails; a shorter one after it works as
    before, and no backward run uses what the failed one gave back."""
    from pacific_b200.abi import Adjoint
    sc = S.small_box(1000, seed=4, velocity_sigma=0.1)
    sim = make(gpu_lib, sc, FP64)
    adj = Adjoint(sim, checkpoint_every=1)
    one = np.ones((sc.n, 3))

    def both():
        return adj.forward(6, 1.0e-6), adj.backward(one, one, one)
    first = both()
    with pytest.raises(GrainsError):
        adj.forward(10_000_000, 1.0e-6)
    with pytest.raises(GrainsError):
        adj.backward(one, one, one)
    second = both()
    for a, b in zip(first, second):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
    adj.close()
    sim.close()


def test_contexts_of_several_threads(gpu_lib):
    """Four contexts step at the same time, each in a thread and on a stream of
    its own, with lists rebuilt every few steps by launches that fill the chip: the
    bits of each context alone, and no wait that runs out."""
    import threading
    sc = S.small_box(60000, seed=12, velocity_sigma=2.0, spacing=2.2)
    sc.dt = 2.0e-6
    sims = [make(gpu_lib, sc, MIXED) for _ in range(5)]

    def run(sim):
        sim.initialize_leapfrog(0.0, sc.dt)
        t = 0.0
        for _ in range(5):
            t = sim.step(60, t, sc.dt)
        sim.synchronize()
        out.append(sim.download())
    out = []
    run(sims[0])
    threads = [threading.Thread(target=run, args=(sim,)) for sim in sims[1:]]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert len(out) == 5 and sims[0].launches_per_step() == 3
    for d in out[1:]:
        for k in d:
            assert np.array_equal(d[k], out[0][k]), k
    for sim in sims:
        assert sim.stats()["status"] == 0
        sim.close()
