"""Steps on resident pair lists (spheres among static obstacles) against the
launched pipeline, which lists the contacts anew in every step: the same bits in
every field, the same contact memory, counts and status.  A list capacity below
24, or above twice the memory capacity (24), keeps a context on the launched
pipeline and changes nothing else."""
import numpy as np
import pytest

from pacific_b200 import scenarios as S
from pacific_b200.abi import (CONTACT_ERROR, CONTACT_HANDLED, FP64, HERTZ, HERTZ_MEMORY, HISTORY_FULL, HOOKE,
                              HOOKE_MEMORY, MIXED, MOTION_ERROR, OUT_OF_GRID, GrainsError)

from helpers import make

pytestmark = pytest.mark.gpu

TUNING = dict(cell_factor=1.0, contacts_block=256, forces_block=128, gather_every=16)
LAWS = {
    "memory": None,  # the scenario's HookeMemory
    "rolling": (HOOKE_MEMORY, [1.0e5, 0.9, -1.0, 0.5, 0.8e5, 0.05, 0.1, 0.0]),
    "none": (HOOKE, [1.0e5, 0.9, -1.0, 0.5, 1.0e-3]),
    "hertz": (HERTZ_MEMORY, [2.0e8, 0.9, 0.5, 6.0e7, 0.05, 0.1, 0.0]),
}


def with_law(sc, law):
    if LAWS[law] is not None:
        sc.laws = [[(a, b, *LAWS[law]) for a, b, _, _ in laws] for laws in sc.laws]
    return sc


def run(lib, sc, precision, steps, capacity, resident, basis=False, factor=1.0):
    if basis:
        sc.particles["basis"] = S.quaternion_basis(sc.particles["quaternion"])
    sim = make(lib, sc, precision)
    sim.set_tuning(**{**TUNING, "cell_factor": factor}, list_capacity=capacity)
    assert (sim.launches_per_step() == 3) == resident
    sim.initialize_leapfrog(0.0, sc.dt)
    out, t = [], 0.0
    for n in steps:
        t = sim.step(n, t, sc.dt)
        d, m = sim.download(), sim.contact_memory()
        order = np.lexsort((m["other"], m["owner"], m["system"]))
        out.append({**d, **{"memory " + k: v[order] for k, v in m.items()}})
    sim.synchronize()
    st = sim.stats()
    sim.close()
    return out, st


def check(lib, sc, precision, steps, capacities=(32, 20), **kw):
    a, sa = run(lib, sc, precision, steps, capacities[0], True, **kw)
    b, sb = run(lib, sc, precision, steps, capacities[1], False, **kw)
    for x, y in zip(a, b):
        for k in x:
            assert np.array_equal(x[k], y[k]), k
    for k in sa:
        if k in ("overlap_sum", "overlap_mean"):  # summed by atomics, in any order
            assert abs(sa[k] - sb[k]) <= 1e-12 * abs(sb[k])
        else:
            assert sa[k] == sb[k], k
    return a, sa


# 7 steps: the shortest resident run; 8: an odd number of middle steps; 40: graphs and a remainder
@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("law", list(LAWS))
@pytest.mark.parametrize("n", [1, 2, 33, 257, 1000])
def test_same_bits_as_the_launched_pipeline(gpu_lib, n, law, precision):
    sc = with_law(S.small_box(n, seed=n, velocity_sigma=0.3, radius_range=(0.95, 1.05), spacing=2.07), law)
    sc.dt = 5.0e-6
    check(gpu_lib, sc, precision, (7, 8, 40))


def test_lists_are_rebuilt_and_regathered(gpu_lib):
    """Fast spheres cross cells and half the skin many times; a run longer than
    the gather period."""
    sc = S.small_box(700, seed=3, velocity_sigma=1.5, radius_range=(0.7, 1.3), spacing=2.7, jitter=0.05)
    sc.dt = 2.0e-6
    _, st = check(gpu_lib, sc, MIXED, (1100, 530))
    assert st["n_contacts"] > 0


@pytest.mark.parametrize("factor", [1.0, 1.5])
def test_bases_systems_and_wide_cells(gpu_lib, factor):
    """Several systems with their own laws, given bases, cells wider than the
    largest diameter."""
    sc = S.ensemble_512(n_systems=5, n_min=40, n_max=900)
    rng = np.random.default_rng(1)
    sc.particles["velocity"] = rng.normal(0.0, 0.5, sc.particles["velocity"].shape)
    sc.particles["omega"] = rng.normal(0.0, 20.0, sc.particles["omega"].shape)
    check(gpu_lib, sc, FP64, (200,), basis=True, factor=factor)


def test_crowded_lists_take_a_thinner_skin(gpu_lib):
    """A lattice so tight that every inner sphere touches 32 others (the list
    capacity) and has 56 within the skin: the build halves the skin until the
    lists hold the entries."""
    rng = np.random.default_rng(2)
    n, side, spacing = 1000, 10, 0.777e-3
    sc = S.small_box(n, seed=1, velocity_sigma=0.01)
    sc.laws = [[(a, b, HOOKE_MEMORY, [1.0e2, 0.9, -1.0, 0.5, 0.8e2, 0.0, 0.0, 0.0]) for a, b, _, _ in sc.laws[0]]]
    k = np.arange(n)
    sc.particles["radius"][:] = 0.79e-3
    sc.particles["crust"][:] = 0.45e-3  # overlaps of 0.8 mm are no ContactError
    sc.particles["position"] = 2.5e-3 + spacing * np.stack([k % side, k // side % side, k // side ** 2], 1)
    sc.particles["position"] += rng.uniform(-0.5e-6, 0.5e-6, (n, 3))
    sc.obstacles = [[]]
    sc.domains[0]["gravity"] = (0.0, 0.0, 0.0)
    sc.dt = 1.0e-7
    out, _ = check(gpu_lib, sc, FP64, (12,), capacities=(32, 52))
    assert out[0]["coordination"].max() == 32


def test_what_does_not_run_on_resident_lists(gpu_lib):
    """Convex bodies, moving obstacles and radii far apart stay on the launched
    pipeline."""
    far = S.small_box(30, seed=1, radius_range=(0.2, 1.0))
    for sc in (S.convex_box(27, seed=1), S.pressed_box(27), far):
        sim = make(gpu_lib, sc, FP64)
        assert sim.launches_per_step() > 3
        sim.initialize_leapfrog(0.0, sc.dt)
        sim.step(9, 0.0, sc.dt)
        sim.synchronize()
        sim.close()


def moving_lattice(n, share, contacts, overlap=1.0e-3):
    """Spheres on a cubic lattice, each in touch with its x neighbours (or none),
    that move together by `share` of a radius per step."""
    r, dt, side = 1.0e-3, 1.0e-6, int(np.ceil(n ** (1.0 / 3.0)))
    k = np.arange(n)
    gap = np.array([(2.0 - overlap) * r if contacts else 2.6 * r, 2.6 * r, 2.6 * r])
    x = 5.0e-3 + gap * np.stack([k % side, k // side % side, k // side ** 2], 1)
    sc = S.small_box(8, seed=1)
    v = np.tile([share * r / dt, 0.0, 0.0], (n, 1))
    v += np.random.default_rng(5).normal(0.0, 1.0e-5 * r / dt, (n, 3))
    sc.particles = S._spheres(n, np.full(n, r), 2500.0, x, v, 0.1 * r)
    sc.obstacles = [[]]
    sc.domains = [dict(origin=(0.0,) * 3, size=tuple(x.max(0) + 10.0e-3), cell_size=2.0 * r, gravity=(0.0,) * 3)]
    sc.dt = dt
    return sc


@pytest.mark.parametrize("n,contacts,share,resident", [
    (1000, False, 0.045, True), (1000, False, 0.055, False), (1000, True, 0.045, True), (1000, True, 0.055, False),
    (65000, False, 0.018, True), (65000, False, 0.021, False),
    (110000, False, 0.013, True), (110000, False, 0.0145, False), (110000, True, 0.03, True),
    (110000, True, 0.036, False)])
def test_fast_spheres_take_the_launched_pipeline(gpu_lib, n, contacts, share, resident):
    """Both sides of the rule on the steps between two builds, and the same bits
    on both pipelines; a call that starts slowly goes
    back to the lists."""
    sc = moving_lattice(n, share, contacts)
    out = []
    for capacity in (32, 20):
        sim = make(gpu_lib, sc, MIXED)
        sim.set_tuning(list_capacity=capacity)
        sim.initialize_leapfrog(0.0, sc.dt)
        t, phases = sim.profile_kernels(12, 0.0, sc.dt)
        launches = {k: v[1] for k, v in phases.items()}
        assert (launches["contacts"] == 1) == (resident and capacity == 32)
        sim.step(9, t, sc.dt)
        sim.synchronize()
        out.append(sim.download())
        sim.update({**sc.particles, "velocity": 0.1 * sc.particles["velocity"]})
        sim.initialize_leapfrog(0.0, sc.dt)
        _, phases = sim.profile_kernels(12, 0.0, sc.dt)
        assert (phases["contacts"][1] == 1) == (capacity == 32)
        sim.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("steps", [7, 520])
def test_profiled_steps_are_those_of_a_step_call(gpu_lib, steps):
    """The profile runs the schedule of grains_gpu_step, the permutation after 504
    steps included, and counts its launches."""
    sc = S.small_box(300, seed=6, velocity_sigma=0.5, spacing=2.2)
    sc.dt = 2.0e-6
    out = []
    for profiled in (True, False):
        sim = make(gpu_lib, sc, MIXED)
        sim.initialize_leapfrog(0.0, sc.dt)
        if profiled:
            _, phases = sim.profile_kernels(steps, 0.0, sc.dt)
        else:
            sim.step(steps, 0.0, sc.dt)
            sim.synchronize()
        out.append((sim.download(), sim.stats()))
        sim.close()
    runs = 2 if steps > 504 else 1
    # rebuilds, starts and ends, five per permutation, the sort of the last step
    assert phases["sort_gather"][1] == steps - 1 + 2 * runs + 5 * (runs - 1) + 3
    assert phases["pairs"][1] == phases["sums_kick"][1] == steps
    for k in out[0][0]:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    assert out[0][1]["n_candidate_pairs"] == out[1][1]["n_candidate_pairs"]


def outcome(lib, sc, precision, capacity, resident, steps=40, setup=None, history=0):
    """Status of a run and what it leaves, errors included"""
    sim = make(lib, sc, precision, history_capacity=history)
    sim.set_tuning(list_capacity=capacity)
    assert (sim.launches_per_step() == 3) == resident
    if setup:
        setup(sim)
    codes = []
    for call in (lambda: sim.initialize_leapfrog(0.0, sc.dt), lambda: sim.step(steps, 0.0, sc.dt), sim.synchronize):
        try:
            call()
            codes.append(0)
        except GrainsError as e:
            codes.append(e.code)
    st = sim.stats()
    sim.reset_stats()
    d, m = sim.download(), sim.contact_memory()
    order = np.lexsort((m["other"], m["owner"], m["system"]))
    sim.close()
    return codes, st, {**d, **{"memory " + k: v[order] for k, v in m.items()}}


def same_outcome(lib, sc, precision, capacities=(32, 20), **kw):
    a, b = (outcome(lib, sc, precision, c, c == capacities[0], **kw) for c in capacities)
    assert a[0] == b[0]
    for k in a[1]:
        if k not in ("overlap_sum", "overlap_mean"):  # summed by atomics, in any order
            assert a[1][k] == b[1][k], k
    for k in a[2]:
        assert np.array_equal(a[2][k], b[2][k], equal_nan=True), k
    return a


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("corrected", [False, True])
def test_immersed_spheres(gpu_lib, corrected, precision):
    """Buoyancy, the fluid's forces and torques, with and without the correction
    of the accelerations."""
    sc = S.small_box(300, seed=8, velocity_sigma=0.3, radius_range=(0.9, 1.1), spacing=2.25)
    sc.dt = 5.0e-6
    rng = np.random.default_rng(8)
    force, torque = rng.normal(0.0, 1.0e-4, (300, 3)), rng.normal(0.0, 1.0e-7, (300, 3))

    def setup(sim):
        sim.set_fluid(1000.0, corrected, np.full(300, 2500.0))
        sim.set_hydro_forces(force, torque)
    codes, st, _ = same_outcome(gpu_lib, sc, precision, setup=setup)
    assert codes == [0, 0, 0] and st["n_contacts"] > 0


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_hertz_without_memory(gpu_lib, precision):
    sc = S.small_box(300, seed=9, velocity_sigma=0.3, radius_range=(0.95, 1.05), spacing=2.07)
    sc.laws = [[(a, b, HERTZ, [2.0e8, 0.9, 0.5, 1.0e-3, 6.0e7]) for a, b, _, _ in sc.laws[0]]]
    sc.dt = 2.0e-6
    codes, st, d = same_outcome(gpu_lib, sc, precision)
    assert codes == [0, 0, 0] and st["n_contacts"] > 0 and len(d["memory owner"]) == 0


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_materials_without_a_law(gpu_lib, precision):
    """Pairs of materials that have no law between them meet too; the lists keep
    no pair constants then."""
    sc = S.small_box(300, seed=10, velocity_sigma=0.3, radius_range=(0.95, 1.05), spacing=2.0)
    sc.dt = 2.0e-6
    sc.particles["material"] = (np.arange(300) % 2 * 2).astype(np.int32)  # 0 and 2
    law = sc.laws[0][0][2:]
    sc.laws = [sc.laws[0] + [(2, 2, *law), (1, 2, *law)]]
    codes, st, d = same_outcome(gpu_lib, sc, precision)
    assert codes == [0, 0, 0] and len(d["memory owner"]) > 0


def one_fast(sc, k, velocity, position=None):
    sc.particles["velocity"][k] = velocity
    if position is not None:
        sc.particles["position"][k] = position
    return sc


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("what", ["motion", "grid", "handled", "contact"])
def test_errors_of_a_run(gpu_lib, what, precision):
    """A displacement beyond the crust, a sphere that leaves the grid, overlaps
    beyond the crusts that the retry with ten crusts handles or not: the status
    and the state of the launched pipeline."""
    sc = S.small_box(125, seed=11, velocity_sigma=0.05, radius_range=(0.95, 1.05), spacing=2.2)
    sc.dt = 2.0e-6
    if what == "motion":
        sc.particles["crust"][:] = 1.0e-6
        one_fast(sc, 7, [0.0, 0.0, 0.9])
    elif what == "grid":
        sc.obstacles = [[]]
        one_fast(sc, 0, [-0.5, 0.0, 0.0], [20.0e-6, 4.0e-3, 15.0e-3])
    else:
        crust = 2.0e-5 if what == "handled" else 2.0e-6
        sc.particles["crust"][:] = crust
        for o in sc.obstacles[0]:
            o["crust"] = crust
        x = sc.particles["position"]
        x[1] = x[0] + [sc.particles["radius"][0] + sc.particles["radius"][1] - 1.0e-4, 0.0, 0.0]
    # (the handled pair flies apart: a few steps before it meets the next spheres)
    codes, st, _ = same_outcome(gpu_lib, sc, precision, steps=9 if what == "handled" else 40)
    bit = {"motion": MOTION_ERROR, "grid": OUT_OF_GRID, "handled": CONTACT_HANDLED, "contact": CONTACT_ERROR}[what]
    assert st["status"] & bit
    if what == "handled":
        assert codes == [0, 0, 0] and st["status"] == bit
    else:
        assert codes[2] & bit


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_more_contacts_than_memory_slots(gpu_lib, precision):
    """The sphere of the lowest id owns its 18 contacts, and a row holds 12
    memories: both pipelines say so."""
    side, r, a = 7, 0.7e-3, 0.975e-3  # neighbours at a and sqrt(2) a touch, at sqrt(3) a do not
    n = side ** 3
    sc = S.small_box(n, seed=1)
    k = np.arange(n)
    x = a * np.stack([k % side, k // side % side, k // side ** 2], 1) + 3.0e-3
    sc.particles = S._spheres(n, np.full(n, r), 2500.0, x, np.zeros((n, 3)), 0.5e-3)
    ids = np.arange(1, n + 1, dtype=np.int32)
    ids[n // 2] = 0
    sc.particles["id"] = ids
    sc.laws = [[(p, q, HOOKE_MEMORY, [1.0e2, 0.9, -1.0, 0.5, 0.8e2, 0.0, 0.0, 0.0]) for p, q, _, _ in sc.laws[0]]]
    sc.obstacles, sc.dt = [[]], 1.0e-8
    for capacity in (24, 20):
        codes, st, d = outcome(gpu_lib, sc, precision, capacity, capacity == 24, history=12)
        assert d["coordination"].max() == 18
        assert codes[0] == codes[2] == st["status"] == HISTORY_FULL


@pytest.mark.parametrize("share", [0.04, 0.06])
def test_the_speed_outlives_force_evaluations_and_rest(gpu_lib, share):
    """Force evaluations that do not permute the particles leave the speed that
    the choice of the pipeline goes by; particles put to rest are slow."""
    sc = moving_lattice(1000, share, False)
    sim = make(gpu_lib, sc, MIXED)

    def resident():
        t, phases = sim.profile_kernels(8, 0.0, sc.dt)
        return phases["contacts"][1] == 1
    sim.initialize_leapfrog(0.0, sc.dt)
    for _ in range(3):
        sim.compute_forces(0.0, sc.dt)
    assert resident() == (share < 0.05)
    sim.compute_forces(0.0, sc.dt)
    sim.reset_stats()
    sim.synchronize()
    assert resident() == (share < 0.05)
    sim.update({**sc.particles, "velocity": 0.0 * sc.particles["velocity"]})
    sim.initialize_leapfrog(0.0, sc.dt)
    assert resident()
    sim.close()
