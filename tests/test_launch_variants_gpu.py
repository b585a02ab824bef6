"""Kernels that take another form at another size: the same bits on both sides
of the line."""
import numpy as np
import pytest

from pacific_b200 import scenarios as S
from pacific_b200.abi import FP64, GJK, GJK_SV, MIXED

from helpers import make

pytestmark = pytest.mark.gpu

STATE = ["position", "quaternion", "velocity", "omega", "force", "torque", "coordination"]


def first(p, n):
    return {k: (None if v is None else v[:n]) for k, v in p.items()}


@pytest.mark.parametrize("convex", [False, True])
@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_contact_lists_by_eight_lanes_and_by_one_thread(gpu_lib, precision, convex):
    """Lists are built by eight lanes per particle up to 28,000 spheres (40,000
    convex bodies) and by one thread above: one particle more leaves the forces
    on all particles out of its reach as they were."""
    if convex:
        m, sc = 40000, S.convex_box(40001, seed=2, spacing=3.4)
    else:
        m, sc = 28000, S.small_box(28001, seed=2, velocity_sigma=0.1, radius_range=(0.95, 1.05), spacing=2.0)
    out = []
    for n in (m + 1, m):
        few = S.Scenario(**{**sc.__dict__, "particles": first(sc.particles, n)})
        sim = make(gpu_lib, few, precision)
        sim.initialize_leapfrog(0.0, sc.dt)
        d = sim.download()
        out.append((d, sim.stats()))
        sim.close()
    x = sc.particles["position"]
    apart = np.linalg.norm(x[:m] - x[m], axis=1) > (8.0e-3 if convex else 5.0e-3)
    assert apart.sum() > 0.97 * m and (convex or out[0][0]["coordination"].max() >= 4)
    assert not convex or out[1][1]["n_gjk_calls"] > 10000  # pairs listed and tested
    for k in STATE:
        assert np.array_equal(out[0][0][k][:m][apart], out[1][0][k][apart]), k
    assert out[0][1]["status"] == out[1][1]["status"]


def copies(sc, k):
    """k systems, each a copy of the scenario's one"""
    p = {key: (None if v is None else np.concatenate([v] * k)) for key, v in sc.particles.items()}
    p["system"] = np.repeat(np.arange(k, dtype=np.int32), sc.n)
    return S.Scenario(**{**sc.__dict__, "domains": sc.domains * k, "laws": sc.laws * k,
                         "obstacles": sc.obstacles * k, "particles": p})


@pytest.mark.parametrize("algorithm", [GJK, GJK_SV])
@pytest.mark.parametrize("k", [2, 300, 1500])
def test_gjk_runs_spread_over_the_warps(gpu_lib, k, algorithm):
    """One GJK run in a few warps, several lanes of each warp (300 systems),
    more runs than lanes (1,500): every system as when it is alone."""
    one = S.convex_box(27, seed=4, converge_time=1.0e-3)
    one.meta = dict(one.meta or {}, collision=algorithm)
    out = []
    for sc in (one, copies(one, k)):
        sim = make(gpu_lib, sc, MIXED)
        sim.initialize_leapfrog(0.0, sc.dt)
        t = sim.step(150, 0.0, sc.dt)
        sim.reset_stats()
        sim.step(1, t, sc.dt)
        out.append((sim.download(), sim.stats()))
        sim.close()
    (a, sa), (b, sb) = out
    assert sa["n_contacts"] > 0
    assert (sb["n_gjk_calls"] > 148 * 8 * 32) == (k == 1500)  # the lanes of all warps
    for key in ("n_gjk_calls", "n_gjk_iterations", "n_contacts", "status"):
        assert sb[key] == (sa[key] if key == "status" else k * sa[key]), key
    for key in STATE:
        v = b[key].reshape((k,) + a[key].shape)
        assert np.array_equal(v, np.broadcast_to(a[key], v.shape)), key
