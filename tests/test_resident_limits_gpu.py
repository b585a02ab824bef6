"""Resident pair lists at their limits: more entries than the lists hold."""
import numpy as np
import pytest

from pacific_b200 import scenarios as S
from pacific_b200.abi import CUDA_ERROR, MIXED, PAIR_OVERFLOW, TIMEOUT, GrainsError

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
