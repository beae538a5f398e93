"""One forward-Euler step a call on 2-D grids around the size up to which a kernel
of one thread a cell takes it (2^19 cells) and beyond, mixed with longer runs:
the oracle's bits, ghosts included (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,block,periodic", [([1, 1], [1, 1], [True, False]), ([24, 15], [8, 5], [False, True]),
                                                  ([1024, 512], [64, 32], [False, False]),
                                                  ([1025, 512], [41, 64], [True, False])])
def test_single_steps(sched, orc, cells, block, periodic):
    grid = L.CartesianGrid(cells, block, [0.0, 0.0], [0.1, 0.1]).with_periodic(periodic)
    sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(0.7), L.ForwardEuler(), sched, L.CudaAllocator("f64"))
    u0 = with_ghosts(np.random.default_rng(5).standard_normal((grid.num_blocks(),) + tuple(reversed(block))), 1)
    sim.state.upload("u", u0)
    ref = orc.State(orc.Grid(cells, block, [0.0, 0.0], [0.1, 0.1], periodic), [1])
    ref.set(0, u0)
    dt, done = 0.0009, 0
    for steps in (1, 1, 2, 1, 3, 1):
        sim.run(dt, steps)
        done += steps
        ref.heat_run(0, 0.7, 0.0, dt, steps, threads=8)
        ref.fill_ghosts(0)
        assert np.array_equal(sim.state.download("u"), ref.get(0))
    assert sim.step_index() == done
