"""Every tile shape of the marching heat kernel: grids that the plan gives the
shapes for narrow x, narrow y and both, and the tile of four rows a thread
(112^3 and up), windows one cell off the tile widths, mirror and periodic
edges, the double, the odd single step and both halves of RungeKutta4.  FP64
interiors and ghosts are the oracle's bits (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

SHAPES = [
    ([8, 160, 300], [8, 16, 20], [True, True, False]),    # 8 x 80
    ([9, 162, 100], [9, 27, 10], [False, False, True]),
    ([300, 8, 200], [20, 8, 20], [False, True, True]),    # 60 x 8
    ([242, 7, 160], [22, 7, 16], [True, False, False]),
    ([8, 8, 2000], [8, 8, 16], [True, False, True]),      # 8 x 8
    ([5, 9, 1500], [5, 3, 50], [False, False, False]),
    ([112, 112, 112], [16, 16, 16], [False, False, False]),  # 28 x 28
    ([115, 113, 114], [23, 113, 57], [True, False, True]),
]


@pytest.mark.parametrize("cells,block,periodic", SHAPES)
@pytest.mark.parametrize("method", ["euler", "rk4"])
def test_has_the_oracle_bits(sched, orc, cells, block, periodic, method):
    grid = L.CartesianGrid(cells, block, [0.0] * 3, [0.1] * 3).with_periodic(periodic)
    u0 = with_ghosts(np.random.default_rng(5).standard_normal((grid.num_blocks(),) + tuple(reversed(block))), 1)
    dt = 0.0009
    for steps in (1, 5) if method == "euler" else (2,):
        sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(0.7),
                           L.ForwardEuler() if method == "euler" else L.RungeKutta4(), sched, L.CudaAllocator("f64"))
        sim.state.upload("u", u0)
        sim.run(dt, steps, graph=steps > 2)
        ref = orc.State(orc.Grid(cells, block, [0.0] * 3, [0.1] * 3, periodic), [1])
        ref.set(0, u0)
        (ref.heat_run if method == "euler" else ref.heat_run_rk4)(0, 0.7, 0.0, dt, steps, threads=8)
        ref.fill_ghosts(0)
        assert np.array_equal(sim.state.download("u"), ref.get(0))
