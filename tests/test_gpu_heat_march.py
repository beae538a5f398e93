"""The marching heat kernel (2-D and 3-D, two stages per launch) where its
tiling can go wrong: windows one cell off the tile widths (34 x 18 and 32 x
16 columns in 3-D, 126 and 124 in 2-D), blocks narrower than the halo, mirror
and periodic edges, odd step counts, several march chunks.  The kernel keeps
the oracle's operand order, so FP64 interiors and the ghosts filled after a run
are its bits (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

SHAPES = [
    ([1, 1], [1, 1], [True, False]),
    ([3, 2, 1], [1, 1, 1], [False, True, True]),
    ([2, 3, 4], [2, 1, 2], [True, False, False]),
    ([33, 17, 5], [11, 17, 1], [False, False, False]),
    ([32, 16, 7], [8, 8, 7], [True, True, False]),
    ([35, 19, 6], [5, 19, 3], [True, False, True]),
    ([66, 33, 40], [33, 11, 8], [False, True, True]),
    ([124, 9], [31, 3], [False, True]),
    ([125, 40], [25, 8], [True, False]),
    ([253, 6], [253, 2], [False, False]),
    ([378, 300], [63, 50], [True, True]),
]


def _pair(sched, orc, cells, block, periodic, method):
    D = len(cells)
    grid = L.CartesianGrid(cells, block, [0.0] * D, [0.1] * D).with_periodic(periodic)
    sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(0.7), method, sched, L.CudaAllocator("f64"))
    u0 = with_ghosts(np.random.default_rng(5).standard_normal((grid.num_blocks(),) + tuple(reversed(block))), 1)
    sim.state.upload("u", u0)
    ref = orc.State(orc.Grid(cells, block, [0.0] * D, [0.1] * D, periodic), [1])
    ref.set(0, u0)
    return sim, ref


@pytest.mark.parametrize("cells,block,periodic", SHAPES)
@pytest.mark.parametrize("steps,graph", [(1, False), (2, False), (3, True), (14, True)])
def test_forward_euler(sched, orc, cells, block, periodic, steps, graph):
    sim, ref = _pair(sched, orc, cells, block, periodic, L.ForwardEuler())
    dt = 0.0009
    sim.run(dt, steps, graph=graph)
    ref.heat_run(0, 0.7, 0.0, dt, steps)
    ref.fill_ghosts(0)
    assert np.array_equal(sim.state.download("u"), ref.get(0))


@pytest.mark.parametrize("cells,block,periodic", SHAPES)
@pytest.mark.parametrize("steps,graph", [(1, False), (4, True)])
def test_rk4(sched, orc, cells, block, periodic, steps, graph):
    sim, ref = _pair(sched, orc, cells, block, periodic, L.RungeKutta4())
    dt = 0.0009
    sim.run(dt, steps, graph=graph)
    ref.heat_run_rk4(0, 0.7, 0.0, dt, steps)
    ref.fill_ghosts(0)
    assert np.array_equal(sim.state.download("u"), ref.get(0))
