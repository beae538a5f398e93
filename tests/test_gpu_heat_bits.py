"""Heat steps as integers: fields of signed zeros and of subnormal values on a
coarse grid, where a dimension's term underflows to a zero of either sign, and
NaN and infinities; the oracle's bits, ghosts included (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

H = 4.0


def _bits(a):
    return np.where(np.isnan(a), 0x7ff8000000000000, a.view(np.int64))


@pytest.mark.parametrize("cells,block,periodic", [([24, 15], [8, 5], [False, True]),
                                                  ([16, 12, 10], [8, 6, 5], [True, False, False])])
@pytest.mark.parametrize("method", ["euler", "rk4"])
@pytest.mark.parametrize("kind", ["zeros", "subnormal", "special"])
def test_has_the_oracle_bits(sched, orc, cells, block, periodic, method, kind):
    D, dt = len(cells), 0.5
    grid = L.CartesianGrid(cells, block, [0.0] * D, [H] * D).with_periodic(periodic)
    rng = np.random.default_rng(9)
    shape = (grid.num_blocks(),) + tuple(reversed(block))
    zeros = np.copysign(0.0, rng.choice([-1.0, 1.0], shape))
    if kind == "zeros":
        u = zeros
    elif kind == "subnormal":
        u = np.where(rng.random(shape) < 0.5, zeros, 2.0 ** -1074 * rng.integers(-3, 4, shape))
    else:
        u = rng.standard_normal(shape)
        u.flat[5], u.flat[40], u.flat[77] = np.nan, np.inf, -np.inf
    u = with_ghosts(u, 1)
    for steps in (1, 2, 3):
        sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(0.7),
                           L.ForwardEuler() if method == "euler" else L.RungeKutta4(), sched, L.CudaAllocator("f64"))
        sim.state.upload("u", u)
        sim.run(dt, steps)
        ref = orc.State(orc.Grid(cells, block, [0.0] * D, [H] * D, periodic), [1])
        ref.set(0, u)
        (ref.heat_run if method == "euler" else ref.heat_run_rk4)(0, 0.7, 0.0, dt, steps)
        ref.fill_ghosts(0)
        assert np.array_equal(_bits(sim.state.download("u")), _bits(ref.get(0)))
