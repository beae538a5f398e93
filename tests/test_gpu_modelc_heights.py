"""FP32 multi-grain steps at the unit heights their plan chooses (6, 10, 12, 20
and 24 rows beside the powers of two; blocks that no height divides), and
batches at theirs: every height has the values of the two-row units, within the few
rounding steps by which the units' first faces may be contracted differently
(needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

H, STEPS = 0.4, 6
# a handful of FP32 roundings (6e-8) a step on values of order one
TOLERANCE = STEPS * 8 * 2.0 ** -24


def _multi_grain(sched, n, b, rows):
    grid = L.CartesianGrid([n, n], [b, b], [0.0, 0.0], [H, H])
    model = L.ModelC(0.05, 3.19, 0.02)
    model.with_orientations()
    sim = L.Simulation(grid, L.FiniteVolume(), model, L.EulerMaruyama(9), sched, L.CudaAllocator("f32"))
    rng = np.random.default_rng(4)
    shape = (grid.num_blocks(), b, b)
    for f in ("phi", "u"):
        sim.state.upload(f, with_ghosts(0.3 * rng.standard_normal(shape), 1))
    sim.state.upload("theta0", rng.uniform(0.0, 1.5, (shape[0], 1, 1)) * np.ones(shape))
    model.set_orientations(sim.state)
    sim.run(0.001, STEPS, graph=True, variant=1000 * rows)
    return [sim.state.download(f) for f in ("phi", "u")]


@pytest.mark.parametrize("n,b,rows", [(100, 50, (6, 10, 12, 20, 24, 32, 0)), (500, 100, (0,)), (720, 48, (0,)),
                                      (1260, 126, (0,)), (1500, 100, (0,))])
def test_multi_grain(sched, n, b, rows):
    ref = _multi_grain(sched, n, b, 2)
    for r in rows:
        got = _multi_grain(sched, n, b, r)
        assert all(np.abs(x - y).max() <= TOLERANCE for x, y in zip(got, ref)), r


@pytest.mark.parametrize("instances,n,b", [(5, 20, 10), (48, 144, 48), (64, 256, 64)])
def test_batched(sched, instances, n, b):
    # an instance alone is stepped in the shortest units
    grid = L.CartesianGrid([n, n], [b, b], [0.0, 0.0], [H, H])
    rng = np.random.default_rng(6)
    fields = [(0.3 * rng.standard_normal((instances, n, n))).astype(np.float32) for _ in range(2)]

    def run(which):
        e = L.Ensemble(grid, L.ModelC(0.05, 3.19, 0.02), [0.03 + 0.0005 * i for i in which], list(which), sched, "f32")
        for f, a in zip(("phi", "u"), fields):
            e.set(f, a[which])
        e.run(0.001, STEPS)
        return [e.get(f) for f in ("phi", "u")]

    every = run(list(range(instances)))
    for i in (0, instances // 2, instances - 1):
        one = run([i])
        assert all(np.abs(x[i] - y[0]).max() <= TOLERANCE for x, y in zip(every, one))
