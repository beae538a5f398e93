"""The Model C launch plan where it changes hands: unit heights of 2 to 32
rows, blocks lower than a group of rows, widths around a strip, one wave and
more (the work list), steps chained through plain launches and graphs.  The
default variant has the reference-order kernel's bits without noise, and with
noise too (the same Gaussians), FP64; multi-grain likewise against itself
stepped one launch at a time (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

H = 0.4


def _run(sched, cells, block, noise, orient, runs, variant, dtype="f64"):
    grid = L.CartesianGrid(cells, block, [0.0, 0.0], [H, H]).with_periodic([True, False])
    model = L.ModelC(0.05, 3.19, noise)
    if orient:
        model.with_orientations()
    sim = L.Simulation(grid, L.FiniteVolume(), model, L.EulerMaruyama(9), sched, L.CudaAllocator(dtype))
    rng = np.random.default_rng(4)
    shape = (grid.num_blocks(), block[1], block[0])
    for f, a in enumerate([np.tanh(3.0 * rng.standard_normal(shape)), 0.3 * rng.standard_normal(shape)]):
        sim.state.upload(f, with_ghosts(a, 1))
    if orient:
        sim.state.upload("theta0", rng.uniform(0.0, 1.5, (shape[0], 1, 1)) * np.ones(shape))
        model.set_orientations(sim.state)
    for steps, graph in runs:
        sim.run(0.008, steps, graph=graph, variant=variant)
    return [sim.state.download(f) for f in ("phi", "u")]


@pytest.mark.parametrize("noise", [0.0, 0.02])
@pytest.mark.parametrize("cells,block", [([6, 3], [3, 1]), ([31, 4], [31, 2]), ([66, 9], [33, 3]), ([32, 10], [32, 5]),
                                         ([130, 14], [65, 7]), ([512, 512], [64, 64]), ([1008, 1008], [126, 126]),
                                         ([1536, 1280], [96, 160]), ([2048, 2044], [128, 73])])
def test_default_has_the_reference_order_bits(sched, cells, block, noise):
    got = _run(sched, cells, block, noise, False, [(3, False), (6, True), (1, False)], 0)
    ref = _run(sched, cells, block, noise, False, [(10, False)], 1)
    assert all(np.array_equal(a[:, 1:-1, 1:-1], b[:, 1:-1, 1:-1]) for a, b in zip(got, ref))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("cells,block", [([6, 3], [3, 1]), ([66, 9], [33, 3]), ([504, 252], [126, 63]),
                                         ([1536, 1280], [96, 160])])
def test_multi_grain_steps_one_by_one(sched, cells, block, dtype):
    got = _run(sched, cells, block, 0.02, True, [(7, False), (8, True)], 0, dtype)
    ref = _run(sched, cells, block, 0.02, True, [(1, False)] * 15, 0, dtype)
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


def test_noise_follows_the_state_time(sched):
    # the device keeps the time between runs; a run after set_time, after an
    # autotune or on a fresh state starts from the state's own time
    def sim_of():
        grid = L.CartesianGrid([64, 32], [32, 16], [0.0, 0.0], [H, H])
        return L.Simulation(grid, L.FiniteVolume(), L.ModelC(0.05, 3.19, 0.02), L.EulerMaruyama(9), sched,
                            L.CudaAllocator("f64"))

    a = sim_of()
    rng = np.random.default_rng(2)
    fields = [with_ghosts(0.1 * rng.standard_normal((4, 16, 32)), 1) for _ in range(2)]
    for f in (0, 1):
        a.state.upload(f, fields[f])
    t = None
    for leg, (start, steps) in enumerate([(None, 3), (None, 2), (5.25, 1), (0.0, 4), (None, 3)]):
        if start is not None:
            a.state.set_time(start, 0)
        if leg == 4:
            a.autotune(0.008, trial_steps=1)
        t, k = a.state.time
        b = sim_of()
        for f in (0, 1):
            b.state.upload(f, fields[f])
        b.state.set_time(t, k)
        for s in (a, b):
            s.run(0.008, steps, variant=5)
        assert a.state.time == b.state.time
        fields = [a.state.download(f) for f in (0, 1)]
        assert all(np.array_equal(x, b.state.download(f)) for f, x in enumerate(fields))
