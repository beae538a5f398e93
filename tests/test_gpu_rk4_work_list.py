"""RungeKutta4 of Model C on grids of more units than one wave holds, where the
four stages of a step take theirs from the list and leave it reset for the
next, read the running sum that other units' warps wrote in the stage before,
and blocks of 32, 64, 126, 128 and 256 columns have their own instantiations:
FP64 has the oracle's bits, plain and as a graph (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L

pytestmark = pytest.mark.gpu

H, STEPS = 0.4, 6


@pytest.mark.parametrize("cells,block", [([1764, 1764], [126, 126]), ([1536, 1664], [128, 128]),
                                         ([1600, 1500], [100, 75]), ([1280, 1024], [32, 64]), ([1280, 1088], [64, 34]),
                                         ([1536, 1280], [256, 160])])
@pytest.mark.parametrize("orient", [False, True])
def test_has_the_oracle_bits(sched, orc, cells, block, orient):
    grid = L.CartesianGrid(cells, block, [0.0, 0.0], [H, H])
    model = L.ModelC(0.05, 3.19)
    if orient:
        model.with_orientations()
    rng = np.random.default_rng(2)
    grains = [(rng.uniform(0, H * cells[0]), rng.uniform(0, H * cells[1]), rng.uniform(4, 20), rng.uniform(0, 1.5))
              for _ in range(25)]
    ref = orc.State(orc.Grid(cells, block, [0.0, 0.0], [H, H]), [1, 1, 0] if orient else [1, 1])
    ref.initialize_grains([g[:3] for g in grains], 0.55)
    if orient:
        ref.initialize_orientations(2, grains)
    sims = []
    for _ in range(2):
        sim = L.Simulation(grid, L.FiniteVolume(), model, L.RungeKutta4(), sched, L.CudaAllocator("f64"))
        model.initialize_grains(grid, sim.state, [L.Grain(g[:2], g[2], g[3] if orient else 0.0) for g in grains], 0.55)
        sims.append(sim)
    sims[0].run(0.008, STEPS, graph=True)
    for _ in range(STEPS):
        sims[1].run(0.008, 1)
    p = orc.modelc_params(eps4=0.05, lam=3.19, d_thermal=model.d_thermal)
    ref.modelc_run_rk4(p, 0.0, 0.008, STEPS, theta_field=2 if orient else -1, threads=16)
    for sim in sims:
        for f in (0, 1):
            assert np.array_equal(sim.state.interior(f), ref.interior(f))
        sim.state._destroy()


def test_fp32_repeats(sched):
    # the stages race for units, yet a run has the same bits each time, plain
    # and as a graph
    n, b = 1764, 126
    grid = L.CartesianGrid([n, n], [b, b], [0.0, 0.0], [H, H])
    rng = np.random.default_rng(2)
    fields = [np.tanh(rng.standard_normal((196, b + 2, b + 2))).astype(np.float32) for _ in range(2)]
    out = []
    for graph in (True, False, True):
        sim = L.Simulation(grid, L.FiniteVolume(), L.ModelC(0.05, 3.19), L.RungeKutta4(), sched, L.CudaAllocator("f32"))
        for f in (0, 1):
            sim.state.upload(f, fields[f])
        sim.run(0.001, STEPS, graph=graph)
        out.append([sim.state.interior(f) for f in (0, 1)])
        sim.state._destroy()
    assert np.isfinite(out[0]).all()
    assert all(np.array_equal(a, b) for one in out[1:] for a, b in zip(out[0], one))
