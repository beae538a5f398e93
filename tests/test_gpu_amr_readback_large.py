"""Reading back blocks of far more entries than a CTA has threads, alone and
beside small ones: every entry of every slab, ghosts included (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,block,patches", [
    ([1024, 1024], [1024, 1024], []),
    ([63, 62], [63, 62], []),  # 65 x 64 entries, one over 4096
    ([600, 257], [300, 257], [[((100, 100), (116, 104)), ((300, 40), (900, 340))]]),
])
def test_round_trip(sched, cells, block, patches):
    base = L.CartesianGrid(cells, block, [0.0, 0.0], [0.4, 0.4])
    grid = L.AmrGrid.from_patches(base, [2] * len(patches), [[L.CellBox(lo, hi) for lo, hi in p] for p in patches])
    sim = L.AmrSimulation(grid, L.FiniteVolume(), L.ModelC(0.05, 3.19, 0.0), L.Subcycling(3), sched,
                          L.CudaAllocator("f64"))
    rng = np.random.default_rng(8)
    want = [[rng.standard_normal(a.shape) for a in sim.get(f)] for f in ("phi", "u")]
    for f in (0, 1):
        sim.set(f, want[f])
    for f in (0, 1):
        got = sim.get(f)
        other = sim.get(f)
        for a in other:  # a read's arrays are its own
            a[...] = 7.0
        assert len(got) == len(want[f]) and all(np.array_equal(a, b) for a, b in zip(got, want[f]))
