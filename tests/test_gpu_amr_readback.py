"""Reading an AMR field back: every block's slab, ghosts included, in block
order, whatever the block sizes, the number of levels and the buffers that the
levels' states are in (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,block,ratios,patches", [
    ([4, 4], [4, 4], [], []),
    ([36, 20], [12, 5], [2], [[((8, 8), (10, 26))]]),
    ([64, 32], [16, 16], [2, 2], [[((16, 16), (64, 48)), ((64, 16), (80, 40))], [((40, 40), (100, 70))]]),
    ([512, 512], [8, 8], [2], [[((100, 100), (356, 104))]]),
])
def test_round_trip(sched, cells, block, ratios, patches):
    base = L.CartesianGrid(cells, block, [0.0, 0.0], [0.4, 0.4])
    grid = L.AmrGrid.from_patches(base, ratios, [[L.CellBox(lo, hi) for lo, hi in level] for level in patches])
    sim = L.AmrSimulation(grid, L.FiniteVolume(), L.ModelC(0.05, 3.19, 0.0), L.Subcycling(3), sched,
                          L.CudaAllocator("f64"))
    rng = np.random.default_rng(8)
    for steps in (0, 1, 2):  # each step moves the levels to their other buffers
        if steps:
            sim.run(0.004, steps)
        want = [[np.tanh(rng.standard_normal(a.shape)) for a in sim.get(f)] for f in ("phi", "u")]
        assert [a.shape for a in want[0]] == [(hi[1] - lo[1] + 2, hi[0] - lo[0] + 2) for _, lo, hi in sim.patches()]
        for f in (1, 0):
            sim.set(f, want[f])
        for f in (0, 1):
            got = sim.get(f)
            assert len(got) == len(want[f]) and all(np.array_equal(a, b) for a, b in zip(got, want[f]))
