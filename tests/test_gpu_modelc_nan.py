"""NaN of either sign and infinities in a quiet region: the far-field test of
the paired rows must not take them for flat, so that one and two noise-free
FP64 steps have the oracle's values cell for cell, and FP32 steps its NaN
cells (needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

CELLS, BLOCK, H = [96, 24], [48, 12], 0.4
NAN = {"+nan": 0x7ff8000000000000, "-nan": 0xfff8000000000000}


def _value(kind):
    return np.array(NAN[kind], np.uint64).view(np.float64) if kind in NAN else np.float64(kind)


def _pair(sched, orc, dtype, field, kind, x, y):
    grid = L.CartesianGrid(CELLS, BLOCK, [0.0, 0.0], [H, H])
    sim = L.Simulation(grid, L.FiniteVolume(), L.ModelC(0.05, 3.19), L.EulerMaruyama(3), sched, L.CudaAllocator(dtype))
    ref = orc.State(orc.Grid(CELLS, BLOCK, [0.0, 0.0], [H, H]), [1, 1])
    for f in (0, 1):
        a = np.full((4, BLOCK[1], BLOCK[0]), -1.0 if f == 0 else -0.5)
        if f == field:
            a[y // BLOCK[1] * 2 + x // BLOCK[0], y % BLOCK[1], x % BLOCK[0]] = _value(kind)
        sim.state.upload(f, with_ghosts(a, 1).astype(sim.state.alloc.numpy_dtype))
        ref.set(f, with_ghosts(a, 1))
    return sim, ref, orc.modelc_params(eps4=0.05, lam=3.19, d_thermal=sim.model.d_thermal)


# inside a strip, on a strip's and a block's edge, on both rows of a pass
@pytest.mark.parametrize("x,y", [(10, 4), (11, 5), (31, 6), (47, 11), (48, 12)])
@pytest.mark.parametrize("kind", ["+nan", "-nan", "inf", "-inf"])
@pytest.mark.parametrize("variant", [0, 1, 5, 15])
def test_fp64_has_the_oracle_values(sched, orc, variant, kind, x, y):
    for field in (0, 1):
        sim, ref, p = _pair(sched, orc, "f64", field, kind, x, y)
        for _ in range(2):
            t = sim.time()
            sim.run(0.008, 1, variant=variant)
            with np.errstate(all="ignore"):
                ref.modelc_run(p, t, 0.008, 3, 1, False)
            for f in (0, 1):
                assert np.array_equal(sim.state.interior(f), ref.interior(f), equal_nan=True)


@pytest.mark.parametrize("kind", ["+nan", "-nan"])
@pytest.mark.parametrize("variant", [0, 5, 15])
def test_fp32_has_the_oracle_nan_cells(sched, orc, variant, kind):
    sim, ref, p = _pair(sched, orc, "f32", 0, kind, 31, 6)
    for _ in range(2):
        t = sim.time()
        sim.run(0.008, 1, variant=variant)
        with np.errstate(all="ignore"):
            ref.modelc_run(p, t, 0.008, 3, 1, False)
        for f in (0, 1):
            assert np.array_equal(np.isnan(sim.state.interior(f)), np.isnan(ref.interior(f)))
