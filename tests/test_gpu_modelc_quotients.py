"""Model C's shared-reciprocal quotients and far-field test where they can go
wrong: gradients on both sides of the tolerance, differences small and large
enough to leave the range of the reciprocal, exact zeros, tolerances of zero
and below, no anisotropy.  One noise-free FP64 step has the oracle's bits
(needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

CELLS, BLOCK, H = [96, 24], [48, 12], 0.4


def _fields(kind, scale):
    rng = np.random.default_rng(11)
    shape = (4, BLOCK[1], BLOCK[0])
    if kind == "zero":
        return np.full(shape, -1.0), np.zeros(shape)
    if kind == "tolerance":  # differences around |grad phi| = 0.01, where |grad phi|^4 is the tolerance
        return -1.0 + 0.01 * scale * rng.integers(0, 2, shape), rng.standard_normal(shape)
    return scale * rng.standard_normal(shape), rng.standard_normal(shape)


@pytest.mark.parametrize("variant", [1, 2, 5, 15])
@pytest.mark.parametrize("eps4,flux_tol,tol", [(0.05, 1e-8, 1e-8), (0.0, 1e-8, 1e-4), (0.06, 0.0, -1.0)])
@pytest.mark.parametrize("kind,scale", [("zero", 0.0), ("tolerance", 1.0), ("tolerance", 1.0 - 2.0 ** -50),
                                        ("tolerance", 0.7071067811865476), ("random", 1e-170), ("random", 1e-70),
                                        ("random", 1e-3), ("random", 1.0), ("random", 1e60), ("random", 1e150)])
def test_one_step(sched, orc, variant, eps4, flux_tol, tol, kind, scale):
    grid = L.CartesianGrid(CELLS, BLOCK, [0.0, 0.0], [H, H])
    model = L.ModelC(eps4, 3.19)
    model.anisotropy_tol = tol
    sim = L.Simulation(grid, L.FiniteVolume(tol=flux_tol), model, L.EulerMaruyama(3), sched, L.CudaAllocator("f64"))
    ref = orc.State(orc.Grid(CELLS, BLOCK, [0.0, 0.0], [H, H]), [1, 1])
    for f, a in enumerate(_fields(kind, scale)):
        sim.state.upload(f, with_ghosts(a, 1))
        ref.set(f, with_ghosts(a, 1))
    sim.run(0.008, 1, variant=variant)
    p = orc.modelc_params(eps4=eps4, lam=3.19, d_thermal=model.d_thermal, noise=0.0, tol=tol, flux_tol=flux_tol)
    with np.errstate(all="ignore"):
        ref.modelc_run(p, 0.0, 0.008, 3, 1, False)
    for f in (0, 1):
        assert np.array_equal(sim.state.interior(f), ref.interior(f), equal_nan=True)
