"""One noise-free FP64 Model C step has the oracle's bits, compared as integers
so that the sign of a zero counts: fields of signed zeros, fields at the end
of the exponent range, tiny steps beside large ones (a face's quotient out of
the shared reciprocal's range), negative a_bar, parameters out of its range
(needs a GPU)."""
import math

import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

pytestmark = pytest.mark.gpu

CELLS, BLOCK, H = [96, 24], [48, 12], 0.4
SHAPE = (4, BLOCK[1], BLOCK[0])


def _fields(kind):
    rng = np.random.default_rng(17)
    sign = lambda: rng.choice([-1.0, 1.0], SHAPE)  # noqa: E731
    if kind == "zeros":
        return np.copysign(0.0, sign()), np.copysign(0.0, sign())
    if kind == "few":  # zeros with a few tiny values
        return [np.where(rng.random(SHAPE) < 0.1, rng.standard_normal(SHAPE) * 1e-310, np.copysign(0.0, sign()))
                for _ in range(2)]
    if kind.startswith("2^"):
        return [rng.standard_normal(SHAPE) * math.ldexp(1.0, int(kind[2:])) for _ in range(2)]
    # rows of constants with one row of tiny values in four: a large y
    # difference beside a tiny x difference, and transposed
    small = math.ldexp(1.0, int(kind.split("^")[1]))
    if kind.startswith("rows"):
        phi = np.where((np.arange(SHAPE[1]) % 4 == 1)[None, :, None], small * rng.standard_normal(SHAPE), 0.5)
    else:
        phi = np.where((np.arange(SHAPE[2]) % 4 == 1)[None, None, :], small * rng.standard_normal(SHAPE), -0.5)
    return phi, small * rng.standard_normal(SHAPE)


KINDS = ["zeros", "few", "2^-300", "2^-520", "2^-980", "2^-1015", "2^-1040", "2^-1060", "2^200", "rows^-330",
         "rows^-980", "rows^-1020", "rows^-1055", "columns^-330", "columns^-990", "columns^-1020", "columns^-1060"]


def _bits(a):
    return np.where(np.isnan(a), 0x7ff8000000000000, a.view(np.int64))


@pytest.mark.parametrize("form", [1, 2, 5, 15, "multi-grain", "rk4"])
@pytest.mark.parametrize("eps4,tol", [(0.05, 1e-8), (0.0, 1e-8), (0.45, 1e-8), (0.05, -1.0), (1e-30, 1e-8)])
@pytest.mark.parametrize("dt", [0.008, 1024.0])  # the longer one shows every bit of the drift
def test_one_step(sched, orc, form, eps4, tol, dt):
    for kind in KINDS:
        _check(sched, orc, form, eps4, tol, dt, kind)


def _check(sched, orc, form, eps4, tol, dt, kind):
    grid = L.CartesianGrid(CELLS, BLOCK, [0.0, 0.0], [H, H])
    model = L.ModelC(eps4, 3.19)
    model.anisotropy_tol = tol
    if form == "multi-grain":
        model.with_orientations()
    method = L.RungeKutta4() if form == "rk4" else L.EulerMaruyama(3)
    sim = L.Simulation(grid, L.FiniteVolume(tol=tol), model, method, sched, L.CudaAllocator("f64"))
    ref = orc.State(orc.Grid(CELLS, BLOCK, [0.0, 0.0], [H, H]), [1, 1, 0] if form == "multi-grain" else [1, 1])
    for f, a in enumerate(_fields(kind)):
        sim.state.upload(f, with_ghosts(a, 1))
        ref.set(f, with_ghosts(a, 1))
    if form == "multi-grain":
        theta = np.random.default_rng(1).uniform(0.0, 1.5, (4, 1, 1)) * np.ones(SHAPE)
        sim.state.upload("theta0", theta)
        model.set_orientations(sim.state)
        ref.set(2, theta)
    p = orc.modelc_params(eps4=eps4, lam=3.19, d_thermal=model.d_thermal, noise=0.0, tol=tol, flux_tol=tol)
    sim.run(dt, 1, variant=form if isinstance(form, int) else 0)
    if form == "rk4":
        ref.modelc_run_rk4(p, 0.0, dt, 1)
    elif form == "multi-grain":
        ref.modelc_run_oriented(p, 2, 0.0, dt, 3, 1, False)
    else:
        ref.modelc_run(p, 0.0, dt, 3, 1, False)
    for f in (0, 1):
        assert np.array_equal(_bits(sim.state.interior(f)), _bits(ref.interior(f))), kind
