"""The marching heat kernel with 64-bit column offsets and coordinates (a layer
of blocks of more than 2^28 entries): forward Euler, double and single steps,
and RungeKutta4 against the same operations in torch on the device, bit for
bit; and 1-D grids, which have kernels of their own, against the oracle (2.2 GB
a buffer; needs a GPU)."""
import numpy as np
import pytest

import legendre_b200 as L
from util import with_ghosts

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

KAPPA, H = 0.7, 0.1


class _Arena:
    def __init__(self, address, shape, strides):
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr="<f8", data=(address, False),
                                             version=3)


def _global(sim, cells, block):
    """The field as one array (z,) y, x: a view of the blocks' interiors, permuted."""
    D = len(cells)
    nb = [c // b for c, b in zip(cells, block)]
    address, _ = sim.state.slab_pointer(0, 0)
    strides, step = [], 8
    for b in block:
        strides.append(step)
        step *= b + 2
    step = sim.state.slab_pointer(1, 0)[0] - address  # slabs are padded
    for n in nb:
        strides.append(step)
        step *= n
    shape = tuple(reversed(nb)) + tuple(b + 2 for b in reversed(block))
    slabs = torch.as_tensor(_Arena(address, shape, tuple(reversed(strides))), device="cuda")
    for d in range(D):
        slabs = slabs.narrow(D + d, 1, block[D - 1 - d])
    return slabs.permute([v for d in range(D) for v in (d, d + D)])


def _drift(u, periodic):
    """kappa lap(u), dimension 0 (the last axis) first, each operation rounded."""
    acc = torch.zeros_like(u)
    ih = 1.0 / (H * H)
    twice = u + u
    for d, wrap in enumerate(periodic):
        axis = u.dim() - 1 - d
        n = u.shape[axis]
        lo = u.narrow(axis, n - 1, 1) if wrap else u.narrow(axis, 0, 1)
        hi = u.narrow(axis, 0, 1) if wrap else u.narrow(axis, n - 1, 1)
        up = torch.cat([u.narrow(axis, 1, n - 1), hi], axis)
        down = torch.cat([lo, u.narrow(axis, 0, n - 1)], axis)
        acc += ((up - twice) + down) * ih
    return acc * KAPPA


@pytest.mark.parametrize("cells,block,periodic", [
    ([16416, 16401], [8208, 16401], [False, True]),
    ([3520, 3520, 16], [20, 20, 16], [True, False, False]),
])
@pytest.mark.parametrize("method", ["euler", "rk4"])
def test_large_layer(sched, cells, block, periodic, method):
    D, dt = len(cells), 0.0009
    layer = np.prod([b + 2 for b in block]) * np.prod([c // b for c, b in zip(cells[:-1], block[:-1])])
    assert layer >= 1 << 28
    grid = L.CartesianGrid(cells, block, [0.0] * D, [H] * D).with_periodic(periodic)
    sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(KAPPA),
                       L.ForwardEuler() if method == "euler" else L.RungeKutta4(), sched, L.CudaAllocator("f64"))
    gen = torch.Generator(device="cuda").manual_seed(5)
    shape = tuple(reversed(cells))
    u = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
    view = _global(sim, cells, block)
    view.copy_(u.view(view.shape))
    torch.cuda.synchronize()
    sim.state.fill_ghosts(0)
    steps = 3 if method == "euler" else 1
    sim.run(dt, steps)
    sched.sync()
    for _ in range(steps):
        k = _drift(u, periodic)
        if method == "euler":
            u = u + dt * k
            continue
        acc = u + dt / 6.0 * k
        for c, s in ((0.5 * dt, dt / 3.0), (0.5 * dt, dt / 3.0), (dt, dt / 6.0)):
            k = _drift(u + c * k, periodic)
            acc = acc + s * k
        u = acc
    view = _global(sim, cells, block)
    assert torch.equal(view.reshape(shape), u)
    sim.state._destroy()


@pytest.mark.parametrize("cells,block,periodic", [([7], [7], [True]), ([600], [300], [False]), ([1024], [8], [True])])
@pytest.mark.parametrize("method", ["euler", "rk4"])
def test_one_dimension(sched, orc, cells, block, periodic, method):
    grid = L.CartesianGrid(cells, block, [0.0], [H]).with_periodic(periodic)
    sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(KAPPA),
                       L.ForwardEuler() if method == "euler" else L.RungeKutta4(), sched, L.CudaAllocator("f64"))
    ref = orc.State(orc.Grid(cells, block, [0.0], [H], periodic), [1])
    u0 = with_ghosts(np.random.default_rng(5).standard_normal((grid.num_blocks(), block[0])), 1)
    sim.state.upload("u", u0)
    ref.set(0, u0)
    sim.run(0.0009, 5, graph=True)
    (ref.heat_run if method == "euler" else ref.heat_run_rk4)(0, KAPPA, 0.0, 0.0009, 5)
    assert np.array_equal(sim.state.interior("u"), ref.interior(0))
