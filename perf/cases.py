"""The measured work: what a user of this framework has it do.

Every case is one call (a ``run`` of a number of steps, or a gradient) through
the public classes, from a state in the middle of a run: grains that have
grown to different radii with the fluctuations the noise keeps up, a diffusing
field, a refined hierarchy.  Step counts are those between two looks at the
state.  ``exact`` repeats the uniform-grid and gradient cases with plain torch
in 64 bits.
"""
import math

import numpy as np
import torch

import legendre_b200 as L

H = 0.4                      # grid spacing of every Model C configuration
MASK = (1 << 64) - 1


def listed():
    return [
        # one interactive step of a small grid: the smallest call, all latency
        dict(name="model_c_step_64", kind="model_c", nx=64, ny=64, bx=32, by=32, dtype="f64", noise=0.01,
             steps=1, graph=False, method="em", orient=False, periodic=False),
        # a parameter study's grid: launches and a short critical path
        dict(name="model_c_512", kind="model_c", nx=512, ny=512, bx=64, by=64, dtype="f64", noise=0.01,
             steps=20, graph=True, method="em", orient=False, periodic=False),
        # the full-scale run: 101.6 million cells in 126^2 blocks
        dict(name="model_c_10080", kind="model_c", nx=10080, ny=10080, bx=126, by=126, dtype="f64", noise=0.01,
             steps=4, graph=True, method="em", orient=False, periodic=False),
        # single precision at 4096^2
        dict(name="model_c_4096_f32", kind="model_c", nx=4096, ny=4096, bx=256, by=256, dtype="f32", noise=0.01,
             steps=16, graph=True, method="em", orient=False, periodic=False),
        # deterministic, periodic, odd block widths, plain launches
        dict(name="model_c_ragged_quiet", kind="model_c", nx=2002, ny=2002, bx=91, by=77, dtype="f64", noise=0.0,
             steps=8, graph=False, method="em", orient=False, periodic=True),
        # many grains, each in its own crystal frame
        dict(name="model_c_grains_2520", kind="model_c", nx=2520, ny=2520, bx=126, by=126, dtype="f64", noise=0.02,
             steps=8, graph=True, method="em", orient=True, periodic=False),
        # fourth-order time steps
        dict(name="model_c_rk4_2048", kind="model_c", nx=2048, ny=2048, bx=128, by=128, dtype="f64", noise=0.0,
             steps=4, graph=True, method="rk4", orient=False, periodic=False),
        # 3-D heat: the cache-resident cube and the large one
        dict(name="heat_96", kind="heat", dim=3, nx=96, ny=96, nz=96, bx=16, by=16, bz=16, steps=50, graph=True,
             method="fe", periodic=True),
        dict(name="heat_512", kind="heat", dim=3, nx=512, ny=512, nz=512, bx=16, by=16, bz=16, steps=10, graph=True,
             method="fe", periodic=True),
        # a 2-D plate with insulated edges and odd blocks, fourth order
        dict(name="heat_plate_rk4", kind="heat", dim=2, nx=1425, ny=1001, nz=1, bx=75, by=77, bz=1, steps=10,
             graph=True, method="rk4", periodic=False),
        # adaptive refinement, one regrid per call, the hierarchy read back
        dict(name="amr_512", kind="amr", n=512, block=32, levels=3, radius=16.0, every=25, steps=25),
        # gradients of a batch of realisations against a target
        dict(name="gradient_32x128", kind="gradient", instances=32, n=128, block=64, dtype="f32", steps=200, ckpt=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model_c"] * 5 + ["heat"] * 3 + ["amr", "gradient"])
    if kind == "model_c":
        bx, by = _log_int(rng, 16, 256), _log_int(rng, 16, 256)
        if rng.random() < 0.4:
            bx = by = rng.choice([32, 64, 126, 128, 256])
        target = _log_int(rng, 4096, 40_000_000)
        side = math.sqrt(target)
        nbx, nby = max(1, round(side / bx)), max(1, round(side / by))
        method = "rk4" if rng.random() < 0.15 else "em"
        noise = 0.0 if method == "rk4" else rng.choice([0.0, 0.01, 0.01, 0.02])
        return dict(kind=kind, nx=nbx * bx, ny=nby * by, bx=bx, by=by, dtype=rng.choice(["f64", "f64", "f32"]),
                    noise=noise, steps=rng.randint(1, 20) if target < 4_000_000 else rng.randint(1, 6),
                    graph=rng.random() < 0.6, method=method, orient=rng.random() < 0.2 and target < 8_000_000,
                    periodic=rng.random() < 0.3)
    if kind == "heat":
        dim = 3 if rng.random() < 0.65 else 2
        if dim == 3:
            b = [rng.randint(8, 32) for _ in range(3)]
            if rng.random() < 0.5:
                b = [rng.choice([8, 16, 24, 32])] * 3
            side = _log_int(rng, 40, 400)
        else:
            b = [_log_int(rng, 16, 256), _log_int(rng, 16, 256), 1]
            side = _log_int(rng, 64, 4000)
        n = [max(1, round(side / v)) * v for v in b]
        if dim == 2:
            n[2] = 1
        return dict(kind=kind, dim=dim, nx=n[0], ny=n[1], nz=n[2], bx=b[0], by=b[1], bz=b[2],
                    steps=rng.randint(2, 40) if side < 200 else rng.randint(2, 10), graph=rng.random() < 0.6,
                    method=rng.choice(["fe", "fe", "rk4"]), periodic=rng.random() < 0.5)
    if kind == "amr":
        return dict(kind=kind, n=rng.choice([256, 384, 512]), block=rng.choice([16, 32]), levels=rng.randint(1, 3),
                    radius=round(rng.uniform(8.0, 20.0), 2), every=rng.choice([10, 25]), steps=rng.randint(10, 30))
    block = rng.choice([16, 24, 32, 48, 64])
    return dict(kind=kind, instances=rng.randint(4, 48), n=block * rng.randint(2, max(2, 144 // block)), block=block,
                dtype=rng.choice(["f32", "f64"]), steps=rng.randint(40, 160), ckpt=rng.choice([8, 10, 20]))


# ------------------------------------------------------------ device memory
class _Memory:
    """The device memory of a program, given back with its last holder."""

    def __init__(self, destroy):
        self.destroy = destroy

    def __del__(self):
        self.destroy()


class _Fields:
    """Torch views of the interiors of a device state, which they keep alive."""

    def __init__(self, sim, memory, names):
        self.sim, self.memory, self.names, self.views = sim, memory, names, {}

    def get(self):
        st = self.sim.state
        at, _ = st.slab_pointer(0, 0)
        got = self.views.get(at)
        if got is None:
            got = self.views[at] = {k: self._view(st, k) for k in self.names}
        return got

    def _view(self, st, name):
        size = 8 if st.alloc.dtype == "f64" else 4
        g = st.specs[st._index(name)].ghost
        p0, _ = st.slab_pointer(0, name)
        blocks = st.grid.num_blocks()
        stride = (st.slab_pointer(1, name)[0] - p0) if blocks > 1 else size
        n = st.grid.block_cells
        strides, offset, step = [], 0, size
        for d in range(len(n)):
            strides.append(step)
            offset += g * step
            step *= n[d] + 2 * g
        return torch.as_tensor(_Interface(self.memory, p0 + offset, (blocks,) + tuple(reversed(n)),
                                          (stride,) + tuple(reversed(strides)), "<f%d" % size), device="cuda")


class _Interface:
    def __init__(self, owner, address, shape, strides, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=kind, data=(address, False),
                                             version=3)


class _Program:
    """What a program keeps between calls."""

    def __init__(self, **kept):
        self.__dict__.update(kept)


_scheduler = None


def scheduler():
    global _scheduler
    if _scheduler is None:
        torch.zeros(1, device="cuda")
        _scheduler = L.CudaScheduler(0)
    return _scheduler


def blocked(a, block):
    """A global array (..., y, x) as the blocks in order, (blocks, ..., by, bx)."""
    if a.dim() == 2:
        (ny, nx), (bx, by) = a.shape, block
        return a.view(ny // by, by, nx // bx, bx).permute(0, 2, 1, 3).reshape(-1, by, bx)
    (nz, ny, nx), (bx, by, bz) = a.shape, block
    return a.view(nz // bz, bz, ny // by, by, nx // bx, bx).permute(0, 2, 4, 1, 3, 5).reshape(-1, bz, by, bx)


# ------------------------------------------------------------ initial states
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _grains(nx, ny, seed, instances=1):
    """Positions, radii and orientations of one grain per 10^5 cells."""
    rs = np.random.RandomState((int(seed) * 9973 + nx) % (1 << 31))
    n = max(1, nx * ny // 100_000)
    r = rs.uniform(4.0, 20.0, n) if n > 1 else np.array([0.15 * H * min(nx, ny)])
    return np.stack([rs.uniform(0, H * nx, n), rs.uniform(0, H * ny, n), r, rs.uniform(0, math.pi / 2, n)], 1)


def _grown(nx, ny, grains, u0, noise, gen):
    """phi and u (ny, nx): tanh fronts, the solid near its melting point, and the
    fluctuations that the noise keeps up around both wells."""
    phi = torch.full((ny, nx), -1.0, dtype=torch.float64, device="cuda")
    for cx, cy, r, _ in grains:
        reach = r + 27.0
        i0, i1 = max(0, int((cx - reach) / H)), min(nx, int((cx + reach) / H) + 2)
        j0, j1 = max(0, int((cy - reach) / H)), min(ny, int((cy + reach) / H) + 2)
        x = (torch.arange(i0, i1, dtype=torch.float64, device="cuda") + 0.5) * H - cx
        y = (torch.arange(j0, j1, dtype=torch.float64, device="cuda") + 0.5) * H - cy
        d = torch.sqrt(x[None, :] ** 2 + y[:, None] ** 2)
        w = phi[j0:j1, i0:i1]
        w.copy_(torch.maximum(w, -torch.tanh((d - r) / math.sqrt(2.0))))
    u = -u0 * (0.5 - 0.5 * phi)
    if noise:
        phi += 0.14 * noise * torch.randn(ny, nx, dtype=torch.float64, device="cuda", generator=gen)
    return phi, u


def _model(case):
    model = L.ModelC(0.05, 2.0 / 0.6267, case["noise"])
    model.d_thermal = 2.0
    return model


def _orientation(nx, ny, grains):
    """theta0 of every cell: the nearest grain's."""
    best = torch.full((ny, nx), float("inf"), dtype=torch.float64, device="cuda")
    theta = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")
    x = (torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5) * H
    y = (torch.arange(ny, dtype=torch.float64, device="cuda") + 0.5) * H
    for cx, cy, _, th in grains:
        d = (x[None, :] - cx) ** 2 + (y[:, None] - cy) ** 2
        near = d < best
        best = torch.where(near, d, best)
        theta = torch.where(near, torch.full_like(theta, th), theta)
    return theta


def _model_c_inputs(case, seed):
    grains = _grains(case["nx"], case["ny"], seed)
    phi, u = _grown(case["nx"], case["ny"], grains, 0.55, case["noise"], _generator(seed))
    theta = _orientation(case["nx"], case["ny"], grains) if case["orient"] else None
    kind = torch.float64 if case["dtype"] == "f64" else torch.float32
    block = (case["bx"], case["by"])
    return [None if a is None else blocked(a, block).to(kind) for a in (phi, u, theta)]


def _heat_input(case, seed):
    n, b = _extent(case)
    g = [(torch.arange(v, dtype=torch.float64, device="cuda") + 0.5) / v for v in n]
    out = torch.ones(tuple(reversed(n)), dtype=torch.float64, device="cuda")
    for d, x in enumerate(g):
        shape = [1] * len(n)
        shape[len(n) - 1 - d] = n[d]
        out *= torch.cos(2 * math.pi * x + 0.1 * (d + 1)).view(shape)
    out += 1e-3 * (2.0 * torch.rand(out.shape, dtype=torch.float64, device="cuda", generator=_generator(seed)) - 1.0)
    return blocked(out, b)


def _extent(case):
    if case["dim"] == 2:
        return (case["nx"], case["ny"]), (case["bx"], case["by"])
    return (case["nx"], case["ny"], case["nz"]), (case["bx"], case["by"], case["bz"])


def _gradient_inputs(case, seed):
    n, m = case["n"], case["instances"]
    rs = np.random.RandomState(seed % (1 << 31))
    eps4, delta = rs.uniform(0.02, 0.07, m), rs.uniform(0.45, 0.65, m)
    x = (np.arange(n) + 0.5) * H - 0.5 * n * H
    d = np.sqrt(x[None, :] ** 2 + x[:, None] ** 2)
    r = rs.uniform(0.12, 0.2, m) * n * H
    phi = -np.tanh((d[None] - r[:, None, None]) / math.sqrt(2.0))
    u = np.repeat(-delta, n * n).reshape(m, n, n)
    target = -np.tanh((d[None] - 1.1 * r[:, None, None]) / math.sqrt(2.0))
    return eps4, [int(s) for s in rs.randint(1, 1 << 31, m)], phi, u, target


GRADIENT_NOISE, GRADIENT_DT, MODEL_DT = 0.005, 0.008, 0.008


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind, sched = case["kind"], scheduler()
    if kind == "model_c":
        grid = L.CartesianGrid([case["nx"], case["ny"]], [case["bx"], case["by"]], [0.0, 0.0], [H, H])
        if case["periodic"]:
            grid = grid.with_periodic([True, False])
        model = _model(case)
        if case["orient"]:
            model.with_orientations()
        step = L.RungeKutta4() if case["method"] == "rk4" else L.EulerMaruyama(seed & MASK)
        sim = L.Simulation(grid, L.FiniteVolume(), model, step, sched, L.CudaAllocator(case["dtype"]))
        names = ["phi", "u"]
        memory = _Memory(sim.state._destroy)
        views = _Fields(sim, memory, names + (["theta0"] if case["orient"] else []))
        for name, a in zip(["phi", "u", "theta0"], _model_c_inputs(case, seed)):
            if a is not None:
                views.get()[name].copy_(a)
        torch.cuda.synchronize()
        if case["orient"]:
            model.set_orientations(sim.state)
        return _Program(sim=sim, fields=_Fields(sim, memory, names), dt=MODEL_DT, steps=case["steps"],
                        graph=case["graph"], kind="grid")
    if kind == "heat":
        n, b = _extent(case)
        h = 1.0 / max(n)
        grid = L.CartesianGrid(n, b, [0.0] * len(n), [h] * len(n))
        if case["periodic"]:
            grid = grid.with_periodic([True] * len(n))
        step = L.RungeKutta4() if case["method"] == "rk4" else L.ForwardEuler()
        sim = L.Simulation(grid, L.FiniteDifference(), L.Heat(1.0), step, sched, L.CudaAllocator("f64"))
        views = _Fields(sim, _Memory(sim.state._destroy), ["u"])
        views.get()["u"].copy_(_heat_input(case, seed))
        torch.cuda.synchronize()
        return _Program(sim=sim, fields=views, dt=0.15 * h * h, steps=case["steps"], graph=case["graph"],
                        kind="grid")
    if kind == "amr":
        n, b = case["n"], case["block"]
        base = L.CartesianGrid([n, n], [b, b], [0.0, 0.0], [H, H])
        model = _model(dict(noise=0.0))
        adapt = L.BergerOliger(L.GradientTagger("phi", 0.05),
                               L.RegridPolicy(case["every"], 2, L.ClusterParams(0.8, 4)))
        sim = L.AmrSimulation(L.AmrGrid.from_patches(base, [2] * case["levels"], []), L.FiniteVolume(), model,
                              L.Subcycling(0), sched, L.CudaAllocator("f64"), adapt)
        rs = np.random.RandomState(seed % (1 << 31))
        c = (0.5 + rs.uniform(-0.1, 0.1, 2)) * n * H
        for f in ("phi", "u"):
            slabs = []
            for k in range(sim.num_blocks):
                x, y = sim.centers(k)
                phi = np.full((b + 2, b + 2), -1.0)
                phi[1:-1, 1:-1] = -np.tanh((np.hypot(x - c[0], y - c[1]) - case["radius"]) / math.sqrt(2.0))
                slabs.append(phi if f == "phi" else -0.55 * (0.5 - 0.5 * phi))
            sim.set(f, slabs)
        dt = sim.stable_dt()
        sim.run(dt, case["every"] * case["levels"] + 1, graph=True)  # each regrid adds a level around the front
        # the buffers that the hierarchy is read into: base blocks, then patches
        room = n * n + 4 * sum(_front_cells(case, level) for level in range(1, case["levels"] + 1))
        return _Program(sim=sim, dt=dt, steps=case["steps"], memory=_Memory(sim._destroy), kind="amr",
                        read={f: np.zeros(room) for f in ("phi", "u")})
    eps4, seeds, phi, u, target = _gradient_inputs(case, seed)
    grid = L.CartesianGrid([case["n"]] * 2, [case["block"]] * 2, [0.0, 0.0], [H, H])
    ens = L.Ensemble(grid, _model(dict(noise=GRADIENT_NOISE)), eps4, seeds, sched, dtype=case["dtype"])
    ens.set("phi", phi)
    ens.set("u", u)
    return _Program(ens=ens, target=target, steps=case["steps"], ckpt=case["ckpt"],
                    memory=_Memory(ens._destroy), kind="gradient")


# ---------------------------------------------------------------------- run
def run(p):
    if p.kind == "grid":
        p.sim.run(p.dt, p.steps, graph=p.graph)
        return p.fields.get()
    if p.kind == "amr":
        p.sim.run(p.dt, p.steps, graph=True)
        for f, room in p.read.items():
            at = 0
            for a in p.sim.get(f):
                cells = (a.shape[0] - 2) * (a.shape[1] - 2)
                room[at:at + cells].reshape(a.shape[0] - 2, -1)[:] = a[1:-1, 1:-1]
                at += cells
            room[at:] = 0.0
        return p.read
    return p.ens.value_and_grad(GRADIENT_DT, p.steps, p.ckpt, p.target)


# --------------------------------------------------------------------- work
def _front_cells(case, level):
    """Cells of a refined level: the band around the front that the tagger and
    its buffer cover."""
    return int(2 * math.pi * case["radius"] / H * 2 ** level * 24)


def work(case):
    """Each pass reads its state once and writes it once; operations are counted
    per cell and step (additions, multiplications, divisions, roots and
    transcendentals one each)."""
    if case["kind"] == "model_c":
        cells, size = case["nx"] * case["ny"], 8 if case["dtype"] == "f64" else 4
        drift = 118 + (90 if case["orient"] else 0)
        per_step = 4 * (drift + 5) if case["method"] == "rk4" else drift + 4 + (12 if case["noise"] else 0)
        return {"bytes": cells * size * (4 + (1 if case["orient"] else 0)), "flops": cells * case["steps"] * per_step}
    if case["kind"] == "heat":
        cells = case["nx"] * case["ny"] * case["nz"]
        drift = 5 * case["dim"] + 1
        return {"bytes": cells * 16, "flops": cells * case["steps"] * (4 * (drift + 4) if case["method"] == "rk4" else drift + 2)}
    if case["kind"] == "amr":
        cells, steps = case["n"] ** 2, case["n"] ** 2 * case["steps"]
        for level in range(1, case["levels"] + 1):
            band = _front_cells(case, level)
            cells += band
            steps += band * case["steps"] * 2 ** level
        return {"bytes": cells * 32, "flops": steps * 122}
    cells, size = case["instances"] * case["n"] ** 2, 8 if case["dtype"] == "f64" else 4
    return {"bytes": cells * (4 * size + 3 * 8), "flops": cells * case["steps"] * (122 + 400)}


# -------------------------------------------------------------------- exact
def _signed(v):
    v &= MASK
    return v - (1 << 64) if v >> 63 else v


def _mix(z):
    """SplitMix64 of an int64 tensor."""
    def shifted(a, k):
        return (a >> k) & ((1 << (64 - k)) - 1)
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ shifted(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ shifted(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ shifted(z, 31)


def _normals(seed, t, blocks, by, bx):
    """The Wiener increments' Gaussians of one step, (blocks, by, bx)."""
    salt = int(np.float64(t).view(np.int64))
    s = torch.tensor([_signed(seed)], dtype=torch.int64, device="cuda")
    s = _mix(_mix(_mix(s) ^ salt) ^ (1 << 32))
    key = _mix(s ^ torch.arange(blocks, dtype=torch.int64, device="cuda"))
    cell = torch.arange(by * bx, dtype=torch.int64, device="cuda")
    a = _mix(_mix(key[:, None] ^ cell[None, :]))
    b = _mix(a ^ _signed(0xD1B54A32D192ED03))
    uniform = lambda v: (((v >> 11) & ((1 << 53) - 1)) + 1).double() * 2.0 ** -53  # noqa: E731
    r = torch.sqrt(-2.0 * torch.log(uniform(a))) * torch.cos(2 * math.pi * uniform(b))
    return r.view(blocks, by, bx)


def _padded(a, periodic_x):
    """(..., ny, nx) with one ghost cell around: wrapped or mirrored in x, mirrored in y."""
    left, right = (a[..., -1:], a[..., :1]) if periodic_x else (a[..., :1], a[..., -1:])
    a = torch.cat([left, a, right], -1)
    return torch.cat([a[..., :1, :], a, a[..., -1:, :]], -2)


def _anisotropy(dx, dy, eps4, tol=1e-8):
    a_bar = 1.0 - 3.0 * eps4
    x2, y2 = dx * dx, dy * dy
    mag = (x2 + y2) ** 2
    flat = mag <= tol
    safe = torch.where(flat, torch.ones_like(mag), mag)
    a = torch.where(flat, a_bar + 0.0 * mag, a_bar + 3.0 * eps4 * (x2 * x2 + y2 * y2) / safe)
    da = torch.where(flat, 0.0 * mag, -12.0 * eps4 * dx * dy * (x2 - y2) / safe)
    return a, da


def _drift(phi, u, eps4, lam, d_thermal, periodic_x, trig):
    p, w = _padded(phi, periodic_x), _padded(u, periodic_x)
    at = lambda q, i, j: q[..., 1 + j:q.shape[-2] - 1 + j, 1 + i:q.shape[-1] - 1 + i]  # noqa: E731
    P = lambda i, j: at(p, i, j)  # noqa: E731
    c, s = trig if trig is not None else (None, None)

    def face(dx, dy, along_x):
        a, da = _anisotropy(dx, dy, eps4) if trig is None else _anisotropy(c * dx + s * dy, c * dy - s * dx, eps4)
        return a * (a * dx - da * dy) if along_x else a * (a * dy + da * dx)

    def x_face(i):
        return face(P(i + 1, 0) - P(i, 0), 0.25 * (P(i + 1, 1) - P(i + 1, -1) + P(i, 1) - P(i, -1)), True)

    def y_face(j):
        return face(0.25 * (P(1, j + 1) - P(-1, j + 1) + P(1, j) - P(-1, j)), P(0, j + 1) - P(0, j), False)

    flux = (x_face(0) - x_face(-1) + y_face(0) - y_face(-1)) / (H * H)
    dx, dy = 0.5 * (P(1, 0) - P(-1, 0)), 0.5 * (P(0, 1) - P(0, -1))
    a, _ = _anisotropy(dx, dy, eps4) if trig is None else _anisotropy(c * dx + s * dy, c * dy - s * dx, eps4)
    k_phi = (flux + phi - phi ** 3 - lam * u * (1 - phi * phi) ** 2) / (a * a)
    lap = (at(w, 1, 0) + at(w, -1, 0) + at(w, 0, 1) + at(w, 0, -1) - 4.0 * u) / (H * H)
    return k_phi, d_thermal * lap + 0.5 * k_phi


def _global(a, nx, ny):
    by, bx = a.shape[-2:]
    return a.view(ny // by, nx // bx, by, bx).permute(0, 2, 1, 3).reshape(ny, nx)


def _exact_model_c(case, seed):
    nx, ny, bx, by = case["nx"], case["ny"], case["bx"], case["by"]
    phi, u, theta = [None if a is None else _global(a.double(), nx, ny) for a in _model_c_inputs(case, seed)]
    trig = None if theta is None else (torch.cos(theta), torch.sin(theta))
    dt, t, lam = MODEL_DT, 0.0, 2.0 / 0.6267
    f = lambda p, w: _drift(p, w, 0.05, lam, 2.0, case["periodic"], trig)  # noqa: E731
    for _ in range(case["steps"]):
        k = f(phi, u)
        if case["method"] == "rk4":
            k2 = f(phi + 0.5 * dt * k[0], u + 0.5 * dt * k[1])
            k3 = f(phi + 0.5 * dt * k2[0], u + 0.5 * dt * k2[1])
            k4 = f(phi + dt * k3[0], u + dt * k3[1])
            phi, u = (q + dt / 6 * (a + 2 * b + 2 * c + d) for q, a, b, c, d in zip((phi, u), k, k2, k3, k4))
        else:
            phi, u = phi + dt * k[0], u + dt * k[1]
            if case["noise"]:
                n = _normals(seed, t, (nx // bx) * (ny // by), by, bx)
                phi = phi + math.sqrt(dt) * case["noise"] * _global(n, nx, ny)
        t += dt
    return {"phi": blocked(phi, (bx, by)), "u": blocked(u, (bx, by))}


def _exact_heat(case, seed):
    n, b = _extent(case)
    u = _heat_input(case, seed)
    nb = [v // w for v, w in zip(n, b)]
    shape = list(reversed(nb)) + list(reversed(b))
    order = [v for d in range(len(n)) for v in (d, d + len(n))]
    u = u.view(shape).permute(order).reshape(tuple(reversed(n)))
    h = 1.0 / max(n)
    dt = 0.15 * h * h

    def f(a):
        out = 0.0
        for d in range(a.dim()):
            size = a.shape[d]
            if case["periodic"]:
                lo, hi = a.narrow(d, size - 1, 1), a.narrow(d, 0, 1)
            else:
                lo, hi = a.narrow(d, 0, 1), a.narrow(d, size - 1, 1)
            w = torch.cat([lo, a, hi], d)
            out = out + (w.narrow(d, 2, size) - 2.0 * a + w.narrow(d, 0, size))
        return out / (h * h)

    for _ in range(case["steps"]):
        k1 = f(u)
        if case["method"] == "rk4":
            k2 = f(u + 0.5 * dt * k1)
            k3 = f(u + 0.5 * dt * k2)
            u = u + dt / 6 * (k1 + 2 * k2 + 2 * k3 + f(u + dt * k3))
        else:
            u = u + dt * k1
    return {"u": blocked(u.contiguous(), b)}


def _exact_gradient(case, seed):
    from torch.utils.checkpoint import checkpoint

    eps4, seeds, phi, u, target = _gradient_inputs(case, seed)
    m, n, b = case["instances"], case["n"], case["block"]
    kind = torch.float64 if case["dtype"] == "f64" else torch.float32
    leaf = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda").requires_grad_()  # noqa: E731
    column = lambda v: v.view(m, 1, 1)  # noqa: E731
    e, lam, d = leaf(eps4), leaf(np.full(m, 2.0 / 0.6267)), leaf(np.full(m, 2.0))
    p0, u0 = (torch.tensor(v, device="cuda").to(kind).double().requires_grad_() for v in (phi, u))
    dt, blocks = GRADIENT_DT, (n // b) ** 2

    def noise(t):
        every = [_global(_normals(s, t, blocks, b, b), n, n) for s in seeds]
        return math.sqrt(dt) * GRADIENT_NOISE * torch.stack(every)

    def stretch(p, w, e, lam, d, t, k):
        for _ in range(k):
            kp, ku = _drift(p, w, column(e), column(lam), column(d), False, None)
            p, w = p + dt * kp + noise(t), w + dt * ku
            t += dt
        return p, w

    p, w, t, left = p0, u0, 0.0, case["steps"]
    while left:
        k = min(10, left)
        p, w = checkpoint(stretch, p, w, e, lam, d, t, k, use_reentrant=False)
        for _ in range(k):
            t += dt
        left -= k
    loss = ((p - torch.tensor(target, device="cuda")) ** 2).sum((1, 2))
    loss.sum().backward()
    return {"loss": loss.detach(), "lambda": lam.grad, "d_thermal": d.grad, "eps4": e.grad,
            "delta": -u0.grad.sum((1, 2)), "phi0": p0.grad, "u0": u0.grad}


def exact(case, seed):
    if case["kind"] == "model_c":
        return _exact_model_c(case, seed)
    if case["kind"] == "heat":
        return _exact_heat(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    return None
