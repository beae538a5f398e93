"""The ghost fill of a block of more than 2^28 ghost entries, whose numbers it
counts in 64 bits: a periodic plate one cell thick, compared on the device
(1.6 GB a buffer; needs a GPU)."""
import pytest

import legendre_b200 as L

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


class _Slab:
    def __init__(self, address, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(address, False), version=3)


def test_thin_plate(sched):
    n = 11600  # two ghost planes of 11602^2
    assert 2 * (n + 2) ** 2 > 1 << 28
    grid = L.CartesianGrid([n, n, 1], [n, n, 1], [0.0] * 3, [1.0] * 3).with_periodic([True, True, True])
    st = L.DeviceState(grid, sched, L.CudaAllocator("f32"), [L.FieldSpec("f", 1)])
    address, _ = st.slab_pointer(0, 0)
    slab = torch.as_tensor(_Slab(address, (3, n + 2, n + 2)), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    slab[1, 1:-1, 1:-1] = torch.rand((n, n), generator=gen, device="cuda")
    torch.cuda.synchronize()
    st.fill_ghosts(0)
    sched.sync()
    inner = slab[1, 1:-1, 1:-1]
    for z in range(3):
        assert torch.equal(slab[z, 1:-1, 1:-1], inner)
        assert torch.equal(slab[z, 1:-1, 0], inner[:, -1]) and torch.equal(slab[z, 1:-1, -1], inner[:, 0])
        assert torch.equal(slab[z, 0, 1:-1], inner[-1]) and torch.equal(slab[z, -1, 1:-1], inner[0])
        corners = [slab[z, j, i].item() for j in (0, -1) for i in (0, -1)]
        assert corners == [inner[j, i].item() for j in (-1, 0) for i in (-1, 0)]
    del slab, inner
    st._destroy()
