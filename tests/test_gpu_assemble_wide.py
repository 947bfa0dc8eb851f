"""The 2D assembly with a thread per edge (up to a tile per SM) against the one with a
thread per node: a mesh by itself takes the first, as many copies of it in one pack as
exceed the SMs the second.  The same arithmetic on the same values: bit-identical.
Meshes smaller than a tile, of whole tiles and ragged."""
import numpy as np
import pytest

from test_gpu_resident import _device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape,copies", [("diode", (2, 2), 150), ("diode", (33, 9), 40),
                                               ("mosfet", (96, 48), 9), ("mosfet", (101, 60), 6)])
def test_wide_assembly_is_bit_identical(kind, shape, copies):
    import torch
    from tcad_b200.batch import DeviceBatch
    one = _device(kind, shape)
    many = DeviceBatch([_device(kind, shape) for _ in range(copies)]).pack
    pk = one.pack
    rng = np.random.default_rng(3)
    n = pk.N
    state = [rng.uniform(-20, 20, n), 10.0 ** rng.uniform(-12, 2, n), 10.0 ** rng.uniform(-12, 2, n)]
    for mode in (0, 1, 2):
        pk.assemble(mode, *[torch.tensor(v, device="cuda") for v in state])
        many.assemble(mode, *[torch.tensor(np.tile(v, copies), device="cuda") for v in state])
        for a, b in ((pk.F, many.F), (pk.J, many.J)):
            a = a.cpu().numpy().reshape(-1, 1, n)
            b = b.cpu().numpy().reshape(-1, copies, n)
            np.testing.assert_array_equal(b, np.broadcast_to(a, b.shape))
