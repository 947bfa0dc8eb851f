"""The resident single-launch solves (one CTA per SM, rows in shared memory,
vectors in registers) against the launch-per-step loops at the sizes where
their layout changes: one and two slots per thread, rows in shared memory and
not, a last block of a few slots, odd rows (pad slots), the smallest meshes.
Same bodies, scalar updates and order of sums: bit-identical."""
import numpy as np
import pytest

from test_gpu_redblack import _scaled_system, _solve_counted

pytestmark = pytest.mark.gpu

SIZES = [("diode", (2, 2)), ("diode", (21, 10)), ("mosfet", (301, 260)), ("mosfet", (385, 385)),
         ("trigate", (9, 7, 5)), ("trigate", (57, 45, 39)), ("trigate", (56, 48, 46))]


def _device(kind, shape):
    import tcad_b200 as tb
    from tcad_b200 import workloads as W
    if kind == "diode":
        x = np.linspace(0.0, 2e-4, shape[0])
        y = np.linspace(0.0, 1e-4, shape[1])
        dev = tb.Device2D(tb.Mesh2D(x, y), np.where(np.meshgrid(x, y)[0] < 1e-4, -1e17, 1e18))
        dev.add_contact("anode", np.zeros(shape[1], int), np.arange(shape[1]))
        return dev
    if kind == "mosfet":
        return W.mosfet2d(tb.Device2D, *shape)
    return W.trigate3d(tb.Device3D, *shape)


@pytest.mark.parametrize("kind,shape", SIZES)
def test_resident_schur_solve_bit_identical_to_per_step(kind, shape):
    pk = _scaled_system(_device(kind, shape))
    for rtol, maxit in ((1e-6, 400), (1e-30, 25)):
        xa, ita, sta, rra, na = _solve_counted(pk, 2, rtol, maxit, fused=False)
        xb, itb, stb, rrb, nb = _solve_counted(pk, 2, rtol, maxit, fused=True)
        assert (ita, sta, rra) == (itb, stb, rrb)
        assert np.array_equal(xa.cpu().numpy(), xb.cpu().numpy())
        assert nb == 2 and na > 2           # colour repack + the single launch
