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


@pytest.mark.parametrize("kind,shape", SIZES + [("diode", (301, 511)), ("trigate", (96, 57, 40)),
                                                ("trigate", (131, 80, 50))])
def test_resident_equilibrium_bit_identical_to_per_step(kind, shape):
    """One to eight slots per thread; the whole equilibrium Newton."""
    res = []
    for fused in (0, 1):
        dev = _device(kind, shape)
        lib = dev.pack.lib
        prev = lib.tcad_set_krylov_fused(fused)
        try:
            n0 = lib.tcad_launch_count()
            dev.solve_equilibrium()
            eq = dev.last_equilibrium
            assert eq["converged"]
            res.append((dev.psi, dev.n, dev.p, eq["iters"], eq["krylov_iters"],
                        lib.tcad_launch_count() - n0))
        finally:
            lib.tcad_set_krylov_fused(prev)
    for a, b in zip(res[0][:5], res[1][:5]):
        assert np.array_equal(a, b)
    assert res[1][5] <= 3 * res[1][3] + 2 < res[0][5]   # assembly, solve, update per step


def test_resident_equilibrium_give_up_falls_back():
    dev = _device("diode", (21, 10))
    lib = dev.pack.lib
    dev.solve_equilibrium()
    want, g0 = dev.psi, lib.tcad_krylov_fused_gave_up()
    prev = lib.tcad_set_krylov_fused_test(1)
    try:
        import tcad_b200 as tb
        import warnings
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")     # one Newton step: not converged
            dev.solve_equilibrium(tb.NewtonOptions(max_iter=1))
        assert lib.tcad_krylov_fused_gave_up() == g0 + 1
    finally:
        lib.tcad_set_krylov_fused_test(prev)
    dev.solve_equilibrium()
    assert np.array_equal(dev.psi, want)
