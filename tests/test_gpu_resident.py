"""The resident single-launch solves (one CTA per SM, rows in shared memory,
vectors in registers) against the launch-per-step loops at the sizes where
their layout changes: a cluster of 8 or 16 CTAs and the whole grid, one and two
slots per thread, rows in shared memory and not, a last block of a few slots, odd
rows (pad slots), the smallest meshes.
Same bodies, scalar updates and order of sums: bit-identical."""
import numpy as np
import pytest

from test_gpu_redblack import _scaled_system, _solve_counted

pytestmark = pytest.mark.gpu

SIZES = [("diode", (2, 2)), ("diode", (21, 10)), ("diode", (126, 122)), ("diode", (129, 119)),
         ("trigate", (31, 22, 16)), ("trigate", (32, 22, 16)), ("mosfet", (301, 260)), ("mosfet", (385, 385)),
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


@pytest.mark.parametrize("kind,shape", SIZES + [("diode", (257, 254)), ("diode", (261, 252)),
                                                ("diode", (301, 511)), ("trigate", (96, 57, 40)),
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


def _batch_system(devs):
    """The block-scaled Newton systems of several devices in one pack, each
    at its bulk-guess state."""
    import torch
    from tcad_b200 import _lib
    from tcad_b200.pack import Pack
    pk = Pack([d.setup for d in devs])
    g = np.concatenate([d.setup.bulk_guess().ravel() for d in devs])
    ns = np.concatenate([d.setup.nie_s.ravel() for d in devs])
    for t, a in ((pk.psi, g), (pk.n, ns * np.exp(g)), (pk.p, ns * np.exp(-g))):
        t.copy_(torch.from_numpy(a))
    pk.set_bias()
    pk.assemble(_lib.MODE_ELIMINATE)
    st = torch.zeros(len(devs), dtype=torch.int32, device=pk.device)
    _lib.check(pk.lib.tcad_block_jacobi_setup_rel(pk.pref, _lib.ptr(pk.J), _lib.ptr(pk.F),
                                                  _lib.ptr(st), _lib.ptr(pk.n), _lib.ptr(pk.p),
                                                  1e-10, pk.sp()), "bj")
    assert not st.any()
    return pk


def _batch_solve(pk, rtol, maxit, fused):
    import ctypes
    import torch
    from tcad_b200 import _lib
    ni = len(pk.setups)
    x = torch.full_like(pk.du, float("nan"))
    it, st, rr = (ctypes.c_int32 * ni)(), (ctypes.c_int32 * ni)(), (ctypes.c_double * ni)()
    prev = pk.lib.tcad_set_krylov_fused(fused)
    try:
        _lib.check(pk.lib.tcad_block_krylov(pk.pref, _lib.ptr(pk.J), _lib.ptr(pk.F),
                                            _lib.ptr(x), 2, rtol, maxit, 0, _lib.ptr(pk.work),
                                            pk.work.numel(), it, st, rr, pk.sp()), "krylov")
    finally:
        pk.lib.tcad_set_krylov_fused(prev)
    torch.cuda.synchronize()
    return x, list(it), list(st), list(rr)


STREAMED = [[("trigate", (131, 80, 51))], [("mosfet", (801, 400))], [("trigate", (161, 97, 79))],
            [("trigate", (57, 45, 39)), ("trigate", (9, 7, 5)), ("trigate", (56, 48, 46))],
            [("diode", (401, 351)), ("diode", (21, 10)), ("diode", (300, 203))]]


@pytest.mark.parametrize("devs", STREAMED, ids=lambda d: "+".join(str(q[1]) for q in d))
def test_streamed_schur_solve_meets_the_full_systems_test(devs):
    """Packs of more blocks than SMs (J streamed through shared memory): one
    instance and ragged ones, odd rows, partial tiles and blocks."""
    import torch
    from tcad_b200 import _lib
    pk = _batch_system([_device(*d) for d in devs])
    rtol = 1e-9
    x, it, st, rr = _batch_solve(pk, rtol, 20000, 1)
    assert bool(x.isfinite().all())
    y = torch.empty_like(x)
    _lib.check(pk.lib.tcad_block_spmv(pk.pref, _lib.ptr(pk.J), _lib.ptr(x), _lib.ptr(y),
                                      pk.sp()), "spmv")
    r, b = (pk.F - y).view(3, -1), pk.F.view(3, -1)
    for i, s in enumerate(pk.setups):
        a = slice(int(pk.node_off[i]), int(pk.node_off[i]) + s.N)
        rel = float(torch.linalg.norm(r[:, a]) / torch.linalg.norm(b[:, a]))
        assert abs(rel - rr[i]) <= 1e-3 * rtol + 0.01 * rr[i], (rel, rr[i])
        if st[i] == _lib.TCAD_OK:          # block Jacobi stalls on some MOSFETs
            assert rel <= 1.01 * rtol
    x, it, st, rr = _batch_solve(pk, 1e-30, 17, 1)
    assert it == [17] * len(devs) and st == [_lib.TCAD_ERR_NOCONV] * len(devs)


@pytest.mark.parametrize("devs", [[("diode", (21, 10)), ("mosfet", (64, 41)), ("diode", (2, 2))],
                                  [("trigate", (9, 7, 5)), ("trigate", (24, 16, 13))],
                                  [("trigate", (9, 7, 5)), ("trigate", (40, 24, 22))]],
                         ids=lambda d: "+".join(str(q[1]) for q in d))
def test_cluster_batches_equal_alone(devs):
    """A cluster per instance (or, where one is too large for it, the per-step
    kernels): equilibrium and the coupled solve of every instance as alone."""
    import tcad_b200 as tb
    from tcad_b200.batch import DeviceBatch
    opts = tb.NewtonOptions(precond="block_jacobi")
    b = DeviceBatch([_device(*d) for d in devs])
    b.solve_equilibrium(opts)
    eq = [b.state(i)[0] for i in range(len(devs))]
    name = {"diode": "anode", "mosfet": "drain", "trigate": "drain"}
    res = b.solve_bias([{name[d[0]]: 0.05} for d in devs], opts)
    assert all(r["converged"] for r in res)
    for i, d in enumerate(devs):
        dev = _device(*d)
        dev.solve_equilibrium(opts)
        assert np.abs(dev.psi - eq[i]).max() * dev.VT < 1e-10, d
        dev.solve_bias({name[d[0]]: 0.05}, opts)
        assert np.abs(dev.psi - b.state(i)[0]).max() * dev.VT < 1e-9, d
