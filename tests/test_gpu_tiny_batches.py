"""Batches made of tiny meshes, whose slots do not fill warp tiles: every instance's
equilibrium and coupled solve as alone (psi within 1e-10 / 1e-9 V, the batches'
tolerances)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device(*shape):
    """A p-n diode along x with a contact at both ends."""
    import tcad_b200 as tb
    ax = [np.linspace(0.0, 2e-4 if a == 0 else 1e-4, n) for a, n in enumerate(shape)]
    dop = np.where(np.meshgrid(*ax[::-1], indexing="ij")[-1] < 1e-4, -1e17, 1e18)
    dev = (tb.Device2D if len(shape) == 2 else tb.Device3D)(
        (tb.Mesh2D if len(shape) == 2 else tb.Mesh3D)(*ax), dop)
    rest = [q.ravel() for q in np.meshgrid(*[np.arange(n) for n in shape[1:]], indexing="ij")]
    for name, i in (("anode", 0), ("cathode", shape[0] - 1)):
        dev.add_contact(name, np.full(rest[0].size, i), *rest)
    return dev


PACKS = [[(5, 3)] * 2, [(5, 3), (41, 21)], [(2, 2)] * 8, [(5, 5)] * 3, [(9, 7)] * 64,
         [(3, 3, 3)] * 3, [(5, 3), (3, 3), (5, 3)]]


@pytest.mark.parametrize("shapes", PACKS, ids=lambda q: f"{len(q)}x{q[0]}")
def test_tiny_batches_equal_alone(shapes):
    import tcad_b200 as tb
    from tcad_b200.batch import DeviceBatch
    opts = tb.NewtonOptions(precond="block_jacobi")
    b = DeviceBatch([_device(*s) for s in shapes])
    b.solve_equilibrium(opts)
    eq = [b.state(i)[0] for i in range(len(shapes))]
    res = b.solve_bias([{"anode": 0.05}] * len(shapes), opts)
    assert all(r["converged"] for r in res)
    for i, s in enumerate(shapes):
        dev = _device(*s)
        dev.solve_equilibrium(opts)
        assert np.abs(dev.psi - eq[i]).max() * dev.VT < 1e-10, s
        dev.solve_bias({"anode": 0.05}, opts)
        assert np.abs(dev.psi - b.state(i)[0]).max() * dev.VT < 1e-9, s


@pytest.mark.parametrize("n", [2, 18, 64, 400])
def test_clusters_with_empty_blocks_bit_identical_to_per_step(n):
    """Instances of 32 slots: of a cluster's eight CTAs (two of 64, one of 400) only the
    first has any, the others reach the first sum at once.  One block of slots, so the
    sums are the per-step kernels'."""
    from test_gpu_resident import _batch_solve, _batch_system
    pk = _batch_system([_device(8, 8)] * n)
    want = _batch_solve(pk, 1e-9, 200, 0)
    n0 = pk.lib.tcad_launch_count()
    for _ in range(20):
        got = _batch_solve(pk, 1e-9, 200, 1)
        assert got[1:] == want[1:]
        assert np.array_equal(got[0].cpu().numpy(), want[0].cpu().numpy())
    assert pk.lib.tcad_launch_count() - n0 == 40        # colour repack + the clusters
