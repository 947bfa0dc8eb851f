"""The slot-order ILU(0) factor and sweeps that a batch's Newton solves run on
(tests/test_gpu_ilu.py checks the node-order ones): one BiCGStab iteration's
preconditioner is the same as the node-order factor's up to its FP32 records,
so Newton takes every device of a ragged batch to the state that node-block
Jacobi alone reaches -- shorter sides of 2, of 32 and 33 rows (one warp and a
row more), of 256 (the most) and along either axis."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [[(2, 40), (40, 2)], [(33, 40), (40, 32), (3, 3)], [(64, 65), (65, 64), (31, 90)],
          [(300, 256), (12, 10)]]


def _device(nx, ny):
    import tcad_b200 as tb
    x, y = np.linspace(0.0, 2e-5, nx), np.linspace(0.0, 1e-5, ny)
    dev = tb.Device2D(tb.Mesh2D(x, y), np.where(np.meshgrid(x, y)[0] < 1e-5, -1e17, 1e17))
    dev.add_contact("anode", np.zeros(ny, int), np.arange(ny))
    dev.add_contact("cathode", np.full(ny, nx - 1), np.arange(ny))
    return dev


@pytest.mark.parametrize("shapes", SHAPES, ids=str)
def test_ilu_batch_lands_on_the_block_jacobi_state(shapes):
    import tcad_b200 as tb
    from tcad_b200.batch import DeviceBatch
    states, its = [], []
    for precond in ("ilu", "block_jacobi"):
        b = DeviceBatch([_device(*s) for s in shapes])
        opts = tb.NewtonOptions(precond=precond, linsolve_maxiter=20000)
        b.solve_equilibrium(opts)
        for v in (0.2, 0.4):
            res = b.solve_bias([{"anode": v}] * len(shapes), opts)
            assert all(r["converged"] for r in res), precond
        its.append([r["krylov_iters"] for r in res])
        states.append([b.state(i) for i in range(len(shapes))])
    for i, (a, c) in enumerate(zip(*states)):
        VT = b.devices[i].VT
        assert np.abs(a[0] - c[0]).max() * VT < 1e-9, shapes[i]
        for u, w in zip(a[1:], c[1:]):
            assert np.abs(np.log(u / w)).max() * VT < 1e-8, shapes[i]
    # and it is the better preconditioner (2 x 40: contact nodes only, no iterations)
    assert all(a < c or a == c == 0 for a, c in zip(*its))
