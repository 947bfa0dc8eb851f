"""A bulk copy that does not arrive: the bounded wait for it (1 s of device time) runs
out, the solve ends with TCAD_ERR_CUDA whichever pass and instance it was for, and the
next solve is as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _streamed_pack():
    """A pack of more blocks than SMs, streamed: the first instance is the small one."""
    from test_gpu_resident import _batch_system, _device
    return _batch_system([_device("diode", (21, 10)), _device("diode", (401, 351)),
                          _device("diode", (300, 203))])


@pytest.mark.parametrize("hold", [2, 3])
def test_streamed_solve_reports_a_lost_copy(hold):
    from test_gpu_resident import _batch_solve
    pk = _streamed_pack()
    want = _batch_solve(pk, 1e-6, 2000, 1)
    prev = pk.lib.tcad_set_krylov_fused_test(hold)
    try:
        with pytest.raises(RuntimeError, match="CUDA"):
            _batch_solve(pk, 1e-6, 2000, 1)
    finally:
        pk.lib.tcad_set_krylov_fused_test(prev)
    got = _batch_solve(pk, 1e-6, 2000, 1)
    assert got[1:] == want[1:] and np.array_equal(got[0].cpu().numpy(), want[0].cpu().numpy())


def test_ilu_sweep_reports_a_lost_copy():
    import tcad_b200 as tb
    from tcad_b200.batch import DeviceBatch
    from test_gpu_batch import PARAMS, _build
    b = DeviceBatch([_build(q) for q in PARAMS[:2]])
    b.solve_equilibrium()
    lib = b.pack.lib
    prev = lib.tcad_set_krylov_fused_test(3)
    try:
        with pytest.raises(RuntimeError, match="CUDA"):
            b.solve_bias([{"gate": 0.2}] * 2, tb.NewtonOptions())
    finally:
        lib.tcad_set_krylov_fused_test(prev)
    b.solve_equilibrium()
    assert all(r["converged"] for r in b.solve_bias([{"gate": 0.2}] * 2, tb.NewtonOptions()))
