"""A bulk copy that does not arrive: the bounded wait for it (1 s of device time) runs
out, the solve ends with TCAD_ERR_CUDA, and the next solve is as before."""
import pytest

pytestmark = pytest.mark.gpu


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
