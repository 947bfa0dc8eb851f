"""A GMRES cycle in one cooperative launch against the launch-per-step cycle at the sizes
where its layout changes: less than a CTA's 252 rows, one past it, the most rows it
takes and one more (which go step by step), a last CTA of one block; cycles of one, a few and
the most columns; no, 1 x 1, 3 x 3 and 6 x 6 blocks.  Both stop at ||r|| <= 1e-12 ||b|| with
||A^-1|| <= 1, so they differ by at most 2e-12 ||b||.  A launch that gives up is run again
step by step: the same bits as without it."""
import numpy as np
import pytest

from test_gpu_csr import _system

pytestmark = pytest.mark.gpu


def _solve(A, b, fused, **kw):
    from tcad_b200 import _lib
    from tcad_b200.linsolve import solve_linear
    lib = _lib.load()
    prev = lib.tcad_set_krylov_fused(fused)
    try:
        n0 = lib.tcad_launch_count()
        x, info = solve_linear(A, b, method="gmres", rtol=1e-12, **kw)
        return x, info["iterations"], lib.tcad_launch_count() - n0
    finally:
        lib.tcad_set_krylov_fused(prev)


@pytest.mark.parametrize("n,bs,restart", [(2, None, None), (251, None, None), (252, 3, None),
                                          (253, None, 3), (258, 6, None), (504, 6, 1000),
                                          (757, None, 1), (37296, 6, None), (37296, 3, 5),
                                          (37297, None, None), (2000, None, 1001)])
def test_gmres_cycle_matches_steps(n, bs, restart):
    A, b = _system(n, 1)
    kw = dict(block_size=bs, maxiter=2000, **({} if restart is None else dict(restart=restart)))
    xa, ia, na = _solve(A, b, 0, **kw)
    xb, ib, nb = _solve(A, b, 1, **kw)
    assert np.linalg.norm(A @ xb - b) <= 1.01e-12 * np.linalg.norm(b)
    assert np.linalg.norm(xa - xb) <= 2.02e-12 * np.linalg.norm(b)
    assert nb < na or n > 37296 or restart in (1, 1001)


def test_gmres_cycle_that_gives_up_is_run_step_by_step():
    from tcad_b200 import _lib
    lib = _lib.load()
    A, b = _system(900, 4)
    xa, ia, _ = _solve(A, b, 0, block_size=3)
    before = lib.tcad_krylov_fused_gave_up()
    prev = lib.tcad_set_krylov_fused_test(1)
    try:
        xb, ib, _ = _solve(A, b, 1, block_size=3)
    finally:
        lib.tcad_set_krylov_fused_test(prev)
    assert lib.tcad_krylov_fused_gave_up() > before
    assert ia == ib and np.array_equal(xa, xb)
