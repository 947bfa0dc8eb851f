"""The red-black solve of one wave of blocks (above the resident sizes, below the streamed
ones) against the launch-per-step loop: just above the resident bound, odd rows, the
largest of its range in 2D and 3D.  Same expressions and order of sums: bit-identical."""
import numpy as np
import pytest

from test_gpu_redblack import _scaled_system, _solve_counted
from test_gpu_resident import _device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("diode", (401, 380)), ("mosfet", (480, 400)),
                                        ("diode", (591, 511)), ("trigate", (61, 56, 45)),
                                        ("trigate", (80, 56, 40)), ("trigate", (71, 54, 54))])
def test_wave_solve_bit_identical_to_per_step(kind, shape):
    pk = _scaled_system(_device(kind, shape))
    for rtol, maxit in ((1e-5, 200), (1e-30, 13)):
        xa, ita, sta, rra, na = _solve_counted(pk, 2, rtol, maxit, fused=False)
        xb, itb, stb, rrb, nb = _solve_counted(pk, 2, rtol, maxit, fused=True)
        assert (ita, sta, rra) == (itb, stb, rrb)
        assert np.array_equal(xa.cpu().numpy(), xb.cpu().numpy())
        assert nb == 2 and na > 2           # colour repack + the single launch


def test_wave_newton_and_give_up():
    """A bias point whose solves are waves: the same state with one launch per step, and
    with the first wave of each solve given up."""
    import tcad_b200 as tb
    states = []
    for fused, hold in ((0, 0), (1, 0), (1, 1)):
        dev = _device("trigate", (61, 56, 45))
        dev.solve_equilibrium()
        lib = dev.pack.lib
        prev, held = lib.tcad_set_krylov_fused(fused), lib.tcad_set_krylov_fused_test(hold)
        g0 = lib.tcad_krylov_fused_gave_up()
        try:
            dev.solve_bias({"drain": 0.05}, tb.NewtonOptions(max_iter=3 if hold else 50))
        finally:
            lib.tcad_set_krylov_fused(prev)
            lib.tcad_set_krylov_fused_test(held)
        if hold:
            assert lib.tcad_krylov_fused_gave_up() == g0 + 3
            dev.solve_bias({"drain": 0.05})
        assert dev.last_converged
        states.append((dev.psi, dev.n, dev.p))
    for a, b in zip(states[0], states[1]):
        assert np.array_equal(a, b)
    assert np.abs(states[2][0] - states[0][0]).max() * dev.VT < 1e-9
