"""The resident red-black solve with a thread per slot above 256 slots a CTA (3D), whose
upper threads hand the terms of the sums to the lower ones, against the launch-per-step
loop: shares of just over 256 and of 352 slots (rows in shared memory, on a cluster of 8 and
on the grid), of 384 and of 512 (rows from L2).  The same order of sums: bit-identical."""
import numpy as np
import pytest

from test_gpu_redblack import _scaled_system, _solve_counted
from test_gpu_resident import _device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 16, 12), (22, 16, 16), (60, 40, 32), (64, 48, 33),
                                   (64, 50, 33), (82, 58, 31)])
def test_split_resident_solve_bit_identical_to_per_step(shape):
    pk = _scaled_system(_device("trigate", shape))
    for rtol, maxit in ((1e-6, 400), (1e-30, 25)):
        xa, ita, sta, rra, _ = _solve_counted(pk, 2, rtol, maxit, fused=False)
        xb, itb, stb, rrb, nb = _solve_counted(pk, 2, rtol, maxit, fused=True)
        assert (ita, sta, rra) == (itb, stb, rrb) and nb == 2
        assert np.array_equal(xa.cpu().numpy(), xb.cpu().numpy())
