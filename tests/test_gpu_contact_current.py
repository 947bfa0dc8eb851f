"""The terminal-current kernel (a lane per edge, one launch where a cluster of CTAs takes
the node list) against the assembly's unstamped continuity rows at the same nodes.  Both
form a node's terms in the same order, so the residuals agree bit for bit; the sum is in
a fixed order over 256 lanes, within count * 2^-52 of the sum of magnitudes.  Counts
around a CTA's (64 nodes in 2D, 32 in 3D) and a cluster's (512, 256)."""
import numpy as np
import pytest

from test_gpu_resident import _device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("diode", (2, 2)), ("diode", (61, 23)),
                                        ("trigate", (9, 7, 5)), ("trigate", (17, 12, 9))])
def test_contact_current_matches_the_unstamped_rows(kind, shape):
    import torch
    from tcad_b200 import _lib
    pk = _device(kind, shape).pack
    rng = np.random.default_rng(2)
    n = pk.N
    state = [torch.tensor(v, device="cuda") for v in
             (rng.uniform(-20, 20, n), 10.0 ** rng.uniform(-12, 2, n),
              10.0 ** rng.uniform(-12, 2, n))]
    pk.assemble(_lib.MODE_UNSTAMPED, *state)
    f = pk.F.cpu().numpy().reshape(3, -1)
    for count in {c for c in (1, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, n)
                  if c <= n}:
        nodes = np.sort(rng.choice(n, count, replace=False))
        part = torch.zeros(2 * count, dtype=torch.float64, device="cuda")
        out = torch.zeros(1, dtype=torch.float64, device="cuda")
        dn = torch.tensor(nodes, dtype=torch.int64, device="cuda")
        _lib.check(pk.lib.tcad_contact_current(
            pk.pref, *[_lib.ptr(v) for v in state], _lib.ptr(dn), count, _lib.ptr(part),
            part.numel(), _lib.ptr(out), pk.sp()), "tcad_contact_current")
        got = part.cpu().numpy().reshape(2, count)
        np.testing.assert_array_equal(got[0], f[1][nodes])
        np.testing.assert_array_equal(got[1], f[2][nodes])
        total = got[0] + got[1]
        assert abs(out.item() - total.sum()) <= count * 2.0 ** -52 * np.abs(total).sum()
