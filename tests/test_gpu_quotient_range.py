"""The recombination's quotients where the reciprocal of its denominator squared is not
an ordinary number (the square near or past either end of the range, subnormal, zero,
infinite): what a division gives, bit for bit.  And quotients next to the middle of two
numbers, where one residual correction has to round the right way."""
import numpy as np
import pytest

from test_gpu_quotients import _recombination

pytestmark = pytest.mark.gpu


def _run(n, p, nie, tn, tp, ns, r0):
    import torch
    from tcad_b200 import _lib
    lib, m = _lib.load(), len(n)
    par = np.zeros(_lib.NPAR)
    par[:6] = ns, r0, 0.0, 0.0, 1.0, 0.0
    args = [torch.tensor(np.asarray(v, float), device="cuda") for v in (n, p, nie, tn, tp, par)]
    out = torch.empty(3 * m, dtype=torch.float64, device="cuda")
    assert lib.tcad_eval_recombination(*[_lib.ptr(a) for a in args[:5]], m, _lib.ptr(args[5]),
                                       _lib.ptr(out), _lib.stream_ptr()) == _lib.TCAD_OK
    with np.errstate(all="ignore"):
        ref = _recombination(n, p, nie, tn, tp, ns, r0, 0.0, 0.0, False)
    for got, want in zip(out.cpu().numpy().reshape(3, m), ref):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("lo,hi", [(-170, -140), (-156, -153), (-110, -100), (100, 110),
                                   (140, 160), (-320, 308)])
def test_extreme_denominators(lo, hi):
    """Carriers and nie of a cold or depleted semiconductor: den = tau nie from 1e-170."""
    rng = np.random.default_rng(11)
    m = 4000
    nie = 10.0 ** rng.uniform(max(lo, -300), min(hi, 300), m)
    n, p = nie * 10.0 ** rng.uniform(-3, 3, m), nie * 10.0 ** rng.uniform(-3, 3, m)
    t = 10.0 ** rng.uniform(-2, 2, m)
    _run(n, p, nie, t, t * rng.uniform(0.1, 10.0, m), 1.0, 1.0)


def test_quotients_next_to_a_middle():
    """a / b = (odd + delta / b) / 2^54 with |delta| <= 3: R = a by n = 1, p = a,
    tau_n = 0, tau_p = 1, nie = 0; one R0 = b per call."""
    import random
    rnd = random.Random(3)
    seen = 0
    while seen < 60:
        b = (1 << 53) - (rnd.getrandbits(rnd.choice([8, 30, 45, 52])) | 1)
        a = []
        for d in (1, -1, 3, -3):
            q = (-d * pow(b, -1, 1 << 54)) % (1 << 54)
            if q >= 1 << 53 and q % 2 and (1 << 52) <= (q * b + d) >> 54 < 1 << 53:
                a.append(float((q * b + d) >> 54))
        if b >> 52 != 1 or not a:
            continue
        seen += 1
        a = np.array(a)
        one, z = np.ones_like(a), np.zeros_like(a)
        _run(one, a, z, z, one, 1.0, float(b))
