"""Quotients formed from a shared reciprocal are the rounded quotients.

The recombination divides by its denominator squared and by R0 through their
reciprocals (a product and one residual correction, csrc/sg_edge.cuh div_by).  NumPy's
divisions are IEEE, the kernel multiplies and adds without contraction, so the two agree
bit for bit -- also where an operand or the quotient is zero, tiny, infinite or NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recombination(n, p, nie, tn, tp, ns, r0, cn, cp, auger):
    nph, pph = n * ns, p * ns
    excess = nph * pph - nie * nie
    den = tp * (nph + nie) + tn * (pph + nie)
    r = excess / den
    den2 = den * den
    dn, dp = (pph * den - excess * tp) / den2, (nph * den - excess * tn) / den2
    if auger:
        cc = cn * nph + cp * pph
        r = r + cc * excess
        dn = dn + cn * excess + cc * pph
        dp = dp + cp * excess + cc * nph
    return r / r0, dn * ns / r0, dp * ns / r0


@pytest.mark.parametrize("auger", [False, True])
def test_recombination_quotients_are_exact(auger):
    import torch
    from tcad_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(5)
    m = 5000
    n, p = (10.0 ** rng.uniform(-25, 6, m) for _ in range(2))
    n[:6] = [0.0, 0.0, 1e-300, np.inf, np.nan, -1e-20]
    p[:6] = [0.0, 1.0, 1e-300, 1.0, 1.0, 1e-20]
    nie = 10.0 ** rng.uniform(0, 12, m)
    tn, tp = (10.0 ** rng.uniform(-12, -3, m) for _ in range(2))
    ns, r0, cn, cp = 1e17, 3.7e23, 2.8e-31, 9.9e-32
    par = np.zeros(_lib.NPAR)
    par[:6] = ns, r0, cn, cp, 1.0, float(auger)
    args = [torch.tensor(v, device="cuda") for v in (n, p, nie, tn, tp, par)]
    out = torch.empty(3 * m, dtype=torch.float64, device="cuda")
    rc = lib.tcad_eval_recombination(*[_lib.ptr(a) for a in args[:5]], m, _lib.ptr(args[5]),
                                     _lib.ptr(out), _lib.stream_ptr())
    assert rc == _lib.TCAD_OK
    with np.errstate(all="ignore"):
        ref = _recombination(n, p, nie, tn, tp, ns, r0, cn, cp, auger)
    for got, want in zip(out.cpu().numpy().reshape(3, m), ref):
        np.testing.assert_array_equal(got, want)
