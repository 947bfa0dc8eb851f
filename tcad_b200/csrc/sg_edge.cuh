// Scharfetter-Gummel edge quantities.  Compiled with -fmad=false so the
// arithmetic rounds step by step in the reference's order
// (pytcad/kernels.py:88-109, pytcad/device2d.py:1449-1479).
#pragma once

#include "common.cuh"

namespace tcad {

// Clip to [-700, 700] keeping NaN (numpy.clip semantics).
__device__ __forceinline__ double clip700(double x) {
  return x < -700.0 ? -700.0 : (x > 700.0 ? 700.0 : x);
}

// a / b from r = 1/b, bit for bit barring underflow and overflow (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990:
// with r the rounded reciprocal, one residual correction of a quotient within one unit
// of its last place rounds it correctly).  RN(a r) may be 1.5 units off, but not where
// that matters: the correction's error is below 2^-51 units, and where a / b is that
// close to the middle of two numbers RN(a r) is one of the two -- with significands in
// [1, 2), |r - 1/b| <= 2^-54 moves a r by less than a / 2 units, so only an a within
// 2^-51 of 2 could get past them, and then a / b lies next to a number.
__device__ __forceinline__ double div_in_range(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}
// ... of any a and a b whose reciprocal is in range: where a or the quotient is zero,
// infinite, NaN or of a magnitude near the end of the range it is a r.
__device__ __forceinline__ double div_by(double a, double b, double r) {
  const double q = a * r;
  const double c = fma(fma(-q, b, a), r, q);
  return fabs(a) > 1e-270 && fabs(q) > 1e-270 && fabs(q) < 1e270 ? c : q;
}

// A divisor of several quotients and its reciprocal.
struct Divisor {
  double b, r;
  static __device__ __forceinline__ Divisor of(double b) { return Divisor{b, 1.0 / b}; }
  __device__ __forceinline__ double divide(double a) const { return div_by(a, b, r); }
};

// ... and of any b: numerator and divisor are scaled by a power of two where b is far
// from one, so that neither the reciprocal nor the residual leaves the range.
struct WideDivisor {
  Divisor d;
  double s;
  static __device__ __forceinline__ WideDivisor of(double b) {
    // by the exponent: below 2^-700, to 2^700, above
    const unsigned e = (unsigned)__double2hiint(b) >> 20 & 0x7ffu;
    const int k = e < 323u ? 1623 : e > 1723u ? 423 : 1023;
    const double s = __hiloint2double(k << 20, 0);
    return WideDivisor{Divisor::of(b * s), s};
  }
  __device__ __forceinline__ double divide(double a) const { return d.divide(a * s); }
};

// B(x), B'(x) and those of -x of the series band |x| < 1e-4 (kernels.py:92-96,
// 105-109), B = (1 - x/2) + x^2/12 and B' = (-1/2 + x/6) - x^3/180; the terms of
// -x are those of x or their negatives.  (A quotient that underflows is far below
// the last bit of the sum it is added to.)
__device__ __forceinline__ void bern_series(double x, double& Bp, double& Bm, double& dBp,
                                            double& dBm) {
  const double x2 = div_in_range(x * x, 12.0, 1.0 / 12.0);
  const double x1 = div_in_range(x, 6.0, 1.0 / 6.0);
  const double x3 = div_in_range(x * x * x, 180.0, 1.0 / 180.0);
  Bp = (1.0 - x / 2.0) + x2;
  Bm = (1.0 + x / 2.0) + x2;
  dBp = (-0.5 + x1) - x3;
  dBm = (-0.5 - x1) + x3;
}

// B(x), B(-x), B'(x), B'(-x).  Three argument bands:
//
//   |x| < 1e-4          the reference's series (kernels.py:92-96, 105-109);
//   1e-4 <= |x| < 1e-2  the reference's own formulas at +x and at -x
//                       (kernels.py:88-109): B = x / expm1(x) and
//                       B' = B (1/x - 1/(1 - e^-x)), two expm1 and the same
//                       divisions.  Here 1/x - 1/(1 - e^-x) cancels (about
//                       4 digits at 1e-4), so the reference's derivative
//                       carries that cancellation's rounding; reproducing
//                       its steps reproduces its values elementwise.
//   |x| >= 1e-2         ONE expm1 and ONE reciprocal serve all four values.
//                       With a = |x|, e = expm1(a) > 0 and r = 1/e:
//                         S  = B(a)   = a r
//                         L  = B(-a)  = a e^a / (e^a - 1) = S + a
//                         dS = B'(a)  = S (1/a - (1 + r)) = r (1 - a (1 + r))
//                         dL = B'(-a) = L (r - 1/a)       = (1 + r) (S - 1)
//                       (L / a = 1 + r and S / a = r).  In this band the
//                       values agree with the reference's formulas to a few
//                       ulp (derivatives within 1e-13 relative; measured
//                       over 4e5 arguments against kernels.py).
//
// The lanes of a warp are seldom in one band and an edge is mostly its
// exponentials and divisions, so the last two bands share one expm1 and its
// reciprocal, and quotients with a divisor whose reciprocal is at hand (or a
// constant) are a product and its correction: a mixed warp runs 2 expm1 and 3
// divisions (3 and 12 band by band).
__device__ __forceinline__ void bern4(double x, double& Bp, double& Bm, double& dBp,
                                      double& dBm) {
  x = clip700(x);
  const double a = fabs(x);
  if (a < 1e-4) {
    bern_series(x, Bp, Bm, dBp, dBm);
    return;
  }
  const bool mid = a < 1e-2;
  const double e = expm1(mid ? x : a);
  const double r = 1.0 / e;
  if (mid) {
    const double em = expm1(-x);
    const double rm = 1.0 / em, rx = 1.0 / x;
    Bp = div_in_range(x, e, r);
    Bm = div_in_range(-x, em, rm);
    dBp = Bp * (rx + rm);    // B (1/x - 1/(1 - e^-x)), 1 - e^-x = -em
    dBm = Bm * (r - rx);
    return;
  }
  const double r1 = 1.0 + r;
  const double S = a * r;
  const double L = S + a;
  const double dS = r * (1.0 - a * r1);
  const double dL = r1 * (S - 1.0);
  const bool pos = x > 0.0;
  Bp = pos ? S : L;
  Bm = pos ? L : S;
  dBp = pos ? dS : dL;
  dBm = pos ? dL : dS;
}

// Everything the two endpoint rows need from one edge (low -> high node).
struct Edge {
  double f;     // Poisson flux (psi_hi - psi_lo) / h
  double Jn;    // electron SG current an (n_hi B(d) - n_lo B(-d))
  double Jp;    // hole SG current -ap (p_hi B(-d') - p_lo B(d'))
  double npsi;  // dJn/dpsi_hi = an (n_hi B'(d) + n_lo B'(-d))
  double nlo;   // dJn/dn_lo = -an B(-d)
  double nhi;   // dJn/dn_hi = an B(d)
  double ppsi;  // dJp/dpsi_hi = ap (p_hi B'(-d') + p_lo B'(d'))
  double plo;   // dJp/dp_lo = ap B(d')
  double phi;   // dJp/dp_hi = -ap B(-d')
};

__device__ __forceinline__ void zero_edge(Edge& e) {
  e.f = e.Jn = e.Jp = e.npsi = e.nlo = e.nhi = e.ppsi = e.plo = e.phi = 0.0;
}

// d = dpsi + dlnnie (electrons), d' = dpsi - dlnnie (holes):
// pytcad/device2d.py:1451-1479.
__device__ __forceinline__ void sg_edge(double psi_lo, double psi_hi, double n_lo,
                                        double n_hi, double p_lo, double p_hi, double an,
                                        double ap, double dl, Divisor h, Edge& e) {
  const double dpsi = psi_hi - psi_lo;
  e.f = h.divide(dpsi);
  double Bp, Bm, dBp, dBm, Bph, Bmh, dBph, dBmh;
  bern4(dpsi + dl, Bp, Bm, dBp, dBm);
  if (dl == 0.0) {
    Bph = Bp; Bmh = Bm; dBph = dBp; dBmh = dBm;
  } else {
    bern4(dpsi - dl, Bph, Bmh, dBph, dBmh);
  }
  e.Jn = an * (n_hi * Bp - n_lo * Bm);
  e.Jp = -ap * (p_hi * Bmh - p_lo * Bph);
  const double Sn = n_hi * dBp + n_lo * dBm;
  const double Sp = p_hi * dBmh + p_lo * dBph;
  e.npsi = an * Sn;
  e.nlo = -an * Bm;
  e.nhi = an * Bp;
  e.ppsi = ap * Sp;
  e.plo = ap * Bph;
  e.phi = -ap * Bmh;
}

// SRH + Auger recombination, scaled (materials.py:474-518 with the
// device's R0/Ns scaling, pytcad/device2d.py:1482-1508), with the
// reference's divisions: R = excess / den, dR/dn = (p den - excess tau_p) /
// den^2, Rs = R / R0, dRs/dn = dR/dn Ns / R0.
__device__ __forceinline__ void recomb(double n, double p, double nie, double taun,
                                       double taup, const double* par, double& Rs,
                                       double& dRsn, double& dRsp) {
  const double Ns = par[TCAD_P_NS], R0 = par[TCAD_P_R0];
  if (par[TCAD_P_SRH] == 0.0) {
    Rs = dRsn = dRsp = 0.0;
    return;
  }
  const double nph = n * Ns, pph = p * Ns;
  const double excess = nph * pph - nie * nie;
  const double den = taup * (nph + nie) + taun * (pph + nie);
  double R = excess / den;
  const double den2 = den * den;
  const WideDivisor by2 = WideDivisor::of(den2);   // (den^2 of a cold semiconductor's carriers)
  double dRdn = by2.divide(pph * den - excess * taup);
  double dRdp = by2.divide(nph * den - excess * taun);
  if (par[TCAD_P_AUGER] != 0.0) {
    const double Cn = par[TCAD_P_CN], Cp = par[TCAD_P_CP];
    const double cc = Cn * nph + Cp * pph;
    R = R + cc * excess;
    dRdn = dRdn + Cn * excess + cc * pph;
    dRdp = dRdp + Cp * excess + cc * nph;
  }
  const Divisor by0 = Divisor::of(R0);
  Rs = by0.divide(R);
  dRsn = by0.divide(dRdn * Ns);
  dRsp = by0.divide(dRdp * Ns);
}

}  // namespace tcad
