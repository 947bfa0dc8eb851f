// The red-black Schur BiCGStab of a small single-instance pack in one
// cooperative launch with everything resident: one CTA of T threads per SM (and
// per flat block of the slot pack, K T slots at most), the CTA's rows of both
// colours of J in shared memory when they fit (JS), its slots' vectors in
// registers.  Global memory holds only what neighbours read: r, p, v and Tr.
//
// A solve of this size is bound by the latency of its steps, not by bytes: at
// 20k nodes an iteration moves 9 MB through L2 (about 1 us) and took 36 us as
// 20 CTAs of 512 slots that read J from L2 behind an arrival counter with
// back-off; here it takes 12 us (201 x 101 diode, 107 CTAs of 96 slots; the
// 40 x 24 x 16 tri-gate 38 -> 14 us).
// Five steps an iteration, each ended by GridSync: red(p), p + v (alpha),
// red(s), s + t (early, omega), x (rho, beta, convergence); p and s are
// formed on the fly at the neighbours (RbFormPCg / RbFormSCg).  Bodies, scalar
// updates and the order of the sums are those of the per-step kernels, so the
// result is bit-identical to launch_bicgstab_rb's loop over the same blocks.
//
// Instances whose rows fit in the shared memory of one cluster have a cluster
// each (SYNC = ClusterSync, eq_resident.cuh); their blocks are its CTAs' shares,
// with several instances other ones than the per-step loop's 512 slots.
#pragma once

namespace tcad {

// slots per CTA whose J rows of both colours fit in shared memory (227 KB)
constexpr int rb_resident_js_slots(int ne) { return (232448 - 2048) / (16 * ne) / 32 * 32; }
constexpr int kRbResidentMaxSlots = 2 * NT;

// values of the other colour that other CTAs wrote during this launch: read
// through L2
struct RbValCg {
  const double* xi;
  int64_t NS;
  __device__ __forceinline__ double operator()(int m, int c) const {
    return __ldcg(xi + c * NS + m);
  }
};
struct RbFormPCg {
  const double *r, *p, *v;
  int64_t NS;
  double beta, omega;
  int restart;
  __device__ __forceinline__ double operator()(int m, int c) const {
    const double rv = __ldcg(r + c * NS + m);
    return restart ? rv
                   : rv + beta * (__ldcg(p + c * NS + m) - omega * __ldcg(v + c * NS + m));
  }
};
struct RbFormSCg {
  const double *r, *v;
  int64_t NS;
  double alpha;
  __device__ __forceinline__ double operator()(int m, int c) const {
    return __ldcg(r + c * NS + m) - alpha * __ldcg(v + c * NS + m);
  }
};

template <int DIM, int K, int T, bool JS, class SYNC>
__global__ void __launch_bounds__(T, 1)
k_bicgstab_rb_resident(const tcad_pack_t pkb, const RbMap mp, const double* __restrict__ Jn,
                       const double* __restrict__ JR, const double* __restrict__ JB, const double* __restrict__ b,
                       double* __restrict__ x, double* bRg, double* Tr, double* xbg,
                       double* rhsg, double* rg, double* pg, double* vg, KState* ks,
                       double* part, unsigned* bar, double rtol, int maxit,
                       const int32_t* __restrict__ pre_status,
                       const double* __restrict__ rtol_inst, int max_rechecks) {
  constexpr int NE = Stencil<DIM>::NE;
  extern __shared__ __align__(16) double s_rows[];
  SYNC gs;
  gs.init(part, bar);
  const RbShare fb = rb_share(pkb, gs);
  const int inst = fb.inst;
  const RbGeo g = rb_geo(pkb, mp, inst);
  const int64_t NS = pkb.n_nodes, NN = mp.n_full;
  const int nloc = fb.len;
  const double *jr, *jb;   // J rows of the CTA's slots in warp tiles
  if constexpr (JS) {
    // a share is a multiple of 32 slots, so the CTA's rows are whole warp tiles,
    // one contiguous run per colour
    const int n2 = (nloc + 31) / 32 * NE * 16;
    const double2* const gr = reinterpret_cast<const double2*>(JR + rb_jidx<NE>(0, fb.begin));
    const double2* const gb = reinterpret_cast<const double2*>(JB + rb_jidx<NE>(0, fb.begin));
    double2* const s2 = reinterpret_cast<double2*>(s_rows);
    if (Jn) {   // from J in node order (zeros at pads, as k_rb_pack)
      for (int l = threadIdx.x; l < nloc; l += T)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const RbNode q = rb_node(g, fb.begin + l, c);
          double* const dst = s_rows + 2 * c * n2 + rb_jidx<NE>(0, l);
#pragma unroll 13
          for (int e = 0; e < NE; ++e)
            dst[32 * e] = q.real ? Jn[(int64_t)e * NN + q.node] : 0.0;
        }
    } else {
#pragma unroll 8
      for (int i = threadIdx.x; i < n2; i += T) s2[i] = gr[i];
#pragma unroll 8
      for (int i = threadIdx.x; i < n2; i += T) s2[n2 + i] = gb[i];
    }
    jr = s_rows;
    jb = s_rows + 2 * n2;
  } else {
    jr = JR + rb_jidx<NE>(0, fb.begin);
    jb = JB + rb_jidx<NE>(0, fb.begin);
  }
  int mr[K][2 * DIM], mb[K][2 * DIM];
  bool own[K], realr[K], realb[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int q = threadIdx.x + k * T;
    own[k] = q < nloc;
    const int64_t slot = fb.begin + (own[k] ? q : 0);
    const RbNode nr = rb_node(g, slot, 0), nk = rb_node(g, slot, 1);
    realr[k] = own[k] && nr.real;
    realb[k] = own[k] && nk.real;
    int m[6];
    rb_nbrs<DIM>(g, nr, (int)(slot - g.soff), m);
#pragma unroll
    for (int d = 0; d < 2 * DIM; ++d) mr[k][d] = m[d];
    rb_nbrs<DIM>(g, nk, (int)(slot - g.soff), m);
#pragma unroll
    for (int d = 0; d < 2 * DIM; ++d) mb[k][d] = m[d];
  }
  const int64_t q0 = fb.begin + threadIdx.x;     // slot of (k, c): q0 + k NT + c NS
  double r[K][3], rh[K][3], p[K][3], v[K][3], s[K][3], t[K][3], xb[K][3], tr[K][3];
  double tot[3], sum[3] = {0.0, 0.0, 0.0};
  KState S;
  // The sums in the per-step kernels' order: a thread below NT adds the terms of its
  // slots q and q + NT, the latter from operands that the thread which has it (T > NT)
  // hands over (operands, not products: a term is one fused multiply-add).
  constexpr int HI = T > NT ? T - NT : 1;
  __shared__ double s_ops[T > NT ? 6 : 1][HI];
  const bool low = T <= NT || threadIdx.x < NT;
  const auto add = [&](int i, double u, double w, const auto& term) {
    if (low) {
      term(u, w);
    } else {
      s_ops[i][threadIdx.x - NT] = u;
      s_ops[3 + i][threadIdx.x - NT] = w;
    }
  };
  const auto collect = [&](const auto& term) {
    if constexpr (T > NT) {
      __syncthreads();
      if (low && (int)threadIdx.x + NT < nloc)
#pragma unroll
        for (int i = 0; i < 3; ++i) term(s_ops[i][threadIdx.x], s_ops[3 + i][threadIdx.x]);
    }
  };
  const auto product = [&](double u, double w) { sum[0] += u * w; };      // (u, w)
  const auto squares = [&](double u, double w) {                          // (u, u), (w, u), (w, w)
    sum[0] += u * u;
    sum[1] += w * u;
    sum[2] += w * w;
  };
  const auto residual = [&](double u, double w) {                         // (u, w), (w, w), (u, u)
    sum[0] += u * w;
    sum[1] += w * w;
    sum[2] += u * u;
  };

  // red pass: tr = E X, stored for the neighbours
  auto red = [&](const auto& X) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      tr[k][0] = 0.0; tr[k][1] = 0.0; tr[k][2] = 0.0;
      if (realr[k])
        rb_couple_f<DIM>(jr, X, threadIdx.x + k * T, mr[k], tr[k][0], tr[k][1], tr[k][2]);
      if (own[k])
#pragma unroll
        for (int c = 0; c < 3; ++c) Tr[c * NS + q0 + k * T] = tr[k][c];
    }
  };
  // u = F y at slot k (0 at a pad)
  auto black = [&](int k, const double* y, double* u) {
    u[0] = 0.0; u[1] = 0.0; u[2] = 0.0;
    if (realb[k])
      rb_couple_f<DIM>(jb, RbValCg{y + g.soff, NS}, threadIdx.x + k * T, mb[k], u[0], u[1],
                       u[2]);
  };

  // colours of b, ||b||^2
  double bB[K][3];
  sum[0] = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (!own[k]) continue;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const RbNode q = rb_node(g, q0 + k * T, c);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const double bv = q.real ? b[e * NN + q.node] : 0.0;
        if (c) bB[k][e] = bv;
        else bRg[e * NS + q0 + k * T] = bv;
        if (low) sum[0] += bv * bv;
        else s_ops[3 * c + e][threadIdx.x - NT] = bv;
      }
    }
  }
  if constexpr (T > NT) {
    __syncthreads();
    if (low && (int)threadIdx.x + NT < nloc)
#pragma unroll
      for (int i = 0; i < 6; ++i) sum[0] += s_ops[i][threadIdx.x] * s_ops[i][threadIdx.x];
  }
  if (!gs.template sum<1>(sum, tot)) return;
  const double bb = tot[0];
  // rhs = bB - F bR; x = 0, r = rh = rhs, p = v = 0
  sum[0] = 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double u[3];
    black(k, bRg, u);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double y = realb[k] ? bB[k][c] - u[c] : 0.0;
      xb[k][c] = 0.0; r[k][c] = y; rh[k][c] = y; p[k][c] = 0.0; v[k][c] = 0.0;
      s[k][c] = 0.0; t[k][c] = 0.0;
      if (own[k]) {
        const int64_t q = c * NS + q0 + k * T;
        rhsg[q] = y; rg[q] = y; pg[q] = 0.0; vg[q] = 0.0;
        add(c, y, y, product);
      }
    }
  }
  collect(product);
  if (!gs.template sum<1>(sum, tot)) return;
  rb_fin_init(S, tot[0], bb, rtol_inst ? rtol_inst[inst] : rtol, maxit,
              pre_status ? pre_status[inst] : TCAD_OK);

  for (int rechecks = 0;; ++rechecks) {
    while (S.active) {
      red(RbFormPCg{rg + g.soff, pg + g.soff, vg + g.soff, NS, S.beta, S.omega, S.restart});
      if (!gs.template sum<0>(nullptr, nullptr)) return;
      sum[0] = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        double u[3];
        black(k, Tr, u);
        if (!own[k]) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double rv = r[k][c];
          const double pn = S.restart ? rv : rv + S.beta * (p[k][c] - S.omega * v[k][c]);
          if (S.restart) rh[k][c] = rv;
          const double y = realb[k] ? pn - u[c] : 0.0;
          p[k][c] = pn;
          v[k][c] = y;
          pg[c * NS + q0 + k * T] = pn;
          vg[c * NS + q0 + k * T] = y;
          add(c, rh[k][c], y, product);
        }
      }
      collect(product);
      if (!gs.template sum<1>(sum, tot)) return;
      fin_v(S, tot[0]);
      if (!S.active) break;
      red(RbFormSCg{rg + g.soff, vg + g.soff, NS, S.alpha});
      if (!gs.template sum<0>(nullptr, nullptr)) return;
      sum[0] = 0.0; sum[1] = 0.0; sum[2] = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        double u[3];
        black(k, Tr, u);
        if (!own[k]) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double sv = r[k][c] - S.alpha * v[k][c];
          const double y = realb[k] ? sv - u[c] : 0.0;
          s[k][c] = sv;
          t[k][c] = y;
          add(c, sv, y, squares);
        }
      }
      collect(squares);
      if (!gs.template sum<3>(sum, tot)) return;
      fin_s(S, tot[0]);
      fin_t(S, tot[1], tot[2]);
      sum[0] = 0.0; sum[1] = 0.0; sum[2] = 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (!own[k]) continue;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xb[k][c] = xb[k][c] + S.alpha * p[k][c] + S.omega * s[k][c];
          const double rn = s[k][c] - S.omega * t[k][c];
          r[k][c] = rn;
          rg[c * NS + q0 + k * T] = rn;
          add(c, rh[k][c], rn, residual);
        }
      }
      collect(residual);
      if (!gs.template sum<3>(sum, tot)) return;
      fin_x(S, tot[0], tot[1], tot[2]);
    }
    // true Schur residual r = rhs - S x
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (own[k])
#pragma unroll
        for (int c = 0; c < 3; ++c) xbg[c * NS + q0 + k * T] = xb[k][c];
    if (!gs.template sum<0>(nullptr, nullptr)) return;
    red(RbValCg{xbg + g.soff, NS});
    if (!gs.template sum<0>(nullptr, nullptr)) return;
    sum[0] = 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double u[3];
      black(k, Tr, u);
      if (!own[k]) continue;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double y = realb[k] ? xb[k][c] - u[c] : 0.0;
        const double a = rhsg[c * NS + q0 + k * T] - y;
        r[k][c] = a;
        rg[c * NS + q0 + k * T] = a;
        add(c, a, a, product);
      }
    }
    collect(product);
    if (!gs.template sum<1>(sum, tot)) return;
    fin_true(S, tot[0], rechecks < max_rechecks ? 1 : 0);
    if (!S.active) break;
  }
  // full solution: x_r = bR - E x_b, x_b
  const bool idle = pre_status && pre_status[inst] != TCAD_OK;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (!own[k]) continue;
    const RbNode nr = rb_node(g, q0 + k * T, 0), nk = rb_node(g, q0 + k * T, 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (realr[k]) x[c * NN + nr.node] = idle ? 0.0 : bRg[c * NS + q0 + k * T] - tr[k][c];
      if (realb[k]) x[c * NN + nk.node] = idle ? 0.0 : xb[k][c];
    }
  }
  if (fb.lead && threadIdx.x == 0) ks[inst] = S;
}

}  // namespace tcad
