// The equilibrium red-black PCG (k_eqrb_*) of a single-instance pack in one
// cooperative launch with everything resident: one CTA of T threads per SM (and per
// flat block of the slot pack, K T slots at most), the CTA's rows of both
// colours in shared memory, taken straight from the node-order J, its slots'
// vectors in registers; z, p, x and Tr also in global memory for the
// neighbours.
//
// The scalar rows are small (112 bytes a slot pair in 3D), so up to 303k slots
// (600k nodes) stay resident and an iteration is bound by the latency of its
// three steps -- red(p), q (alpha), x (beta) -- instead of four launches and
// two last-block reductions.  240 x 120 MOSFET: 24 -> 4.5 us per iteration.
// Instances of at most kClusterMaxCtas x kEqResidentMaxSlots slots have a cluster
// each instead (SYNC = ClusterSync): barriers inside a cluster cost a fifth, and a
// batch's instances run side by side, each to its own convergence.
// Expressions and the order of the sums are the per-step kernels', so the
// update is bit-identical to launch_cg_rb's loop over the same blocks (of several
// instances: the CTAs' shares, other blocks than the loop's 512 slots).
#pragma once

namespace tcad {

constexpr int kEqResidentMaxSlots = 8 * NT;

template <int DIM, int K, int T, class SYNC>
__global__ void __launch_bounds__(T, 1)
k_eqrb_resident(const tcad_pack_t pkb, const RbMap mp, const double* __restrict__ J,
                const double* __restrict__ F, double* __restrict__ d, double* zg, double* pg,
                double* xg, double* Tr, KState* ks, double* part, unsigned* bar, double rtol,
                int maxit, const uint8_t* __restrict__ active,
                const double* __restrict__ rtol_inst, int rows) {
  constexpr int NE = 1 + 2 * DIM, ND = 2 * DIM;
  extern __shared__ __align__(16) double s_rows[];   // [2][NE][rows]
  SYNC gs;
  gs.init(part, bar);
  const RbShare fb = rb_share(pkb, gs);
  const int inst = fb.inst;
  if (active && !active[inst]) {
    if (fb.lead && threadIdx.x == 0) ks[inst].active = 0;
    return;
  }
  const RbGeo g = rb_geo(pkb, mp, inst);
  const int64_t NN = mp.n_full;
  const int nloc = fb.len, fn = rows;
  double* const sR = s_rows;
  double* const sB = s_rows + (int64_t)NE * fn;
  const int64_t q0 = fb.begin + threadIdx.x;   // slot k of the thread: q0 + k T
  int mr[K][ND], mb[K][ND];
  bool own[K], realr[K], realb[K];
  double x[K], r[K], z[K], p[K], q[K], si[K];
  double sum[2] = {0.0, 0.0}, tot[2];
  KState S;
  // sum[0] = (u, w) over the slots in the per-step kernels' order, sum[1] = (u, u) for
  // TWO: thread l < NT adds the slots l, l + NT, ...; the threads above NT hand it their
  // operands
  constexpr int HI = T > NT ? T - NT : 1;
  __shared__ double s_ops[T > NT ? 2 * K : 1][HI];
  const auto dot = [&](const double (&u)[K], const double (&w)[K], auto two) {
    const auto term = [&](double a, double b) {
      sum[0] += a * b;
      if constexpr (decltype(two)::value) sum[1] += a * a;
    };
    sum[0] = 0.0; sum[1] = 0.0;
    if constexpr (T == NT) {
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (own[k]) term(u[k], w[k]);
    } else {
      if (threadIdx.x >= NT) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          s_ops[2 * k][threadIdx.x - NT] = u[k];
          s_ops[2 * k + 1][threadIdx.x - NT] = w[k];
        }
      }
      __syncthreads();
      if (threadIdx.x < NT) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (own[k]) term(u[k], w[k]);
#pragma unroll
          for (int j = 0; j < T / NT - 1; ++j)
            if ((int)threadIdx.x + k * T + (j + 1) * NT < nloc)
              term(s_ops[2 * k][threadIdx.x + j * NT], s_ops[2 * k + 1][threadIdx.x + j * NT]);
        }
      }
    }
  };

#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int l = threadIdx.x + k * T;
    own[k] = l < nloc;
    const int64_t slot = own[k] ? q0 + k * T : fb.begin;
    const RbNode nr = rb_node(g, slot, 0), nk = rb_node(g, slot, 1);
    realr[k] = own[k] && nr.real;
    realb[k] = own[k] && nk.real;
    int m[6];
    rb_nbrs<DIM>(g, nr, (int)(slot - g.soff), m);
#pragma unroll
    for (int a = 0; a < ND; ++a) mr[k][a] = m[a];
    rb_nbrs<DIM>(g, nk, (int)(slot - g.soff), m);
#pragma unroll
    for (int a = 0; a < ND; ++a) mb[k][a] = m[a];
    r[k] = realr[k] ? F[nr.node] : 0.0;   // F_r here and F_b in q until the start
    q[k] = realb[k] ? F[nk.node] : 0.0;
    if (own[k])
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        sR[e * fn + l] = realr[k] ? J[(int64_t)e * NN + nr.node] : 0.0;
        sB[e * fn + l] = realb[k] ? J[(int64_t)e * NN + nk.node] : 0.0;
      }
    // Sinv = 1 / diag(S), as k_eqrb_diag; a neighbour's row is J at its node
    double sd = 0.0;
    if (realb[k]) {
      const int64_t sxy = (int64_t)g.nx * g.ny;
      const int64_t step[6] = {-1, 1, -(int64_t)g.nx, g.nx, -sxy, sxy};
      sd = -J[nk.node];
#pragma unroll
      for (int a = 0; a < ND; ++a) {
        const double jbd = J[(int64_t)(1 + a) * NN + nk.node];
        if (jbd != 0.0) {
          const int64_t n = nk.node + step[a];
          const double jrb = J[(int64_t)(1 + (a ^ 1)) * NN + n];
          sd -= (jbd * jrb) / (-J[n]);
        }
      }
    }
    si[k] = (realb[k] && sd != 0.0) ? 1.0 / sd : 0.0;
  }

  // red pass: t = A_rr^-1 (vr - A_rb X) at the thread's red slots
  auto red = [&](int k, const auto& X, double vr) {
    double t = 0.0;
    if (realr[k]) {
      const int l = threadIdx.x + k * T;
      double a = 0.0;
#pragma unroll
      for (int e = 0; e < ND; ++e) a += sR[(1 + e) * fn + l] * X(mr[k][e]);
      const double arr = -sR[l];
      t = (vr + a) / arr;
    }
    return t;
  };
  // black coupling: -sum_d J_bd Tr(m_d)
  auto black = [&](int k) {
    const int l = threadIdx.x + k * T;
    const double* const ti = Tr + g.soff;
    double a = 0.0;
#pragma unroll
    for (int e = 0; e < ND; ++e) a += sB[(1 + e) * fn + l] * __ldcg(ti + mb[k][e]);
    return -a;
  };

  // start: Tr = A_rr^-1 F_r, rhs = F_b - A_br Tr; x = 0, r = rhs, z = p = Sinv r
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (own[k]) Tr[q0 + k * T] = red(k, [](int) { return 0.0; }, r[k]);
  if (!gs.template sum<0>(nullptr, nullptr)) return;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    x[k] = 0.0; r[k] = 0.0; z[k] = 0.0; p[k] = 0.0;
    if (!own[k]) continue;
    const double bv = realb[k] ? q[k] - black(k) : 0.0;
    z[k] = bv * si[k];
    r[k] = bv;
    zg[q0 + k * T] = z[k];
    pg[q0 + k * T] = 0.0;
  }
  dot(r, z, std::true_type{});
  if (!gs.template sum<2>(sum, tot)) return;
  fin_cg_init(S, tot[0], tot[1], rtol_inst ? rtol_inst[inst] : rtol, maxit, true);
  S.beta = 0.0;   // the first direction is z: p = z + 0 * 0
  while (S.active) {
    const double beta = S.beta;
    const double* const zi = zg + g.soff;
    const double* const pi = pg + g.soff;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (own[k])
        Tr[q0 + k * T] =
            red(k, [&](int m) { return __ldcg(zi + m) + beta * __ldcg(pi + m); }, 0.0);
    if (!gs.template sum<0>(nullptr, nullptr)) return;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (!own[k]) continue;
      const double pv = z[k] + beta * p[k];
      p[k] = pv;
      pg[q0 + k * T] = pv;
      q[k] = realb[k] ? -sB[threadIdx.x + k * T] * pv + black(k) : 0.0;
    }
    dot(p, q, std::false_type{});
    if (!gs.template sum<1>(sum, tot)) return;
    fin_cg_q(S, tot[0]);
    if (!S.active) break;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (!own[k]) continue;
      x[k] = x[k] + S.alpha * p[k];
      const double rn = r[k] - S.alpha * q[k];
      r[k] = rn;
      z[k] = rn * si[k];
      zg[q0 + k * T] = z[k];
    }
    dot(r, z, std::false_type{});
    if (!gs.template sum<1>(sum, tot)) return;
    fin_cg_x(S, tot[0]);
  }
  // d_r = A_rr^-1 (F_r - A_rb d_b), d_b = x
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (own[k]) xg[q0 + k * T] = x[k];
  if (!gs.template sum<0>(nullptr, nullptr)) return;
  const double* const xi = xg + g.soff;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (!own[k]) continue;
    const RbNode nr = rb_node(g, q0 + k * T, 0), nk = rb_node(g, q0 + k * T, 1);
    if (realr[k]) d[nr.node] = red(k, [&](int m) { return __ldcg(xi + m); }, F[nr.node]);
    if (realb[k]) d[nk.node] = x[k];
  }
  if (fb.lead && threadIdx.x == 0) ks[inst] = S;
}

}  // namespace tcad
