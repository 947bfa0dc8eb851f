// The red-black Schur BiCGStab of a single-instance pack that is too large to be
// resident but whose slot blocks are all on the GPU at once (one wave: two CTAs of 256
// threads per SM, a block of at most 512 slots each), in one cooperative launch.
//
// Vectors and J stay in global memory and are read through L1 (a fifth of the sectors hit)
// and L2, 36 or 54 gathers a slot and pass (the resident kernel's registers do not stretch
// to two slots a thread at two CTAs an SM: 0.9 KB of spills, 49 us an iteration of a 440 x
// 480 diode; here 28, streamed 39).  Within a step no CTA reads what another writes, which the
// restrict qualifiers of the steps' bodies tell the compiler, and the solver's state is in
// shared memory: both slots' gathers then fit in the registers (60 x 56 x 46 tri-gate 40
// us with the state in every thread, 32).  The five steps of an iteration and their sums
// are the resident kernel's (rb_resident.cuh), with GridSync between them: bit-identical
// to launch_bicgstab_rb's per-step loop over the same blocks.
#pragma once

namespace tcad {

// p = r + beta (p - omega v) (restart: r) and s = r - alpha v, formed at the other
// colour's slots from vectors that no CTA writes in that step
struct RbFormP {
  const double* __restrict__ r;
  const double* __restrict__ p;
  const double* __restrict__ v;
  int64_t NS;
  double beta, omega;
  int restart;
  __device__ __forceinline__ double operator()(int m, int c) const {
    const double rv = r[c * NS + m];
    return restart ? rv : rv + beta * (p[c * NS + m] - omega * v[c * NS + m]);
  }
};
struct RbFormS {
  const double* __restrict__ r;
  const double* __restrict__ v;
  int64_t NS;
  double alpha;
  __device__ __forceinline__ double operator()(int m, int c) const {
    return r[c * NS + m] - alpha * v[c * NS + m];
  }
};

// red pass: Tr = E X
template <int DIM, class XF>
__device__ __forceinline__ void rb_wave_red(const RbGeo& g, const FlatBlock& fb, int64_t NS,
                                            const double* __restrict__ JR, const XF& X,
                                            double* __restrict__ Tr) {
  for (int64_t slot = fb.begin + threadIdx.x; slot < fb.end; slot += NT) {
    const RbNode q = rb_node(g, slot, 0);
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
    if (q.real) {
      int m[6];
      rb_nbrs<DIM>(g, q, (int)(slot - g.soff), m);
      rb_couple_f<DIM>(JR, X, slot, m, y0, y1, y2);
    }
    Tr[slot] = y0; Tr[NS + slot] = y1; Tr[2 * NS + slot] = y2;
  }
}

// p, v = S p (Tr = E p), (rh, v); restart: rh = p = r
template <int DIM>
__device__ __forceinline__ double rb_wave_v(const RbGeo& g, const FlatBlock& fb, int64_t NS,
                                            const double* __restrict__ JB,
                                            const double* __restrict__ Tr, const BiVec& w,
                                            double beta, double omega, int restart) {
  const double* __restrict__ R = w.r;
  double* __restrict__ P = w.p;
  double* __restrict__ V = w.v;
  double* __restrict__ RH = w.rh;
  double sum = 0.0;
  for (int64_t slot = fb.begin + threadIdx.x; slot < fb.end; slot += NT) {
    double u[3];
    const bool real = rb_black_u<DIM>(g, JB, Tr, slot, NS, u);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = c * NS + slot;
      const double rv = R[i];
      const double pn = restart ? rv : rv + beta * (P[i] - omega * V[i]);
      const double h = restart ? rv : RH[i];
      const double y = real ? pn - u[c] : 0.0;
      if (restart) RH[i] = rv;
      P[i] = pn;
      V[i] = y;
      sum += h * y;
    }
  }
  return sum;
}

// s = r - alpha v, t = S s (Tr = E s); (s, s), (t, s), (t, t)
template <int DIM>
__device__ __forceinline__ void rb_wave_t(const RbGeo& g, const FlatBlock& fb, int64_t NS,
                                          const double* __restrict__ JB,
                                          const double* __restrict__ Tr, const BiVec& w,
                                          double alpha, double (&sum)[3]) {
  const double* __restrict__ R = w.r;
  const double* __restrict__ V = w.v;
  double* __restrict__ S = w.s;
  double* __restrict__ T = w.t;
  sum[0] = 0.0; sum[1] = 0.0; sum[2] = 0.0;
  for (int64_t slot = fb.begin + threadIdx.x; slot < fb.end; slot += NT) {
    double u[3];
    const bool real = rb_black_u<DIM>(g, JB, Tr, slot, NS, u);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = c * NS + slot;
      const double sv = R[i] - alpha * V[i];
      const double y = real ? sv - u[c] : 0.0;
      S[i] = sv;
      T[i] = y;
      sum[0] += sv * sv;
      sum[1] += y * sv;
      sum[2] += y * y;
    }
  }
}

template <int DIM>
__global__ void __launch_bounds__(NT, 2)
k_bicgstab_rb_wave(const tcad_pack_t pkb, const RbMap mp, const double* __restrict__ JR,
                   const double* __restrict__ JB, const double* __restrict__ b, double* x,
                   double* bR, double* bB, double* Tr, double* xb, double* rhs, BiVec w,
                   KState* ks, double* part, unsigned* bar, double rtol, int maxit,
                   const int32_t* __restrict__ pre_status, const double* __restrict__ rtol_inst,
                   int max_rechecks) {
  GridSync gs;
  gs.init(part, bar);
  const FlatBlock fb = flat_block(pkb, blockIdx.x);
  const int inst = fb.inst;
  const RbGeo g = rb_geo(pkb, mp, inst);
  const int64_t NS = pkb.n_nodes;
  double tot[3];
  __shared__ KState S;   // thread 0's, read by all after a barrier
  double sum[1] = {rb_split_body<DIM>(pkb, mp, fb, b, bR, bB)};
  if (!gs.template sum<1, 2>(sum, tot)) return;
  const double bb = tot[0];
  sum[0] = rb_init_body<DIM>(pkb, mp, fb, JB, bR, bB, rhs, xb, w);
  if (!gs.template sum<1, 2>(sum, tot)) return;
  if (threadIdx.x == 0)
    rb_fin_init(S, tot[0], bb, rtol_inst ? rtol_inst[inst] : rtol, maxit,
                pre_status ? pre_status[inst] : TCAD_OK);
  __syncthreads();
  for (int rechecks = 0;; ++rechecks) {
    while (S.active) {
      rb_wave_red<DIM>(g, fb, NS, JR,
                       RbFormP{w.r + g.soff, w.p + g.soff, w.v + g.soff, NS, S.beta, S.omega,
                               S.restart},
                       Tr);
      if (!gs.template sum<0, 2>(nullptr, nullptr)) return;
      sum[0] = rb_wave_v<DIM>(g, fb, NS, JB, Tr, w, S.beta, S.omega, S.restart);
      if (!gs.template sum<1, 2>(sum, tot)) return;
      if (threadIdx.x == 0) fin_v(S, tot[0]);
      __syncthreads();
      if (!S.active) break;
      rb_wave_red<DIM>(g, fb, NS, JR, RbFormS{w.r + g.soff, w.v + g.soff, NS, S.alpha}, Tr);
      if (!gs.template sum<0, 2>(nullptr, nullptr)) return;
      double s3[3];
      rb_wave_t<DIM>(g, fb, NS, JB, Tr, w, S.alpha, s3);
      if (!gs.template sum<3, 2>(s3, tot)) return;
      if (threadIdx.x == 0) {
        fin_s(S, tot[0]);
        fin_t(S, tot[1], tot[2]);
      }
      __syncthreads();
      bi_x_body<double>(pkb, fb, xb, w, S.alpha, S.omega, s3);
      if (!gs.template sum<3, 2>(s3, tot)) return;
      if (threadIdx.x == 0) fin_x(S, tot[0], tot[1], tot[2]);
      __syncthreads();
    }
    // true Schur residual r = rhs - S x
    rb_wave_red<DIM>(g, fb, NS, JR, RbVal{xb + g.soff, NS}, Tr);
    if (!gs.template sum<0, 2>(nullptr, nullptr)) return;
    sum[0] = rb_true_body<DIM>(pkb, mp, fb, JB, Tr, rhs, xb, w.r);
    if (!gs.template sum<1, 2>(sum, tot)) return;
    if (threadIdx.x == 0) fin_true(S, tot[0], rechecks < max_rechecks ? 1 : 0);
    __syncthreads();
    if (!S.active) break;
  }
  rb_merge_body<DIM>(pkb, mp, fb, bR, Tr, xb, x, pre_status && pre_status[inst] != TCAD_OK);
  if (blockIdx.x == 0 && threadIdx.x == 0) ks[inst] = S;
}

}  // namespace tcad
