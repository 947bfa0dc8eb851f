// The red-black BiCGStab of a pack larger than one wave of blocks: J streamed
// through shared memory.
//
// A pass (red: t = E x, black: x - F t) is one read of a colour's J (312 bytes a
// slot in 3D, 232 in 2D) against 70 to 120 bytes of vectors that mostly stay in
// L2, so it should run at the copy rate.  With J loaded where it is used
// (k_rb_red, k_rb_v, k_rb_t) a thread's 39 row entries compete with its gathers
// for registers: at 48 registers and 5 CTAs per SM the 983k-node tri-gate's
// passes read J at 2.6 to 3.6 TB/s.  Here one CTA of 16 warps per SM walks the
// flat blocks, each warp owns one warp tile of a block (a contiguous run of
// 10 KB), and lane 0 copies the warp's tile of the NEXT block with
// cp.async.bulk as soon as the present one is consumed: up to 160 KB in flight
// per SM without a register, next to the gathers.  J is read with an
// evict-first policy, so that it does not push the vectors out of L2.  (8 warps
// of two buffers each wait for their gathers, 6.6 of 11 stall cycles per issue,
// and take 28.5 / 36 / 33 us a pass.)
//
// Successive launches overlap (programmatic dependent launch): J does not depend
// on the vectors, so a CTA of the next kernel starts as soon as its SM is free,
// copies its first tiles, and only then waits for the present kernel to end.
//
// Two sequences run an iteration:
//   formed (vectors that fit in L2 together): red(p), v, red(s), t, x -- p and s
//     are formed where they are gathered, and s is never stored;
//   stored: k_bi_p, red, v, k_bi_s, red, t, k_bi_x.
// Tried and slower: the formed sequence in one cooperative launch (195 us per
// iteration of the 983k-node tri-gate against 160: a static split leaves every
// grid barrier 4 to 8 us of waiting for the slowest SM).
#pragma once

namespace tcad {

constexpr int kRbStreamSlots = 512;       // most slots of a flat block
constexpr int NTS = 512;                  // threads: one slot each
// passes: red(p) and red(s) formed, red(X); v and t formed, and stored; the true
// residual
enum RbPass { kRbRedP, kRbRedS, kRbRed, kRbV, kRbT, kRbVs, kRbTs, kRbTrue };
constexpr bool rb_is_red(int pass) { return pass <= kRbRed; }
constexpr int rb_sums(int pass) { return pass == kRbT ? 3 : pass == kRbTs ? 2 : 1; }
// the formed sequence up to this many slots: its x, r, rh, p, v, t and red result
// (168 bytes a slot) then stay in L2 (126 MB).  Per iteration, formed / stored:
// 491k slots 160 / 180 us, 983k slots 335 / 322 us.
constexpr int64_t kRbFormSlots = 600000;

template <int DIM>
constexpr size_t rb_stream_smem() {
  return (size_t)(NTS / 32) * Stencil<DIM>::NE * 32 * sizeof(double);
}

// J of more than this many bytes is read evict-first; less stays in L2 (126 MB)
// from one pass to the next along with the vectors
constexpr int64_t kRbKeepBytes = (int64_t)80 << 20;

__device__ __forceinline__ uint64_t stream_policy(bool keep) {
  uint64_t p;
  if (keep)
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  else
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// rb_couple_f on gathered values xv[d][c]; Jt: the slot's column of its tile
template <int DIM>
__device__ __forceinline__ void rb_couple_r(const double* Jt, const double (&xv)[2 * DIM][3],
                                            double& y0, double& y1, double& y2) {
  double t0 = 0.0, t1 = 0.0, t2 = 0.0;
#pragma unroll
  for (int d = 0; d < 2 * DIM; ++d) {
    const int e = 9 + 5 * d;
    t0 += Jt[32 * e] * xv[d][0];
    t1 += Jt[32 * (e + 1)] * xv[d][0] + Jt[32 * (e + 2)] * xv[d][1];
    t2 += Jt[32 * (e + 3)] * xv[d][0] + Jt[32 * (e + 4)] * xv[d][2];
  }
  double d[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) d[e] = Jt[32 * e];
  y0 = d[0] * t0 + d[1] * t1 + d[2] * t2;
  y1 = d[3] * t0 + d[4] * t1 + d[5] * t2;
  y2 = d[6] * t0 + d[7] * t1 + d[8] * t2;
}

// a flat block of the slot pack
struct RbBlk {
  int64_t id, begin;
  int len, inst;   // len 0: nothing to do
};

__device__ __forceinline__ RbBlk rb_blk(const tcad_pack_t& pkb, int64_t id) {
  const FlatBlock fb = flat_block(pkb, id);
  return RbBlk{id, fb.begin, (int)(fb.end - fb.begin), fb.inst};
}

// shared memory of a streaming CTA (next to the dynamic tiles)
struct RbStreamShared {
  uint64_t bar[NTS / 32];
  double sum[2][3][NTS / 32];
};

template <int DIM>
struct RbStreamer {
  static constexpr int NE = Stencil<DIM>::NE, NW = NTS / 32, ND = 2 * DIM;
  const tcad_pack_t& pkb;
  const RbMap& mp;
  const double *JR, *JB;
  RbStreamShared& sh;
  double* tile;      // the warp's buffer
  uint64_t policy;
  int lane, warp, par;
  int64_t pend;      // block whose tile the buffer holds or waits for (-1: none)
  int pcol;          // and its colour
  unsigned phase;
  bool lost;         // a copy did not arrive within its limit

  __device__ __forceinline__ RbStreamer(const tcad_pack_t& pkb_, const RbMap& mp_,
                                        const double* JR_, const double* JB_,
                                        RbStreamShared& sh_, double* tiles)
      : pkb(pkb_), mp(mp_), JR(JR_), JB(JB_), sh(sh_) {
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    tile = tiles + (size_t)warp * NE * 32;
    policy = stream_policy(pkb.n_nodes * (2 * NE * 8) <= kRbKeepBytes);
    par = 0;
    pend = -1;
    pcol = 0;
    phase = 0u;
    lost = false;
    if (lane == 0) {
      mbar_init(&sh.bar[warp]);
      fence_async();
    }
    __syncwarp();
  }

  // start copying the warp's tile of block q, colour col (every lane has
  // read the buffer); hold: a copy that never comes (test hook)
  __device__ __forceinline__ void issue(const RbBlk& q, int col, bool hold = false) {
    pend = -1;
    if (warp * 32 >= q.len) return;
    pend = q.id;
    pcol = col;
    if (lane == 0 && !lost) {
      constexpr unsigned n = NE * 32 * sizeof(double);
      mbar_expect(&sh.bar[warp], n);
      if (!hold)
        bulk_copy(tile, (col ? JB : JR) + ((q.begin >> 5) + warp) * (NE * 32), n, &sh.bar[warp],
                  policy);
    }
  }
  __device__ __forceinline__ void arrive() {
    if (!lost) {
      lost = !mbar_wait(&sh.bar[warp], phase);
      if (!lost) phase ^= 1u;
    }
    pend = -1;
  }
  // at the kernel's end: whether a copy was lost (lane 0 has then waited for it again)
  __device__ __forceinline__ bool end() {
    if (lost && lane == 0) (void)mbar_wait(&sh.bar[warp], phase);
    return lost;
  }

  // block sums of v (all threads) into out[0..NS): warp sums, then the 16 of
  // them pairwise
  template <int NS>
  __device__ __forceinline__ void block_sums(double (&v)[NS], double* out) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
      if (lane == 0) sh.sum[par][q][warp] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < NS) {
      const double* const e = sh.sum[par][threadIdx.x];
      double s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = e[i] + e[i + 8];
      out[threadIdx.x] = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    }
    par ^= 1;   // (the next sums go to the other buffer, across a barrier)
  }

  // one block of a pass; nxt, ncol: what the warp's buffer is for after it;
  // S: the instance's state.  Between x and v, w.p holds p - omega v: a
  // neighbour's p is then formed from two values, r + beta w.p, the bits of
  // r + beta (p - omega v); s is formed from r and v and never stored.
  //   kRbRedP, kRbRedS, kRbRed:  Tr = E p, E s, E X
  //   kRbV:    w.p = p, w.v = p - F Tr; (rh, v)   (restart: rh = r)
  //   kRbT:    w.t = s - F Tr; (s, s), (t, s), (t, t)
  //   kRbVs, kRbTs: the same with p and s as stored, without (s, s)
  //   kRbTrue: w.r = rhs - (X - F Tr); (r, r)
  template <int PASS>
  __device__ __forceinline__ void block(const RbBlk& q, const RbBlk& nxt, int ncol,
                                        const KState& S, const double* X, double* Tr,
                                        const BiVec& w, const double* rhs, double* partial) {
    constexpr int NS = rb_sums(PASS), col = rb_is_red(PASS) ? 0 : 1;
    const int64_t VS = pkb.n_nodes;
    const RbGeo g = rb_geo(pkb, mp, q.inst);
    const double alpha = S.alpha, beta = S.beta;
    const int restart = S.restart;
    const bool here = warp * 32 < q.len;
    if (pend >= 0 && (!here || pend != q.id || pcol != col)) arrive();
    if (here && pend < 0) issue(q, col);
    double v[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) v[k] = 0.0;
    const int64_t slot = q.begin + threadIdx.x;
    const bool mine = (int)threadIdx.x < q.len;
    bool real = false;
    double xv[ND][3], own[3][3];
    if (mine) {
      const RbNode nd = rb_node(g, slot, col);
      real = nd.real;
      if (real) {
        int m[6];
        rb_nbrs<DIM>(g, nd, (int)(slot - g.soff), m);
#pragma unroll
        for (int d = 0; d < ND; ++d)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int64_t a = c * VS + g.soff + m[d];
            if (PASS == kRbRedP) {
              const double rv = w.r[a], pv = w.p[a];
              xv[d][c] = restart ? rv : rv + beta * pv;
            } else if (PASS == kRbRedS) {
              xv[d][c] = w.r[a] - alpha * w.v[a];
            } else {
              xv[d][c] = PASS == kRbRed ? X[a] : Tr[a];
            }
          }
      }
      if (!rb_is_red(PASS)) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int64_t a = c * VS + slot;
          own[0][c] = PASS == kRbTrue ? X[a] : PASS == kRbVs ? w.p[a] : PASS == kRbTs ? w.s[a]
                                                                                     : w.r[a];
          if (PASS == kRbV) own[1][c] = w.p[a];
          if (PASS == kRbT) own[1][c] = w.v[a];
          if (PASS == kRbTrue) own[1][c] = rhs[a];
          if (PASS == kRbV || PASS == kRbVs) own[2][c] = w.rh[a];
        }
      }
    }
    if (here) arrive();
    double u[3] = {0.0, 0.0, 0.0};
    if (real) rb_couple_r<DIM>(tile + lane, xv, u[0], u[1], u[2]);
    __syncwarp();
    issue(nxt, ncol);
    if (mine) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t a = c * VS + slot;
        if (rb_is_red(PASS)) {
          Tr[a] = u[c];
        } else if (PASS == kRbV) {
          const double rv = own[0][c], pn = restart ? rv : rv + beta * own[1][c];
          const double hv = restart ? rv : own[2][c];
          const double y = real ? pn - u[c] : 0.0;
          if (restart) w.rh[a] = rv;
          w.p[a] = pn;
          w.v[a] = y;
          v[0] += hv * y;
        } else if (PASS == kRbT) {
          const double sv = own[0][c] - alpha * own[1][c];
          const double y = real ? sv - u[c] : 0.0;
          w.t[a] = y;
          v[0] += sv * sv;
          v[NS - 2] += y * sv;
          v[NS - 1] += y * y;
        } else if (PASS == kRbVs) {
          const double y = real ? own[0][c] - u[c] : 0.0;
          w.v[a] = y;
          v[0] += own[2][c] * y;
        } else if (PASS == kRbTs) {
          const double y = real ? own[0][c] - u[c] : 0.0;
          w.t[a] = y;
          v[0] += y * own[0][c];
          v[NS - 1] += y * y;
        } else {
          const double y = real ? own[0][c] - u[c] : 0.0;
          const double r = own[1][c] - y;
          w.r[a] = r;
          v[0] += r * r;
        }
      }
    }
    if (!rb_is_red(PASS)) block_sums<NS>(v, partial + q.id * 4);
  }

  // the vectors of the x step, loaded one block ahead
  struct XVec {
    double e[6][3];   // x, p, r, v, t, rh
  };
  __device__ __forceinline__ void x_load(const RbBlk& q, const double* X, const BiVec& w,
                                         XVec& o) {
    if ((int)threadIdx.x >= q.len) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t a = c * pkb.n_nodes + q.begin + threadIdx.x;
      o.e[0][c] = X[a]; o.e[1][c] = w.p[a]; o.e[2][c] = w.r[a];
      o.e[3][c] = w.v[a]; o.e[4][c] = w.t[a]; o.e[5][c] = w.rh[a];
    }
  }
  // x += alpha p + omega s, r = s - omega t, w.p = p - omega v; (rh, r), (r, r),
  // (rh, rh)
  __device__ __forceinline__ void x_block(const RbBlk& q, const XVec& o, const KState& S,
                                          double* X, const BiVec& w, double* partial) {
    const double alpha = S.alpha, omega = S.omega;
    double v[3] = {0.0, 0.0, 0.0};
    if ((int)threadIdx.x < q.len)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int64_t a = c * pkb.n_nodes + q.begin + threadIdx.x;
        const double sv = o.e[2][c] - alpha * o.e[3][c], hv = o.e[5][c];
        X[a] = o.e[0][c] + alpha * o.e[1][c] + omega * sv;
        const double r = sv - omega * o.e[4][c];
        w.r[a] = r;
        w.p[a] = o.e[1][c] - omega * o.e[3][c];
        v[0] += hv * r;
        v[1] += r * r;
        v[2] += hv * hv;
      }
    block_sums<3>(v, partial + q.id * 4);
  }
};

// sums over instance inst's blocks of partial[b * 4 + q], valid in thread 0
template <int NS>
__device__ __forceinline__ void rb_totals(const tcad_pack_t& pkb, int inst, const double* partial,
                                          double (&sum)[NS][NTS / 32], double* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t b1 = pkb.flat_off[inst + 1];
  double v[NS];
#pragma unroll
  for (int q = 0; q < NS; ++q) v[q] = 0.0;
  for (int64_t b = pkb.flat_off[inst] + threadIdx.x; b < b1; b += NTS)
#pragma unroll
    for (int q = 0; q < NS; ++q) v[q] += __ldcg(&partial[b * 4 + q]);
#pragma unroll
  for (int q = 0; q < NS; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    if (lane == 0) sum[q][warp] = v[q];
  }
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      double s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = sum[q][i] + sum[q][i + 8];
      tot[q] = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    }
}

// ---- one step per launch over nblk blocks (blk: their numbers, null: all) of the
// instances still iterating (all: of every instance).  A CTA adds its count of
// blocks to the instance's ticket once; the last CTA takes the totals into ks.
// Where a copy did not arrive within its limit a word of its own says so, which the host
// reads with the states.
struct RbTicket {
  unsigned count = 0u;
  int inst = -1;
};

template <int NS, class FIN>
__device__ __forceinline__ void rb_flush(const tcad_pack_t& pkb, RbTicket& tk, double* partial,
                                         unsigned* ticket, const FIN& fin) {
  __shared__ double s_tot[NS][NTS / 32];
  __shared__ int s_last;
  if (threadIdx.x < 32) {      // the threads that stored the CTA's partials
    __threadfence();
    __syncwarp();
  }
  if (threadIdx.x == 0) {
    const unsigned nb = (unsigned)(pkb.flat_off[tk.inst + 1] - pkb.flat_off[tk.inst]);
    s_last = atomicAdd(&ticket[tk.inst], tk.count) + tk.count == nb;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    double tot[NS];
    rb_totals<NS>(pkb, tk.inst, partial, s_tot, tot);
    if (threadIdx.x == 0) {
      ticket[tk.inst] = 0u;
      fin(tk.inst, tot);
    }
  }
  __syncthreads();
  tk.count = 0u;
}

// the i-th block; len 0 when its instance takes no part (ks null: all do)
__device__ __forceinline__ RbBlk rb_fetch(const tcad_pack_t& pkb, const KState* ks, int64_t i,
                                          int64_t nblk, const int32_t* blk) {
  RbBlk q{-1, 0, 0, 0};
  if (i < nblk) {
    q = rb_blk(pkb, blk ? (int64_t)blk[i] : i);
    if (ks && !ks[q.inst].active) q.len = 0;
  }
  return q;
}

template <int DIM, int PASS>
__global__ void __launch_bounds__(NTS, 1)
k_rb_stream(const tcad_pack_t pkb, const RbMap mp, const double* __restrict__ JR,
            const double* __restrict__ JB, const double* X, double* Tr, BiVec w,
            const double* rhs, KState* ks, bool all, double* partial, unsigned* ticket,
            int rearm, int64_t nblk, const int32_t* __restrict__ blk, unsigned* lost, bool hold) {
  constexpr int NS = rb_sums(PASS), col = rb_is_red(PASS) ? 0 : 1;
  extern __shared__ __align__(128) double s_tiles[];
  __shared__ RbStreamShared sh;
  RbStreamer<DIM> st(pkb, mp, JR, JB, sh, s_tiles);
  auto fin = [&](int inst, const double* tot) {
    if (PASS == kRbV || PASS == kRbVs) fin_v(ks[inst], tot[0]);
    if (PASS == kRbT) fin_s(ks[inst], tot[0]);
    if (PASS == kRbT || PASS == kRbTs) fin_t(ks[inst], tot[NS > 1 ? NS - 2 : 0], tot[NS - 1]);
    if (PASS == kRbTrue) fin_true(ks[inst], tot[0], rearm);
  };
  RbTicket tk;
  // J and the tables are older than the kernel before this one; its states and
  // vectors are not
  RbBlk cur = rb_fetch(pkb, nullptr, blockIdx.x, nblk, blk);
  st.issue(cur, col, hold && blockIdx.x == 0 && st.warp == 0);
  launch_dependents();
  wait_prior();
  if (!all && !ks[cur.inst].active) cur.len = 0;
  for (int64_t i = blockIdx.x; i < nblk; i += gridDim.x) {
    const RbBlk nxt = rb_fetch(pkb, all ? nullptr : ks, i + gridDim.x, nblk, blk);
    if (cur.len > 0) {
      if (!rb_is_red(PASS)) {
        if (tk.inst >= 0 && tk.inst != cur.inst) rb_flush<NS>(pkb, tk, partial, ticket, fin);
        tk.inst = cur.inst;
        ++tk.count;
      }
      st.template block<PASS>(cur, nxt, col, ks[cur.inst], X, Tr, w, rhs, partial);
    } else {
      if (st.pend >= 0) st.arrive();
      st.issue(nxt, col);
    }
    cur = nxt;
  }
  if (tk.inst >= 0) rb_flush<NS>(pkb, tk, partial, ticket, fin);
  if (st.end()) *lost = 1u;
}

template <int DIM>
__global__ void __launch_bounds__(NTS, 1)
k_rb_stream_x(const tcad_pack_t pkb, const RbMap mp, double* X, BiVec w, KState* ks,
              double* partial, unsigned* ticket, int64_t nblk, const int32_t* __restrict__ blk) {
  __shared__ RbStreamShared sh;
  RbStreamer<DIM> st(pkb, mp, nullptr, nullptr, sh, nullptr);
  typename RbStreamer<DIM>::XVec a, b;
  auto fin = [&](int inst, const double* tot) { fin_x(ks[inst], tot[0], tot[1], tot[2]); };
  RbTicket tk;
  launch_dependents();
  wait_prior();
  RbBlk cur = rb_fetch(pkb, ks, blockIdx.x, nblk, blk);
  st.x_load(cur, X, w, a);
  for (int64_t i = blockIdx.x; i < nblk; i += gridDim.x) {
    const RbBlk nxt = rb_fetch(pkb, ks, i + gridDim.x, nblk, blk);
    st.x_load(nxt, X, w, b);
    if (cur.len > 0) {
      if (tk.inst >= 0 && tk.inst != cur.inst) rb_flush<3>(pkb, tk, partial, ticket, fin);
      tk.inst = cur.inst;
      ++tk.count;
      st.x_block(cur, a, ks[cur.inst], X, w, partial);
    }
    cur = nxt;
    a = b;
  }
  if (tk.inst >= 0) rb_flush<3>(pkb, tk, partial, ticket, fin);
}

}  // namespace tcad
