// The red and black passes of the red-black BiCGStab as persistent kernels
// that stream the colour rows of J through shared memory.
//
// These passes are one read of a colour's J (312 bytes a slot in 3D, 232 in
// 2D) against 70 to 120 bytes of vectors that mostly stay in L2, so they should
// run at the copy rate.  With J loaded where it is used (k_rb_red, k_rb_v,
// k_rb_t) a thread's 39 row entries compete with its gathers for registers:
// at 48 registers and 5 CTAs per SM the 983k-node tri-gate's passes read J at
// 2.6 to 3.6 TB/s.  Here one CTA per SM walks the flat blocks, each warp owns
// two of a block's sixteen warp tiles, and lane 0 copies the warp's tiles of the
// NEXT block (contiguous runs of 10 KB) with cp.async.bulk as soon as the
// present ones are consumed: 80 to 160 KB in flight per SM without a register,
// while the gathers have 255 registers a thread to be in flight together.
// J is read with an evict-first policy, so that it does not push the vectors
// out of L2.  983k-node tri-gate, one instance: red 42.7 -> 28.5 us (153 MB of J:
// 3.6 -> 5.4 TB/s), v 58.0 -> 36.1, t 53.4 -> 33.3; an iteration 240 -> 166 us.
//
// Expressions, the slots of a thread and the order of every sum are those of
// the per-step kernels: bit-identical to them.  A CTA adds its count of blocks
// to the instance's ticket once (not once per block).
#pragma once

namespace tcad {

constexpr int kRbStreamSlots = 2 * NT;   // the flat block these kernels take
constexpr int kRbRed = 0, kRbV = 1, kRbT = 2, kRbTrue = 3;

template <int DIM>
constexpr size_t rb_stream_smem() {
  return (size_t)2 * (NT / 32) * Stencil<DIM>::NE * 32 * sizeof(double);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}

// bulk copy of n bytes (a multiple of 16) global -> shared, completing on b
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned n, uint64_t* b,
                                          uint64_t policy) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)),
               "r"(n)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1], %2, [%3], %4;" ::"r"(smem_addr(dst)),
      "l"(src), "r"(n), "r"(smem_addr(b)), "l"(policy)
      : "memory");
}

__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// wait for the phase, at most `tries` polls (each suspends for a while)
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, unsigned tries) {
  const unsigned a = smem_addr(b);
  for (unsigned i = 0; i < tries; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
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

// PASS kRbRed:  out = E X (X black, all instances when ks is null)
//      kRbV:    w.v = w.p - F X (X = E p); (rh, v)
//      kRbT:    w.t = w.s - F X (X = E s); (t, s), (t, t)
//      kRbTrue: out = rhs - (xb - F X) (X = E xb); (r, r), every instance
// `fail`: the states of all instances (status TCAD_ERR_CUDA when a copy did
// not arrive within its limit)
template <int DIM, int PASS>
__global__ void __launch_bounds__(NT, 1)
k_rb_stream(const tcad_pack_t pkb, const RbMap mp, const double* __restrict__ Jc,
            const double* __restrict__ X, double* __restrict__ out, BiVec w,
            const double* __restrict__ rhs, const double* __restrict__ xb, const KState* ks,
            KState* fail, double* partial, unsigned* ticket, int rearm, int64_t nblk,
            const int32_t* __restrict__ blk) {
  constexpr int NE = Stencil<DIM>::NE, NW = NT / 32, ND = 2 * DIM;
  constexpr int NS = PASS == kRbT ? 2 : 1;
  constexpr unsigned kBytes = NE * 32 * sizeof(double);
  extern __shared__ __align__(128) double s_tiles[];   // [NW][2][NE * 32]
  __shared__ uint64_t s_bar[NW][2];
  __shared__ double s_sum[2][NS][NW];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* const tile = s_tiles + (size_t)warp * 2 * NE * 32;
  const int64_t VS = pkb.n_nodes;
  const uint64_t policy = evict_first_policy();
  if (lane == 0) {
    mbar_init(&s_bar[warp][0]);
    mbar_init(&s_bar[warp][1]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();

  struct Blk {
    FlatBlock fb;
    int64_t id;
    bool on;
  };
  auto fetch = [&](int64_t i) {
    Blk q;
    q.on = false;
    if (i < nblk) {
      q.id = blk ? (int64_t)blk[i] : i;
      q.fb = flat_block(pkb, q.id);
      q.on = !ks || ks[q.fb.inst].active;
    }
    return q;
  };
  auto has = [&](const Blk& q, int h) {
    return q.on && q.fb.begin + (warp + h * NW) * 32 < q.fb.end;
  };
  auto issue = [&](const Blk& q, int h) {
    if (lane == 0 && has(q, h))
      bulk_load(tile + h * NE * 32, Jc + ((q.fb.begin >> 5) + warp + h * NW) * (NE * 32), kBytes,
                &s_bar[warp][h], policy);
  };
  // once the CTA has stored all its partials of an instance: its ticket, and
  // the totals by the last CTA
  auto flush = [&](int inst, unsigned count) {
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned nb = (unsigned)(pkb.flat_off[inst + 1] - pkb.flat_off[inst]);
      s_last = atomicAdd(&ticket[inst], count) + count == nb;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      double tot[NS];
      Reduce<NS>::total(pkb, inst, partial, tot);
      if (threadIdx.x == 0) {
        ticket[inst] = 0u;
        if (PASS == kRbV) fin_v(fail[inst], tot[0]);
        if (PASS == kRbT) fin_t(fail[inst], tot[0], tot[NS - 1]);
        if (PASS == kRbTrue) fin_true(fail[inst], tot[0], rearm);
      }
    }
    __syncthreads();
  };

  unsigned phase[2] = {0u, 0u}, tries = 1u << 20, count = 0u;
  int cinst = -1, par = 0;
  Blk cur = fetch(blockIdx.x);
  issue(cur, 0);
  issue(cur, 1);
  for (int64_t i = blockIdx.x; i < nblk; i += gridDim.x) {
    const Blk nxt = fetch(i + gridDim.x);
    double v[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) v[q] = 0.0;
    if (cur.on) {
      const RbGeo g = rb_geo(pkb, mp, cur.fb.inst);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!has(cur, h)) {
          issue(nxt, h);
          continue;
        }
        const int64_t slot = cur.fb.begin + (warp + h * NW) * 32 + lane;
        const bool mine = slot < cur.fb.end;
        bool real = false;
        double xv[ND][3], own[2][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) { own[0][c] = 0.0; own[1][c] = 0.0; }
        if (mine) {
          const RbNode q = rb_node(g, slot, PASS == kRbRed ? 0 : 1);
          real = q.real;
          if (real) {
            int m[6];
            rb_nbrs<DIM>(g, q, (int)(slot - g.soff), m);
            const double* __restrict__ xi = X + g.soff;
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
              for (int c = 0; c < 3; ++c) xv[d][c] = xi[c * VS + m[d]];
          }
          if (PASS != kRbRed) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const int64_t a = c * VS + slot;
              own[0][c] = PASS == kRbV ? w.p[a] : PASS == kRbT ? w.s[a] : xb[a];
              if (PASS == kRbV) own[1][c] = w.rh[a];
              if (PASS == kRbTrue) own[1][c] = rhs[a];
            }
          }
        }
        if (!mbar_wait(&s_bar[warp][h], phase[h], tries)) {
          if (lane == 0) {
            fail[cur.fb.inst].status = TCAD_ERR_CUDA;
            fail[cur.fb.inst].active = 0;
          }
          tries = 64u;
        }
        phase[h] ^= 1u;
        double u[3] = {0.0, 0.0, 0.0};
        if (real) rb_couple_r<DIM>(tile + h * NE * 32 + lane, xv, u[0], u[1], u[2]);
        __syncwarp();
        issue(nxt, h);
        if (mine) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const int64_t a = c * VS + slot;
            if (PASS == kRbRed) {
              out[a] = u[c];
            } else if (PASS == kRbV) {
              const double y = real ? own[0][c] - u[c] : 0.0;
              w.v[a] = y;
              v[0] += own[1][c] * y;
            } else if (PASS == kRbT) {
              const double y = real ? own[0][c] - u[c] : 0.0;
              w.t[a] = y;
              v[0] += y * own[0][c];
              v[NS - 1] += y * y;
            } else {
              const double y = real ? own[0][c] - u[c] : 0.0;
              const double r = own[1][c] - y;
              out[a] = r;
              v[0] += r * r;
            }
          }
        }
      }
      if (PASS != kRbRed) {
        if (cinst >= 0 && cinst != cur.fb.inst) {
          flush(cinst, count);
          count = 0u;
        }
        cinst = cur.fb.inst;
        ++count;
#pragma unroll
        for (int q = 0; q < NS; ++q) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
          if (lane == 0) s_sum[par][q][warp] = v[q];
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
          for (int q = 0; q < NS; ++q) {
            double r = lane < NW ? s_sum[par][q][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
            if (lane == 0) partial[cur.id * 4 + q] = r;
          }
        }
        par ^= 1;
      }
    } else {
      issue(nxt, 0);
      issue(nxt, 1);
    }
    cur = nxt;
  }
  if (PASS != kRbRed && cinst >= 0) flush(cinst, count);
}

}  // namespace tcad
