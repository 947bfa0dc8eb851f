// General-CSR Krylov path of linsolve.solve_linear (pytcad/linsolve.py:725-985):
// GMRES(m) and BiCGStab, right node-block-Jacobi preconditioning
// (pytcad/linsolve.py:363-427), convergence on the true residual norm.
//
// One linear system per call.  SpMV assigns a group of 8 lanes to a row
// (device Jacobians carry ~10 entries per row), so a warp reads four rows'
// entries with unit stride.  Dot products reduce per block; the last block
// to finish sums the block partials in block order (deterministic) and
// updates the solver's state on the device (BiCGStab's scalars; GMRES's column
// of H, its Givens rotations and residual norm), so an iteration runs without
// the host, which looks at the state every few iterations.  Once a state is
// done, the kernels already queued return at once.
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "grid_sync.cuh"

namespace tcad {
namespace csr {

constexpr int NT = 256;
constexpr int kRowsPerBlock = NT / 8;
constexpr int64_t kGridBlocks = 592;   // 4 per SM: most blocks of a reducing kernel

struct Sys {
  int64_t n;
  const int32_t* ptr;
  const int32_t* idx;
  const double* val;
};

__global__ void __launch_bounds__(NT) k_spmv(Sys A, const double* x, double* y) {
  chain_in();
  const int64_t row = (int64_t)blockIdx.x * kRowsPerBlock + (threadIdx.x >> 3);
  const int lane = threadIdx.x & 7;
  double s = 0.0;
  if (row < A.n) {
    const int a = A.ptr[row], b = A.ptr[row + 1];
    for (int q = a + lane; q < b; q += 8) s += A.val[q] * x[A.idx[q]];
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
  if (row < A.n && lane == 0) y[row] = s;
}

// Node-block-Jacobi: invert the bs x bs diagonal blocks (bs = 3; bs = 1 is
// point Jacobi).  flag[0] != 0 when a block is singular (|det| < 1e-300) or
// non-finite -- the caller then falls back to point Jacobi like the
// reference falls through its preconditioner chain.
__global__ void k_bj_setup(Sys A, int bs, double* __restrict__ inv, int* __restrict__ flag) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nb = A.n / bs;
  if (b >= nb) return;
  double a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int r = 0; r < bs; ++r) {
    const int64_t row = b * bs + r;
    for (int q = A.ptr[row]; q < A.ptr[row + 1]; ++q) {
      const int64_t c = A.idx[q] - b * bs;
      if (c >= 0 && c < bs) a[r * bs + c] += A.val[q];
    }
  }
  if (bs == 1) {
    const bool ok = isfinite(a[0]) && fabs(a[0]) >= 1e-300;
    if (!ok) atomicExch(flag, 1);
    inv[b] = ok ? 1.0 / a[0] : 1.0;
    return;
  }
  const double c00 = a[4] * a[8] - a[5] * a[7];
  const double c01 = a[5] * a[6] - a[3] * a[8];
  const double c02 = a[3] * a[7] - a[4] * a[6];
  const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
  bool ok = isfinite(det) && fabs(det) >= 1e-300;
  if (!ok) atomicExch(flag, 1);
  const double id = ok ? 1.0 / det : 0.0;
  double* o = inv + 9 * b;
  o[0] = c00 * id;
  o[1] = (a[2] * a[7] - a[1] * a[8]) * id;
  o[2] = (a[1] * a[5] - a[2] * a[4]) * id;
  o[3] = c01 * id;
  o[4] = (a[0] * a[8] - a[2] * a[6]) * id;
  o[5] = (a[2] * a[3] - a[0] * a[5]) * id;
  o[6] = c02 * id;
  o[7] = (a[1] * a[6] - a[0] * a[7]) * id;
  o[8] = (a[0] * a[4] - a[1] * a[3]) * id;
}

// 6 x 6 node blocks (the real-equivalent form of a complex 3 x 3 node block:
// the AC small-signal systems), inverted by Gauss-Jordan elimination with
// partial pivoting in registers.
__global__ void k_bj_setup6(Sys A, double* __restrict__ inv, int* __restrict__ flag) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nb = A.n / 6;
  if (b >= nb) return;
  double a[36], o[36];
#pragma unroll
  for (int q = 0; q < 36; ++q) {
    a[q] = 0.0;
    o[q] = (q % 7 == 0) ? 1.0 : 0.0;
  }
  for (int r = 0; r < 6; ++r) {
    const int64_t row = b * 6 + r;
    for (int q = A.ptr[row]; q < A.ptr[row + 1]; ++q) {
      const int64_t c = A.idx[q] - b * 6;
      if (c >= 0 && c < 6) a[r * 6 + c] += A.val[q];
    }
  }
  double scale = 0.0;
#pragma unroll
  for (int q = 0; q < 36; ++q) scale = fmax(scale, fabs(a[q]));
  bool ok = isfinite(scale) && scale > 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    int piv = k;
    double best = fabs(a[k * 6 + k]);
#pragma unroll
    for (int r = k + 1; r < 6; ++r)
      if (fabs(a[r * 6 + k]) > best) { best = fabs(a[r * 6 + k]); piv = r; }
    if (!(best > 1e-300 * scale)) ok = false;
    if (piv != k) {
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        double t = a[k * 6 + c]; a[k * 6 + c] = a[piv * 6 + c]; a[piv * 6 + c] = t;
        t = o[k * 6 + c]; o[k * 6 + c] = o[piv * 6 + c]; o[piv * 6 + c] = t;
      }
    }
    const double ip = ok ? 1.0 / a[k * 6 + k] : 0.0;
#pragma unroll
    for (int c = 0; c < 6; ++c) { a[k * 6 + c] *= ip; o[k * 6 + c] *= ip; }
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      if (r == k) continue;
      const double f = a[r * 6 + k];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        a[r * 6 + c] -= f * a[k * 6 + c];
        o[r * 6 + c] -= f * o[k * 6 + c];
      }
    }
  }
  if (!ok) atomicExch(flag, 1);
  double* out = inv + 36 * b;
#pragma unroll
  for (int q = 0; q < 36; ++q) out[q] = ok ? o[q] : 0.0;
}

// z = M^-1 r (bs = 3 or 6 blocks, bs = 1 diagonal, bs = 0 identity)
__global__ void k_bj_apply(int64_t n, int bs, const double* __restrict__ inv,
                           const double* __restrict__ r, double* __restrict__ z) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (bs == 3) {
    if (t >= n / 3) return;
    const double* m = inv + 9 * t;
    const double a = r[3 * t], b = r[3 * t + 1], c = r[3 * t + 2];
    z[3 * t] = m[0] * a + m[1] * b + m[2] * c;
    z[3 * t + 1] = m[3] * a + m[4] * b + m[5] * c;
    z[3 * t + 2] = m[6] * a + m[7] * b + m[8] * c;
  } else if (bs == 6) {
    if (t >= n / 6) return;
    const double* m = inv + 36 * t;
    double v[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] = r[6 * t + c];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      double acc = 0.0;
#pragma unroll
      for (int c = 0; c < 6; ++c) acc += m[6 * q + c] * v[c];
      z[6 * t + q] = acc;
    }
  } else if (t < n) {
    z[t] = bs == 1 ? inv[t] * r[t] : r[t];
  }
}

// y = a*x + b*y
__global__ void k_axpby(int64_t n, double a, const double* __restrict__ x, double b,
                        double* __restrict__ y) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a * x[i] + b * y[i];
}

// ---- the last block of a grid to finish (ticket), for its totals
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (threadIdx.x == 0) *ticket = 0u;
  return true;
}

// NS block sums into partial[q gridDim.x + block]; in the last block, the
// totals (valid in thread 0)
template <int NS, int T = NT>
__device__ __forceinline__ bool grid_sums(double (&v)[NS], double* partial, unsigned* ticket,
                                          double* tot) {
  __shared__ double sm[32];
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    const double r = block_sum<T>(v[q], sm);
    if (threadIdx.x == 0) partial[(size_t)q * gridDim.x + blockIdx.x] = r;
  }
  if (!last_block(ticket)) return false;
#pragma unroll
  for (int q = 0; q < NS; ++q) {
    double s = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += T)
      s += __ldcg(&partial[(size_t)q * gridDim.x + b]);
    tot[q] = block_sum<T>(s, sm);
  }
  return true;
}

// out = sum_i v[i]^2
__global__ void __launch_bounds__(NT) k_norm2(int64_t n, const double* __restrict__ v,
                                              double* partial, unsigned* ticket, double* out) {
  double s[1] = {0.0}, tot[1];
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * NT)
    s[0] += v[i] * v[i];
  if (grid_sums<1>(s, partial, ticket, tot) && threadIdx.x == 0) out[0] = tot[0];
}

// z = M^-1 r at one block row (bs = 3, 6), or one row
__device__ __forceinline__ void prec_row(int bs, const double* __restrict__ inv, int64_t t,
                                         const double* v, double* z) {
  if (bs == 3) {
    const double* m = inv + 9 * t;
#pragma unroll
    for (int q = 0; q < 3; ++q) z[q] = m[3 * q] * v[0] + m[3 * q + 1] * v[1] + m[3 * q + 2] * v[2];
  } else if (bs == 6) {
    const double* m = inv + 36 * t;
    for (int q = 0; q < 6; ++q) {
      double acc = 0.0;
#pragma unroll
      for (int c = 0; c < 6; ++c) acc += m[6 * q + c] * v[c];
      z[q] = acc;
    }
  } else {
    z[0] = bs == 1 ? inv[t] * v[0] : v[0];
  }
}

// ---- GMRES(m), right preconditioned: one iteration in five launches
//   spmv   w = A z
//   dots   h1 = V^T w
//   sub    w -= V h1, h2 = V^T w      (classical Gram-Schmidt, twice)
//   norm   w -= V h2, ||w||; the last block: column h1 + h2 of H, its Givens
//          rotations, the residual norm |g[j + 1]|
//   next   V_{j+1} = w / ||w||, z = M^-1 V_{j+1}
// A Jacobian of a few thousand nodes gives the V products 50 blocks of 256 rows,
// so they are bound by the latency of their loads, one basis vector after the
// other: a block has 32 warps, which take two vectors at a time for V^T w (w in
// shared memory, one warp reduction per vector and 256 rows), and four groups
// of 256 threads, which take every fourth vector for w -= V h.  13,824 rows, up
// to 100 vectors: 180 us per iteration with the host in it, 44 us with 8 warps and
// one group, 32 us with this.
struct GState {
  int j, done;      // columns finished; 1: residual at the tolerance or breakdown
  double inv;       // 1 / ||w|| (0 when it vanished)
};
struct Gmres {
  int64_t n;
  int m;
  double *V, *w, *h1, *h2, *R, *cs, *sn, *g;   // R: column j at R + j (m + 1)
  double* partial;                              // [m + 1][blocks]
  unsigned* ticket;
  GState* st;
};

constexpr int NTG = 4 * NT;   // threads of the V products' blocks

// partial sums of h = V^T w over the block's cnt <= 256 rows sw from row0 (0 past cnt)
__device__ __forceinline__ void gm_dots(const Gmres& G, int nv, int64_t row0, int cnt,
                                        const double* sw, bool first, double* partial) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double wv[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) wv[u] = sw[lane + 32 * u];   // 0 past the end
  // two vectors at a time: sixteen loads a lane in flight
  for (int i = 2 * warp; i < nv; i += 2 * (NTG / 32)) {
    const bool two = i + 1 < nv;
    const double* const Vi = G.V + (int64_t)i * G.n + row0;
    const double* const Vk = two ? Vi + G.n : Vi;
    double x[8], y[8], v = 0.0, q = 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const bool in = lane + 32 * u < cnt;
      x[u] = in ? Vi[lane + 32 * u] : 0.0;
      y[u] = in ? Vk[lane + 32 * u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      v += x[u] * wv[u];
      q += y[u] * wv[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_down_sync(0xffffffffu, v, o);
      q += __shfl_down_sync(0xffffffffu, q, o);
    }
    if (lane == 0) {
      double* const d = &partial[(size_t)i * gridDim.x + blockIdx.x];
      *d = first ? v : *d + v;
      if (two) d[gridDim.x] = first ? q : d[gridDim.x] + q;
    }
  }
}

// h = the blocks' partial sums
__device__ __forceinline__ void gm_totals(int nv, const double* partial, double* h) {
  const int lane = threadIdx.x & 7;   // 8 lanes a vector
  for (int i0 = 0; i0 < nv; i0 += NTG / 8) {
    const int i = i0 + (threadIdx.x >> 3);
    double v = 0.0;
    if (i < nv) {
#pragma unroll 8
      for (unsigned b = lane; b < gridDim.x; b += 8)
        v += __ldcg(&partial[(size_t)i * gridDim.x + b]);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, 8);
    if (i < nv && lane == 0) h[i] = v;
  }
}

// w[l] - sum_i h[i] V_i[row0 + l] of the block's cnt <= 256 rows, in the threads l < NT
// (0 past cnt); s4: [4][NT]
__device__ __forceinline__ double gm_minus(const Gmres& G, int nv, const double* h, int64_t row0,
                                           int cnt, const double* w, double (*s4)[NT]) {
  const int l = threadIdx.x & (NT - 1), grp = threadIdx.x / NT;
  double a = 0.0;
  if (l < cnt) {
    const double* const Vr = G.V + row0 + l;
#pragma unroll 8
    for (int i = grp; i < nv; i += 4) a += h[i] * Vr[(int64_t)i * G.n];
  }
  s4[grp][l] = a;
  __syncthreads();
  if (grp != 0 || l >= cnt) return 0.0;
  return w[l] - ((s4[0][l] + s4[1][l]) + (s4[2][l] + s4[3][l]));
}

template <bool SUB>
__global__ void __launch_bounds__(NTG) k_gm_dots(Gmres G) {
  chain_in();
  __shared__ double sw[NT], s4[4][NT];
  if (G.st->done || G.st->j >= G.m) return;
  const int nv = G.st->j + 1;
  bool first = true;
  for (int64_t row0 = (int64_t)blockIdx.x * NT; row0 < G.n; row0 += (int64_t)gridDim.x * NT) {
    const int64_t row = row0 + threadIdx.x;
    const int cnt = (int)min((int64_t)NT, G.n - row0);
    const bool mine = (int)threadIdx.x < cnt;
    double w = 0.0;
    if (SUB) w = gm_minus(G, nv, G.h1, row0, cnt, G.w + row0, s4);
    else if (mine) w = G.w[row];
    if (SUB && mine) G.w[row] = w;
    if (threadIdx.x < NT) sw[threadIdx.x] = w;
    __syncthreads();
    gm_dots(G, nv, row0, cnt, sw, first, G.partial);
    __syncthreads();
    first = false;
  }
  if (last_block(G.ticket)) gm_totals(nv, G.partial, SUB ? G.h2 : G.h1);
}

__global__ void __launch_bounds__(NTG) k_gm_norm(Gmres G, double tol) {
  chain_in();
  __shared__ double s4[4][NT];
  if (G.st->done || G.st->j >= G.m) return;
  const int j = G.st->j;
  double v[1] = {0.0}, tot[1];
  for (int64_t row0 = (int64_t)blockIdx.x * NT; row0 < G.n; row0 += (int64_t)gridDim.x * NT) {
    const int cnt = (int)min((int64_t)NT, G.n - row0);
    const double w = gm_minus(G, j + 1, G.h2, row0, cnt, G.w + row0, s4);
    if ((int)threadIdx.x < cnt) G.w[row0 + threadIdx.x] = w;
    v[0] += w * w;
    __syncthreads();
  }
  if (!grid_sums<1, NTG>(v, G.partial, G.ticket, tot)) return;
  // column j: the rotations so far (through shared memory: the chain in thread
  // 0 then waits for arithmetic only), then the new one
  double* const sh = s4[0];
  double* const sc = s4[1];
  double* const ss = s4[2];
  double* const r = G.R + (size_t)j * (G.m + 1);
  double a = G.h1[0] + G.h2[0];
  for (int i0 = 0; i0 < j; i0 += NT) {
    const int i = i0 + threadIdx.x;
    __syncthreads();
    if (threadIdx.x < NT && i < j) {
      sh[threadIdx.x] = G.h1[i + 1] + G.h2[i + 1];
      sc[threadIdx.x] = G.cs[i];
      ss[threadIdx.x] = G.sn[i];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int k = 0; k < min(NT, j - i0); ++k) {
        r[i0 + k] = sc[k] * a + ss[k] * sh[k];
        a = -ss[k] * a + sc[k] * sh[k];
      }
  }
  if (threadIdx.x != 0) return;
  const double hn = sqrt(tot[0]);
  const double den = hypot(a, hn);
  const double c = den > 0.0 ? a / den : 1.0, s = den > 0.0 ? hn / den : 0.0;
  r[j] = den;
  G.cs[j] = c;
  G.sn[j] = s;
  const double gj = G.g[j], gn = -s * gj;
  G.g[j + 1] = gn;
  G.g[j] = c * gj;
  G.st->inv = hn > 0.0 ? 1.0 / hn : 0.0;
  G.st->done = (fabs(gn) <= tol || !(den > 0.0)) ? 1 : 0;
  G.st->j = j + 1;
}

// V_j = w inv (j the new column), z = M^-1 V_j
__global__ void __launch_bounds__(NT) k_gm_next(Gmres G, int bs, const double* __restrict__ inv,
                                                double* z) {
  chain_in();
  if (G.st->done || G.st->j >= G.m) return;
  const int64_t t = (int64_t)blockIdx.x * NT + threadIdx.x;
  const int b = bs > 1 ? bs : 1;
  if (t >= G.n / b) return;
  const double a = G.st->inv;
  double* const Vj = G.V + (int64_t)G.st->j * G.n;
  double v[6], q[6];
  for (int c = 0; c < b; ++c) {
    v[c] = a * G.w[b * t + c];
    Vj[b * t + c] = v[c];
  }
  prec_row(bs, inv, t, v, q);
  for (int c = 0; c < b; ++c) z[b * t + c] = q[c];
}

// ---- a whole restart cycle in one cooperative launch, for systems of at most
// kGmCycleCtas x kGmRows rows
//
// Five launches of such an iteration are latency (30 us at 13,824 rows, chained; 20
// here).  Whole solves, five launches an iteration / one a cycle: 288 rows 1.6 / 1.05
// ms, 13,824 rows 28.4 / 19.8, 36,960 rows 68.5 / 43.2; above 37,296 a CTA would
// need more rows than its shared memory and registers are laid out for.  Here a CTA keeps kGmRows rows of w in shared memory and an
// iteration is four grid barriers: h1 = V^T A z; w -= V h1, h2 = V^T w; w -= V h2,
// ||w||; V_{j+1}, z (whose neighbours' rows the next product reads).  Every CTA adds
// the partial sums for itself and applies the Givens rotations to its own copy of the
// column -- the same numbers everywhere -- in one warp while the others form V_{j+1}
// and z.  kGmRows: whole 3 x 3 and 6 x 6 blocks.  Needs V_0 and z (k_gm_start,
// k_gm_next); leaves G.w as it was, so that a cycle whose barrier gave up can be run
// again step by step.
constexpr int kGmRows = 252;
constexpr int kGmCycleCtas = 148;
constexpr int kGmCycleCols = 1000;   // columns of a cycle whose state fits in shared memory
constexpr size_t gm_cycle_smem(int m) { return 4 * (size_t)(m + 1) * sizeof(double); }

__global__ void __launch_bounds__(NTG, 1)
k_gm_cycle(Sys A, Gmres G, int bs, const double* __restrict__ inv, double* z, double tol, double g0,
           unsigned* bar) {
  extern __shared__ double s_dyn[];   // h1, h2, cs, sn
  __shared__ double sw[NT], s4[4][NT], sm[32], s_norm, s_g;
  __shared__ int ok, s_done;
  double* const h1 = s_dyn;
  double* const h2 = h1 + (G.m + 1);
  double* const cs = h2 + (G.m + 1);
  double* const sn = cs + (G.m + 1);
  GridBarrier gb{bar, 0u};
  double* const part[2] = {G.partial, G.partial + (size_t)gridDim.x * (G.m + 1)};
  double* const pnorm = G.partial + 2 * (size_t)gridDim.x * (G.m + 1);
  const int64_t row0 = (int64_t)blockIdx.x * kGmRows;
  const int cnt = (int)min((int64_t)kGmRows, G.n - row0);
  const int tid = threadIdx.x, b = bs > 1 ? bs : 1;
  if (tid == 0) {
    s_g = g0;
    s_done = 0;
  }
  if (tid < NT) sw[tid] = 0.0;
  __syncthreads();
  for (int j = 0; j < G.m; ++j) {
    // w = A z, eight lanes a row
    for (int r0 = 0; r0 < cnt; r0 += NTG / 8) {
      const int r = r0 + (tid >> 3);
      double s = 0.0;
      if (r < cnt) {
        const int e = A.ptr[row0 + r + 1];
        for (int q = A.ptr[row0 + r] + (tid & 7); q < e; q += 8) s += A.val[q] * __ldcg(z + A.idx[q]);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
      if (r < cnt && (tid & 7) == 0) sw[r] = s;
    }
    __syncthreads();
    gm_dots(G, j + 1, row0, cnt, sw, true, part[0]);
    if (!gb.wait(&ok)) return;
    gm_totals(j + 1, part[0], h1);
    __syncthreads();
    double w = gm_minus(G, j + 1, h1, row0, cnt, sw, s4);
    __syncthreads();
    if (tid < NT) sw[tid] = w;
    __syncthreads();
    gm_dots(G, j + 1, row0, cnt, sw, true, part[1]);
    if (!gb.wait(&ok)) return;
    gm_totals(j + 1, part[1], h2);
    __syncthreads();
    w = gm_minus(G, j + 1, h2, row0, cnt, sw, s4);
    __syncthreads();
    if (tid < NT) sw[tid] = w;
    double tot = block_sum<NTG>(w * w, sm);
    if (tid == 0) pnorm[blockIdx.x] = tot;
    if (!gb.wait(&ok)) return;
    tot = block_sum<NTG>(tid < (int)gridDim.x ? __ldcg(pnorm + tid) : 0.0, sm);
    if (tid == 0) s_norm = sqrt(tot);
    __syncthreads();
    const double hn = s_norm, a1 = hn > 0.0 ? 1.0 / hn : 0.0;
    // V_{j+1}, z; meanwhile the last thread: column j's rotations
    if (tid < cnt / b) {
      const int64_t t = row0 / b + tid;
      double* const Vj = G.V + (int64_t)(j + 1) * G.n;
      double v[6], q[6];
      for (int c = 0; c < b; ++c) {
        v[c] = a1 * sw[b * tid + c];
        Vj[b * t + c] = v[c];
      }
      prec_row(bs, inv, t, v, q);
      for (int c = 0; c < b; ++c) z[b * t + c] = q[c];
    } else if (tid == NTG - 1) {
      const bool out = blockIdx.x == 0;
      double* const r = G.R + (size_t)j * (G.m + 1);
      double a = h1[0] + h2[0];
      for (int k = 0; k < j; ++k) {
        const double hk = h1[k + 1] + h2[k + 1];
        if (out) r[k] = cs[k] * a + sn[k] * hk;
        a = -sn[k] * a + cs[k] * hk;
      }
      const double den = hypot(a, hn);
      const double c = den > 0.0 ? a / den : 1.0, s = den > 0.0 ? hn / den : 0.0;
      cs[j] = c;
      sn[j] = s;
      const double gj = s_g, gn = -s * gj;
      s_g = gn;
      s_done = (fabs(gn) <= tol || !(den > 0.0)) ? 1 : 0;
      if (out) {
        r[j] = den;
        G.g[j] = c * gj;
        G.g[j + 1] = gn;
        *G.st = GState{j + 1, s_done, a1};
      }
    }
    if (!gb.wait(&ok)) return;
    if (s_done) return;
  }
}

// start of a cycle: g = (rn, 0, ...), no columns, w = the residual
__global__ void k_gm_start(Gmres G, double rn) {
  for (int i = threadIdx.x; i <= G.m; i += blockDim.x) G.g[i] = i == 0 ? rn : 0.0;
  if (threadIdx.x == 0) *G.st = GState{0, 0, 1.0 / rn};
}

// ---- BiCGStab, right preconditioned: one iteration in five launches, each
// ended by its scalars (last block)
struct BState {
  double rho, alpha, omega, beta, rn;   // rn: the residual norm (of s on an early exit)
  int it, done;                         // done: converged, out of iterations or broken down
};
struct Bicg {
  int64_t n;
  double *r, *rh, *p, *v, *ph, *s, *sh, *t, *x;
  double* partial;
  unsigned* ticket;
  BState* st;
  double tol;
  int maxit;
};

// the test at the top of an iteration on (rh, r): rho, beta for it
__device__ __forceinline__ void bi_top(BState& st, double rhr, double tol, int maxit) {
  if (!(st.rn > tol) || st.it >= maxit || rhr == 0.0 || !isfinite(rhr)) st.done = 1;
  st.beta = (rhr / st.rho) * (st.alpha / st.omega);
  st.rho = rhr;
}

// p = r + beta p - beta omega v, ph = M^-1 p
__global__ void __launch_bounds__(NT) k_cb_p(Bicg B, int bs, const double* __restrict__ inv) {
  chain_in();
  const BState st = *B.st;
  if (st.done) return;
  const int64_t t = (int64_t)blockIdx.x * NT + threadIdx.x;
  const int b = bs > 1 ? bs : 1;
  if (t >= B.n / b) return;
  const double bw = -st.beta * st.omega;
  double v[6], q[6];
  for (int c = 0; c < b; ++c) {
    const int64_t i = b * t + c;
    v[c] = B.r[i] + st.beta * B.p[i] + bw * B.v[i];
    B.p[i] = v[c];
  }
  prec_row(bs, inv, t, v, q);
  for (int c = 0; c < b; ++c) B.ph[b * t + c] = q[c];
}

// s = r - alpha v, sh = M^-1 s; (s, s): early exit
__global__ void __launch_bounds__(NT) k_cb_s(Bicg B, int bs, const double* __restrict__ inv) {
  chain_in();
  const BState st = *B.st;
  if (st.done) return;
  const int b = bs > 1 ? bs : 1;
  double sum[1] = {0.0}, tot[1];
  for (int64_t t = (int64_t)blockIdx.x * NT + threadIdx.x; t < B.n / b;
       t += (int64_t)gridDim.x * NT) {
    double v[6], q[6];
    for (int c = 0; c < b; ++c) {
      const int64_t i = b * t + c;
      v[c] = B.r[i] - st.alpha * B.v[i];
      B.s[i] = v[c];
      sum[0] += v[c] * v[c];
    }
    prec_row(bs, inv, t, v, q);
    for (int c = 0; c < b; ++c) B.sh[b * t + c] = q[c];
  }
  if (grid_sums<1>(sum, B.partial, B.ticket, tot) && threadIdx.x == 0) {
    ++B.st->it;
    if (sqrt(tot[0]) <= B.tol) {
      B.st->rn = sqrt(tot[0]);
      B.st->done = 2;               // x += alpha ph is left to do
    }
  }
}

// one row of A x by its 8 lanes (valid in lane 0)
__device__ __forceinline__ double row_dot(const Sys& A, int64_t row, const double* __restrict__ x,
                                          int lane) {
  double s = 0.0;
  if (row < A.n) {
    const int a = A.ptr[row], b = A.ptr[row + 1];
    for (int q = a + lane; q < b; q += 8) s += A.val[q] * x[A.idx[q]];
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, 8);
  return s;
}

// v = A ph, (rh, v) -> alpha;  T: t = A sh, (t, t), (s, t) -> omega
template <bool T>
__global__ void __launch_bounds__(NT) k_cb_spmv(Sys A, Bicg B) {
  chain_in();
  if (B.st->done) return;
  const int lane = threadIdx.x & 7;
  double sum[2] = {0.0, 0.0}, tot[2];
  for (int64_t r0 = (int64_t)blockIdx.x * kRowsPerBlock; r0 < A.n;
       r0 += (int64_t)gridDim.x * kRowsPerBlock) {
    const int64_t row = r0 + (threadIdx.x >> 3);
    const double y = row_dot(A, row, T ? B.sh : B.ph, lane);
    if (row < A.n && lane == 0) {
      if (T) {
        B.t[row] = y;
        sum[0] += y * y;
        sum[1] += B.s[row] * y;
      } else {
        B.v[row] = y;
        sum[0] += B.rh[row] * y;
      }
    }
  }
  if (!grid_sums<2>(sum, B.partial, B.ticket, tot) || threadIdx.x != 0) return;
  if (T) {
    // tot[0] = (t, t), tot[1] = (s, t)
    B.st->omega = tot[0] > 0.0 ? tot[1] / tot[0] : 0.0;
  } else if (tot[0] == 0.0 || !isfinite(tot[0])) {
    B.st->done = 1;
  } else {
    B.st->alpha = B.st->rho / tot[0];
  }
}

// x += alpha ph + omega sh, r = s - omega t; (r, r), (rh, r)
__global__ void __launch_bounds__(NT) k_cb_x(Bicg B) {
  chain_in();
  const BState st = *B.st;
  if (st.done) return;
  double sum[2] = {0.0, 0.0}, tot[2];
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < B.n;
       i += (int64_t)gridDim.x * NT) {
    B.x[i] = st.alpha * B.ph[i] + B.x[i] + st.omega * B.sh[i];
    const double r = B.s[i] - st.omega * B.t[i];
    B.r[i] = r;
    sum[0] += r * r;
    sum[1] += B.rh[i] * r;
  }
  if (!grid_sums<2>(sum, B.partial, B.ticket, tot) || threadIdx.x != 0) return;
  B.st->rn = sqrt(tot[0]);
  if (st.omega == 0.0) B.st->done = 1;
  bi_top(*B.st, tot[1], B.tol, B.maxit);
}

// rh = r, p = v = 0; (r, r): the first iteration's scalars
__global__ void __launch_bounds__(NT) k_cb_start(Bicg B) {
  double sum[1] = {0.0}, tot[1];
  for (int64_t i = (int64_t)blockIdx.x * NT + threadIdx.x; i < B.n;
       i += (int64_t)gridDim.x * NT) {
    const double r = B.r[i];
    B.rh[i] = r;
    B.p[i] = 0.0;
    B.v[i] = 0.0;
    sum[0] += r * r;
  }
  if (!grid_sums<1>(sum, B.partial, B.ticket, tot) || threadIdx.x != 0) return;
  *B.st = BState{1.0, 1.0, 1.0, 0.0, sqrt(tot[0]), 0, 0};
  bi_top(*B.st, tot[0], B.tol, B.maxit);
}

// x += sum_i c[i] Z_i  (Z_i = M^-1 V_i folded later) -- here: y = sum_i c[i] V_i
__global__ void k_lincomb(int64_t n, const double* __restrict__ V, int m,
                          const double* __restrict__ c, double* __restrict__ y) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s = 0.0;
  for (int i = 0; i < m; ++i) s += c[i] * V[(int64_t)i * n + k];
  y[k] = s;
}

}  // namespace csr
}  // namespace tcad

using namespace tcad;
using namespace tcad::csr;

namespace {

struct Ctx {
  Sys A;
  int bs;
  double* inv;
  cudaStream_t s;
  double* partial;
  unsigned* ticket;
  double* scal;  // device scalars
  int nblk;
};

inline unsigned g1(int64_t n) { return (unsigned)((n + NT - 1) / NT); }

int spmv(const Ctx& c, const double* x, double* y) {
  launch_chained(c.s, (unsigned)((c.A.n + kRowsPerBlock - 1) / kRowsPerBlock), NT, 0, k_spmv, c.A, x,
                 y);
  note_launch();
  return TCAD_OK;
}

int prec(const Ctx& c, const double* r, double* z) {
  const int64_t n = c.A.n;
  k_bj_apply<<<g1(c.bs == 3 ? n / 3 : (c.bs == 6 ? n / 6 : n)), NT, 0, c.s>>>(n, c.bs,
                                                                               c.inv, r, z);
  note_launch();
  return TCAD_OK;
}

int norm(const Ctx& c, const double* v, double& out) {
  k_norm2<<<c.nblk, NT, 0, c.s>>>(c.A.n, v, c.partial, c.ticket, c.scal);
  note_launch();
  TCAD_CUDA_CHECK(cudaMemcpyAsync(&out, c.scal, sizeof(double), cudaMemcpyDeviceToHost, c.s));
  TCAD_CUDA_CHECK(cudaStreamSynchronize(c.s));
  out = std::sqrt(out);
  return TCAD_OK;
}

int axpby(const Ctx& c, double a, const double* x, double b, double* y) {
  k_axpby<<<g1(c.A.n), NT, 0, c.s>>>(c.A.n, a, x, b, y);
  note_launch();
  return TCAD_OK;
}

// one cycle by k_gm_cycle, its state into st; done = false: it did not run to its end
int gm_cycle(const Ctx& c, const Gmres& G, double* z, double tol, double rn, GState& st,
             bool& done) {
  done = false;
  unsigned* const bar = c.ticket + 32;
  unsigned h[4] = {0u, 0u, 0u, krylov_fused_hold() ? 1u : 0u};
  TCAD_CUDA_CHECK(cudaMemcpyAsync(bar, h, sizeof(h), cudaMemcpyHostToDevice, c.s));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((G.n + kGmRows - 1) / kGmRows));
  cfg.blockDim = dim3(NTG);
  cfg.dynamicSmemBytes = gm_cycle_smem(G.m);
  cfg.stream = c.s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k_gm_cycle, c.A, G, c.bs, (const double*)c.inv, z, tol, rn, bar) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return TCAD_OK;
  }
  note_launch();
  TCAD_CUDA_CHECK(cudaMemcpyAsync(&st, G.st, sizeof(st), cudaMemcpyDeviceToHost, c.s));
  TCAD_CUDA_CHECK(cudaMemcpyAsync(h, bar, sizeof(h), cudaMemcpyDeviceToHost, c.s));
  TCAD_CUDA_CHECK(cudaStreamSynchronize(c.s));
  if (h[2] != 0u) {
    krylov_note_gave_up();
    st = GState{0, 0, 0.0};
  } else {
    done = true;
  }
  return TCAD_OK;
}

}  // namespace

extern "C" size_t tcad_csr_workspace_bytes(int64_t n, int method, int restart) {
  const int m = restart > 0 ? restart : 100;
  size_t vec = (size_t)n * sizeof(double);
  size_t v = 9 * (size_t)n * sizeof(double);        // block inverses (upper bound: 3n
                                                     // for 3 x 3 blocks, 6n for 6 x 6)
  if (method == 0) v += 8 * vec;                     // BiCGStab vectors
  else v += (size_t)(m + 1) * vec + 3 * vec;         // GMRES basis + work
  v += 4096 * 4 * sizeof(double) + 64 * sizeof(double) + 256;
  v += (size_t)4096 * (m + 1) * sizeof(double);      // Gram-Schmidt partials
  v += (size_t)(m + 1) * sizeof(double) + vec;       // coefficients, true residual
  if (method != 0) {
    // H, rotations and sums of the min(restart, n) columns that are used lie in what the
    // partials leave (kGridBlocks of 4096 a column); past 3,500 columns H is larger
    const int64_t c = std::min<int64_t>(m, n);
    const int64_t more = (c + 1) * (c + 5) - (4096 - kGridBlocks) * ((int64_t)m + 1);
    if (more > 0) v += (size_t)more * sizeof(double);
  }
  return v + (1u << 20);                             // alignment slack
}

extern "C" int tcad_csr_krylov(int64_t n, const int32_t* indptr, const int32_t* indices,
                               const double* data, const double* b, double* x,
                               int method, int block_size, double rtol, double atol,
                               int maxiter, int restart, void* work, size_t work_bytes,
                               int32_t* iters_out, double* resid_out, int32_t* precond_out,
                               void* stream) {
  if (n <= 0 || !indptr || !indices || !data || !b || !x || !work) return TCAD_ERR_ARG;
  if (method != 0 && method != 1) return TCAD_ERR_ARG;
  if (work_bytes < tcad_csr_workspace_bytes(n, method, restart)) return TCAD_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  char* base = reinterpret_cast<char*>(work);
  size_t used = 0;
  auto take = [&](size_t bytes) {
    char* p = base + used;
    used += (bytes + 255) & ~(size_t)255;
    return p;
  };
  const int m = restart > 0 ? (int)std::min<int64_t>(restart, n) : (int)std::min<int64_t>(100, n);
  Ctx c;
  c.A = Sys{n, indptr, indices, data};
  c.s = s;
  c.inv = reinterpret_cast<double*>(take(9 * (size_t)n * sizeof(double)));
  c.nblk = (int)std::min<int64_t>(4096, (n + NT - 1) / NT);
  c.partial = reinterpret_cast<double*>(take(4096 * 4 * sizeof(double)));
  c.scal = reinterpret_cast<double*>(take(64 * sizeof(double)));
  c.ticket = reinterpret_cast<unsigned*>(take(256));
  int* flag = reinterpret_cast<int*>(c.ticket + 16);
  TCAD_CUDA_CHECK(cudaMemsetAsync(c.ticket, 0, 256, s));
  // preconditioner: node blocks, else point Jacobi, else none
  c.bs = ((block_size == 3 || block_size == 6) && n % block_size == 0) ? block_size : 1;
  for (;;) {
    TCAD_CUDA_CHECK(cudaMemsetAsync(flag, 0, sizeof(int), s));
    const int64_t nb = n / c.bs;
    if (c.bs == 6)
      k_bj_setup6<<<g1(nb), NT, 0, s>>>(c.A, c.inv, flag);
    else
      k_bj_setup<<<g1(nb), NT, 0, s>>>(c.A, c.bs, c.inv, flag);
    note_launch();
    int hflag = 0;
    TCAD_CUDA_CHECK(cudaMemcpyAsync(&hflag, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    TCAD_CUDA_CHECK(cudaStreamSynchronize(s));
    if (!hflag) break;
    if (c.bs == 3 || c.bs == 6) c.bs = 1;
    else { c.bs = 0; break; }
  }
  if (precond_out) *precond_out = c.bs;
  const int64_t N = n;
  double bnorm = 0.0;
  int rc = norm(c, b, bnorm);
  if (rc) return rc;
  if (!std::isfinite(bnorm)) return TCAD_ERR_NONFINITE;
  const double tol = std::max(atol, rtol * bnorm);
  int it = 0;
  double rn = 0.0;
  const unsigned gv = (unsigned)std::min<int64_t>(kGridBlocks, (N + NT - 1) / NT);
  if (method == 0) {
    Bicg B;
    double** const vec[8] = {&B.r, &B.rh, &B.p, &B.v, &B.ph, &B.s, &B.sh, &B.t};
    for (double** q : vec) *q = reinterpret_cast<double*>(take(N * 8));
    B.n = N;
    B.x = x;
    B.partial = c.partial;
    B.ticket = c.ticket;
    B.st = reinterpret_cast<BState*>(c.scal + 8);
    B.tol = tol;
    B.maxit = maxiter;
    // r = b - A x
    spmv(c, x, B.r);
    axpby(c, 1.0, b, -1.0, B.r);
    k_cb_start<<<gv, NT, 0, s>>>(B);
    note_launch();
    const unsigned gb = g1(c.bs > 1 ? N / c.bs : N);
    const unsigned gr = (unsigned)std::min<int64_t>(kGridBlocks,
                                                    (N + kRowsPerBlock - 1) / kRowsPerBlock);
    BState st;
    for (int check = 4;; check = std::min(2 * check, 32)) {
      TCAD_CUDA_CHECK(cudaMemcpyAsync(&st, B.st, sizeof(st), cudaMemcpyDeviceToHost, s));
      TCAD_CUDA_CHECK(cudaStreamSynchronize(s));
      if (st.done) break;
      for (int q = 0; q < check; ++q) {
        launch_chained(s, gb, NT, 0, k_cb_p, B, c.bs, c.inv);
        launch_chained(s, gr, NT, 0, k_cb_spmv<false>, c.A, B);
        launch_chained(s, (unsigned)std::min<int64_t>(kGridBlocks, gb), NT, 0, k_cb_s, B, c.bs,
                       c.inv);
        launch_chained(s, gr, NT, 0, k_cb_spmv<true>, c.A, B);
        launch_chained(s, gv, NT, 0, k_cb_x, B);
        note_launch(5);
      }
      TCAD_LAUNCH_CHECK();
    }
    if (st.done == 2) axpby(c, st.alpha, B.ph, 1.0, x);
    rn = st.rn;
    it = st.it;
  } else {
    Gmres G;
    G.n = N;
    G.m = m;
    G.V = reinterpret_cast<double*>(take((size_t)(m + 1) * N * 8));
    G.w = reinterpret_cast<double*>(take(N * 8));
    double* z = reinterpret_cast<double*>(take(N * 8));
    double* y = reinterpret_cast<double*>(take(N * 8));
    G.partial = reinterpret_cast<double*>(take((size_t)kGridBlocks * (m + 1) * 8));
    G.R = reinterpret_cast<double*>(take((size_t)m * (m + 1) * 8));
    double** const vec[5] = {&G.h1, &G.h2, &G.cs, &G.sn, &G.g};
    for (double** q : vec) *q = reinterpret_cast<double*>(take((size_t)(m + 1) * 8));
    if (used > work_bytes) return TCAD_ERR_ARG;
    G.ticket = c.ticket;
    G.st = reinterpret_cast<GState*>(c.scal + 8);
    std::vector<double> R((size_t)m * (m + 1)), g(m + 1), yv(m);
    const unsigned gb = g1(c.bs > 1 ? N / c.bs : N);
    // maxiter counts restart cycles, as scipy's gmres does
    for (int cycle = 0;; ++cycle) {
      // r = b - A x -> V_0
      spmv(c, x, G.w);
      axpby(c, 1.0, b, -1.0, G.w);
      if ((rc = norm(c, G.w, rn))) return rc;
      if (rn <= tol || cycle >= maxiter || !std::isfinite(rn)) break;
      k_gm_start<<<1, NT, 0, s>>>(G, rn);
      k_gm_next<<<gb, NT, 0, s>>>(G, c.bs, c.inv, z);
      note_launch(2);
      GState st{0, 0, 0.0};
      bool whole = N <= (int64_t)kGmCycleCtas * kGmRows && m <= kGmCycleCols && krylov_fused();
      if (whole) {
        if ((rc = gm_cycle(c, G, z, tol, rn, st, whole))) return rc;
        if (!whole) {   // the launch was refused or gave up: the cycle step by step
          k_gm_start<<<1, NT, 0, s>>>(G, rn);
          k_gm_next<<<gb, NT, 0, s>>>(G, c.bs, c.inv, z);
          note_launch(2);
        }
      }
      int queued = 0;
      for (int check = 4; !whole && !st.done && st.j < m; check = std::min(2 * check, 32)) {
        const int todo = std::min(check, m - queued);
        for (int q = 0; q < todo; ++q) {
          spmv(c, z, G.w);
          launch_chained(s, gv, NTG, 0, k_gm_dots<false>, G);
          launch_chained(s, gv, NTG, 0, k_gm_dots<true>, G);
          launch_chained(s, gv, NTG, 0, k_gm_norm, G, tol);
          launch_chained(s, gb, NT, 0, k_gm_next, G, c.bs, c.inv, z);
          note_launch(4);
        }
        queued += todo;
        TCAD_LAUNCH_CHECK();
        TCAD_CUDA_CHECK(cudaMemcpyAsync(&st, G.st, sizeof(st), cudaMemcpyDeviceToHost, s));
        TCAD_CUDA_CHECK(cudaStreamSynchronize(s));
      }
      const int j = st.j;
      it += j;
      // solve the j x j triangle, x += M^-1 (V y)
      TCAD_CUDA_CHECK(cudaMemcpyAsync(R.data(), G.R, sizeof(double) * (size_t)j * (m + 1),
                                      cudaMemcpyDeviceToHost, s));
      TCAD_CUDA_CHECK(cudaMemcpyAsync(g.data(), G.g, sizeof(double) * (m + 1),
                                      cudaMemcpyDeviceToHost, s));
      TCAD_CUDA_CHECK(cudaStreamSynchronize(s));
      for (int i = j - 1; i >= 0; --i) {
        double sacc = g[i];
        for (int k = i + 1; k < j; ++k) sacc -= R[(size_t)k * (m + 1) + i] * yv[k];
        const double d = R[(size_t)i * (m + 1) + i];
        yv[i] = d != 0.0 ? sacc / d : 0.0;
      }
      TCAD_CUDA_CHECK(cudaMemcpyAsync(G.h1, yv.data(), sizeof(double) * j,
                                      cudaMemcpyHostToDevice, s));
      k_lincomb<<<g1(N), NT, 0, s>>>(N, G.V, j, G.h1, y);
      note_launch();
      prec(c, y, z);
      axpby(c, 1.0, z, 1.0, x);
      TCAD_CUDA_CHECK(cudaStreamSynchronize(s));
    }
  }
  // true relative residual ||b - A x|| / ||b|| (the acceptance quantity of
  // pytcad/linsolve.py:973-982)
  double* rt = reinterpret_cast<double*>(take(N * 8));
  spmv(c, x, rt);
  axpby(c, 1.0, b, -1.0, rt);
  double res = 0.0;
  if ((rc = norm(c, rt, res))) return rc;
  TCAD_LAUNCH_CHECK();
  const double true_res = res / std::max(bnorm, 1e-300);
  if (iters_out) *iters_out = it;
  if (resid_out) *resid_out = true_res;
  const bool ok = rn <= tol && std::isfinite(true_res);
  return ok ? TCAD_OK : TCAD_ERR_NOCONV;
}
