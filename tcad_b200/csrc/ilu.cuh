// Block ILU(0) of the node-block-scaled 2D operator, as a right
// preconditioner of the BiCGStab in krylov.cu.  On 3D packs the same
// factorisation is taken plane by plane (the in-plane W/E/S/N couplings of
// each z-plane; the D/U couplings are left to the Krylov iteration): a
// block-diagonal-over-planes preconditioner, one CTA per (instance, plane).
//
// The scaled operator is A^ = I + G_k sum_d B_kd (node k, neighbours
// d = W, E, S, N): G_k is the (row-scaled) inverse diagonal block stored in
// J entries 0..8, B_kd the 5-entry neighbour block (psi<-psi, n<-psi, n<-n,
// p<-psi, p<-p) in entries 9 + 5d + m.  For the 5-point block stencil
// ILU(0) keeps the off-diagonal blocks of A^ and changes only the diagonal
// ones (no fill survives), i.e. M = (D~ + L^) D~^-1 (D~ + U^) with
//   D~_k = I - G_k (B_kW D~_W^-1 G_W B_WE + B_kS D~_S^-1 G_S B_SN)
// (W, S the lower neighbours in the x-fastest natural order).  Q_k = D~_k^-1
// is stored (9 doubles per node).  Applying M^-1 r:
//   forward  a_k = Q_k (r_k - G_k (B_kW a_W + B_kS a_S))
//   backward x_k = a_k - Q_k G_k (B_kE x_E + B_kN x_N)
// Node (i, j) depends on (i-1, j) and (i, j-1) only, so all nodes of an
// anti-diagonal i + j = d are independent: one CTA per instance sweeps the
// nx + ny - 1 anti-diagonals with a block barrier between them (global
// writes of a level are visible to the block after the barrier).
#pragma once

#include "async_copy.cuh"

namespace tcad {

constexpr int kIluThreads = 256;

// C = M * B with B the sparse neighbour block (b0..b4)
__device__ __forceinline__ void mul_dense_nb(const double* M, const double* b, double* C) {
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    C[3 * r + 0] = M[3 * r + 0] * b[0] + M[3 * r + 1] * b[1] + M[3 * r + 2] * b[3];
    C[3 * r + 1] = M[3 * r + 1] * b[2];
    C[3 * r + 2] = M[3 * r + 2] * b[4];
  }
}

// C = B * M with B the sparse neighbour block
__device__ __forceinline__ void mul_nb_dense(const double* b, const double* M, double* C) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    C[0 + c] = b[0] * M[0 + c];
    C[3 + c] = b[1] * M[0 + c] + b[2] * M[3 + c];
    C[6 + c] = b[3] * M[0 + c] + b[4] * M[6 + c];
  }
}

__device__ __forceinline__ void mul33(const double* A, const double* B, double* C) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      C[3 * r + c] = A[3 * r + 0] * B[0 + c] + A[3 * r + 1] * B[3 + c] + A[3 * r + 2] * B[6 + c];
}

// inv = D^-1; the identity and false when D is singular
__device__ __forceinline__ bool inverse33(const double* D, double* inv) {
  const double c00 = D[4] * D[8] - D[5] * D[7];
  const double c01 = D[5] * D[6] - D[3] * D[8];
  const double c02 = D[3] * D[7] - D[4] * D[6];
  const double det = D[0] * c00 + D[1] * c01 + D[2] * c02;
  if (!(isfinite(det) && fabs(det) >= 1e-300)) {
#pragma unroll
    for (int e = 0; e < 9; ++e) inv[e] = (e % 4 == 0) ? 1.0 : 0.0;
    return false;
  }
  const double id = 1.0 / det;
  inv[0] = c00 * id;
  inv[1] = (D[2] * D[7] - D[1] * D[8]) * id;
  inv[2] = (D[1] * D[5] - D[2] * D[4]) * id;
  inv[3] = c01 * id;
  inv[4] = (D[0] * D[8] - D[2] * D[6]) * id;
  inv[5] = (D[2] * D[3] - D[0] * D[5]) * id;
  inv[6] = c02 * id;
  inv[7] = (D[1] * D[6] - D[0] * D[7]) * id;
  inv[8] = (D[0] * D[4] - D[1] * D[3]) * id;
  return true;
}

__device__ __forceinline__ void load9(const double* __restrict__ X, int64_t NN, int64_t k,
                                      int e0, double* out) {
#pragma unroll
  for (int e = 0; e < 9; ++e) out[e] = X[(int64_t)(e0 + e) * NN + k];
}

__device__ __forceinline__ void load_nb(const double* __restrict__ J, int64_t NN, int64_t k,
                                        int d, double* b) {
#pragma unroll
  for (int m = 0; m < 5; ++m) b[m] = J[(int64_t)(9 + 5 * d + m) * NN + k];
}

// y += B v (sparse neighbour block)
__device__ __forceinline__ void add_nb_vec(const double* b, double v0, double v1, double v2,
                                           double& y0, double& y1, double& y2) {
  y0 += b[0] * v0;
  y1 += b[1] * v0 + b[2] * v1;
  y2 += b[3] * v0 + b[4] * v2;
}

// ---------------------------------------------------------------------------
// Coalesced sweep (2D packs whose shorter side fits the block).
//
// The sweeps touch one node per row per anti-diagonal level, so in node
// order every access of a level is a separate memory sector.  The factor
// therefore also writes what the sweeps read in ANTI-DIAGONAL-MAJOR order:
// node (c, w) -- row c of the shorter side, position w along it -- of the
// plane whose first node is `base` sits in slot 2*base + (c + w)*Lc + c.
// A plane with Lc <= Lw rows has (Lc + Lw - 1) Lc <= 2 Lc Lw slots, so the
// slots of all planes fit in 2 * n_nodes.  Each sweep has an array of records, one
// per slot: two 3 x 3 products (FP32, a preconditioner needs no more) --
// Q G B_walk, Q G B_cross forward, Q G B_walk', Q G B_cross' backward -- and a
// vector (FP64), so that
//   forward  a = Q r - (Q G B_walk) a_prev - (Q G B_cross) a_cross
//   backward x = a - (Q G B_walk') x_next - (Q G B_cross') x_cross'
// and all that a level reads is one contiguous run, copied in bulk.  Q r is formed
// node-parallel while r is permuted into the forward records; the forward sweep
// leaves a in the backward records and the backward one x in their place.
constexpr int kIluRec = 28;   // floats of a record (7 x 16 bytes: an odd stride, no
                              // bank conflicts): 18, 2 of pad, 3 doubles, 1 of pad
constexpr int kIluVec = 20;   // where the vector starts
__device__ __forceinline__ double2* ilu_vec(float* M, int64_t slot) {
  return reinterpret_cast<double2*>(M + slot * kIluRec + kIluVec);
}
constexpr int kIluStages = 16;
constexpr int kIluSweepThreads = 4 * 128 + 32;   // 4 groups of 128 rows, or 2 of 256

struct IluGeo {
  bool byj;      // rows are j (ny <= nx), walk along i
  int Lc, Lw;    // rows, positions per row
  int64_t soff;  // first slot of the plane
};

__device__ __forceinline__ IluGeo ilu_geo(const Inst& g, int64_t base) {
  IluGeo q;
  q.byj = g.ny <= g.nx;
  q.Lc = q.byj ? g.ny : g.nx;
  q.Lw = q.byj ? g.nx : g.ny;
  q.soff = 2 * base;
  return q;
}

// slot of node (i, j) of the plane
__device__ __forceinline__ int64_t ilu_slot(const IluGeo& q, int i, int j) {
  const int c = q.byj ? j : i, w = q.byj ? i : j;
  return q.soff + (int64_t)(c + w) * q.Lc + c;
}

// Factor: Q_k for every node of each instance whose pre_status is TCAD_OK;
// status[inst] = TCAD_ERR_SINGULAR when a D~ block is singular.
__global__ void __launch_bounds__(kIluThreads)
k_ilu2d_factor(const tcad_pack_t pk, const double* __restrict__ J, double* __restrict__ Q,
               const int32_t* __restrict__ pre_status, int32_t* __restrict__ status,
               int nzmax) {
  const int inst = blockIdx.x / nzmax, z = blockIdx.x % nzmax;
  if (pre_status && pre_status[inst] != TCAD_OK) return;
  const Inst g = load_inst(pk, inst);
  if (z >= g.nz) return;
  const int64_t base = g.off + (int64_t)z * g.nx * g.ny;  // this z-plane (2D: the instance)
  const int64_t NN = pk.n_nodes;
  const int nx = g.nx, ny = g.ny;
  for (int d = 0; d < nx + ny - 1; ++d) {
    const int jlo = d - (nx - 1) > 0 ? d - (nx - 1) : 0;
    const int jhi = d < ny - 1 ? d : ny - 1;
    for (int j = jlo + threadIdx.x; j <= jhi; j += kIluThreads) {
      const int i = d - j;
      const int64_t k = base + (int64_t)j * nx + i;
      double S[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      double b[5], G[9], Qm[9], T1[9], T2[9], T3[9];
      if (i > 0) {  // W: term B_kW Q_W G_W B_WE
        const int64_t m = k - 1;
        load9(J, NN, m, 0, G);
        load_nb(J, NN, m, 1, b);
        mul_dense_nb(G, b, T1);
        load9(Q, NN, m, 0, Qm);
        mul33(Qm, T1, T2);
        load_nb(J, NN, k, 0, b);
        mul_nb_dense(b, T2, T3);
#pragma unroll
        for (int e = 0; e < 9; ++e) S[e] += T3[e];
      }
      if (j > 0) {  // S: term B_kS Q_S G_S B_SN
        const int64_t m = k - nx;
        load9(J, NN, m, 0, G);
        load_nb(J, NN, m, 3, b);
        mul_dense_nb(G, b, T1);
        load9(Q, NN, m, 0, Qm);
        mul33(Qm, T1, T2);
        load_nb(J, NN, k, 2, b);
        mul_nb_dense(b, T2, T3);
#pragma unroll
        for (int e = 0; e < 9; ++e) S[e] += T3[e];
      }
      load9(J, NN, k, 0, G);
      double D[9];
      mul33(G, S, D);
#pragma unroll
      for (int e = 0; e < 9; ++e) D[e] = (e % 4 == 0 ? 1.0 : 0.0) - D[e];
      double inv[9];
      if (!inverse33(D, inv) && status) atomicExch(&status[inst], TCAD_ERR_SINGULAR);
#pragma unroll
      for (int e = 0; e < 9; ++e) Q[(int64_t)e * NN + k] = inv[e];
    }
    __syncthreads();
  }
}

// out = M^-1 rin for every instance still iterating (ks[inst].active);
// instances with mask[inst] == 0 are not preconditioned (out = rin).
template <class T>
__global__ void __launch_bounds__(kIluThreads)
k_ilu2d_apply(const tcad_pack_t pk, const double* __restrict__ J, const double* __restrict__ Q,
              const T* __restrict__ rin, T* __restrict__ out, const KState* ks,
              const uint8_t* __restrict__ mask, int nzmax) {
  const int inst = blockIdx.x / nzmax, z = blockIdx.x % nzmax;
  if (ks && !ks[inst].active) return;
  const Inst g = load_inst(pk, inst);
  if (z >= g.nz) return;
  const int64_t base = g.off + (int64_t)z * g.nx * g.ny;  // this z-plane (2D: the instance)
  const int64_t NN = pk.n_nodes;
  if (mask && !mask[inst]) {
    const int64_t end = base + (int64_t)g.nx * g.ny;
    for (int64_t k = base + threadIdx.x; k < end; k += kIluThreads) {
      out[k] = rin[k];
      out[NN + k] = rin[NN + k];
      out[2 * NN + k] = rin[2 * NN + k];
    }
    return;
  }
  const int nx = g.nx, ny = g.ny;
  const int nd = nx + ny - 1;
  // Fast path when every anti-diagonal fits the block (min(nx, ny) <=
  // threads).  Each thread owns one row c of the shorter dimension (j, or i
  // when nx < ny) and walks along it, one node per anti-diagonal level: the
  // previous node of its own row is in a register, the other lower
  // neighbour (row c-1, same position) comes from a shared-memory front,
  // and the node data of the next two positions of its row is already in
  // flight, so each level costs only the dependent arithmetic and a barrier.
  const bool byj = ny <= nx;
  const int Lc = byj ? ny : nx, Lw = byj ? nx : ny;
  if (Lc <= kIluThreads) {
    __shared__ double fr[2][kIluThreads][3];
    // rows by parity: warps 0..3 own the even rows, warps 4..7 the odd ones,
    // so (d - c) has one parity across a warp and the slot choice below
    // never diverges inside a warp
    const int tid = threadIdx.x, half = kIluThreads / 2;
    const int c = tid < half ? 2 * tid : 2 * (tid - half) + 1;
    const bool lane = c < Lc;
    // neighbour directions: along the row (walk) and across rows (cross)
    const int dwp = byj ? 0 : 2, dcp = byj ? 2 : 0;   // forward: W/S
    const int dwn = byj ? 1 : 3, dcn = byj ? 3 : 1;   // backward: E/N
    auto node = [&](int w) -> int64_t {
      return byj ? base + (int64_t)c * nx + w : base + (int64_t)w * nx + c;
    };
    struct Nd {
      double G[9], Q[9], bw[5], bc[5], v[3];
    };
    // forward data of position w (v = r)
    auto load_f = [&](int w, Nd& o) {
      if (!lane || w < 0 || w >= Lw) return;
      const int64_t k = node(w);
      load9(J, NN, k, 0, o.G);
      load9(Q, NN, k, 0, o.Q);
      if (w > 0) load_nb(J, NN, k, dwp, o.bw);
      if (c > 0) load_nb(J, NN, k, dcp, o.bc);
      o.v[0] = rin[k]; o.v[1] = rin[NN + k]; o.v[2] = rin[2 * NN + k];
    };
    // backward data of position w (v = a from the forward sweep)
    auto load_b = [&](int w, Nd& o) {
      if (!lane || w < 0 || w >= Lw) return;
      const int64_t k = node(w);
      load9(J, NN, k, 0, o.G);
      load9(Q, NN, k, 0, o.Q);
      if (w < Lw - 1) load_nb(J, NN, k, dwn, o.bw);
      if (c < Lc - 1) load_nb(J, NN, k, dcn, o.bc);
      o.v[0] = out[k]; o.v[1] = out[NN + k]; o.v[2] = out[2 * NN + k];
    };
    // two register slots: position w lives in slot (w & 1); after a
    // position is used its slot is reloaded with position w + 2 (no copies,
    // so a pending load is waited for only where its data is used)
    Nd A, B;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;   // own previous result
    int cur = 0;
    auto fstep = [&](const Nd& X, int w) {
      const int pv = cur ^ 1;
      double u0 = 0.0, u1 = 0.0, u2 = 0.0;
      if (w > 0) add_nb_vec(X.bw, p0, p1, p2, u0, u1, u2);
      if (c > 0) {
        const double* f = fr[pv][c - 1];
        add_nb_vec(X.bc, f[0], f[1], f[2], u0, u1, u2);
      }
      const double t0 = X.v[0] - (X.G[0] * u0 + X.G[1] * u1 + X.G[2] * u2);
      const double t1 = X.v[1] - (X.G[3] * u0 + X.G[4] * u1 + X.G[5] * u2);
      const double t2 = X.v[2] - (X.G[6] * u0 + X.G[7] * u1 + X.G[8] * u2);
      p0 = X.Q[0] * t0 + X.Q[1] * t1 + X.Q[2] * t2;
      p1 = X.Q[3] * t0 + X.Q[4] * t1 + X.Q[5] * t2;
      p2 = X.Q[6] * t0 + X.Q[7] * t1 + X.Q[8] * t2;
      double* f = fr[cur][c];
      f[0] = p0; f[1] = p1; f[2] = p2;
      const int64_t k = node(w);
      out[k] = (T)p0; out[NN + k] = (T)p1; out[2 * NN + k] = (T)p2;
    };
    auto bstep = [&](const Nd& X, int w) {
      const int pv = cur ^ 1;
      double u0 = 0.0, u1 = 0.0, u2 = 0.0;
      if (w < Lw - 1) add_nb_vec(X.bw, p0, p1, p2, u0, u1, u2);
      if (c < Lc - 1) {
        const double* f = fr[pv][c + 1];
        add_nb_vec(X.bc, f[0], f[1], f[2], u0, u1, u2);
      }
      const double t0 = X.G[0] * u0 + X.G[1] * u1 + X.G[2] * u2;
      const double t1 = X.G[3] * u0 + X.G[4] * u1 + X.G[5] * u2;
      const double t2 = X.G[6] * u0 + X.G[7] * u1 + X.G[8] * u2;
      p0 = X.v[0] - (X.Q[0] * t0 + X.Q[1] * t1 + X.Q[2] * t2);
      p1 = X.v[1] - (X.Q[3] * t0 + X.Q[4] * t1 + X.Q[5] * t2);
      p2 = X.v[2] - (X.Q[6] * t0 + X.Q[7] * t1 + X.Q[8] * t2);
      double* f = fr[cur][c];
      f[0] = p0; f[1] = p1; f[2] = p2;
      const int64_t k = node(w);
      out[k] = (T)p0; out[NN + k] = (T)p1; out[2 * NN + k] = (T)p2;
    };
    // ---- forward: a_k = Q_k (r_k - G_k (B_walk a_prev + B_cross a_cross))
    load_f(0, A);
    load_f(1, B);
    for (int d = 0; d < nd; ++d) {
      const int w = d - c;
      if (lane && w >= 0 && w < Lw) {
        if ((w & 1) == 0) {
          fstep(A, w);
          load_f(w + 2, A);
        } else {
          fstep(B, w);
          load_f(w + 2, B);
        }
      }
      __syncthreads();
      cur ^= 1;
    }
    // ---- backward: x_k = a_k - Q_k G_k (B_walk x_next + B_cross x_cross)
    if (((Lw - 1) & 1) == 0) {
      load_b(Lw - 1, A);
      load_b(Lw - 2, B);
    } else {
      load_b(Lw - 1, B);
      load_b(Lw - 2, A);
    }
    for (int d = nd - 1; d >= 0; --d) {
      const int w = d - c;
      if (lane && w >= 0 && w < Lw) {
        if ((w & 1) == 0) {
          bstep(A, w);
          load_b(w - 2, A);
        } else {
          bstep(B, w);
          load_b(w - 2, B);
        }
      }
      __syncthreads();
      cur ^= 1;
    }
    return;
  }
  // forward: a_k = Q_k (r_k - G_k (B_kW a_W + B_kS a_S))
  for (int d = 0; d < nd; ++d) {
    const int jlo = d - (nx - 1) > 0 ? d - (nx - 1) : 0;
    const int jhi = d < ny - 1 ? d : ny - 1;
    for (int j = jlo + threadIdx.x; j <= jhi; j += kIluThreads) {
      const int i = d - j;
      const int64_t k = base + (int64_t)j * nx + i;
      double u0 = 0.0, u1 = 0.0, u2 = 0.0, b[5];
      if (i > 0) {
        load_nb(J, NN, k, 0, b);
        add_nb_vec(b, out[k - 1], out[NN + k - 1], out[2 * NN + k - 1], u0, u1, u2);
      }
      if (j > 0) {
        load_nb(J, NN, k, 2, b);
        add_nb_vec(b, out[k - nx], out[NN + k - nx], out[2 * NN + k - nx], u0, u1, u2);
      }
      double G[9], Qk[9];
      load9(J, NN, k, 0, G);
      load9(Q, NN, k, 0, Qk);
      const double t0 = rin[k] - (G[0] * u0 + G[1] * u1 + G[2] * u2);
      const double t1 = rin[NN + k] - (G[3] * u0 + G[4] * u1 + G[5] * u2);
      const double t2 = rin[2 * NN + k] - (G[6] * u0 + G[7] * u1 + G[8] * u2);
      out[k] = (T)(Qk[0] * t0 + Qk[1] * t1 + Qk[2] * t2);
      out[NN + k] = (T)(Qk[3] * t0 + Qk[4] * t1 + Qk[5] * t2);
      out[2 * NN + k] = (T)(Qk[6] * t0 + Qk[7] * t1 + Qk[8] * t2);
    }
    __syncthreads();
  }
  // backward: x_k = a_k - Q_k G_k (B_kE x_E + B_kN x_N), in place
  for (int d = nd - 1; d >= 0; --d) {
    const int jlo = d - (nx - 1) > 0 ? d - (nx - 1) : 0;
    const int jhi = d < ny - 1 ? d : ny - 1;
    for (int j = jlo + threadIdx.x; j <= jhi; j += kIluThreads) {
      const int i = d - j;
      const int64_t k = base + (int64_t)j * nx + i;
      double u0 = 0.0, u1 = 0.0, u2 = 0.0, b[5];
      if (i < nx - 1) {
        load_nb(J, NN, k, 1, b);
        add_nb_vec(b, out[k + 1], out[NN + k + 1], out[2 * NN + k + 1], u0, u1, u2);
      }
      if (j < ny - 1) {
        load_nb(J, NN, k, 3, b);
        add_nb_vec(b, out[k + nx], out[NN + k + nx], out[2 * NN + k + nx], u0, u1, u2);
      }
      double G[9], Qk[9];
      load9(J, NN, k, 0, G);
      load9(Q, NN, k, 0, Qk);
      const double t0 = G[0] * u0 + G[1] * u1 + G[2] * u2;
      const double t1 = G[3] * u0 + G[4] * u1 + G[5] * u2;
      const double t2 = G[6] * u0 + G[7] * u1 + G[8] * u2;
      out[k] = (T)((double)out[k] - (Qk[0] * t0 + Qk[1] * t1 + Qk[2] * t2));
      out[NN + k] = (T)((double)out[NN + k] - (Qk[3] * t0 + Qk[4] * t1 + Qk[5] * t2));
      out[2 * NN + k] = (T)((double)out[2 * NN + k] - (Qk[6] * t0 + Qk[7] * t1 + Qk[8] * t2));
    }
    __syncthreads();
  }
}

}  // namespace tcad

namespace tcad {

constexpr int NT_ILU_FLAT = 256;  // flat (node-parallel) permutation kernels

// Factor of the 2D instances with slot data: thread c owns row c and walks
// along it, level by level as the sweeps do.  Its own previous Q G B_walk' is in
// registers and the row below's Q G B_cross' in shared memory -- the terms of
// the recursion and, rounded to FP32, the backward records -- and the next
// position's blocks of J are loaded while this one is worked on.  (Recomputing
// the neighbours' products from J and Q in global memory at every level took
// 609 us on a batch of up to 120 x 60 devices, this takes 174.)
__global__ void __launch_bounds__(kIluThreads)
k_ilu_factor_rows(const tcad_pack_t pk, const double* __restrict__ J, double* __restrict__ Q,
                  const int32_t* __restrict__ pre_status, float* __restrict__ Mf,
                  float* __restrict__ Mb) {
  const int inst = blockIdx.x;
  if (pre_status[inst] != TCAD_OK) return;
  const Inst g = load_inst(pk, inst);
  const IluGeo q = ilu_geo(g, g.off);
  const int Lc = q.Lc, Lw = q.Lw, nd = Lc + Lw - 1, c = threadIdx.x;
  const int64_t NN = pk.n_nodes;
  // neighbour directions (W 0, E 1, S 2, N 3): along the row and across rows
  const int dwp = q.byj ? 0 : 2, dcp = q.byj ? 2 : 0, dwn = q.byj ? 1 : 3, dcn = q.byj ? 3 : 1;
  __shared__ double tn[2][9][kIluThreads];
  struct Nd {
    double G[9], b[4][5];
  };
  auto node = [&](int w) { return g.off + (q.byj ? (int64_t)c * g.nx + w : (int64_t)w * g.nx + c); };
  auto valid = [&](int d) { return c < Lc && d - c >= 0 && d - c < Lw; };
  auto load = [&](int d, Nd& o) {
    if (!valid(d)) return;
    const int w = d - c;
    const int64_t k = node(w);
    load9(J, NN, k, 0, o.G);
    const int dir[4] = {dwp, dcp, dwn, dcn};
    const bool has[4] = {w > 0, c > 0, w < Lw - 1, c < Lc - 1};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (has[m]) load_nb(J, NN, k, dir[m], o.b[m]);
      else
#pragma unroll
        for (int e = 0; e < 5; ++e) o.b[m][e] = 0.0;
    }
  };
  double tw[9];   // Q G B_walk' of the previous position
#pragma unroll
  for (int e = 0; e < 9; ++e) tw[e] = 0.0;
  Nd cur;
  load(0, cur);
  for (int d = 0; d < nd; ++d) {
    Nd nxt;
    load(d + 1, nxt);
    if (valid(d)) {
      const int w = d - c;
      double S[9], T[9], D[9], Qk[9], QG[9];
      mul_nb_dense(cur.b[0], tw, S);
      if (c > 0) {
        double tc[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) tc[e] = tn[(d & 1) ^ 1][e][c - 1];
        mul_nb_dense(cur.b[1], tc, T);
#pragma unroll
        for (int e = 0; e < 9; ++e) S[e] += T[e];
      }
      mul33(cur.G, S, D);
#pragma unroll
      for (int e = 0; e < 9; ++e) D[e] = (e % 4 == 0 ? 1.0 : 0.0) - D[e];
      inverse33(D, Qk);
      const int64_t k = node(w);
#pragma unroll
      for (int e = 0; e < 9; ++e) Q[(int64_t)e * NN + k] = Qk[e];
      mul33(Qk, cur.G, QG);
      float rec[2][kIluVec];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        mul_dense_nb(QG, cur.b[m], T);
#pragma unroll
        for (int e = 0; e < 9; ++e) {
          rec[m >> 1][9 * (m & 1) + e] = (float)T[e];
          if (m == 2) tw[e] = T[e];
          if (m == 3) tn[d & 1][e][c] = T[e];
        }
      }
      const int64_t sl = q.soff + (int64_t)d * Lc + c;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        rec[h][18] = rec[h][19] = 0.0f;
        float4* const dst = reinterpret_cast<float4*>((h ? Mb : Mf) + sl * kIluRec);
#pragma unroll
        for (int e = 0; e < kIluVec / 4; ++e)
          dst[e] = make_float4(rec[h][4 * e], rec[h][4 * e + 1], rec[h][4 * e + 2],
                               rec[h][4 * e + 3]);
      }
    }
    __syncthreads();
    cur = nxt;
  }
}

// the forward records' vectors = Q r for the instances preconditioned here
template <class T>
__global__ void __launch_bounds__(NT_ILU_FLAT)
k_ilu_perm(const tcad_pack_t pk, const double* __restrict__ Q, const T* r,
           float* __restrict__ Mf, const KState* ks, const uint8_t* __restrict__ mask,
           const int32_t* __restrict__ blk) {
  chain_in();
  const int64_t fbi = blk ? (int64_t)blk[blockIdx.x] : (int64_t)blockIdx.x;
  const FlatBlock fb = flat_block(pk, fbi);
  if (ks && !ks[fb.inst].active) return;
  if (mask && !mask[fb.inst]) return;
  const Inst g = load_inst(pk, fb.inst);
  const IluGeo q = ilu_geo(g, g.off);
  const int64_t NN = pk.n_nodes;
  for (int64_t k = fb.begin + threadIdx.x; k < fb.end; k += NT_ILU_FLAT) {
    const unsigned loc = (unsigned)(k - g.off);
    const int j = (int)(loc / (unsigned)g.nx), i = (int)(loc - (unsigned)j * (unsigned)g.nx);
    double Qk[9];
    load9(Q, NN, k, 0, Qk);
    const double r0 = (double)r[k], r1 = (double)r[NN + k], r2 = (double)r[2 * NN + k];
    double2* const dst = ilu_vec(Mf, ilu_slot(q, i, j));
    dst[0] = make_double2(Qk[0] * r0 + Qk[1] * r1 + Qk[2] * r2,
                          Qk[3] * r0 + Qk[4] * r1 + Qk[5] * r2);
    dst[1] = make_double2(Qk[6] * r0 + Qk[7] * r1 + Qk[8] * r2, 0.0);
  }
}

// out (node order) = the backward records' vectors; instances not preconditioned:
// out = r
template <class T>
__global__ void __launch_bounds__(NT_ILU_FLAT)
k_ilu_unperm(const tcad_pack_t pk, float* Mb, const T* r,
             T* out, const KState* ks, const uint8_t* __restrict__ mask,
             const int32_t* __restrict__ blk) {
  chain_in();
  const int64_t fbi = blk ? (int64_t)blk[blockIdx.x] : (int64_t)blockIdx.x;
  const FlatBlock fb = flat_block(pk, fbi);
  if (ks && !ks[fb.inst].active) return;
  const int64_t NN = pk.n_nodes;
  if (mask && !mask[fb.inst]) {
    for (int64_t k = fb.begin + threadIdx.x; k < fb.end; k += NT_ILU_FLAT) {
      out[k] = r[k]; out[NN + k] = r[NN + k]; out[2 * NN + k] = r[2 * NN + k];
    }
    return;
  }
  const Inst g = load_inst(pk, fb.inst);
  const IluGeo q = ilu_geo(g, g.off);
  for (int64_t k = fb.begin + threadIdx.x; k < fb.end; k += NT_ILU_FLAT) {
    const unsigned loc = (unsigned)(k - g.off);
    const int j = (int)(loc / (unsigned)g.nx), i = (int)(loc - (unsigned)j * (unsigned)g.nx);
    const double2* const src = ilu_vec(Mb, ilu_slot(q, i, j));
    const double2 a = src[0], b = src[1];
    out[k] = (T)a.x; out[NN + k] = (T)a.y; out[2 * NN + k] = (T)b.x;
  }
}

// The sweeps, one CTA per 2D instance (Lc <= rows <= kIluThreads).
//
// A sweep is a chain of nx + ny - 1 levels, so what counts is a level's
// dependent part: the values of the level before from shared memory, five
// dependent multiply-adds and the store of the result.  Everything else is kept
// off it:
// - GROUPS groups of `rows` threads take the levels in turn (thread c of a group:
//   row c).  Only the group whose turn it is waits for the one before (a named
//   barrier that the latter arrives at without waiting); the others meanwhile
//   wait for their next level's records, read them and convert them (18 FP32 to
//   FP64 conversions a thread: 200 cycles of that pipe, more than the level).
// - One more warp fills a ring of up to kIluStages levels in shared memory with
//   bulk copies, one contiguous run a level.  (Its thread takes about as long as a
//   level: one more wait of it per level cost a third of the sweep.)
// Devices of up to 120 x 60, both sweeps: 175 us with one group of 256 threads that loaded
// two levels ahead into registers from 30 arrays; 54 us now.
// `ring`: bytes of dynamic shared memory, at least GROUPS levels of the longest Lc.
template <int GROUPS>
__global__ void __launch_bounds__(kIluSweepThreads)
k_ilu_sweep(const tcad_pack_t pk, float* Mf, float* Mb, KState* ks,
            const uint8_t* __restrict__ mask, int rows, int ring, bool hold) {
  chain_in();
  extern __shared__ __align__(128) unsigned char s_ring[];
  __shared__ uint64_t s_full[kIluStages], s_empty[kIluStages];
  __shared__ double fr[2][3][kIluThreads];
  const int inst = blockIdx.x;
  if (!ks[inst].active) return;
  if (mask && !mask[inst]) return;
  const Inst g = load_inst(pk, inst);
  const IluGeo q = ilu_geo(g, g.off);
  const int Lc = q.Lc, Lw = q.Lw, nd = Lc + Lw - 1;
  const int level = Lc * kIluRec * (int)sizeof(float);
  const int D = min(kIluStages, ring / level);
  if (threadIdx.x == 0) {
    for (int i = 0; i < D; ++i) {
      mbar_init(&s_full[i]);
      mbar_init(&s_empty[i], rows / 32);   // one arrival per warp of a group
    }
    fence_async();
  }
  for (int i = threadIdx.x; i < 2 * 3 * kIluThreads; i += blockDim.x) (&fr[0][0][0])[i] = 0.0;
  __syncthreads();
  // A wait that runs out: the thread does not say that it has read a level from then
  // on, so the copying thread's own wait runs out and it starts no more copies.
  bool lost = false;
  int issued = 0;                                 // levels whose copy was started
  auto wait = [&](uint64_t* b, unsigned parity) {
    if (!mbar_wait(b, parity, lost)) lost = true;
  };
  const int grp = threadIdx.x / rows;             // GROUPS: the copying warp
  const int c = threadIdx.x - grp * rows, lane = threadIdx.x & 31;
  auto sweep = [&](bool fwd, int base) {          // base: levels of the ring used so far
    auto at = [&](int s) { return fwd ? s : nd - 1 - s; };
    if (grp == GROUPS) {
      if (lane != 0) return;
      const float* const M = fwd ? Mf : Mb;
      int st = base % D;
      unsigned par = (base / D) & 1;
      int s = 0;
      if (hold) {                                 // (test hook: a copy that never comes)
        mbar_expect(&s_full[st], level);
        if (++st == D) { st = 0; par ^= 1u; }
        s = 1;
      }
      for (; s < nd; ++s) {
        if (!mbar_wait(&s_empty[st], par ^ 1u)) {   // the first round finds them empty
          lost = true;
          break;
        }
        mbar_expect(&s_full[st], level);
        bulk_copy(s_ring + st * level, M + (q.soff + (int64_t)at(s) * Lc) * kIluRec, level,
                  &s_full[st]);
        if (++st == D) { st = 0; par ^= 1u; }
      }
      issued = base + s;
      return;
    }
    const int cn = fwd ? max(c - 1, 0) : min(c + 1, Lc - 1);   // (its record is 0 at the edge)
    int st = (base + grp) % D;
    unsigned par = ((base + grp) / D) & 1;
    for (int s = grp; s < nd; s += GROUPS) {
      const int w = at(s) - c;
      const bool mine = c < Lc && w >= 0 && w < Lw;
      wait(&s_full[st], par);
      double mw[9], mc[9], a[3];
      if (mine) {
        const float4* const m4 =
            reinterpret_cast<const float4*>(s_ring + st * level + c * 4 * kIluRec);
        float f[kIluVec];
#pragma unroll
        for (int e = 0; e < kIluVec / 4; ++e) {
          const float4 v = m4[e];
          f[4 * e] = v.x; f[4 * e + 1] = v.y; f[4 * e + 2] = v.z; f[4 * e + 3] = v.w;
        }
#pragma unroll
        for (int e = 0; e < 9; ++e) { mw[e] = (double)f[e]; mc[e] = (double)f[9 + e]; }
        const double2* const r2 = reinterpret_cast<const double2*>(m4 + kIluVec / 4);
        const double2 u = r2[0], v = r2[1];
        a[0] = u.x; a[1] = u.y; a[2] = v.x;
      }
      __syncwarp();
      if (lane == 0 && !lost) mbar_arrive(&s_empty[st]);
      st += GROUPS;
      if (st >= D) { st -= D; par ^= 1u; }
      // level s - 1 is in fr (its group arrived; the first level has none)
      if (s > 0)
        asm volatile("bar.sync %0, %1;" ::"r"(1 + s % GROUPS), "r"(2 * rows) : "memory");
      if (mine) {
        const double(*const f)[kIluThreads] = fr[(s & 1) ^ 1];
        const double p0 = f[0][c], p1 = f[1][c], p2 = f[2][c];
        const double x0 = f[0][cn], x1 = f[1][cn], x2 = f[2][cn];
        const bool first = fwd ? w == 0 : w == Lw - 1;   // no position before this one
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const double ow = mw[3 * e] * p0 + mw[3 * e + 1] * p1 + mw[3 * e + 2] * p2;
          const double ox = mc[3 * e] * x0 + mc[3 * e + 1] * x1 + mc[3 * e + 2] * x2;
          a[e] = (a[e] - (first ? 0.0 : ow)) - ox;
          fr[s & 1][e][c] = a[e];
        }
      }
      if (s + 1 < nd)
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + (s + 1) % GROUPS), "r"(2 * rows) : "memory");
      if (mine) {
        double2* const dst = ilu_vec(Mb, q.soff + (int64_t)at(s) * Lc + c);
        dst[0] = make_double2(a[0], a[1]);
        dst[1] = make_double2(a[2], 0.0);
      }
    }
  };
  sweep(true, 0);
  __threadfence();
  fence_async();   // the forward results, before the bulk copies that read them
  if (!__syncthreads_or(lost)) sweep(false, nd);
  if (!__syncthreads_or(lost)) return;
  // the copies in flight: the last D that were started
  if (grp == GROUPS && lane == 0)
    for (int i = max(issued - D, 0); i < issued; ++i)
      (void)mbar_wait(&s_full[i % D], (i / D) & 1);
  if (lost) {
    ks[inst].status = TCAD_ERR_CUDA;
    ks[inst].active = 0;
  }
}

}  // namespace tcad
