// Grid barrier that carries the dot products, for the single-launch solves
// whose CTAs are all resident (cooperative launch, at most kSyncMaxCtas).
//
// A CTA stores its partial sums, one thread adds an arrival to a monotonic
// counter (acquire-release) and polls it without backing off, and every CTA
// then reads all partials: each thread takes one, so the totals are in every
// thread after one block reduction.  Measured per step on 16 to 148 CTAs: 1.06
// to 1.14 us without sums, 1.6 to 1.7 with one, 1.8 with three.  Tried and
// slower at 148 CTAs: every CTA polling every other CTA's word with the sums
// in it (one trip instead of two, but 148 x 148 polls contend: 4.1 / 5.3 /
// 7.4 us), the same with private inboxes (2.3 / 2.6 / 6.4), a reduction
// instead of the returning atomic (1.24 / 1.82 / 1.98).
//
// The sums are taken in the order of block_sum / Reduce::total, so a solve
// gives the per-step kernels' bits.  Partials alternate between two buffers
// by step parity: a CTA stores step k + 2 only after all have arrived at
// k + 1, i.e. after all have read step k.
//
// Every wait is bounded (kBarrierNs of device time, or another CTA's give-up
// flag); sum() then returns false in every thread of the CTA and the kernel
// returns.
#pragma once

namespace tcad {

constexpr int kSyncMaxCtas = 2 * kFlatThreads;             // two partials per thread
constexpr int kSyncSums = 3;                               // sums per step, at most

// doubles of the partials' two buffers
constexpr size_t sync_doubles() { return 2 * kSyncSums * (size_t)kSyncMaxCtas; }

__device__ __forceinline__ unsigned atom_add_acq_rel(unsigned* p, unsigned v) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
               : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The barrier alone, for CTAs of any size.  bar[0]: arrivals; [2]: a CTA gave
// up; [3]: the give-up test hook, an arrival to wait for that never comes.
struct GridBarrier {
  unsigned* bar;
  unsigned round;

  // thread 0's part, between two CTA barriers
  __device__ __forceinline__ int arrive_and_wait() {
    const unsigned target = round * gridDim.x + ld_acquire(&bar[3]);
    if (atom_add_acq_rel(&bar[0], 1u) + 1u == target) return 1;
    unsigned long long t0 = 0;
    for (unsigned it = 1; (int)(ld_acquire(&bar[0]) - target) < 0; ++it) {
      if ((it & 255u) != 0u) continue;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (ld_acquire(&bar[2]) != 0u) return 0;
      if (now - t0 > kBarrierNs || it > (1u << 30)) {
        atomicExch(&bar[2], 1u);
        return 0;
      }
    }
    return 1;
  }

  // ok: a shared word.  Orders all global writes before it, of any thread of
  // the grid, before all reads after it.
  __device__ __forceinline__ bool wait(int* ok) {
    ++round;
    __syncthreads();
    if (threadIdx.x == 0) *ok = arrive_and_wait();
    __syncthreads();
    return *ok != 0;
  }
};

struct GridSync {
  double* partial;   // sync_doubles()
  GridBarrier gb;

  __device__ __forceinline__ void init(double* part, unsigned* b) {
    partial = part;
    gb = GridBarrier{b, 0u};
  }

  // tot = the sums over the grid (of at most PER x kFlatThreads CTAs) of the first
  // kFlatThreads threads' v, valid in every thread; NQ = 0: a barrier alone.  Orders all
  // global writes before it, of any thread of the grid, before all reads after it.
  template <int NQ, int PER = 1>
  __device__ __forceinline__ bool sum(const double* v, double* tot) {
    static_assert(NQ <= kSyncSums, "sums per step");
    static_assert(PER * kFlatThreads <= kSyncMaxCtas, "partials per thread");
    constexpr int NT = kFlatThreads, NW = NT / 32, NS = NQ > 0 ? NQ : 1;
    __shared__ double sa[NS][NW], sb[NS][NW];
    __shared__ int ok;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned G = gridDim.x;
    // the last tree of block_sum: 8 warp sums, halves added pairwise
    const auto tree = [](const double* w) {
      const double a = w[0] + w[4], b = w[1] + w[5], c = w[2] + w[6], d = w[3] + w[7];
      return (a + c) + (b + d);
    };
    const auto warps = [&](double (*dst)[NW], double* r) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r[q] += __shfl_down_sync(0xffffffffu, r[q], o);
        if (lane == 0 && warp < NW) dst[q][warp] = r[q];
      }
    };
    ++gb.round;
    double* const buf = partial + (gb.round & 1u) * (size_t)(kSyncSums * kSyncMaxCtas);
    double r[NS];
#pragma unroll
    for (int q = 0; q < NQ; ++q) r[q] = v[q];
    warps(sa, r);
    __syncthreads();   // the CTA's sums are in sa, its global writes are issued
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) buf[q * kSyncMaxCtas + blockIdx.x] = tree(sa[q]);
      ok = gb.arrive_and_wait();
    }
    __syncthreads();
    if (!ok) return false;
    if constexpr (NQ > 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        r[q] = 0.0 + (threadIdx.x < G ? __ldcg(&buf[q * kSyncMaxCtas + threadIdx.x]) : 0.0);
        if (PER > 1 && threadIdx.x < NT && threadIdx.x + NT < G)
          r[q] += __ldcg(&buf[q * kSyncMaxCtas + NT + threadIdx.x]);
      }
      warps(sb, r);
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NQ; ++q) tot[q] = tree(sb[q]);
    }
    return true;
  }
};

// The same for one thread-block cluster (hardware barrier, no bound needed: the
// CTAs of a cluster are always resident together, and a barrier of it cannot be
// waited for by fewer).  A CTA stores its sums into every peer's shared memory
// before it arrives, so the totals are at hand after the wait.  Per step on 8 / 16
// CTAs: 0.21 us without sums, 0.65 / 0.78 with one, 0.76 / 1.09 with three.
constexpr int kClusterMaxCtas = 16;

struct ClusterSync {
  unsigned rank, ctas;
  int par;

  __device__ __forceinline__ void init(double*, unsigned*) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
    par = 0;
    // a peer's shared memory may be written once the peer runs (a CTA without slots
    // of its own would get to its first sum before that)
    barrier();
  }

  __device__ __forceinline__ void barrier() {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }

  template <int NQ>
  __device__ __forceinline__ bool sum(const double* v, double* tot) {
    static_assert(NQ <= kSyncSums, "sums per step");
    constexpr int NT = kFlatThreads, NW = NT / 32, NS = NQ > 0 ? NQ : 1;
    __shared__ double sa[NS][NW], slot[2][NS][kClusterMaxCtas];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (NQ > 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double r = v[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        if (lane == 0 && warp < NW) sa[q][warp] = r;
      }
      __syncthreads();
      if (threadIdx.x < ctas) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          const double* const w = sa[q];   // (the last tree of block_sum)
          const double r = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
          unsigned peer;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                       : "=r"(peer)
                       : "r"((unsigned)__cvta_generic_to_shared(&slot[par][q][rank])),
                         "r"(threadIdx.x));
          asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer), "d"(r) : "memory");
        }
      }
      __syncwarp();
    }
    barrier();
    if constexpr (NQ > 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double r = 0.0 + (lane < (int)ctas ? slot[par][q][lane] : 0.0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        tot[q] = __shfl_sync(0xffffffffu, r, 0);
      }
      par ^= 1;
    }
    return true;
  }
};

// A resident CTA's share of the slot pack: a flat block of the grid, or of a
// cluster that has an instance to itself
struct RbShare {
  int inst, len;
  int64_t begin;
  bool lead;   // writes the instance's state
};
template <class SYNC>
__device__ __forceinline__ RbShare rb_share(const tcad_pack_t& pkb, const SYNC&) {
  const FlatBlock fb = flat_block(pkb, blockIdx.x);
  return RbShare{fb.inst, (int)(fb.end - fb.begin), fb.begin, blockIdx.x == 0};
}
__device__ __forceinline__ RbShare rb_share(const tcad_pack_t& pkb, const ClusterSync& cs) {
  const int inst = (int)(blockIdx.x / cs.ctas);
  const int64_t slots = (int64_t)pkb.shape[3 * inst] * pkb.shape[3 * inst + 1];
  const int64_t chunk = ((slots + cs.ctas - 1) / cs.ctas + 31) / 32 * 32;
  const int64_t at = cs.rank * chunk;
  const int64_t len = slots - at < chunk ? slots - at : chunk;
  return RbShare{inst, (int)(len > 0 ? len : 0), pkb.node_off[inst] + (len > 0 ? at : 0),
                 cs.rank == 0};
}

}  // namespace tcad
