// psbx_gridsync.cuh -- reductions over all blocks of a cooperative launch
// that are the grid barrier at the same time.
//
// Every block reduces its values, warp 0 publishes them, and every block reads
// all blocks' values and adds them in block order: the totals hold the same
// bits everywhere, so all blocks take the same branches and none broadcasts
// anything.  Two ways of publishing, by the number of blocks:
//
// up to GS_TAG_BLOCKS: each value goes into the block's slot -- a 128-byte line
//   of its own -- in one 16-byte word with the sequence number of the
//   reduction, and the blocks read all slots until their numbers match.  One
//   exchange through L2: two sums over 7 blocks of 256 threads 1.3 us in all,
//   against 2.2 us with the counter.
// more: one thread adds to a counter with release order and waits for it to
//   reach the number of blocks, then warp 0 reads all slots.  With 148 blocks
//   polling 148 slots the polls hold up the late stores: 3.7 us against 2.9 us
//   (measured in the solver's loop, two sums).
// The line between them, us an iteration of CG and of BiCGSTAB with tags and with
// the counter: 9 blocks 5.7 / 6.6 and 9.9 / 11.2; 32 6.6 / 6.8 and 11.4 / 11.5; 42
// 6.75 / 6.82 and 11.5 / 11.4; 48 6.85 / 6.82 and 11.7 / 11.4; 62 7.0 / 6.8 and
// 12.0 / 11.4; 148 13.0 / 11.0 and 23.7 / 19.7.
//
// Two slot buffers alternate: a block publishes reduction s + 2 only after it
// has seen every block's s + 1, which a block publishes after it has read all
// of s.  Waits are bounded (GS_WAIT_NS): past the bound `bad` is set, and the
// kernel returns with a timeout status.
#pragma once

#include "psbx_internal.cuh"

#define GS_MAXV 8                        // 8-byte values a reduction carries: 2 per sum, 1 per max
#define GS_MAXWARPS 16                   // warps of a block
#define GS_WAIT_NS 10000000000ull        // 10 s: far beyond any phase, and finite

// Shared memory of the reductions of one block.
struct GsShared {
  double red[2][GS_MAXV][GS_MAXWARPS];   // per-warp values, by parity of the sequence number
  double tot[2][GS_MAXV][GS_MAXWARPS];   // per-warp values of the slots read
  int bad;
};

struct GridSync {
  ulonglong2 *slots;                     // [2][nblocks][GS_SLOT] and the counter, zero at launch, 128-byte aligned
  GsShared *sh;
  unsigned long long seq;
  int nblocks;
};
#define GS_SLOT 8                        // 16-byte words of a slot
#define GS_TAG_BLOCKS 40
#define GS_MAXB 160                      // blocks of a launch: one per SM
#define GS_BYTES(nblocks) (sizeof(ulonglong2) * GS_SLOT * (2 * (size_t)(nblocks) + 2))

__device__ __forceinline__ void gs_store(ulonglong2 *p, double v, unsigned long long tag) {
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ ulonglong2 gs_load(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void gs_arrive(unsigned *p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned gs_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void gs_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ unsigned long long gs_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ dd_t dd_shfl_xor(dd_t v, int o) {
  dd_t u;
  u.s = __shfl_xor_sync(0xffffffffu, v.s, o);
  u.c = __shfl_xor_sync(0xffffffffu, v.c, o);
  return u;
}

// Warp sum / max, the result in every lane (merging is commutative to the
// bit, so all lanes agree).
template <int NS, int NM>
__device__ __forceinline__ void gs_warp(dd_t *s, double *m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < NS; k++) s[k] = dd_merge(s[k], dd_shfl_xor(s[k], o));
#pragma unroll
    for (int k = 0; k < NM; k++) m[k] = fmax(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
  }
}

// Sums S values and maximises M values over the grid (arrays of length
// max(1, .)); every thread gets the totals.  FENCE: what any thread wrote to
// global memory before it is visible to every thread after it.  Every thread
// of every block calls it.
template <int S, int M, bool FENCE>
__device__ __forceinline__ void grid_reduce(GridSync &g, dd_t (&s)[S > 0 ? S : 1], double (&m)[M > 0 ? M : 1]) {
  constexpr int NV = 2 * S + M, NW = NV > 0 ? NV : 1;
  static_assert(NV <= GS_MAXV && GS_MAXV <= GS_SLOT, "values per reduction");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int par = (int)(g.seq & 1);
  GsShared &sh = *g.sh;  // (its arrays hold GS_MAXWARPS warps: the launch bound of the kernels that use it)
  auto from_warps = [&]() {
#pragma unroll
    for (int k = 0; k < S; k++)
      s[k] = lane < nw ? dd_t{sh.red[par][2 * k][lane], sh.red[par][2 * k + 1][lane]} : dd_t{0.0, 0.0};
#pragma unroll
    for (int k = 0; k < M; k++) m[k] = lane < nw ? sh.red[par][2 * S + k][lane] : 0.0;
    gs_warp<S, M>(s, m);
  };
  if (NV > 0) {
    gs_warp<S, M>(s, m);
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < S; k++) sh.red[par][2 * k][warp] = s[k].s, sh.red[par][2 * k + 1][warp] = s[k].c;
#pragma unroll
      for (int k = 0; k < M; k++) sh.red[par][2 * S + k][warp] = m[k];
    }
  }
  __syncthreads();
  g.seq++;
  if (g.nblocks == 1) {
    if (NV > 0) from_warps();  // every warp for itself
    return;
  }
  ulonglong2 *buf = g.slots + (size_t)par * g.nblocks * GS_SLOT;
  const int np = (g.nblocks + 31) >> 5;
  if (g.nblocks > GS_TAG_BLOCKS) {
    // counter: slots hold plain values, value k of block b at part[k*nblocks + b]
    double *part = (double *)buf;
    if (warp == 0) {
      if (NV > 0) {
        from_warps();
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < S; k++) {
            part[(2 * k) * g.nblocks + blockIdx.x] = s[k].s;
            part[(2 * k + 1) * g.nblocks + blockIdx.x] = s[k].c;
          }
#pragma unroll
          for (int k = 0; k < M; k++) part[(2 * S + k) * g.nblocks + blockIdx.x] = m[k];
        }
      }
      // every lane waits, on the one word, and they leave together: a wait by
      // lane 0 alone left the warp split at the shuffles below (7 us)
      unsigned *counter = (unsigned *)(g.slots + (size_t)2 * g.nblocks * GS_SLOT);
      __syncwarp();
      if (lane == 0) gs_arrive(counter);
      __syncwarp();
      const unsigned want = (unsigned)g.seq * (unsigned)g.nblocks;
      unsigned spins = 0;
      unsigned long long t0 = 0;
      while (!__all_sync(0xffffffffu, (int)(gs_acquire(counter) - want) >= 0)) {
        if ((++spins & 1023u) == 0) {
          const unsigned long long now = gs_now();
          if (t0 == 0) t0 = now;
          if (__any_sync(0xffffffffu, now - t0 > GS_WAIT_NS)) {
            if (lane == 0) sh.bad = 1;
            break;
          }
        }
      }
      __syncwarp();
      if (NV > 0) {
        constexpr int B = GS_MAXB / 32;
        double v[B][NW];
#pragma unroll
        for (int u = 0; u < B; u++)
#pragma unroll
          for (int k = 0; k < NV; k++)
            v[u][k] = lane + 32 * u < g.nblocks ? __ldcg(part + k * g.nblocks + lane + 32 * u) : 0.0;
#pragma unroll
        for (int k = 0; k < S; k++) s[k] = dd_t{v[0][2 * k], v[0][2 * k + 1]};
#pragma unroll
        for (int k = 0; k < M; k++) m[k] = v[0][2 * S + k];
#pragma unroll
        for (int u = 1; u < B; u++) {
#pragma unroll
          for (int k = 0; k < S; k++) s[k] = dd_merge(s[k], dd_t{v[u][2 * k], v[u][2 * k + 1]});
#pragma unroll
          for (int k = 0; k < M; k++) m[k] = fmax(m[k], v[u][2 * S + k]);
        }
        gs_warp<S, M>(s, m);
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < S; k++) sh.tot[par][2 * k][0] = s[k].s, sh.tot[par][2 * k + 1][0] = s[k].c;
#pragma unroll
          for (int k = 0; k < M; k++) sh.tot[par][2 * S + k][0] = m[k];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < S; k++) s[k] = dd_t{sh.tot[par][2 * k][0], sh.tot[par][2 * k + 1][0]};
#pragma unroll
    for (int k = 0; k < M; k++) m[k] = sh.tot[par][2 * S + k][0];
    return;
  }
  if (warp == 0) {
    double mine = 0.0;
    if (NV > 0) {
      from_warps();
#pragma unroll
      for (int k = 0; k < S; k++) mine = lane == 2 * k ? s[k].s : lane == 2 * k + 1 ? s[k].c : mine;
#pragma unroll
      for (int k = 0; k < M; k++) mine = lane == 2 * S + k ? m[k] : mine;
    }
    if (lane < NW) {
      if (FENCE) gs_fence();
      gs_store(buf + (size_t)blockIdx.x * GS_SLOT + lane, mine, g.seq);
    }
    __syncwarp();
  }
#pragma unroll
  for (int k = 0; k < S; k++) s[k] = dd_t{0.0, 0.0};
#pragma unroll
  for (int k = 0; k < M; k++) m[k] = 0.0;
  // slots t, t + blockDim, ... by thread t, in block order within a thread (one
  // slot as GS_TAG_BLOCKS stands; written without the loop, the solver's
  // registers come out 3 to 6 % slower).
  // The lanes of a warp leave the wait together, those without a slot too:
  // with some lanes ahead at the shuffles below, a reduction took 7 us.
  const int nread = np < nw ? np : nw;  // warps that read slots
  for (int b = threadIdx.x; warp < nread && b - lane < g.nblocks; b += blockDim.x) {
    const ulonglong2 *p = buf + (size_t)b * GS_SLOT;
    const bool mine = b < g.nblocks;
    ulonglong2 v[NW];
    unsigned spins = 0;
    unsigned long long t0 = 0;
    for (;;) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < NW; k++) v[k] = mine ? gs_load(p + k) : make_ulonglong2(0, g.seq);
#pragma unroll
      for (int k = 0; k < NW; k++) ok &= v[k].y == g.seq;
      if (__all_sync(0xffffffffu, ok)) break;
      if ((++spins & 1023u) == 0) {
        const unsigned long long now = gs_now();
        if (t0 == 0) t0 = now;
        if (__any_sync(0xffffffffu, now - t0 > GS_WAIT_NS)) {
          if (lane == 0) sh.bad = 1;
          break;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < S; k++) {
      const dd_t u = {__longlong_as_double(v[2 * k].x), __longlong_as_double(v[2 * k + 1].x)};
      s[k] = b < (int)blockDim.x ? u : dd_merge(s[k], u);
    }
#pragma unroll
    for (int k = 0; k < M; k++) m[k] = fmax(m[k], __longlong_as_double(v[2 * S + k].x));
    if (FENCE) gs_fence();
  }
  __syncwarp();
  if (NV > 0 && warp < nread) {
    gs_warp<S, M>(s, m);
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < S; k++) sh.tot[par][2 * k][warp] = s[k].s, sh.tot[par][2 * k + 1][warp] = s[k].c;
#pragma unroll
      for (int k = 0; k < M; k++) sh.tot[par][2 * S + k][warp] = m[k];
    }
  }
  __syncthreads();
  if (NV > 0) {
#pragma unroll
    for (int k = 0; k < S; k++) s[k] = dd_t{sh.tot[par][2 * k][0], sh.tot[par][2 * k + 1][0]};
#pragma unroll
    for (int k = 0; k < M; k++) m[k] = sh.tot[par][2 * S + k][0];
    for (int w = 1; w < nread; w++) {
#pragma unroll
      for (int k = 0; k < S; k++) s[k] = dd_merge(s[k], dd_t{sh.tot[par][2 * k][w], sh.tot[par][2 * k + 1][w]});
#pragma unroll
      for (int k = 0; k < M; k++) m[k] = fmax(m[k], sh.tot[par][2 * S + k][w]);
    }
  }
}

// The barrier alone: all writes before it are visible after it.
__device__ __forceinline__ void grid_barrier(GridSync &g) {
  dd_t s[1];
  double m[1];
  grid_reduce<0, 0, true>(g, s, m);
}
