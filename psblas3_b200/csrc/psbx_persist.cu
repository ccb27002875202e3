// psbx_persist.cu -- psb_krylov('CG' | 'BICGSTAB') with the diagonal
// preconditioner as one cooperative kernel, for systems whose vectors fit the
// shared memory of the SMs (krylov/psb_dcg.F90:218-295,
// krylov/psb_dcgstab.f90:226-365, stop test
// krylov/psb_d_krylov_conv_mod.f90:205-356).
//
// What bounds such a solve is latency, not bytes: as a kernel per step
// (psbx_krylov.cu) an iteration on 64,000 rows took 15 us (CG) and 23 us
// (BiCGSTAB), most of it kernel boundaries (2 us each) and the tails of the
// reductions (fence, ticket, second read: about 6 us each), for data that L2
// delivers in about 1 us.  Here a block keeps a run of 32-row slices for the
// whole solve: its part of every vector lives in shared memory, and so does
// its part of the matrix as far as it fits (columns and values of a slice
// side by side, read once); only the vector that the products gather from
// goes through L2.  Reductions are one exchange between all blocks
// (psbx_gridsync.cuh), every block updates the scalars itself, and restarts
// after a breakdown run in the kernel too, so a solve is one launch.  An
// iteration, kernel per step and here, 7-point operators: CG 13.7 / 5.9 us on
// 1,728 rows, 18.3 / 7.9 on 64,000, 42 / 17.5 on 512,000; BiCGSTAB 22.5 /
// 10.0, 26.3 / 13.1 and 71 / 34.
//
// Operation order and roundings are those of psbx_krylov.cu's kernels: rows
// sum their entries in stored order, updates are rounded multiplies and
// adds, dots are compensated; only the order in which the partial sums of a
// dot meet differs.
#include "psbx_krylov.cuh"
#include "psbx_gridsync.cuh"

#include <string.h>

#define PS_MAXT 512   // (1024 threads at 64 registers: 3 to 15 % slower)
static_assert(PS_MAXT / 32 <= GS_MAXWARPS, "warps of a block");
#define PS_SMEM (212 * 1024)  // dynamic shared memory of a block at most
// Largest itmax taken here (the kernel-per-step drivers take the rest): the
// host waits for the one kernel, so a solve that never converges should end
// in seconds.  100,000 iterations are 1.8 s (CG) and 3.4 s (BiCGSTAB) on 512,000
// rows of the 7-point operators, more by the unstaged entries that ps_limit lets
// through.
#define PS_MAXIT 100000

struct PsOut {         // the solve's result, in page-locked host memory
  double errnum, errden;
  int itx, timeout, declined;
};

// Entries of storage row s: the j-th at v[j*st], column p[j*st].
struct RowPtr {
  const double *v;
  const int *p;
  int st, n;
};
__device__ __forceinline__ RowPtr row_ptr(const HllView &A, int s) {
  const int h = A.hksz == 32 ? s >> 5 : s / A.hksz;
  const int off = ld_ro(A.hkoffs + h) + (s - h * A.hksz);
  return {A.val + off, A.ja + off, A.hksz, ld_ro(A.irn + s)};
}
__device__ __forceinline__ RowPtr row_ptr(const EllView &A, int r) {
  return {A.val + r, A.ja + r, A.pitch, ld_ro(A.irn + r)};
}
__device__ __forceinline__ RowPtr row_ptr(const CsrView &A, int r) {
  const int b = ld_ro(A.irp + r) - A.base;
  return {A.val + b, A.ja + b, 1, ld_ro(A.irp + r + 1) - A.base - b};
}

struct PsArgs {
  const double *dinv, *b;
  double *x;
  double *g;           // the vector the products gather from, n entries (matrix row order)
  ulonglong2 *slots;   // of the reductions (psbx_gridsync.cuh)
  PsOut *out;
  int nslices, max_slices;  // of the system; of a block
  int mat_entries;     // matrix entries a block's shared memory holds
  int itmax, istop;
  double eps;
  double most, per_mean, per_longest;  // what a block may read through L2 (PsLoad)
};

// What a block's products read through L2, in quarters of an entry: the
// entries of its slices that are not staged, weighted.  A block's SM reads
// them alone in every iteration, so the solve is as slow as the fullest block
// -- long rows side by side, or rows too many for the staging area -- while
// the kernel-per-step drivers spread the same rows over all SMs.
//   1.5 for rows of more than 8 entries (a slice's average) that are held one
//     after the other (CSR): a warp's loads touch a line per lane, more than the
//     L1 that the staging area leaves can hold;
//   else 0.25 + 0.75 * lines / lanes, for the lines of x that a gather touches
//     (seen at the middle entry of each row): 0.3 for a stencil, 1 at random.
struct PsLoad {
  unsigned long long cost, entries;  // weighted and unstaged; all
  int longest;
};

// Most a block may carry for the kernel to go on: a + m * (entries of an
// average block) + r * (longest row); the drivers' own time grows with
// both.  Fitted to 593 solves (length-sorted power-law rows up to 128 entries,
// rows that are long in one part of a banded matrix, random rows, 7- and
// 27-point grids; 60,000 to 690,000 rows; CSR, ELL, HLL), each timed both ways.  us an
// iteration here and with a kernel per step: CG, CSR, length-sorted rows up to 69
// entries on 480,000 rows (144,000 entries unstaged) 402 and 70; BiCGSTAB 801 and
// 115; CG, HLL, 27-point 84^3 72 and 56, 67^3 30 and 41; CG, 7-point 88^3 (31,000 unstaged)
// 22 and 34.  With the staging area beyond PS_SMEM_L1 the SM's L1 has only
// 28 KB left for the gathers and their cost doubles (200,000 rows, BiCGSTAB: 50 us
// at 184 KB, 98 at 190).
#define PS_SMEM_L1 (188 * 1024)
static void ps_limit(PsArgs &P, size_t smem) {
  const bool l1 = smem <= PS_SMEM_L1;
  P.most = l1 ? 20480.0 : 18432.0;
  P.per_mean = l1 ? 0.75 : 0.125;
  P.per_longest = l1 ? 320.0 : 128.0;
}

// A block's rows and their data in shared memory.
struct Blk {
  int s0, ns;          // first storage row, slices
  double *sv;          // staged values, slice after slice, entry-major
  int *sj;             // staged columns (0-based)
  int *len;            // row lengths
  int *off;            // per slice: start of its staged entries, or -1
};

// Row sums in stored order against the vector x (plain loads: x is written by
// other blocks during the kernel, so it must not go through the read-only
// path); f(l, i, sum) for each row: local row l, matrix row i.
template <class View, class F>
__device__ __forceinline__ void each_product(const Blk &B, const View &A, const double *x, F &&f) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  constexpr int U = 8;
  for (int k = threadIdx.x >> 5; k < B.ns; k += nw) {
    const int l = k * 32 + lane, s = B.s0 + l;
    if (s >= A.rows) continue;
    const int n = B.len[l], o = B.off[k];
    double acc = 0.0;
    if (o >= 0) {
      const double *vp = B.sv + o + lane;
      const int *jp = B.sj + o + lane;
      for (int j = 0; j < n; j += U) {
        double xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) xv[u] = j + u < n ? x[jp[(j + u) * 32]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (j + u < n) acc = radd(acc, rmul(vp[(j + u) * 32], xv[u]));
      }
    } else {
      const RowPtr r = row_ptr(A, s);
      for (int j = 0; j < n; j += U) {
        int c[U];
        double v[U], xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const bool ok = j + u < n;
          c[u] = ok ? ld_ro(r.p + (size_t)(j + u) * r.st) - A.base : 0;
          v[u] = ok ? ld_ro(r.v + (size_t)(j + u) * r.st) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) xv[u] = j + u < n ? x[c[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
          if (j + u < n) acc = radd(acc, rmul(v[u], xv[u]));
      }
    }
    f(l, out_row(A, s), acc);
  }
}

// f(l, i) for each row of the block (local row, matrix row), by the thread
// that also forms the row's product.
template <class View, class F>
__device__ __forceinline__ void each_row(const Blk &B, const View &A, F &&f) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int k = threadIdx.x >> 5; k < B.ns; k += nw) {
    const int l = k * 32 + lane, s = B.s0 + l;
    if (s < A.rows) f(l, out_row(A, s));
  }
}

// The load of a block whose rows are staged.  (A loop of its own, not
// unrolled: inside the staging loop it cost HLL's CG 2 to 20 % an iteration
// through the register allocation of the products.)
template <class View>
__device__ __forceinline__ void slice_loads(const Blk &B, const View &A, PsLoad &load) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll 1
  for (int k = warp; k < B.ns; k += nw) {
    const int l = k * 32 + lane, s = B.s0 + l, o = B.off[k], n = B.len[l];
    const unsigned e = __reduce_add_sync(0xffffffffu, (unsigned)n);
    const int w = __reduce_max_sync(0xffffffffu, n);
    unsigned long long cost = 0;
    if (o < 0) {
      RowPtr r = {nullptr, nullptr, 0, 0};
      if (n > 0) r = row_ptr(A, s);
      const int line = n > 0 ? ld_ro(r.p + (size_t)(n / 2) * r.st) >> 4 : -1;
      const unsigned lanes = __popc(__ballot_sync(0xffffffffu, n > 0));
      const unsigned first = __ffs(__match_any_sync(0xffffffffu, line)) - 1;
      const unsigned lines = __popc(__ballot_sync(0xffffffffu, n > 0 && (int)first == lane));
      const bool by_row = __any_sync(0xffffffffu, r.st == 1);
      cost = by_row && e > 8 * lanes ? 6ull * e : e + 3ull * e * lines / lanes;
    }
    if (lane == 0) {
      atomicAdd(&load.entries, (unsigned long long)e);
      atomicAdd(&load.cost, cost);
      atomicMax(&load.longest, w);
    }
  }
}

// Row lengths, slice offsets, and the matrix entries of the slices that fit.
template <class View>
__device__ __forceinline__ void stage(Blk &B, const View &A, int cap) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = warp; k < B.ns; k += nw) {
    const int l = k * 32 + lane, s = B.s0 + l;
    const int n = s < A.rows ? row_ptr(A, s).n : 0;
    B.len[l] = n;
    const int w = __reduce_max_sync(0xffffffffu, n);
    if (lane == 0) B.off[k] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long at = 0;
    for (int k = 0; k < B.ns; k++) {
      const long long e = (long long)B.off[k] * 32;
      if (at + e <= cap) {
        B.off[k] = (int)at;
        at += e;
      } else {
        B.off[k] = -1;
      }
    }
  }
  __syncthreads();
  for (int k = warp; k < B.ns; k += nw) {
    const int l = k * 32 + lane, s = B.s0 + l, o = B.off[k];
    if (s >= A.rows || o < 0) continue;
    const RowPtr r = row_ptr(A, s);
    for (int j = 0; j < r.n; j++) {
      B.sv[o + j * 32 + lane] = ld_ro(r.v + (size_t)j * r.st);
      B.sj[o + j * 32 + lane] = ld_ro(r.p + (size_t)j * r.st) - A.base;
    }
  }
}

// The scalars of the stop test, the same in every thread.
struct Conv {
  double bn2, bni, ani, r0n2, errnum, errden;
  int itx;
};

__device__ __forceinline__ bool conv_stop(const PsArgs &P, Conv &c, double rr, double amax_r, double amax_x) {
  if (P.istop == 1) {
    c.errnum = amax_r;
    c.errden = c.ani * amax_x + c.bni;
  } else {
    c.errnum = sqrt(rr);
    c.errden = P.istop == 2 ? c.bn2 : c.r0n2;
  }
  const bool res = (c.errden == 0.0) ? (c.errnum <= P.eps) : (c.errnum <= P.eps * c.errden);
  return res || P.itmax <= c.itx;
}

template <class View, bool BICG>
__global__ void __launch_bounds__(PS_MAXT, 1) k_persist(View A, PsArgs P) {
  __shared__ GsShared gsh;
  extern __shared__ __align__(16) unsigned char dyn[];
  constexpr int NVEC = BICG ? 7 : 5;
  Blk B;
  const int k0 = (int)((long long)P.nslices * blockIdx.x / gridDim.x);
  const int k1 = (int)((long long)P.nslices * (blockIdx.x + 1) / gridDim.x);
  B.s0 = k0 * 32;
  B.ns = k1 - k0;
  const int nloc = P.max_slices * 32;
  double *vec = (double *)dyn;
  double *lx = vec, *lr = vec + nloc, *lp = vec + 2 * nloc, *lq = vec + 3 * nloc, *ld = vec + 4 * nloc;
  double *lv = BICG ? vec + 5 * nloc : nullptr, *lt = BICG ? vec + 6 * nloc : nullptr;
  B.sv = vec + (size_t)NVEC * nloc;
  B.sj = (int *)(B.sv + P.mat_entries);
  B.len = B.sj + P.mat_entries;
  B.off = B.len + nloc;
  __shared__ PsLoad load;
  if (threadIdx.x == 0) {
    gsh.bad = 0;
    load.cost = load.entries = 0;
    load.longest = 0;
  }
  stage(B, A, P.mat_entries);
  slice_loads(B, A, load);
  __syncthreads();
  GridSync G = {P.slots, &gsh, 0, (int)gridDim.x};
  const bool norms = P.istop == 1;  // the stop test needs max|r| and max|x|

  Conv c = {0, 0, 0, 0, 0, 0, 0};
  {
    dd_t s[2] = {{0.0, 0.0}, {0.0, 0.0}};
    double m[4] = {0.0, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0) {
      s[1].s = (double)load.entries;
      m[2] = (double)load.cost;
      m[3] = (double)load.longest;
    }
    each_row(B, A, [&](int l, int i) {
      const double bi = P.b[i];
      lx[l] = P.x[i];
      ld[l] = P.dinv ? P.dinv[i] : 1.0;  // 1*v is v to the bit
      dd_add_prod(s[0], bi, bi);
      if (norms) {
        m[0] = fmax(m[0], fabs(bi));
        double t = 0.0;
        const RowPtr r = row_ptr(A, B.s0 + l);
        for (int j = 0; j < r.n; j++) t = radd(t, fabs(r.v[(size_t)j * r.st]));
        m[1] = fmax(m[1], t);
      }
    });
    grid_reduce<2, 4, false>(G, s, m);
    c.bn2 = sqrt(dd_value(s[0]));
    c.bni = m[0];
    c.ani = m[1];
    if (!gsh.bad && 0.25 * m[2] > P.most + P.per_mean * dd_value(s[1]) / gridDim.x + P.per_longest * m[3]) {
      if (blockIdx.x == 0 && threadIdx.x == 0) P.out->declined = 1;
      return;  // nothing written: the drivers take the solve
    }
  }
  bool restarted = false;
  int r0set = 0;
  // restart loop (psb_dcg.F90:218-225, psb_dcgstab.f90:226-237)
  while (c.itx < P.itmax && !gsh.bad) {
    if (restarted) {  // x as it stands, for the product below
      each_row(B, A, [&](int l, int i) { P.x[i] = lx[l]; });
      grid_barrier(G);
    }
    restarted = true;
    double rho = 0.0, beta = 0.0, alpha = 0.0, omega = 0.0;
    {
      dd_t s[2] = {{0.0, 0.0}, {0.0, 0.0}};
      double m[2] = {0.0, 0.0};
      each_product(B, A, P.x, [&](int l, int i, double ax) {
        const double ri = radd(rmul(-1.0, ax), P.b[i]);
        lr[l] = ri;
        if (BICG) lq[l] = ri;
        else dd_add_prod(s[1], ri, rmul(ld[l], ri));
        dd_add_prod(s[0], ri, ri);
        if (BICG && norms) {
          m[0] = fmax(m[0], fabs(ri));
          m[1] = fmax(m[1], fabs(lx[l]));
        }
      });
      grid_reduce<2, 2, false>(G, s, m);
      if (gsh.bad) break;
      const double rr = dd_value(s[0]);
      if (BICG) {
        if (P.istop == 3 && !r0set) c.r0n2 = sqrt(rr);  // once, before the restart loop
        r0set = 1;
        if (conv_stop(P, c, rr, m[0], m[1])) break;
        c.itx += 1;
        rho = rr;
        if (rr == 0.0) continue;  // psb_dcgstab.f90:267
      } else {
        if (P.istop == 3) c.r0n2 = sqrt(rr);
        c.itx += 1;
        rho = dd_value(s[1]);
      }
    }
    bool first = true, stop = false;
    for (;;) {
      dd_t s1[1] = {{0.0, 0.0}}, s2[2] = {{0.0, 0.0}, {0.0, 0.0}};
      double m0[1], m[2] = {0.0, 0.0};
      if (!BICG) {
        // p = z (first) or p = z + beta p, z = M^-1 r
        each_row(B, A, [&](int l, int i) {
          const double z = rmul(ld[l], lr[l]);
          const double p = first ? z : radd(z, rmul(beta, lp[l]));
          lp[l] = p;
          P.g[i] = p;
        });
        grid_barrier(G);
        // q = A p ; sigma = (p,q)
        each_product(B, A, P.g, [&](int l, int, double t) {
          lq[l] = t;
          dd_add_prod(s1[0], lp[l], t);
        });
        grid_reduce<1, 0, false>(G, s1, m0);
        const double sigma = dd_value(s1[0]);
        if (gsh.bad || sigma == 0.0) break;  // psb_dcg.F90:265-270
        alpha = rho / sigma;
        // x = alpha p + x ; r = -alpha q + r ; (r,z) and the stop test
        const double malpha = -alpha;
        each_row(B, A, [&](int l, int) {
          const double x = radd(rmul(alpha, lp[l]), lx[l]);
          const double r = radd(rmul(malpha, lq[l]), lr[l]);
          lx[l] = x;
          lr[l] = r;
          dd_add_prod(s2[0], r, rmul(ld[l], r));
          dd_add_prod(s2[1], r, r);
          if (norms) {
            m[0] = fmax(m[0], fabs(r));
            m[1] = fmax(m[1], fabs(x));
          }
        });
      } else {
        // p = r (first) or p = r + beta (p - omega v) ; f = M^-1 p
        const double momega = -omega;
        each_row(B, A, [&](int l, int i) {
          double p = lr[l];
          if (!first) p = radd(p, rmul(beta, radd(rmul(momega, lv[l]), lp[l])));
          lp[l] = p;
          P.g[i] = rmul(ld[l], p);
        });
        grid_barrier(G);
        // v = A f ; sigma = (q,v)
        each_product(B, A, P.g, [&](int l, int, double t) {
          lv[l] = t;
          dd_add_prod(s1[0], lq[l], t);
        });
        grid_reduce<1, 0, false>(G, s1, m0);
        const double sigma = dd_value(s1[0]);
        if (gsh.bad || sigma == 0.0) break;  // psb_dcgstab.f90:298
        alpha = rho / sigma;
        // s = -alpha v + r (kept in r) ; z = M^-1 s.  Every block has formed
        // its product with f (the reduction above), so g is free.
        const double malpha = -alpha;
        each_row(B, A, [&](int l, int i) {
          const double s = radd(rmul(malpha, lv[l]), lr[l]);
          lr[l] = s;
          P.g[i] = rmul(ld[l], s);
        });
        grid_barrier(G);
        // t = A z ; sigma = (t,t) ; tau = (t,s)
        dd_t s3[2] = {{0.0, 0.0}, {0.0, 0.0}};
        each_product(B, A, P.g, [&](int l, int, double t) {
          lt[l] = t;
          dd_add_prod(s3[0], t, t);
          dd_add_prod(s3[1], t, lr[l]);
        });
        grid_reduce<2, 0, false>(G, s3, m0);
        const double tt = dd_value(s3[0]);
        if (gsh.bad || tt == 0.0) break;  // psb_dcgstab.f90:328
        omega = dd_value(s3[1]) / tt;
        if (omega == 0.0) break;  // psb_dcgstab.f90:346
        // x = alpha f + x ; x = omega z + x ; r = -omega t + s ; (q,r)
        const double mo = -omega;
        each_row(B, A, [&](int l, int) {
          double x = radd(rmul(alpha, rmul(ld[l], lp[l])), lx[l]);
          x = radd(rmul(omega, rmul(ld[l], lr[l])), x);
          const double r = radd(rmul(mo, lt[l]), lr[l]);
          lx[l] = x;
          lr[l] = r;
          dd_add_prod(s2[0], lq[l], r);
          dd_add_prod(s2[1], r, r);
          if (norms) {
            m[0] = fmax(m[0], fabs(r));
            m[1] = fmax(m[1], fabs(x));
          }
        });
      }
      if (norms) grid_reduce<2, 2, false>(G, s2, m);
      else grid_reduce<2, 0, false>(G, s2, m0);
      if (gsh.bad) break;
      if (conv_stop(P, c, dd_value(s2[1]), m[0], m[1])) {
        stop = true;
        break;
      }
      c.itx += 1;
      first = false;
      const double rho_old = rho;
      rho = dd_value(s2[0]);
      if (BICG) {
        if (rho == 0.0) break;  // psb_dcgstab.f90:267
        beta = (rho / rho_old) * (alpha / omega);
      } else {
        if (rho_old == 0.0) break;  // psb_dcg.F90:253-258
        beta = rho / rho_old;
      }
    }
    if (stop) break;
    // a breakdown: back to the restart test
  }
  each_row(B, A, [&](int l, int i) { P.x[i] = lx[l]; });
  if (threadIdx.x == 0) {
    if (gsh.bad) P.out->timeout = 1;
    if (blockIdx.x == 0) {
      P.out->itx = c.itx;
      P.out->errnum = c.errnum;
      P.out->errden = c.errden;
    }
  }
}

// ------------------------------------------------------------------ host
template <class View>
static int nslices_of(const View &A) { return (A.rows + 31) / 32; }

// Blocks: enough rows each that an exchange between fewer blocks is not the
// cheaper choice, at most one per SM.  (4 and 16 slices a block instead of 8:
// 10 and 1 % slower on 13,824 rows, 2 and 7 % on 1,728.)
#define PS_MIN_SLICES 8
static int ps_blocks(int nslices) {
  const int sms = psbx_ctx().sms;
  const int g = (nslices + PS_MIN_SLICES - 1) / PS_MIN_SLICES;
  const int most = sms < GS_MAXB ? sms : GS_MAXB;
  return g < 1 ? 1 : (g > most ? most : g);
}

static size_t ps_fixed_bytes(int max_slices, bool bicg) {
  return (size_t)max_slices * (32 * (sizeof(double) * (bicg ? 7 : 5) + sizeof(int)) + sizeof(int));
}

template <class View>
static bool fits(const View &A, bool bicg) {
  if (A.rows <= 0) return false;
  const int ns = nslices_of(A), g = ps_blocks(ns);
  return ps_fixed_bytes((ns + g - 1) / g, bicg) <= PS_SMEM;
}

template <class View, bool BICG>
static int run(const View &A, const double *dinv, const double *b, double *x, psbx_SolverOptions *opt, int *ran) {
  PsbxCtx &c = psbx_ctx();
  cudaStream_t st = c.stream;
  *ran = 0;
  if (opt->itmax > PS_MAXIT) return SPGPU_SUCCESS;
  PsArgs P;
  P.nslices = nslices_of(A);
  const int g = ps_blocks(P.nslices);
  P.max_slices = (P.nslices + g - 1) / g;
  const size_t fixed = ps_fixed_bytes(P.max_slices, BICG);
  // room for the matrix entries of an average block and a little more, as far
  // as PS_SMEM goes; a block that holds more reads the rest through L2
  const size_t entry = sizeof(double) + sizeof(int);
  size_t room = (size_t)((double)A.entries / P.nslices * P.max_slices * 1.1) + 1024;
  if (room * entry > PS_SMEM - fixed) room = (PS_SMEM - fixed) / entry;
  P.mat_entries = (int)(room / 2 * 2);  // sj stays 8-byte aligned
  const size_t smem = fixed + P.mat_entries * entry;
  int threads = P.max_slices * 32;
  threads = threads < 256 ? 256 : (threads > PS_MAXT ? PS_MAXT : threads);
  cudaError_t e = cudaFuncSetAttribute(k_persist<View, BICG>, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_SMEM);
  if (e != cudaSuccess) return psbx_cuda_status(e, "k_persist (attributes)");
  // workspace (256-byte aligned): the slots of the reductions, the gathered vector
  char *ws = nullptr;
  PSBX_CK(psbx_malloc_async(&ws, GS_BYTES(g) + sizeof(double) * (size_t)A.rows, st));
  P.slots = (ulonglong2 *)ws;
  P.g = (double *)(ws + GS_BYTES(g));
  P.dinv = dinv;
  P.b = b;
  P.x = x;
  static_assert(sizeof(PsOut) <= 64 * sizeof(double), "the result fits the pinned staging area");
  P.out = (PsOut *)c.h_res;
  P.itmax = opt->itmax;
  P.istop = opt->istop;
  P.eps = opt->eps;
  ps_limit(P, smem);
  memset(P.out, 0, sizeof(PsOut));
  e = cudaMemsetAsync(ws, 0, GS_BYTES(g), st);
  View Av = A;
  void *args[] = {&Av, &P};
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel((const void *)k_persist<View, BICG>, dim3(g), dim3(threads), args, smem, st);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs are ours than the device has: the kernel-per-step path
    cudaGetLastError();
    cudaFreeAsync(ws, st);
    return SPGPU_SUCCESS;
  }
  psbx_count_launch();
  cudaFreeAsync(ws, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return psbx_cuda_status(e, "k_persist");
  if (P.out->declined && !P.out->timeout) return SPGPU_SUCCESS;
  *ran = 1;
  if (P.out->timeout) {
    psbx_set_error("psbx_dkrylov: a wait between the blocks of the solve ran past its bound");
    return PSBX_TIMEOUT;
  }
  opt->iter = P.out->itx;
  opt->err = P.out->errden == 0.0 ? P.out->errnum : P.out->errnum / P.out->errden;
  return SPGPU_SUCCESS;
}

#define PSBX_PERSIST(View)                                                                                     \
  bool persist_fits(const View &A, bool bicg) { return fits(A, bicg); }                                        \
  int persist_solve(const View &A, bool bicg, const double *dinv, const double *b, double *x,                  \
                    psbx_SolverOptions *opt, int *ran) {                                                       \
    return bicg ? run<View, true>(A, dinv, b, x, opt, ran) : run<View, false>(A, dinv, b, x, opt, ran);        \
  }
PSBX_PERSIST(HllView)
PSBX_PERSIST(EllView)
PSBX_PERSIST(CsrView)
#undef PSBX_PERSIST
