// cg.cuh -- the conjugate gradients of divergence cleaning (matlab/+induction_eq/clean_div.m
// :36-79) in three launches: k_cg_begin (r = div B on the interior, the zeroed vectors,
// partials of <r, r>), k_cg_loop (every iteration, one cooperative launch) and k_cg_project
// (B += grad phi).
//
// Measured on B200 (wide stencil, 4th order, 50 iterations): 1.84 ms a cleaning at 128^3 against
// 3.78 for one kernel per pass inside a graph loop node, 15 against 40 us an iteration at 96 x
// 81 x 70.  At 128^3 an iteration is pass A 17 us, pass B 8, two barriers 5.4 and the sums 1.6
// (80 B a node, mostly from L2); pass A is bound by the latency of its one barrier and one
// prefetched plane per step at 16 warps an SM, not by a pipe (shared memory 40 %, FP64 25 %).
//
// k_cg_loop.  An iteration is two passes over the grid that each end in a dot product every
// block needs, so its blocks meet at two grid barriers per iteration instead of at two
// kernel boundaries and a graph loop node (about 10 us of launches per iteration, more than
// the arithmetic up to about 64^3):
//   pass A  direction u = beta u + r (formed where it is loaded, written to the other buffer
//           of a pair), lap = (-Laplace) u, <u, lap>;
//   pass B  phi += alpha u, r -= alpha lap, <r, r>.
// Every block adds the block partials in the same order, so alpha, beta and the decision to
// go on are the same value everywhere without a broadcast.
//
// Pass A marches a 32 x 16 (W > 9: 32 x 8) tile of x-y columns through a chunk of z planes: the column's
// values sit in a register queue, plane z with its halos in shared memory (double buffered,
// one barrier per plane), and the loads of plane z + 1 are in flight while plane z is summed.
// Boundary rows take no second path: a thread's x row is fixed for its whole column and kept
// in registers, the y and z rows are warp-uniform (interior: kernel parameters, boundary:
// a shared-memory table).  The three axes are summed apart, which breaks the dependent chain
// of 3 W additions into three.
#pragma once
#include "misc_kernels.cuh"
#include "stage_kernel.cuh"

namespace ieq {

// the grid barrier of one loop launch: arrivals since the state was reset (a multiple of the
// grid between launches), the arrivals up to which blocks may go on (a line of its own: the
// waiting blocks' polls would slow the arrivals down), and whether a wait gave up
struct CgSync {
  unsigned arrived;
  unsigned pad0[31];
  unsigned released;
  int timeout;
  unsigned pad1[30];
};

struct CgDevice {
  CgState state;
  CgSync sync;
};

constexpr long long kCgSpinLimit = 4000000;   // polls of about 0.6 us: a few seconds
constexpr int kCgThreads = kCgTX * kCgTY;

template <int W>
struct CgLoopArgs {
  int nx, ny, nz, off, gx, gy, gz, nb, periodic;
  int inner_y, inner_z;  // nb, or -1 where an axis is too short to have an interior row
  double Li[3][W];       // interior row of each axis, divided by DX^2, DY^2, DZ^2
  const double *Ls;      // [3][2nb+1][W], divided likewise
  double *phi, *r, *u0, *u1, *lap;
  double *partials_a, *partials_b;   // one entry per block each
  const double *rr0;     // partials of <r, r> before the first iteration (k_cg_begin's)
  int n_rr0;
  CgState *cs;
  CgSync *sync;
  double *history;
  double tol;
  int max_it;
  int first;             // 1: the loop starts here (rr from rr0), 0: it goes on from *cs
  int launch_it;         // iterations this launch may do
  unsigned extra;        // arrivals its barriers wait for beyond the grid (0; a test sets 1 to
  long long spin_limit;  // make every wait run out) and the polls of a wait before it gives up
  int tiles_x, tiles_y, chunks, tz;
};

// every block of the (cooperative) launch arrives; false if the wait gave up.  The
// arrival releases the block's earlier writes, the poll acquires those of every block.
__device__ __forceinline__ bool cg_barrier(CgSync *s, unsigned &target, unsigned extra, long long spin_limit) {
  __shared__ int ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    unsigned n;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(n) : "l"(&s->arrived) : "memory");
    if (n + 1u == target + extra) {
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&s->released), "r"(target) : "memory");
    } else {
      for (long long spins = 0;; ++spins) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&s->released) : "memory");
        if (n == target) break;
        if (spins > 256) {
          if (*(volatile int *)&s->timeout || spins > spin_limit) {
            *(volatile int *)&s->timeout = 1;
            ok = 0;
            break;
          }
          __nanosleep(64);
        }
      }
    }
  }
  __syncthreads();
  return ok != 0;
}

// the block's sum of v in a fixed order, to partials[blockIdx.x]
__device__ __forceinline__ void cg_block_partial(double v, double *partials) {
  __shared__ double sm[kCgThreads / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kCgThreads / 32; ++w) s += sm[w];
    __stcg(partials + blockIdx.x, s);
  }
}
// the sum of np partials that other blocks wrote, the same value in every thread of every block
__device__ __forceinline__ double cg_total(const double *partials, int np) {
  __shared__ double sm[kCgThreads / 32];
  double v = 0.0;
  for (int i = threadIdx.x; i < np; i += kCgThreads) v += __ldcg(partials + i);
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < kCgThreads / 32; ++w) s += sm[w];
  return s;
}

// y rows per thread of pass A: two share the loads of their y columns and the halo of a tile
// twice as deep (W = 9 at 128^3: 17 us against 23 with one row and three blocks per SM), where
// both queues fit the registers
template <int W>
__host__ __device__ constexpr int cg_rows_per_thread() {
  return W <= 9 ? 2 : 1;
}
template <int W>
__host__ __device__ constexpr int cg_ty() {
  return kCgTY * cg_rows_per_thread<W>();
}
// resident blocks per SM the register allocation is made for: the queues and the x row take
// 2 W (rows + 1) registers of a thread
template <int W>
__host__ __device__ constexpr int cg_min_blocks() {
  return W <= 15 ? 2 : 1;
}

// rows of the widest operator with a Laplacian of width W, for the shared-memory tables
template <int W>
__host__ __device__ constexpr int cg_max_rows() {
  return W <= 3 ? 5 : W <= 5 ? 9 : W <= 7 ? 9 : W <= 9 ? 13 : W <= 11 ? 13 : W <= 13 ? 17 : W <= 15 ? 19 : W <= 17 ? 19 : 23;
}

// A stencil point outside a box reads the node itself.  The coefficients there are zero unless
// the axis is shorter than its two boundary closures: they then count for the node's own.
template <int W>
__device__ __forceinline__ void cg_fold_outside(double *row, int i, int n, int periodic) {
  constexpr int C0 = (W - 1) / 2;
  if (periodic) return;
#pragma unroll
  for (int c = 0; c < W; ++c) {
    if (i + c - C0 < 0 || i + c - C0 >= n) {
      if (c != C0) {
        row[C0] += row[c];
        row[c] = 0.0;
      }
    }
  }
}

// where a block's threads are in one item of pass A (a tile of columns and a chunk of planes):
// the positions in a plane of the thread's own columns and of its halo points (-1 outside a
// box, wrapped on a periodic grid), their places in the plane buffer, and the thread's rows
template <int W>
struct CgItem {
  static constexpr int C0 = (W - 1) / 2, RPT = cg_rows_per_thread<W>(), TY = cg_ty<W>();
  static constexpr int NH = 2 * C0 * (kCgTX + TY);                 // halo points of a plane
  static constexpr int NS = (NH + kCgThreads - 1) / kCgThreads;    // of a thread
  int zb, ze, own[RPT], ry[RPT], hoff[NS], hpos[NS];
  bool mine[RPT];
  double lx[W];

  __device__ __forceinline__ void set(const CgLoopArgs<W> &a, int item) {
    const int nx = a.nx, ny = a.ny;
    const int tx = threadIdx.x % kCgTX, ty = RPT * (threadIdx.x / kCgTX);
    const int bx = item % a.tiles_x, by = (item / a.tiles_x) % a.tiles_y, bz = item / (a.tiles_x * a.tiles_y);
    const int x0 = a.off + bx * kCgTX, y0 = a.off + by * TY, ix = x0 + tx;
    zb = a.off + bz * a.tz;
    ze = min(zb + a.tz, a.off + a.gz);
    auto at = [&](int x, int y) -> int {
      if (a.periodic) {
        x += x < 0 ? nx : 0; x -= x >= nx ? nx : 0;
        y += y < 0 ? ny : 0; y -= y >= ny ? ny : 0;
      }
      return x >= 0 && x < nx && y >= 0 && y < ny ? x + nx * y : -1;
    };
#pragma unroll
    for (int e = 0; e < RPT; ++e) {
      const int iy = y0 + ty + e;
      own[e] = at(ix, iy);
      mine[e] = ix < a.off + a.gx && iy < a.off + a.gy;
      ry[e] = a.periodic ? a.nb : sbp_row(min(iy, ny - 1), ny, a.nb);
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const int h = threadIdx.x + s * kCgThreads;
      hoff[s] = -1;
      hpos[s] = -1;
      if (h < NH) {
        int px, py;
        if (h < 2 * C0 * kCgTX) {   // C0 rows below and above the tile
          py = h / kCgTX;
          py += py >= C0 ? TY : 0;
          px = C0 + h % kCgTX;
        } else {                    // C0 columns on each side of its rows
          const int g = h - 2 * C0 * kCgTX;
          px = g % (2 * C0);
          px += px >= C0 ? kCgTX : 0;
          py = C0 + g / (2 * C0);
        }
        hoff[s] = at(x0 - C0 + px, y0 - C0 + py);
        hpos[s] = py * (kCgTX + 2 * C0) + px;
      }
    }
    const int rx = a.periodic ? a.nb : sbp_row(min(ix, nx - 1), nx, a.nb);
#pragma unroll
    for (int c = 0; c < W; ++c) lx[c] = __ldg(a.Ls + (long long)rx * W + c);
    cg_fold_outside<W>(lx, ix, nx, a.periodic);
  }
};

// pass A over the block's items; a block with a single one keeps its CgItem from iteration to
// iteration (`set` is false then)
template <int W>
__device__ __forceinline__ double cg_pass_a(const CgLoopArgs<W> &a, CgItem<W> &t, bool set, const double *uo, double *un, double beta,
                            double (&pl)[2][cg_ty<W>() + W - 1][kCgTX + W - 1],
                            const double (&tab)[2][cg_max_rows<W>()][W]) {
  constexpr int C0 = (W - 1) / 2;
  constexpr int RPT = cg_rows_per_thread<W>(), TY = cg_ty<W>(), NS = CgItem<W>::NS;
  const int nz = a.nz;
  const long long plane = (long long)a.nx * a.ny;
  const int tx = threadIdx.x % kCgTX, ty = RPT * (threadIdx.x / kCgTX);
  auto z_of = [&](int z) -> int {
    if (a.periodic) {
      z += z < 0 ? nz : 0; z -= z >= nz ? nz : 0;
    }
    return z >= 0 && z < nz ? z : -1;
  };
  double prod = 0.0;
  const int items = a.tiles_x * a.tiles_y * a.chunks;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    if (set) t.set(a, item);
    const int zb = t.zb, ze = t.ze;
    double q[RPT][W];
    // the direction at a position of plane z (0 outside the grid)
    auto dir = [&](int o, int zz) -> double {
      if (o < 0 || zz < 0) return 0.0;
      const long long j = o + plane * zz;
      return __fma_rn(beta, __ldcg(uo + j), __ldcg(a.r + j));
    };
    double nq[RPT], hv[NS];
#pragma unroll
    for (int k = 0; k < W - 1; ++k)
#pragma unroll
      for (int e = 0; e < RPT; ++e) q[e][k + 1] = dir(t.own[e], z_of(zb - C0 + k));
#pragma unroll
    for (int e = 0; e < RPT; ++e) nq[e] = dir(t.own[e], z_of(zb + C0));
#pragma unroll
    for (int s = 0; s < NS; ++s) hv[s] = dir(t.hoff[s], z_of(zb));
    for (int z = zb; z < ze; ++z) {
      double(&p)[TY + W - 1][kCgTX + W - 1] = pl[z & 1];
#pragma unroll
      for (int e = 0; e < RPT; ++e) {
#pragma unroll
        for (int k = 0; k < W - 1; ++k) q[e][k] = q[e][k + 1];
        q[e][W - 1] = nq[e];
        p[ty + e + C0][tx + C0] = q[e][C0];
      }
#pragma unroll
      for (int s = 0; s < NS; ++s)
        if (t.hpos[s] >= 0) (&p[0][0])[t.hpos[s]] = hv[s];
      // the values of the next plane, in flight while this one is summed
      const int zn = z + 1 < ze ? z_of(z + 1) : -1, zq = z + 1 < ze ? z_of(z + 1 + C0) : -1;
      double nu[RPT], nr[RPT], hu[NS], hr[NS];
#pragma unroll
      for (int e = 0; e < RPT; ++e) {
        nu[e] = nr[e] = 0.0;
        if (t.own[e] >= 0 && zq >= 0) {
          nu[e] = __ldcg(uo + t.own[e] + plane * zq);
          nr[e] = __ldcg(a.r + t.own[e] + plane * zq);
        }
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        hu[s] = hr[s] = 0.0;
        if (t.hoff[s] >= 0 && zn >= 0) {
          hu[s] = __ldcg(uo + t.hoff[s] + plane * zn);
          hr[s] = __ldcg(a.r + t.hoff[s] + plane * zn);
        }
      }
      __syncthreads();
      if (t.mine[0]) {   // (rows are in order: no later row is inside if the first is not)
        const int rz = a.periodic ? a.nb : sbp_row(z, nz, a.nb);
        double vx[RPT], vy[RPT], vz[RPT];
#pragma unroll
        for (int e = 0; e < RPT; ++e) {
          vx[e] = vy[e] = vz[e] = 0.0;
#pragma unroll
          for (int c = 0; c < W; ++c) vx[e] += (c == C0 ? q[e][C0] : p[ty + e + C0][tx + c]) * t.lx[c];
        }
        // the column of y values serves every row of the thread
        bool inner = true;
#pragma unroll
        for (int e = 0; e < RPT; ++e) inner = inner && t.ry[e] == a.inner_y;
        auto y_sums = [&](auto coef) {
#pragma unroll
          for (int c = 0; c < W + RPT - 1; ++c) {
            const bool center = c >= C0 && c < C0 + RPT;
            const double v = center ? q[center ? c - C0 : 0][C0] : p[ty + c][tx + C0];
#pragma unroll
            for (int e = 0; e < RPT; ++e)
              if (c - e >= 0 && c - e < W) vy[e] += v * coef(e, c - e);
          }
        };
        if (inner) y_sums([&](int, int c) { return a.Li[1][c]; });
        else y_sums([&](int e, int c) { return tab[0][t.ry[e]][c]; });
        if (rz == a.inner_z) {
#pragma unroll
          for (int c = 0; c < W; ++c)
#pragma unroll
            for (int e = 0; e < RPT; ++e) vz[e] += q[e][c] * a.Li[2][c];
        } else {
#pragma unroll
          for (int c = 0; c < W; ++c) {
            const double cf = tab[1][rz][c];
#pragma unroll
            for (int e = 0; e < RPT; ++e) vz[e] += q[e][c] * cf;
          }
        }
#pragma unroll
        for (int e = 0; e < RPT; ++e) {
          if (!t.mine[e]) continue;
          const double val = (vx[e] + vy[e]) + vz[e];
          const long long j = t.own[e] + plane * z;
          __stcg(un + j, q[e][C0]);
          __stcg(a.lap + j, val);
          prod += q[e][C0] * val;
        }
      }
#pragma unroll
      for (int e = 0; e < RPT; ++e) nq[e] = __fma_rn(beta, nu[e], nr[e]);
#pragma unroll
      for (int s = 0; s < NS; ++s) hv[s] = __fma_rn(beta, hu[s], hr[s]);
    }
    __syncthreads();   // the next item fills the plane buffers again
  }
  return prod;
}

// pass B over the interior rows, one warp a row, four values of each vector in flight
template <int W>
__device__ double cg_pass_b(const CgLoopArgs<W> &a, const double *u, double alpha) {
  const int warps = gridDim.x * (kCgThreads / 32);
  const int lane = threadIdx.x & 31;
  const int rows = a.gy * a.gz;
  double rr = 0.0;
  for (int row = blockIdx.x * (kCgThreads / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
    const long long base = a.off + (long long)a.nx * (a.off + row % a.gy + (long long)a.ny * (a.off + row / a.gy));
    for (int x = lane; x < a.gx; x += 128) {
      double p[4], d[4], r[4], l[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const long long j = base + x + 32 * k;
        const bool in = x + 32 * k < a.gx;
        p[k] = in ? __ldcg(a.phi + j) : 0.0;
        d[k] = in ? __ldcg(u + j) : 0.0;
        r[k] = in ? __ldcg(a.r + j) : 0.0;
        l[k] = in ? __ldcg(a.lap + j) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (x + 32 * k < a.gx) {
          const long long j = base + x + 32 * k;
          __stcg(a.phi + j, p[k] + alpha * d[k]);
          const double rn = r[k] + (-alpha) * l[k];
          __stcg(a.r + j, rn);
          rr += rn * rn;
        }
      }
    }
  }
  return rr;
}

template <int W>
__global__ void __launch_bounds__(kCgThreads, cg_min_blocks<W>()) k_cg_loop(const __grid_constant__ CgLoopArgs<W> a) {
  __shared__ double pl[2][cg_ty<W>() + W - 1][kCgTX + W - 1];
  __shared__ double tab[2][cg_max_rows<W>()][W];   // the y and z rows
  const int rows = 2 * a.nb + 1;
  for (int i = threadIdx.x; i < 2 * rows * W; i += kCgThreads) {
    const int ax = i / (rows * W), k = i % (rows * W);
    tab[ax][k / W][k % W] = __ldg(a.Ls + (long long)(ax + 1) * rows * W + k);
  }
  __syncthreads();
  if (a.inner_y < 0)   // a short axis has every row once
    for (int i = threadIdx.x; i < a.ny; i += kCgThreads) cg_fold_outside<W>(tab[0][sbp_row(i, a.ny, a.nb)], i, a.ny, 0);
  if (a.inner_z < 0)
    for (int i = threadIdx.x; i < a.nz; i += kCgThreads) cg_fold_outside<W>(tab[1][sbp_row(i, a.nz, a.nb)], i, a.nz, 0);
  __syncthreads();
  double rr, old;
  int it;
  if (a.first) {
    rr = cg_total(a.rr0, a.n_rr0);
    old = 1.0;
    it = 0;
  } else {
    rr = a.cs->rr;
    old = a.cs->old;
    it = a.cs->it;
  }
  const bool writer = blockIdx.x == 0 && threadIdx.x == 0;
  if (a.first && writer) a.history[0] = rr;
  // no block may arrive before every block has read *cs and the barrier's state
  unsigned target = 0;   // (arrivals are a multiple of the grid when the launch starts)
  {
    const unsigned seen = *(volatile unsigned *)&a.sync->arrived;
    target = seen - seen % gridDim.x;
  }
  CgItem<W> item;
  const bool many = a.tiles_x * a.tiles_y * a.chunks > (int)gridDim.x;
  if (!many) item.set(a, blockIdx.x);
  bool ok = cg_barrier(a.sync, target, a.extra, a.spin_limit);
  for (int k = 0; ok && k < a.launch_it && rr > a.tol && it < a.max_it; ++k) {
    const double *uo = (it & 1) ? a.u1 : a.u0;
    double *un = (it & 1) ? a.u0 : a.u1;
    cg_block_partial(cg_pass_a<W>(a, item, many, uo, un, rr / old, pl, tab), a.partials_a);
    if (!(ok = cg_barrier(a.sync, target, a.extra, a.spin_limit))) break;
    const double alpha = rr / cg_total(a.partials_a, gridDim.x);
    cg_block_partial(cg_pass_b<W>(a, un, alpha), a.partials_b);
    if (!(ok = cg_barrier(a.sync, target, a.extra, a.spin_limit))) break;
    old = rr;
    rr = cg_total(a.partials_b, gridDim.x);
    ++it;
    if (writer) a.history[it] = rr;
  }
  if (writer) {
    a.cs->rr = rr;
    a.cs->old = old;
    a.cs->tol = a.tol;
    a.cs->it = it;
    a.cs->max_it = a.max_it;
    a.cs->done = !(rr > a.tol && it < a.max_it);
  }
}

// ---- before and after the loop: one node per thread.  A node whose row of an axis is the
// interior one sums its 2 RI points with the coefficients from the parameters; boundary rows
// load every coefficient and then every value before the first sum (a zero coefficient loads
// nothing, as in diff_rt).  Rows are multiplied by 1 / DX.
// The field is the caller's records or, in the time loop, the fused state (row pitch px).
template <typename R, typename F>
struct CgEndArgs {
  int nx, ny, nz, px, off, gx, gy, gz, periodic;
  const double *D;     // derivative (or adjoint) rows [2nb+1][SW]
  double Dint[7];      // the interior row, offsets -RI .. RI
  double inv_d[3];
  double sign;
  F b;
  double *phi, *r, *u0, *u1;
  double *partials;    // of <r, r>, one per block
  CgSync *sync;
};

// sum_c D[row][c] f(i + c - C0) / DX of one axis; load(o) is the value o nodes along the axis
template <int OP, typename R, typename F, typename Load>
__device__ __forceinline__ double cg_axis(const CgEndArgs<R, F> &a, int ax, int i, int n, const Load &load) {
  constexpr int NB = Op<OP>::NB, SW = Op<OP>::SW, C0 = (SW - 1) / 2, RI = Op<OP>::RI;
  double v = 0.0;
  if (i >= (NB > RI ? NB : RI) && i < n - (NB > RI ? NB : RI)) {
    double f[2 * RI];
#pragma unroll
    for (int o = 0; o < RI; ++o) {
      f[o] = load(o - RI);
      f[RI + o] = load(o + 1);
    }
#pragma unroll
    for (int o = 0; o < RI; ++o) v += a.Dint[o] * f[o];
#pragma unroll
    for (int o = 0; o < RI; ++o) v += a.Dint[RI + 1 + o] * f[RI + o];
  } else {
    const int row = a.periodic ? NB : sbp_row(i, n, NB);
    double cf[SW], f[SW];
#pragma unroll
    for (int c = 0; c < SW; ++c) cf[c] = __ldg(a.D + row * SW + c);
#pragma unroll
    for (int c = 0; c < SW; ++c) f[c] = cf[c] != 0.0 ? load(nbr_rt<double>(i, c - C0, n, a.periodic) - i) : 0.0;
#pragma unroll
    for (int c = 0; c < SW; ++c)
      if (cf[c] != 0.0) v += cf[c] * f[c];
  }
  return v * a.inv_d[ax];
}

// r = div B on the interior; phi, r outside it and both directions zero; partials of <r, r>
template <typename R, typename F, int OP>
__global__ void __launch_bounds__(kCgThreads) k_cg_begin(const __grid_constant__ CgEndArgs<R, F> a) {
  if (blockIdx.x == 0 && threadIdx.x == 0) a.sync->arrived = a.sync->released = 0u;
  const int lane = threadIdx.x & 31, rows = a.ny * a.nz;
  double rr = 0.0;
  for (int row = blockIdx.x * (kCgThreads / 32) + (threadIdx.x >> 5); row < rows;
       row += gridDim.x * (kCgThreads / 32)) {
    const int iy = row % a.ny, iz = row / a.ny;
    const bool in_yz = iy >= a.off && iy < a.off + a.gy && iz >= a.off && iz < a.off + a.gz;
    for (int ix = lane; ix < a.nx; ix += 32) {
      const long long j = (long long)a.nx * row + ix;
      double v = 0.0;
      if (in_yz && ix >= a.off && ix < a.off + a.gx) {
        const Idx<F> jb = ix + (Idx<F>)a.px * row, sy = a.px, sz = (Idx<F>)a.px * a.ny;
        const double vx = cg_axis<OP>(a, 0, ix, a.nx, [&](int o) { return (double)ldc<R, F>(a.b, jb + o, 0); });
        const double vy = cg_axis<OP>(a, 1, iy, a.ny, [&](int o) { return (double)ldc<R, F>(a.b, jb + o * sy, 1); });
        const double vz = cg_axis<OP>(a, 2, iz, a.nz, [&](int o) { return (double)ldc<R, F>(a.b, jb + o * sz, 2); });
        v = (vx + vy) + vz;
        rr += v * v;
      }
      a.r[j] = v;
      a.phi[j] = 0.0;
      a.u0[j] = 0.0;
      a.u1[j] = 0.0;
    }
  }
  cg_block_partial(rr, a.partials);
}

// B += grad(phi), or B -= grad_adj(phi) (sign = -1, D the adjoint rows), the xyz components.  B
// stays as it is if a barrier of the loop gave up: phi is then a part of an iteration
template <typename R>
__device__ __forceinline__ void cg_store_xyz(const AoS<R> &f, long long j, V3<R> v) {   // .w untouched, as the
  R *q = reinterpret_cast<R *>(f.p + j);                                                // reference's .xyz store
  if constexpr (sizeof(R) == 8) *reinterpret_cast<double2 *>(q) = make_double2(v.x, v.y);
  else *reinterpret_cast<float2 *>(q) = make_float2(v.x, v.y);
  q[2] = v.z;
}
template <typename R>
__device__ __forceinline__ void cg_store_xyz(const SoA<R> &f, int j, V3<R> v) {
  stf(f, j, v);
}
template <typename R, typename F, int OP>
__global__ void __launch_bounds__(kCgThreads) k_cg_project(const __grid_constant__ CgEndArgs<R, F> a) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x;
  const int iy = blockIdx.y * blockDim.y + threadIdx.y;
  const int iz = blockIdx.z * blockDim.z + threadIdx.z;
  if (ix >= a.nx || iy >= a.ny || iz >= a.nz || a.sync->timeout) return;
  const long long plane = (long long)a.nx * a.ny, j = ix + (long long)a.nx * iy + plane * iz;
  const double *p = a.phi + j;
  const double gx = cg_axis<OP>(a, 0, ix, a.nx, [&](int o) { return __ldg(p + o); });
  const double gy = cg_axis<OP>(a, 1, iy, a.ny, [&](int o) { return __ldg(p + (long long)o * a.nx); });
  const double gz = cg_axis<OP>(a, 2, iz, a.nz, [&](int o) { return __ldg(p + o * plane); });
  const Idx<F> jb = ix + (Idx<F>)a.px * (iy + (Idx<F>)a.ny * iz);
  const V3<R> B = ldf_plain(a.b, jb);
  cg_store_xyz(a.b, jb, V3<R>{(R)((double)B.x + a.sign * gx), (R)((double)B.y + a.sign * gy),
                              (R)((double)B.z + a.sign * gz)});
}

}  // namespace ieq
