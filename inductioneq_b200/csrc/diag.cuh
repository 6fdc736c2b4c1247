// diag.cuh -- the per-step diagnostics of the time loop in one pass.
//
// compute_numerical_solution.m:153-173 (save_integrals_over_time) records before every
// step the energy norm2(b), the divergence norm sqrt(norm2_S(calc_div(b))) and the error
// sqrt(norm2_diff(b, analytical_b(time))) -- four kernels, three reductions and a host
// sum each.  k_diag_partials evaluates the three per-node terms in one pass over b (the
// divergence with the SBP rows of calc_div, the exact field at time[0]) and writes one
// partial per block and quantity; k_diag_final adds them in a fixed order and appends
// the three totals to a device series.  The per-node terms and the summation order are
// those of the stand-alone reductions (k_reduce_partials / k_reduce_final), so each entry
// equals what ieq_norm2_value, ieq_norm2_S_value of calc_div and ieq_norm2_diff_value of
// analytical_b return for the same field (up to the compiler's FMA contraction).
#pragma once
#include "misc_kernels.cuh"
#include "stage_kernel.cuh"

namespace ieq {

template <typename R, typename F>
struct DiagArgs {
  Mesh m;
  F b;
  long long n;
  const R *wx, *wy, *wz;   // per-axis mass weights (norm2 of kernel_operator.cl)
  const Tables<R> *tab;    // derivative rows (calc_div)
  int periodic;
  R dS[3];                 // (REAL)DX ...
  int tc;                  // testcase of analytical_b
  const R *time;           // analytical_b at time[0] ...
  R t;                     // ... or, without one, at t
};

// d/d(axis) of that axis' component (calc_div, kernel_operator.cl:145): the row's non-zero
// entries, all loads free to issue before the first sum
template <typename R, typename F, int OP>
__device__ __forceinline__ R diag_axis(const DiagArgs<R, F> &a, int ax, int i, int n, Idx<F> ib, Idx<F> st) {
  const int row = a.periodic ? Op<OP>::NB : sbp_row(i, n, Op<OP>::NB);
  R v = 0;
#pragma unroll
  for (int t = 0; t < Op<OP>::ND; ++t) {
    const R c = __ldg(&a.tab->nd[row][t]);
    int o = __ldg(&a.tab->nd_off[row][t]);
    if (a.periodic) o = nbr<true>(i, o, n) - i;
    R f = 0;
    if (c != (R)0) f = ldc<R, F>(a.b, ib + o * st, ax);
    v += c * f;
  }
  return v / a.dS[ax];
}

// the terms of node (ix, iy, iz): energy, divergence, error (each as its reduction kernel forms
// it); A: analytical_b there, div: div B, fac: the mass weight
template <typename R, typename F, int OP>
__device__ __forceinline__ void diag_node(const DiagArgs<R, F> &a, int ix, int iy, int iz, double &e, double &dv,
                                          double &er, V3<R> &A, R &div, R &fac) {
  const Idx<F> ib = node_at<F>(a.m, ix, iy, iz);
  fac = (a.wx[ix] * a.wy[iy]) * a.wz[iz];
  const V3<R> B = ldf(a.b, ib);
  e += (double)(fac * ((B.x * B.x + B.y * B.y) + B.z * B.z));
  const R dx = diag_axis<R, F, OP>(a, 0, ix, a.m.nx, ib, 1), dy = diag_axis<R, F, OP>(a, 1, iy, a.m.ny, ib, a.m.px),
          dz = diag_axis<R, F, OP>(a, 2, iz, a.m.nz, ib, (Idx<F>)a.m.px * a.m.ny);
  div = (dx + dy) + dz;
  dv += (double)((fac * div) * div);
  A = b_analytical<R>(a.tc, a.m, ix, iy, iz, a.time ? a.time[0] : a.t);
  const V3<R> w = {B.x - A.x, B.y - A.y, B.z - A.z};
  er += (double)(fac * ((w.x * w.x + w.y * w.y) + w.z * w.z));
}

// partials[k * gridDim.x + block], k = 0 energy, 1 divergence, 2 error; with `results` also 3 the
// norm of analytical_b, and analytical_b and div B of every node to va and sdiv
template <typename R, typename F, int OP>
__global__ void __launch_bounds__(256) k_diag_partials(const __grid_constant__ DiagArgs<R, F> a, double *partials,
                                                       int results, R4<R> *va, R *sdiv) {
  __shared__ double sm[4][8];
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.n; i += stride) {
    V3<R> A;
    R div, fac;
    int ix, iy, iz;
    node_position(i, a.m.nx, a.m.ny, ix, iy, iz);
    diag_node<R, F, OP>(a, ix, iy, iz, acc[0], acc[1], acc[2], A, div, fac);
    if (results) {
      acc[3] += (double)(fac * ((A.x * A.x + A.y * A.y) + A.z * A.z));
      st3(va + i, A);
      sdiv[i] = div;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double v = warp_sum(acc[k]);
    if ((threadIdx.x & 31) == 0) sm[k][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      double v = threadIdx.x < (blockDim.x >> 5) ? sm[k][threadIdx.x] : 0.0;
      v = warp_sum(v);
      if (threadIdx.x == 0 && (k < 3 || results)) partials[k * gridDim.x + blockIdx.x] = v;
    }
  }
}

// the totals of `np` partials each, in the order of k_reduce_final: three appended to
// series[3 * pos .. 3 * pos + 2] (pos = *count, then incremented; nothing is written past
// `capacity` entries), or, without a count, `quantities` totals to series[0 ..]
static __global__ void __launch_bounds__(256) k_diag_final(const double *partials, int np, int quantities,
                                                           double *series, int *count, int capacity) {
  __shared__ double sm[8];
  const int pos = count ? *count : 0;
  for (int k = 0; k < quantities; ++k) {
    double acc = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) acc += partials[k * np + i];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sm[w];
      if (pos < capacity) series[3 * pos + k] = v;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && count) *count = pos + 1;
}

}  // namespace ieq
