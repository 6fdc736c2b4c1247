// stage_kernel.cuh -- the fused Runge-Kutta stage kernel and the curl(B)/rho kernel.
//
// One thread per node.  For every node the kernel evaluates the time derivative DB of
// kernel/kernel_time_integrator.cl:9-31 -- volume terms (induction_Eq_volume.cl),
// Hall volume term, SAT surface terms (induction_Eq_surface.cl) and artificial
// dissipation (artificial_dissipation.cl) -- and applies the stage update of the
// integrator in the same pass (epilogue modes below), so the stage derivative never
// touches memory.
//
// Volume term.  The reference sums the split-form flux F(B_m,u_m,B_k,u_k) over the
// stencil points k of each derivative row.  Every flux form is bilinear in (m, k)
// quantities, so with D applied to the pointwise products the sum factors into
//     sum_k c_k F = w1 D[u_i B_a] + w2 B_a,m D[u_i] + w3 u_i,m D[B_a]
//                 - (v1 D[u_a B_i] + v2 u_a,m D[B_i] + v3 B_i,m D[u_a])
// (plus terms proportional to sum_k c_k, which is zero for every derivative row);
// w and v come from the USE_UIBJ_* / USE_SOURCE_* / USE_UJBI_* switches.  This cuts the
// flops per stencil point from ~40 to 9-21 and changes only the rounding order.
//
// Interior nodes of every axis use the interior row (radius RI = ORDER/2, coefficients
// in kernel parameters); the SBP boundary closures read their rows from a table.
#pragma once
#include "ieq_common.cuh"

namespace ieq {

// ---- field layouts: REAL4 array-of-structs (the reference's layout, used by the per-kernel
// entry points) and structure-of-arrays (x, y, z planes of one allocation, component stride s;
// used by the fused time stepping: a warp's neighbour load is 256 contiguous bytes).
template <typename R>
struct AoS {
  R4<R> *p;
};
template <typename R>
struct SoA {
  R *p;
  long long s;
  int ro;     // (used by SoAcg only) the field is never written during the launch
};
// SoA for a persistent kernel that reads, in a later stage, data other blocks wrote in an
// earlier stage of the same launch.  Such data must not go through the non-coherent
// read-only path (ld.global.nc); ordinary loads (ld.global.ca) issued after the fenced grid
// barrier observe the other blocks' writes.  A field marked `ro` (never written during the
// launch) keeps the read-only path.
template <typename R>
struct SoAcg {
  R *p;
  long long s;
  int ro;
};
template <typename R>
__device__ __forceinline__ V3<R> ldf(const AoS<R> &f, long long j) { return ld3(f.p + j); }
template <typename R>
__device__ __forceinline__ V3<R> ldf(const SoAcg<R> &f, long long j) {
  if (f.ro) return {__ldg(f.p + j), __ldg(f.p + j + f.s), __ldg(f.p + j + 2 * f.s)};
  return {__ldca(f.p + j), __ldca(f.p + j + f.s), __ldca(f.p + j + 2 * f.s)};
}
template <typename R>
__device__ __forceinline__ V3<R> ldf_plain(const SoAcg<R> &f, long long j) {
  return {__ldca(f.p + j), __ldca(f.p + j + f.s), __ldca(f.p + j + 2 * f.s)};
}
template <typename R>
__device__ __forceinline__ void stf(const SoAcg<R> &f, long long j, V3<R> v) {
  f.p[j] = v.x;
  f.p[j + f.s] = v.y;
  f.p[j + 2 * f.s] = v.z;
}
// The type of a node's index.  The fused state's are 32-bit: it holds 27 planes beside the
// caller's fields, and 2^31 nodes of it do not fit 180 GB (the component bases are uniform, so a
// load's address is one multiply-add).  A single field of the caller's records has room for
// more: FP32 records of 2^31 nodes are 34 GB, a curl of them 69 GB.  AoSNear is AoS where the
// grid has fewer nodes, for the stage and curl kernels (with 64-bit indices the stage kernels
// spill: kernel lists 48^3 443 us against 435).
template <typename F>
struct NodeIndex {
  using T = int;
};
template <typename R>
struct AoSNear : AoS<R> {};
template <typename R>
struct NodeIndex<AoS<R>> {
  using T = long long;
};
template <typename F>
using Idx = typename NodeIndex<F>::T;
// node (ix, iy, iz) of a field of layout F
template <typename F>
__device__ __forceinline__ Idx<F> node_at(const Mesh &m, int ix, int iy, int iz) {
  return ix + (Idx<F>)m.px * (iy + (Idx<F>)m.ny * iz);
}
template <typename R>
__device__ __forceinline__ V3<R> ldf(const SoA<R> &f, int j) {
  return {__ldg(f.p + j), __ldg(f.p + f.s + j), __ldg(f.p + 2 * f.s + j)};
}
template <typename R>
__device__ __forceinline__ V3<R> ldf_plain(const AoS<R> &f, long long j) { return ld3_plain(f.p + j); }
template <typename R>
__device__ __forceinline__ V3<R> ldf_plain(const SoA<R> &f, int j) {
  return {f.p[j], (f.p + f.s)[j], (f.p + 2 * f.s)[j]};
}
template <typename R>
__device__ __forceinline__ void stf(const AoS<R> &f, long long j, V3<R> v) { st3(f.p + j, v); }
template <typename R>
__device__ __forceinline__ void stf(const SoA<R> &f, int j, V3<R> v) {
  f.p[j] = v.x;
  (f.p + f.s)[j] = v.y;
  (f.p + 2 * f.s)[j] = v.z;
}

// Rounding written out: a b + c in one rounding, a b and a - b each in their own.  A sum s += c v
// is always one rounding, but which product of two is contracted, and whether one is contracted
// at all into a sum that stands elsewhere, depends on the kernel around it.  The stage kernels
// must round alike whichever of them runs a node, or a z slab would differ from the whole grid in
// its last bits: what follows the sums over a stencil uses these.
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
// s += a v, by component
template <typename R>
__device__ __forceinline__ void mad3(V3<R> &s, R a, const V3<R> &v) {
  s.x = mad(a, v.x, s.x);
  s.y = mad(a, v.y, s.y);
  s.z = mad(a, v.z, s.z);
}

enum EpilogueMode : int {
  EP_X_PLUS_HF = 0,   // out = X + h*F                 SSPRK33_1, SSPRK104, KCL_5, CFR_6
  EP_PX_QYHF = 1,     // out = p*X + q*(Y + h*F)       SSPRK33_2b/3b, SSPRK104_11b
  EP_HF = 2,          // out = h*F                     *_1a, KCL/CFR "a" kernels
  EP_AX_HF = 3,       // out = A*X + h*F               CarpenterKennedy/ToulorgeDesmet "a"
  EP_2N_FUSED = 4,    // t = A*X + h*F; out = t; out2 = Z + Bc*t     ("a" and "b" fused)
  EP_2N_FUSED_FIRST = 5,  // t = h*F; out = t; out2 = Z + Bc*t
  EP_2R_FUSED = 6,    // t = h*F; out = X + A*t; out2 = out + Bc*t; out3 = t (if set)   (2R "a" + "b")
};

enum TimePost : int {
  TP_NONE = 0,
  TP_SET_STAGE = 1,   // time[1] = time[0] + K
  TP_ADVANCE = 2,     // time[0] = time[0] + DT; time[1] = time[0]
};

enum DissKind : int { DISS_NONE = 0, DISS_HO = 1, DISS_FO_OR_AD = 2 };

template <typename R, typename F = AoS<R>>
struct StageArgs {
  Mesh m;
  F bk;                 // field the derivative is taken of
  F J;                  // curl(B)/rho (Hall; the column kernel reads it on faces only)
  F E;                  // (column kernel, Hall) J x B as (Jx By - Jy Bx, Jx Bz - Jz Bx, Jy Bz - Jz By)
  F Hpre;               // (column kernel) the dissipation sum of bk, precomputed by k_curl_e_hod
  F u;
  F X, Y, Z;
  F out, out2, out3;
  const Tables<R> *tab;
  R *time;
  unsigned *counter;    // last-block ticket for the time post-update
  R Dint[7];            // interior derivative row, offsets -RI..RI
  R Hint[7];            // interior dissipation row, offsets -RI..RI
  R two_inv_d[3];       // (REAL)(2.0/DX) ...
  R inv_d[3];           // (REAL)(1.0/DX) ...
  R sat_s[3];           // (REAL)(M_INV[0]/DX) ...
  R dR[3];              // (REAL)DX ...
  R w[6];               // flux-form weights w1 w2 w3 v1 v2 v3
  int need;             // 1: D[u_i B_a], 2: D[u], 4: D[B], 8: D[u_a B_i]
  int conv;             // convection terms present (u not identically zero) ...
  const int *conv_flag; // ... or, if set, read from device memory at kernel start
  int tc;               // testcase (b_boundary of the inflow SAT)
  int diss_form;        // 2 first order, 3 adaptive (DISS_FO_OR_AD)
  R hod_factor;
  double mp2min, mp2max, cmin, cmax;
  int mode;
  R p, q, h, A, Bc;
  int tpost;
  R tK, tDT;
};

// neighbour index along one axis: periodic wrap, or clamp-to-self outside the grid
// (include/utils.h:89-168; the coefficient of a clamped point is zero)
template <bool PER>
__device__ __forceinline__ int nbr(int i, int o, int n) {
  int j = i + o;
  if (PER) {
    j += (j < 0) ? n : 0;
    j -= (j >= n) ? n : 0;
  } else {
    j = (j < 0 || j >= n) ? i : j;
  }
  return j;
}

template <typename R>
struct AxisSums {
  V3<R> SuiBa, SU, SB, SuaB, SH, SHo;
};

// CHK: test the coefficients for zero at run time (boundary rows); the interior rows call
// this with compile-time knowledge instead (only the centre derivative coefficient is zero)
template <typename R, typename F, bool HALL, bool HOD, bool CHK>
__device__ __forceinline__ void accumulate(AxisSums<R> &s, const StageArgs<R, F> &a, int conv, int axis, R cD, R cH,
                                           Idx<F> j) {
  const V3<R> B = ldf(a.bk, j);
  if (conv && (!CHK || cD != (R)0)) {
    const V3<R> U = ldf(a.u, j);
    const R Ba = axis == 0 ? B.x : (axis == 1 ? B.y : B.z);
    const R Ua = axis == 0 ? U.x : (axis == 1 ? U.y : U.z);
    if (a.need & 1) {
      s.SuiBa.x += cD * (U.x * Ba); s.SuiBa.y += cD * (U.y * Ba); s.SuiBa.z += cD * (U.z * Ba);
    }
    if (a.need & 2) { s.SU.x += cD * U.x; s.SU.y += cD * U.y; s.SU.z += cD * U.z; }
    if (a.need & 4) { s.SB.x += cD * B.x; s.SB.y += cD * B.y; s.SB.z += cD * B.z; }
    if (a.need & 8) {
      s.SuaB.x += cD * (Ua * B.x); s.SuaB.y += cD * (Ua * B.y); s.SuaB.z += cD * (Ua * B.z);
    }
  }
  if (HALL && (!CHK || cD != (R)0)) {
    // Hall_volume: D[J_a B - J B_a]; the a-component is J_a B_a - J_a B_a = 0
    const V3<R> Jk = ldf(a.J, j);
    const R Ja = axis == 0 ? Jk.x : (axis == 1 ? Jk.y : Jk.z);
    const R Ba = axis == 0 ? B.x : (axis == 1 ? B.y : B.z);
    if (axis != 0) s.SH.x += cD * (Ja * B.x - Jk.x * Ba);
    if (axis != 1) s.SH.y += cD * (Ja * B.y - Jk.y * Ba);
    if (axis != 2) s.SH.z += cD * (Ja * B.z - Jk.z * Ba);
  }
  if (HOD && (!CHK || cH != (R)0)) {
    s.SHo.x += cH * B.x; s.SHo.y += cH * B.y; s.SHo.z += cH * B.z;
  }
}

template <typename R, typename F>
__device__ __forceinline__ R ldc(const F &f, Idx<F> j, int comp);
template <>
__device__ __forceinline__ double ldc<double, SoA<double>>(const SoA<double> &f, int j, int comp) {
  return __ldg(f.p + comp * f.s + j);
}
template <>
__device__ __forceinline__ float ldc<float, SoA<float>>(const SoA<float> &f, int j, int comp) {
  return __ldg(f.p + comp * f.s + j);
}
template <>
__device__ __forceinline__ double ldc<double, AoS<double>>(const AoS<double> &f, long long j, int comp) {
  return __ldg(reinterpret_cast<const double *>(f.p + j) + comp);
}
template <>
__device__ __forceinline__ float ldc<float, AoS<float>>(const AoS<float> &f, long long j, int comp) {
  return __ldg(reinterpret_cast<const float *>(f.p + j) + comp);
}

template <>
__device__ __forceinline__ double ldc<double, AoSNear<double>>(const AoSNear<double> &f, int j, int comp) {
  return ldc<double, AoS<double>>(f, j, comp);
}
template <>
__device__ __forceinline__ float ldc<float, AoSNear<float>>(const AoSNear<float> &f, int j, int comp) {
  return ldc<float, AoS<float>>(f, j, comp);
}

// kappa of adaptive dissipation for one pair (include/artificial_dissipation.h:23-45): s =
// max(|u1|, |u2|) (b1 - b2)^2 against the thresholds of the distance.  The square root runs only
// between them.  (0 * s carries a NaN, as there.)
__device__ __forceinline__ double ad_kappa(double s, double lo, double hi, double inv) {
  if (s >= hi) return 1.0 + 0.0 * s;
  if (s > lo) return sqrt(sub(s, lo) * inv);
  return 0.0 * s;
}

// adaptive dissipation (artificial_dissipation.cl:83-160) of one axis at a node on the interior
// row, one component at a time (the loop is not unrolled: a warp comes here only where some
// kappa is not zero, and 60 inlined kappas would crowd out the rest of the kernel's code).  The
// 2 RI + 1 points serve the first-order part and the high-order part, whose pairs lie within
// them; the two pairs at the node are in both.  Every operation is that of fo_ad_dissipation's
// general path, which interior nodes of a warp with boundary rows take.
template <typename R, typename F, int OP, bool PER>
__device__ __forceinline__ V3<R> ad_axis_full(const StageArgs<R, F> &a, int ax, int i, int n, Idx<F> idx,
                                              Idx<F> st) {
  constexpr int NB = Op<OP>::NB, RI = Op<OP>::RI, WH = Op<OP>::WH;
  static_assert(WH == RI + 1, "the dissipation pairs lie within the derivative's points");
  const bool wrap = PER && (i < RI || i >= n - RI);
  constexpr R sgn = (Op<OP>::ORDER / 2 + 1) % 2 ? (R)-1 : (R)1;
  const double lo1 = __ldg(&a.tab->ad_lo[ax][1]), hi1 = __ldg(&a.tab->ad_hi[ax][1]), inv1 = __ldg(&a.tab->ad_inv[ax][1]);
  V3<R> out = {0, 0, 0};
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    R b[2 * RI + 1], u[2 * RI + 1], kf[2 * RI + 1];
#pragma unroll
    for (int o = -RI; o <= RI; ++o) {
      const Idx<F> j = wrap ? idx + (nbr<true>(i, o, n) - i) * st : idx + o * st;
      b[o + RI] = ldc<R, F>(a.bk, j, c);
      u[o + RI] = fabs(ldc<R, F>(a.u, j, c));
    }
    // first-order part: sum_k |c_k| kappa max(|u_k|, |u|) (B_k - B) / DX
    R fo = 0, ho = 0;
#pragma unroll
    for (int o = -RI; o <= RI; ++o) {
      if (o == 0) continue;
      const int k = o < 0 ? -o : o;
      const R sg = fmax(u[o + RI], u[RI]), d = b[o + RI] - b[RI];
      kf[o + RI] = (R)ad_kappa((double)((sg * d) * d), __ldg(&a.tab->ad_lo[ax][k]), __ldg(&a.tab->ad_hi[ax][k]),
                               __ldg(&a.tab->ad_inv[ax][k]));
      fo = mad((fabs(a.Dint[o + RI]) * kf[o + RI]) * sg, d, fo);
    }
    // high-order part: (1 - kappa) of the pair (e, e - 1) weights the difference that starts
    // at e - RI (interior row: M_INV = 1, D_HO integer)
#pragma unroll
    for (int e = 0; e <= RI; ++e) {
      R h = 0;
#pragma unroll
      for (int k = 0; k < WH; ++k) h = mad(__ldg(&a.tab->DHO[NB][k]), b[e + k], h);
      R kap;
      if (e == 0) kap = kf[RI - 1];
      else if (e == 1) kap = kf[RI + 1];
      else {
        const R sg = fmax(u[RI + e], u[RI + e - 1]), d = b[RI + e] - b[RI + e - 1];
        kap = (R)ad_kappa((double)((sg * d) * d), lo1, hi1, inv1);
      }
      ho = mad(((R)1 - kap) * a.hod_factor, (__ldg(&a.tab->DHO[NB][e]) * sgn) * h, ho);
    }
    const R v = fo / a.dR[ax] + ho;
    if (c == 0) out.x = v;
    else if (c == 1) out.y = v;
    else out.z = v;
  }
  return out;
}

// whether kappa of a pair of points at distance k may differ from zero in any component
template <typename R>
__device__ __forceinline__ bool ad_test(const V3<R> &b1, const V3<R> &u1, const V3<R> &b2, const V3<R> &u2, R thr) {
  const R dx = b1.x - b2.x, dy = b1.y - b2.y, dz = b1.z - b2.z;
  const R sx = fmax(fabs(u1.x), fabs(u2.x)), sy = fmax(fabs(u1.y), fabs(u2.y)), sz = fmax(fabs(u1.z), fabs(u2.z));
  return (sx * dx) * dx > thr || (sy * dy) * dy > thr || (sz * dz) * dz > thr;
}

// first-order / adaptive dissipation (artificial_dissipation.cl:36-160), evaluated as in
// the reference per stencil point; used only by the DISS_FO_OR_AD instantiation.  Axes in `skip`
// are left out; adaptive axes on which the whole warp sits on the interior row take ad_axis_full,
// which rounds alike.
// (Hall periodic 64^3 with a current sheet, adaptive, 4th order, 20 stages: 2.37 ms with every
// kappa evaluated from the table rows, 0.92 with the interior points loaded once and thresholds
// from the host, 0.79 with the axes whose kappas are all zero summed in col_axis, 0.67 with that
// and the block shape decided as now.)
template <typename R, typename F, int OP, bool PER>
__device__ V3<R> fo_ad_dissipation(const StageArgs<R, F> &a, const int ii[3], const int nn[3],
                                   const Idx<F> st[3], Idx<F> idx, V3<R> Bm, V3<R> um, int skip = 0) {
  constexpr int NB = Op<OP>::NB, SW = Op<OP>::SW, C0 = (SW - 1) / 2, WH = Op<OP>::WH;
  V3<R> acc = {0, 0, 0};
  const bool adaptive = a.diss_form == 3;
  auto kap = [&](unsigned k, R dx, R b1, R b2, R u1, R u2) -> R {
    const R s = (fmax(fabs(u1), fabs(u2)) * (b1 - b2)) * (b1 - b2);
    k = k + (k == 0);
    const double kk = (double)(k * k);
    const double lo = mul(mul(mul(kk, a.mp2min), a.cmin), (double)dx);
    const double hi = mul(mul(mul(kk, a.mp2max), a.cmax), (double)dx);
    return (R)ad_kappa((double)s, lo, hi, 1.0 / fabs(hi - lo));
  };
#pragma unroll 1
  for (int ax = 0; ax < 3; ++ax) {
    if (skip >> ax & 1) continue;
    const int row = PER ? NB : sbp_row(ii[ax], nn[ax], NB);
    if (adaptive && (PER || warp_on_row(row, NB))) {
      const V3<R> v = ad_axis_full<R, F, OP, PER>(a, ax, ii[ax], nn[ax], idx, st[ax]);
      acc.x += v.x; acc.y += v.y; acc.z += v.z;
      continue;
    }
    V3<R> tmp = {0, 0, 0};
    for (int c = 0; c < SW; ++c) {
      const int o = c - C0;
      const R cd = fabs(a.tab->D[row][c]);
      if (cd == (R)0) continue;   // a zero coefficient adds a zero term: skip its loads
      const Idx<F> j = idx + (nbr<PER>(ii[ax], o, nn[ax]) - ii[ax]) * st[ax];
      const V3<R> Bk = ldf(a.bk, j);
      const V3<R> uk = ldf(a.u, j);
      V3<R> sg = {fmax(fabs(uk.x), fabs(um.x)), fmax(fabs(uk.y), fabs(um.y)), fmax(fabs(uk.z), fabs(um.z))};
      if (adaptive) {
        const unsigned k = (unsigned)(o < 0 ? -o : o);
        tmp.x = mad((cd * kap(k, a.dR[ax], Bk.x, Bm.x, uk.x, um.x)) * sg.x, Bk.x - Bm.x, tmp.x);
        tmp.y = mad((cd * kap(k, a.dR[ax], Bk.y, Bm.y, uk.y, um.y)) * sg.y, Bk.y - Bm.y, tmp.y);
        tmp.z = mad((cd * kap(k, a.dR[ax], Bk.z, Bm.z, uk.z, um.z)) * sg.z, Bk.z - Bm.z, tmp.z);
      } else {
        tmp.x += (cd * sg.x) * (Bk.x - Bm.x);
        tmp.y += (cd * sg.y) * (Bk.y - Bm.y);
        tmp.z += (cd * sg.z) * (Bk.z - Bm.z);
      }
    }
    const V3<R> fo = {tmp.x / a.dR[ax], tmp.y / a.dR[ax], tmp.z / a.dR[ax]};
    if (!adaptive) {
      acc.x += fo.x; acc.y += fo.y; acc.z += fo.z;
      continue;
    }
    // high-order part weighted by (1 - kappa) of the neighbouring pair
    V3<R> ho = {0, 0, 0};
    for (int term = -WH + 1; term <= 0; ++term) {
      const Idx<F> j1 = idx + (nbr<PER>(ii[ax], term + WH - 1, nn[ax]) - ii[ax]) * st[ax];
      const Idx<F> j2 = idx + (nbr<PER>(ii[ax], term + WH - 2, nn[ax]) - ii[ax]) * st[ax];
      const V3<R> b1 = ldf(a.bk, j1), b2 = ldf(a.bk, j2), u1 = ldf(a.u, j1), u2 = ldf(a.u, j2);
      // diff_HOD (artificial_dissipation.h:58-101) for this start offset
      const R sgn = (Op<OP>::ORDER / 2 + 1) % 2 ? (R)-1 : (R)1;
      const R c = (a.tab->Minv[row] * a.tab->DHO[row][term + WH - 1]) * sgn;
      V3<R> hod = {0, 0, 0};
      for (int i = 0; i < WH; ++i) {
        const Idx<F> j = idx + (nbr<PER>(ii[ax], i + term, nn[ax]) - ii[ax]) * st[ax];
        mad3(hod, a.tab->DHO[NB][i], ldf(a.bk, j));
      }
      ho.x = mad(((R)1 - kap(1, a.dR[ax], b1.x, b2.x, u1.x, u2.x)) * a.hod_factor, c * hod.x, ho.x);
      ho.y = mad(((R)1 - kap(1, a.dR[ax], b1.y, b2.y, u1.y, u2.y)) * a.hod_factor, c * hod.y, ho.y);
      ho.z = mad(((R)1 - kap(1, a.dR[ax], b1.z, b2.z, u1.z, u2.z)) * a.hod_factor, c * hod.z, ho.z);
    }
    acc.x += fo.x + ho.x; acc.y += fo.y + ho.y; acc.z += fo.z + ho.z;
  }
  return acc;
}

// the inflow factors of a face node (induction_Eq_surface.cl:7-33, upwind against
// b_boundary(t)): f[ax] = sat_s c u_ax on an inflow face of the axis, else 0; whether any is set
template <typename R, typename F>
__device__ __forceinline__ bool sat_inflow(const StageArgs<R, F> &a, const int ii[3], const int nn[3],
                                           const V3<R> &um, R (&f)[3]) {
  bool any = false;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const R ua = ax == 0 ? um.x : (ax == 1 ? um.y : um.z);
    const R c = (ii[ax] == 0 && ua > (R)0 ? (R)-1 : (R)0) + (ii[ax] == nn[ax] - 1 && ua < (R)0 ? (R)1 : (R)0);
    f[ax] = c == (R)0 ? (R)0 : (a.sat_s[ax] * c) * ua;
    any = any || c != (R)0;
  }
  return any;
}
template <typename R>
__device__ __forceinline__ void sat_inflow_add(const R (&f)[3], const V3<R> &df, V3<R> &db) {
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    if (f[ax] == (R)0) continue;
    mad3(db, f[ax], df);
  }
}

// SAT surface terms on the faces of a non-periodic box (added into db)
template <typename R, typename F, bool HALL>
__device__ __forceinline__ void stage_sat(const StageArgs<R, F> &a, const int ii[3], const int nn[3], Idx<F> idx,
                                          const V3<R> &Bm, const V3<R> &um, int conv, V3<R> &db) {
  const int ix = ii[0], iy = ii[1], iz = ii[2], nx = nn[0], ny = nn[1], nz = nn[2];
  const bool face = ix == 0 || iy == 0 || iz == 0 || ix == nx - 1 || iy == ny - 1 || iz == nz - 1;
  if (face) {
    if (HALL) {
      // induction_Eq_surface.cl:35-81 (outflow, directional do-nothing)
      const V3<R> Jm = ldf(a.J, idx);
      const V3<R> tv = {mad((R)0.5, um.x, -Jm.x), mad((R)0.5, um.y, -Jm.y), mad((R)0.5, um.z, -Jm.z)};
      for (int ax = 0; ax < 3; ++ax) {
        const bool l = ii[ax] == 0, r = ii[ax] == nn[ax] - 1;
        if (!l && !r) continue;
        const R tva = ax == 0 ? tv.x : (ax == 1 ? tv.y : tv.z);
        const R Ba = ax == 0 ? Bm.x : (ax == 1 ? Bm.y : Bm.z);
        const R c1 = (l && tva > (R)0 ? (R)-1 : (R)0) + (r && tva < (R)0 ? (R)1 : (R)0);
        const R c2 = (l ? (R)-1 : (R)0) + (r ? (R)1 : (R)0);
        const R f1 = c1 * tva, f2 = c2 * Ba;
        mad3(db, a.sat_s[ax],
             V3<R>{mad(f1, Bm.x, mul(f2, Jm.x)), mad(f1, Bm.y, mul(f2, Jm.y)), mad(f1, Bm.z, mul(f2, Jm.z))});
      }
    } else if (conv) {
      R f[3];
      if (sat_inflow(a, ii, nn, um, f)) {
        const V3<R> bb = b_boundary<R>(a.tc, a.m, ix, iy, iz, a.time[1]);
        sat_inflow_add(f, V3<R>{sub(Bm.x, bb.x), sub(Bm.y, bb.y), sub(Bm.z, bb.z)}, db);
      }
    }
  }
}

// stage_sat of the inflow terms at two x-adjacent nodes (ix even).  b_boundary costs more than
// the rest of a face node (its exponential and trigonometric functions), and a warp that holds
// the ends of a row has one node at x = 0 in one lane and one at x = nx - 1 in another: every
// lane takes its inflow node, whichever of the two it is, in the same pass, and a second pass
// runs only where both nodes of a lane have one (y and z faces).
template <typename R, typename F>
__device__ __forceinline__ void stage_sat_pair(const StageArgs<R, F> &a, int ix, int iy, int iz, const int nn[3],
                                               const V3<R> (&Bm)[2], const V3<R> (&um)[2], V3<R> (&db)[2]) {
  const int i0[3] = {ix, iy, iz}, i1[3] = {ix + 1, iy, iz};
  if (ix != 0 && iy != 0 && iz != 0 && ix + 1 < nn[0] - 1 && iy != nn[1] - 1 && iz != nn[2] - 1) return;
  R f0[3], f1[3];
  // (the last pair of an odd row has one node)
  const bool need0 = sat_inflow(a, i0, nn, um[0], f0), need1 = ix + 1 < nn[0] && sat_inflow(a, i1, nn, um[1], f1);
  if (!need0 && !need1) return;
  const R t = a.time[1];
  int k = need0 ? 0 : 1;
#pragma unroll 1
  for (;;) {
    const V3<R> bb = b_boundary<R>(a.tc, a.m, ix + k, iy, iz, t);
    const V3<R> B = k ? Bm[1] : Bm[0];
    V3<R> d = k ? db[1] : db[0];
    const R f[3] = {k ? f1[0] : f0[0], k ? f1[1] : f0[1], k ? f1[2] : f0[2]};
    sat_inflow_add(f, V3<R>{sub(B.x, bb.x), sub(B.y, bb.y), sub(B.z, bb.z)}, d);
    if (k) {
      db[1] = d;
      break;
    }
    db[0] = d;
    if (!need1) break;
    k = 1;
  }
}

// the stage update of the integrator (EpilogueMode) at one node, split into the loads of
// the fields it combines (which do not depend on DB, so a kernel may issue them early) and
// the arithmetic and stores
template <typename R>
struct EpIn {
  V3<R> X, Y;   // X; Y (EP_PX_QYHF) or Z (the fused 2N modes)
};

template <typename R, typename F>
__device__ __forceinline__ EpIn<R> epilogue_load(const StageArgs<R, F> &a, Idx<F> idx) {
  EpIn<R> e = {{0, 0, 0}, {0, 0, 0}};
  switch (a.mode) {
    case EP_X_PLUS_HF:
    case EP_AX_HF:
    case EP_2R_FUSED:
      e.X = ldf_plain(a.X, idx);
      break;
    case EP_PX_QYHF:
      e.X = ldf_plain(a.X, idx);
      e.Y = ldf_plain(a.Y, idx);
      break;
    case EP_2N_FUSED:
      e.X = ldf_plain(a.X, idx);
      e.Y = ldf_plain(a.Z, idx);
      break;
    case EP_2N_FUSED_FIRST:
      e.Y = ldf_plain(a.Z, idx);
      break;
    default:
      break;
  }
  return e;
}

// the values a mode stores: o1 into out, o2 into out2 (fused 2N / 2R modes), o3 into out3
// (EP_2R_FUSED, if set)
template <typename R>
struct EpOut {
  V3<R> o1, o2, o3;
};
__host__ __device__ constexpr bool epilogue_writes_out2(int mode) {
  return mode == EP_2N_FUSED || mode == EP_2N_FUSED_FIRST || mode == EP_2R_FUSED;
}

template <typename R, typename F>
__device__ __forceinline__ EpOut<R> epilogue_values(const StageArgs<R, F> &a, const V3<R> &db, const EpIn<R> &e) {
  const V3<R> &X = e.X, &Y = e.Y;
  EpOut<R> r = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  switch (a.mode) {
    case EP_X_PLUS_HF:
      r.o1 = V3<R>{mad(a.h, db.x, X.x), mad(a.h, db.y, X.y), mad(a.h, db.z, X.z)};
      break;
    case EP_PX_QYHF:
      r.o1 = V3<R>{mad(a.p, X.x, mul(a.q, mad(a.h, db.x, Y.x))), mad(a.p, X.y, mul(a.q, mad(a.h, db.y, Y.y))),
                   mad(a.p, X.z, mul(a.q, mad(a.h, db.z, Y.z)))};
      break;
    case EP_HF:
      r.o1 = V3<R>{mul(a.h, db.x), mul(a.h, db.y), mul(a.h, db.z)};
      break;
    case EP_AX_HF:
      r.o1 = V3<R>{mad(a.A, X.x, mul(a.h, db.x)), mad(a.A, X.y, mul(a.h, db.y)), mad(a.A, X.z, mul(a.h, db.z))};
      break;
    case EP_2N_FUSED:
    case EP_2N_FUSED_FIRST: {
      V3<R> t;
      t = {mul(a.h, db.x), mul(a.h, db.y), mul(a.h, db.z)};
      if (a.mode == EP_2N_FUSED) t = {mad(a.A, X.x, t.x), mad(a.A, X.y, t.y), mad(a.A, X.z, t.z)};
      r.o1 = t;
      r.o2 = V3<R>{mad(a.Bc, t.x, Y.x), mad(a.Bc, t.y, Y.y), mad(a.Bc, t.z, Y.z)};
      break;
    }
    case EP_2R_FUSED: {
      const V3<R> t = {mul(a.h, db.x), mul(a.h, db.y), mul(a.h, db.z)};
      const V3<R> o = {mad(a.A, t.x, X.x), mad(a.A, t.y, X.y), mad(a.A, t.z, X.z)};
      r.o1 = o;
      r.o2 = V3<R>{mad(a.Bc, t.x, o.x), mad(a.Bc, t.y, o.y), mad(a.Bc, t.z, o.z)};
      r.o3 = t;
      break;
    }
  }
  return r;
}

template <typename R, typename F>
__device__ __forceinline__ void epilogue_store(const StageArgs<R, F> &a, Idx<F> idx, const V3<R> &db,
                                               const EpIn<R> &e) {
  const EpOut<R> r = epilogue_values(a, db, e);
  stf(a.out, idx, r.o1);
  if (epilogue_writes_out2(a.mode)) stf(a.out2, idx, r.o2);
  if (a.mode == EP_2R_FUSED && a.out3.p) stf(a.out3, idx, r.o3);
}

template <typename R, typename F>
__device__ __forceinline__ void stage_epilogue(const StageArgs<R, F> &a, Idx<F> idx, const V3<R> &db) {
  epilogue_store(a, idx, db, epilogue_load(a, idx));
}

// DB and the stage update at one node (ix, iy, iz) inside the grid.
template <typename R, typename F, int OP, bool PER, bool HALL, int DISS, int CONV>
__device__ __forceinline__ void stage_node(const StageArgs<R, F> &a, int ix, int iy, int iz) {
  constexpr int NB = Op<OP>::NB, RI = Op<OP>::RI;
  constexpr bool HOD = DISS == DISS_HO;
  const int nx = a.m.nx, ny = a.m.ny, nz = a.m.nz;
  {
    const Idx<F> idx = node_at<F>(a.m, ix, iy, iz);
    const int ii[3] = {ix, iy, iz};
    const int nn[3] = {nx, ny, nz};
    const Idx<F> st[3] = {1, a.m.px, (Idx<F>)a.m.px * ny};
    const int conv = CONV >= 0 ? CONV : (a.conv_flag ? *a.conv_flag : a.conv);
    const V3<R> Bm = ldf(a.bk, idx);
    V3<R> um = {0, 0, 0};
    if (conv) um = ldf(a.u, idx);
    V3<R> db = {0, 0, 0};
    V3<R> hod = {0, 0, 0};
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      AxisSums<R> s{};
      const int row = PER ? NB : sbp_row(ii[ax], nn[ax], NB);
      if (PER || warp_on_row(row, NB)) {
        // periodic neighbours wrap only within RI of the ends of the axis
        const bool wrap = PER && (ii[ax] < RI || ii[ax] >= nn[ax] - RI);
#pragma unroll
        for (int o = -RI; o <= RI; ++o) {
          const R cD = a.Dint[o + RI];
          const R cH = a.Hint[o + RI];
          Idx<F> j = idx;
          if (o != 0) {
            if (wrap) j = idx + (nbr<true>(ii[ax], o, nn[ax]) - ii[ax]) * st[ax];
            else j = idx + o * st[ax];
            accumulate<R, F, HALL, HOD, false>(s, a, conv, ax, cD, cH, j);
          } else if (HOD) {
            // the interior derivative rows have a zero centre
            accumulate<R, F, false, HOD, false>(s, a, 0, ax, cD, cH, j);
          }
        }
      } else {
        constexpr int NT = HOD ? Op<OP>::NU : Op<OP>::ND;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const R cD = HOD ? __ldg(&a.tab->ud[row][t]) : __ldg(&a.tab->nd[row][t]);
          const R cH = HOD ? __ldg(&a.tab->uh[row][t]) : (R)0;
          const int o = HOD ? __ldg(&a.tab->ud_off[row][t]) : __ldg(&a.tab->nd_off[row][t]);
          if (cD == (R)0 && cH == (R)0) continue;
          accumulate<R, F, HALL, HOD, true>(s, a, conv, ax, cD, cH, idx + o * st[ax]);
        }
      }
      if (conv) {
        const R Ba = ax == 0 ? Bm.x : (ax == 1 ? Bm.y : Bm.z);
        const R Ua = ax == 0 ? um.x : (ax == 1 ? um.y : um.z);
        const R SBa = ax == 0 ? s.SB.x : (ax == 1 ? s.SB.y : s.SB.z);
        const R SUa = ax == 0 ? s.SU.x : (ax == 1 ? s.SU.y : s.SU.z);
        const R *w = a.w;
        V3<R> vol;
        vol.x = w[0] * s.SuiBa.x + w[1] * Ba * s.SU.x + w[2] * um.x * SBa -
                (w[3] * s.SuaB.x + w[4] * Ua * s.SB.x + w[5] * Bm.x * SUa);
        vol.y = w[0] * s.SuiBa.y + w[1] * Ba * s.SU.y + w[2] * um.y * SBa -
                (w[3] * s.SuaB.y + w[4] * Ua * s.SB.y + w[5] * Bm.y * SUa);
        vol.z = w[0] * s.SuiBa.z + w[1] * Ba * s.SU.z + w[2] * um.z * SBa -
                (w[3] * s.SuaB.z + w[4] * Ua * s.SB.z + w[5] * Bm.z * SUa);
        db.x += a.two_inv_d[ax] * vol.x;
        db.y += a.two_inv_d[ax] * vol.y;
        db.z += a.two_inv_d[ax] * vol.z;
      }
      if (HALL) {
        db.x += a.inv_d[ax] * s.SH.x;
        db.y += a.inv_d[ax] * s.SH.y;
        db.z += a.inv_d[ax] * s.SH.z;
      }
      if (HOD) {
        hod.x += s.SHo.x; hod.y += s.SHo.y; hod.z += s.SHo.z;
      }
    }
    if (!PER) stage_sat<R, F, HALL>(a, ii, nn, idx, Bm, um, conv, db);
    if (HOD) {
      mad3(db, a.hod_factor, hod);
    }
    if (DISS == DISS_FO_OR_AD) {
      const V3<R> ds = fo_ad_dissipation<R, F, OP, PER>(a, ii, nn, st, idx, Bm, um);
      db.x += ds.x; db.y += ds.y; db.z += ds.z;
    }
    stage_epilogue<R, F>(a, idx, db);
  }
}

// time bookkeeping of the folded "a"/calc_time kernels, done by the last block to finish
// (every thread of the block must call this)
template <typename R, typename F>
__device__ __forceinline__ void stage_time_post(const StageArgs<R, F> &a) {
  if (a.tpost != TP_NONE) {
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0) {
      __threadfence();
      const unsigned nblocks = gridDim.x * gridDim.y * gridDim.z;
      const unsigned ticket = atomicAdd(a.counter, 1u);
      if (ticket == nblocks - 1) {
        if (a.tpost == TP_SET_STAGE) {
          a.time[1] = a.time[0] + a.tK;
        } else {
          const R t0 = a.time[0] + a.tDT;
          a.time[0] = t0;
          a.time[1] = t0;
        }
        __threadfence();
        *a.counter = 0u;
      }
    }
  }
}

// blocks of 128 threads, five resident (<= 102 registers): at 48^3 the 576 blocks of 256 threads
// were two waves of two per SM.  Confined Hall 48^3, 4th order, high-order dissipation, two steps
// as kernel lists and the results: 428 us (433 with four blocks, 440 with six and spills)
#ifndef IEQ_STAGE_MIN_BLOCKS
#define IEQ_STAGE_MIN_BLOCKS 5
#endif
constexpr int kStageThreads = 128;
template <typename R, typename F, int OP, bool PER, bool HALL, int DISS, int CONV = -1>
__global__ void __launch_bounds__(kStageThreads, IEQ_STAGE_MIN_BLOCKS) k_stage(const __grid_constant__ StageArgs<R, F> a) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x;
  const int iy = blockIdx.y * blockDim.y + threadIdx.y;
  const int iz = blockIdx.z * blockDim.z + threadIdx.z;
  if (ix < a.m.nx && iy < a.m.ny && iz < a.m.nz) stage_node<R, F, OP, PER, HALL, DISS, CONV>(a, ix, iy, iz);
  stage_time_post(a);
}

// curl(b)/rho (kernel_time_integrator.cl:136-208 via SBP_operator.cl:126-135), with the
// same interior/boundary row split; diff_* divide by (REAL)DX as the reference does.
template <typename R, typename F = AoS<R>>
struct CurlArgs {
  Mesh m;
  F b;
  const R *rho;       // nullptr: plain curl (kernel_operator.cl:158 calc_curl)
  F out;
  R4<R> *out_aos;     // (k_curl_rho) if set, the output goes here as records of nx per row
  F jface;      // (k_curl_e) J on the faces of a non-periodic box
  F hout;       // (k_curl_e_hod) the dissipation sum of b (sum over the axes of the H rows)
  R Hint[7];    // (k_curl_e_hod) interior dissipation row, offsets -RI..RI
  const Tables<R> *tab;
  R dR[3];
  R inv_d[3];   // (REAL)(1.0/DX) ...
  R Dint[7];
};

// curl(b)/rho.  Each axis contributes the derivatives of the two components orthogonal to
// it; the derivative rows are multiplied by (REAL)(1/DX) and the curl by 1/rho (within one
// rounding of the reference's divisions).
template <typename R, typename F, int OP, bool PER>
__global__ void __launch_bounds__(256) k_curl_rho(const __grid_constant__ CurlArgs<R, F> a) {
  constexpr int NB = Op<OP>::NB, RI = Op<OP>::RI;
  const int ix = blockIdx.x * blockDim.x + threadIdx.x;
  const int iy = blockIdx.y * blockDim.y + threadIdx.y;
  const int iz = blockIdx.z * blockDim.z + threadIdx.z;
  if (ix >= a.m.nx || iy >= a.m.ny || iz >= a.m.nz) return;
  const Idx<F> idx = node_at<F>(a.m, ix, iy, iz);
  const int ii[3] = {ix, iy, iz};
  const int nn[3] = {a.m.nx, a.m.ny, a.m.nz};
  const Idx<F> st[3] = {1, a.m.px, (Idx<F>)a.m.px * a.m.ny};
  R g[3][3];   // g[axis][component]
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int c1 = (ax + 1) % 3, c2 = (ax + 2) % 3;
    R v1 = 0, v2 = 0;
    const int row = PER ? NB : sbp_row(ii[ax], nn[ax], NB);
    if (PER || warp_on_row(row, NB)) {
      const bool wrap = PER && (ii[ax] < RI || ii[ax] >= nn[ax] - RI);
#pragma unroll
      for (int o = -RI; o <= RI; ++o) {
        if (o == 0) continue;   // the interior row has a zero centre
        const R c = a.Dint[o + RI];
        Idx<F> j;
        if (wrap) j = idx + (nbr<true>(ii[ax], o, nn[ax]) - ii[ax]) * st[ax];
        else j = idx + o * st[ax];
        v1 += c * ldc<R, F>(a.b, j, c1);
        v2 += c * ldc<R, F>(a.b, j, c2);
      }
    } else {
#pragma unroll
      for (int t = 0; t < Op<OP>::ND; ++t) {
        const R c = __ldg(&a.tab->nd[row][t]);
        const Idx<F> j = idx + __ldg(&a.tab->nd_off[row][t]) * st[ax];
        R p1 = 0, p2 = 0;
        if (c != (R)0) {
          p1 = ldc<R, F>(a.b, j, c1);
          p2 = ldc<R, F>(a.b, j, c2);
        }
        v1 += c * p1;
        v2 += c * p2;
      }
    }
    g[ax][c1] = v1 * a.inv_d[ax];
    g[ax][c2] = v2 * a.inv_d[ax];
  }
  V3<R> c = {g[1][2] - g[2][1], g[2][0] - g[0][2], g[0][1] - g[1][0]};
  if (a.rho) {
    const R r = (R)1 / a.rho[idx];
    c = {c.x * r, c.y * r, c.z * r};
  }
  if (a.out_aos) st3(a.out_aos + (ix + a.m.nx * (iy + a.m.ny * iz)), c);
  else stf(a.out, idx, c);
}

// explicit launchers, instantiated per (R, OP) in stage_<r>_o<op>.cu
// conv: -1 decides per launch from StageArgs (conv / conv_flag); 0/1 fixes it at compile time
template <typename R, typename F, int OP>
void launch_stage(const StageArgs<R, F> &a, bool per, bool hall, int diss, int conv, dim3 grid, dim3 block,
                  cudaStream_t s);
template <typename R, typename F, int OP>
void launch_curl(const CurlArgs<R, F> &a, bool per, dim3 grid, dim3 block, cudaStream_t s);

// Vector fields between the caller's REAL4 records and the fused state (entry and exit of the
// fused calls): every field in one launch, field blockIdx.y.  A field without an output is only
// looked at.  If field `check` has a non-zero x, y or z (a NaN counts), *flag = mark; the mark
// changes from call to call, so nothing resets the flag.
struct StateFlag {
  int check;   // -1: none
  int mark;
  int *flag;
};
template <typename R>
struct StateIo {
  unsigned n, nx, px;
  R4<R> *aos[5];
  R *soa[5];
  long long s;
};
template <typename R>
__global__ void __launch_bounds__(256) k_state_in(const __grid_constant__ StateIo<R> a, const StateFlag f) {
  const int k = blockIdx.y;
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  bool set = false;
  if (i < a.n) {
    const V3<R> v = ld3(a.aos[k] + i);
    if (R *out = a.soa[k]) {
      const unsigned j = a.px == a.nx ? i : i + i / a.nx * (a.px - a.nx);
      out[j] = v.x;
      (out + a.s)[j] = v.y;
      (out + 2 * a.s)[j] = v.z;
    }
    set = v.x != (R)0 || v.y != (R)0 || v.z != (R)0;
  }
  if (k == f.check && __syncthreads_or(set) && threadIdx.x == 0 && *(volatile int *)f.flag != f.mark) *f.flag = f.mark;
}
template <typename R>
__global__ void __launch_bounds__(256) k_state_out(const __grid_constant__ StateIo<R> a) {
  const int k = blockIdx.y;
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const R *in = a.soa[k];
  const unsigned j = a.px == a.nx ? i : i + i / a.nx * (a.px - a.nx);
  st3(a.aos[k] + i, V3<R>{in[j], (in + a.s)[j], (in + 2 * a.s)[j]});
}

}  // namespace ieq
