// Order-9 WENO reconstruction of the two cell-edge values of one stencil.
//
// Follows limiter::WenoLimiter<real,9>::compute_limited_edges
// (model/modules/helpers/WenoLimiter.h:349-437):
//   1. smoothness indicators TV_1..TV_5 of the five 5-cell sub-stencils
//      (TransformMatrices.h:429-433, 19841-19880), normalised to sum 1
//      (convexify, WenoLimiter.h:30-34);
//   2. imm_L: TV_5 = max(TV), imm_R: TV_1 = max(TV)  (WenoLimiter.h:430-437);
//   3. per edge: w_k = ideal_k / (TV_k^2 + 1e-20), normalise, optionally
//      apply map_rs (k=6, m=3, s=2000; WenoLimiter.h:75-82) and normalise
//      again, then the weighted sub-stencil edge values (WenoLimiter.h:382-426).
// The arithmetic is rearranged (difference form, see gen_weno9.py): nested
// stencil differences, per window three linear forms that give both its TV
// and its two edge values, one reciprocal shared by both edges for each
// 1/(TV_k^2+1e-20), and the normalisation after map_rs applied once to the
// weighted sum instead of to each weight.
//
// The stencil kernels are bound by the FP32 multiply-add pipe, so the count
// of these operations is what the limiter costs: ~240 per stencil (both
// edges) against ~280 for the earlier form (an LDL^T factorisation of each
// window's TV and separate edge formulas, 118 operations up to the TVs and
// edge values where this one takes 94; MAP_RATIOS below takes 18 more off),
// and ~25 distinct constants instead of ~100.  Both together took the
// 256x256x128 boundary layer from 6.53 to 5.98 ms per step and the 512x512x128
// urban canopy from 24.2 to 22.2 ms.
// In FP32 the reciprocals use rcp.approx.ftz; every operand is a normal
// number there (or t^2 = 0, see MAP_RATIOS): TV_k^2+1e-20 >= 1e-20, the
// normalisation sums exceed 1e-20 on the branch that divides (the weight sums
// always), and the map_rs denominators, divided by 2000, are at least
// ideal_k^6/2000 > 1e-16 or 1/2000.
#pragma once

#include "weno9_tables.cuh"

namespace pu {

template <class R>
__device__ __forceinline__ R fast_rcp(R x) { return R(1) / x; }

template <>
__device__ __forceinline__ float fast_rcp<float>(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---------------------------------------------------------------------------
// Arithmetic of one stencil (float, double) or of two at once (float2, the
// packed FFMA2/FADD2/FMUL2 of sm_100).  Every operation is rounded by itself
// and the limiter below is written once over them, so each lane of the packed
// form gives the scalar form's bits.  A difference in the packed form is
// fma(b, -1, a), which is one operation whether or not the packed add takes a
// negated operand, with the same rounding.
// ---------------------------------------------------------------------------
struct bool2 {
  bool x, y;
};
template <class V>
struct Arith;

template <>
struct Arith<float> {
  using V = float;
  using B = bool;
  static __device__ __forceinline__ V c(double a) { return float(a); }
  static __device__ __forceinline__ V c2(double, double b) { return float(b); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ V fma(V a, V b, V x) { return fmaf(a, b, x); }
  static __device__ __forceinline__ V rcp(V a) { return fast_rcp(a); }
  static __device__ __forceinline__ V neg(V a) { return -a; }
  static __device__ __forceinline__ V max(V a, V b) { return fmaxf(a, b); }
  static __device__ __forceinline__ B gt(V a, float b) { return a > b; }
  static __device__ __forceinline__ V sel(B q, V a, V b) { return q ? a : b; }
  static __device__ __forceinline__ bool any(B q) { return q; }
};

template <>
struct Arith<double> {   // the windows; the rest of the FP64 limiter is below
  using V = double;
  using B = bool;
  static __device__ __forceinline__ V c(double a) { return a; }
  static __device__ __forceinline__ V add(V a, V b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ V mul(V a, V b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ V fma(V a, V b, V x) { return ::fma(a, b, x); }
};

template <>
struct Arith<float2> {
  using V = float2;
  using B = bool2;
  static __device__ __forceinline__ V c(double a) { return make_float2(float(a), float(a)); }
  static __device__ __forceinline__ V c2(double a, double b) { return make_float2(float(a), float(b)); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
  static __device__ __forceinline__ V fma(V a, V b, V x) { return __ffma2_rn(a, b, x); }
  static __device__ __forceinline__ V rcp(V a) { return make_float2(fast_rcp(a.x), fast_rcp(a.y)); }
  static __device__ __forceinline__ V neg(V a) { return make_float2(-a.x, -a.y); }
  static __device__ __forceinline__ V max(V a, V b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
  static __device__ __forceinline__ B gt(V a, float b) { return bool2{a.x > b, a.y > b}; }
  static __device__ __forceinline__ V sel(B q, V a, V b) { return make_float2(q.x ? a.x : b.x, q.y ? a.y : b.y); }
  static __device__ __forceinline__ bool any(B q) { return q.x || q.y; }
};

template <class V>
__device__ __forceinline__ V sum5(const V (&w)[5]) {
  using A = Arith<V>;
  return A::add(A::add(A::add(A::add(w[0], w[1]), w[2]), w[3]), w[4]);
}

// The five windows of a stencil in difference form: X and O, whose sum and
// difference (O scaled by DF_SO) are 1/DF_OUT times the window's right and
// left edge value minus s_4, and tv = 4 TV / DF_CA.
template <class V>
__device__ __forceinline__ void weno9_windows(const V (&s)[9], V (&X)[5], V (&O)[5], V (&tv)[5]) {
  using namespace pu_weno9;
  using A = Arith<V>;
  V d[8], e2[7], e3[6], e4[5];
#pragma unroll
  for (int m = 0; m < 8; m++) d[m] = A::sub(s[m + 1], s[m]);
#pragma unroll
  for (int m = 0; m < 7; m++) e2[m] = A::sub(d[m + 1], d[m]);
#pragma unroll
  for (int m = 0; m < 6; m++) e3[m] = A::sub(e2[m + 1], e2[m]);
#pragma unroll
  for (int m = 0; m < 5; m++) e4[m] = A::sub(e3[m + 1], e3[m]);
  // Second and central first difference at the centre cell: windows 1 to 3
  // hold the centre's neighbours, windows 0 and 4 extend their quartic by one.
  const V lo = A::add(e2[2], A::add(e3[1], e4[0])), nhi = A::sub(A::sub(e3[4], e4[4]), e2[4]);
  const V wm = A::mul(A::c(DF_SW), e2[3]);
  const V hm = A::mul(A::c(DF_OS), A::add(d[3], d[4]));
  const V w[5] = {A::mul(A::c(DF_SW), lo), wm, wm, wm, A::mul(A::c(-DF_SW), nhi)};
  const V h[5] = {A::mul(A::c(DF_OS), A::fma(A::c(2.), d[3], lo)), hm, hm, hm,
                  A::mul(A::c(DF_OS), A::fma(A::c(2.), d[4], nhi))};
  const V a3[5] = {A::fma(A::c(1.5), e4[0], e3[1]), A::fma(A::c(.5), e4[1], e3[2]), A::fma(A::c(.5), e4[2], e3[2]),
                   A::fma(A::c(-.5), e4[3], e3[3]), A::fma(A::c(-1.5), e4[4], e3[4])};
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const V W = A::fma(A::c(DF_CW), e4[k], w[k]);
    O[k] = A::fma(A::c(DF_CO), a3[k], h[k]);
    X[k] = A::fma(A::c(DF_CX), e4[k], W);
    V t = A::mul(A::mul(A::c(DF_C4), e4[k]), e4[k]);
    t = A::fma(a3[k], a3[k], t);
    t = A::fma(W, W, t);
    tv[k] = A::fma(O[k], O[k], t);
  }
}

// From the windows' tv to the reciprocals rk = 1/(TV_k^2 + 1e-20) of the
// normalised TVs (convexify: not normalised where the sum of the TVs is at
// most 1e-20; TV_k^2 is then below 1e-38, and any fixed scale of tv leaves
// rk at 1e20), with the immersed replacements (imm_L: TV_5 = max, imm_R:
// TV_1 = max).
template <class V>
__device__ __forceinline__ void weno9_rk(V (&tv)[5], typename Arith<V>::B imm_L, typename Arith<V>::B imm_R,
                                         V (&rk)[5]) {
  using A = Arith<V>;
  const V tot = sum5(tv);
  const V r = A::sel(A::gt(tot, 4.e-20 / pu_weno9::DF_CA), A::rcp(tot), A::c(1.));
#pragma unroll
  for (int k = 0; k < 5; k++) tv[k] = A::mul(tv[k], r);
  if (A::any(imm_L) || A::any(imm_R)) {
    const V mx = A::max(A::max(A::max(A::max(tv[0], tv[1]), tv[2]), tv[3]), tv[4]);
    tv[4] = A::sel(imm_L, mx, tv[4]);
    tv[0] = A::sel(imm_R, mx, tv[0]);
  }
#pragma unroll
  for (int k = 0; k < 5; k++) rk[k] = A::rcp(A::fma(tv[k], tv[k], A::c(1.e-20)));
}

// Per-lane constants of one edge: SIDE 0 the left edge, 1 the right edge, 2
// (float2) the right edge in lane x and the left edge in lane y.
template <class V, int SIDE>
__device__ __forceinline__ V ideal_of(int k, double scale = 1.) {
  using namespace pu_weno9;
  return Arith<V>::c2(scale * (SIDE == 0 ? IDEAL_L[k] : IDEAL_R[k]), scale * (SIDE == 1 ? IDEAL_R[k] : IDEAL_L[k]));
}
// How many of an edge's five weights are mapped by way of the ratio z = u/t^2,
//   d + t t^6/(t^6 + 2000 u^3) = d + t/(1 + 2000 z^3),
// which takes seven multiply-adds and two reciprocals against ten and one.
// The multiply-add pipe is the busiest of the stencil kernels' (79 % in k_xy
// with none, 77 % with three) and the reciprocals' pipe had room (48 %, now
// 57-64 %): on the 256x256x128 boundary layer 0, 2, 3, 4 of five take 24.58,
// 24.02, 23.94, 24.01 ms for four steps (all five, in a first form of this,
// were slower than three by 1.5 %).  z is infinite where t = 0, and the weight
// then the ideal one.
constexpr int MAP_RATIOS = 3;
template <class V, int SIDE>
__device__ __forceinline__ V odd_of() {
  using namespace pu_weno9;
  return Arith<V>::c2(SIDE == 0 ? -DF_SO : DF_SO, SIDE == 1 ? DF_SO : -DF_SO);
}

// The weights of one edge, negated: -w_k of the ideal-weighted normalised
// reciprocals, or after map_rs the unnormalised -2000 m_k, whose sum the
// caller divides by (r: 1/sum(-2000 m_k), or -1).  The signs spare every
// negated operand in between: with n = -w,  n + d = -(w - d)  and
// n n + n = -w (1 - w) = -u; the factor 2000 spares its multiplication.
// Both sums always pass the reference's test (> 1e-20): rk_k is at least
// 1/(1 + 1e-20) when the TVs were normalised (each is then at most 1 up to a
// rounding) and 1e20 when they were not, so the first is at least the sum of
// the ideal weights, 1; each m_k >= min(w_k, ideal_k) >= 0, and the k with
// w_k >= 1/5 gives m_k >= min_k ideal_k = 1/126.
template <class V, int SIDE>
__device__ __forceinline__ V weno9_neg_weights(const V (&rk)[5], typename Arith<V>::B do_map, V (&n)[5]) {
  using A = Arith<V>;
#pragma unroll
  for (int k = 0; k < 5; k++) n[k] = A::mul(ideal_of<V, SIDE>(k), rk[k]);
  const V rn = A::rcp(A::neg(sum5(n)));
#pragma unroll
  for (int k = 0; k < 5; k++) n[k] = A::mul(n[k], rn);
  V r = A::c(-1.);
  if (A::any(do_map)) {
    V m[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const V t = A::add(n[k], ideal_of<V, SIDE>(k));
      const V t2 = A::mul(t, t);
      const V u = A::fma(n[k], n[k], n[k]);
      const V d2000 = ideal_of<V, SIDE>(k, -2000.);
      if (k < MAP_RATIOS) {
        const V z = A::mul(u, A::rcp(A::neg(t2)));
        const V den = A::fma(A::mul(z, z), z, A::c(1. / 2000.));
        m[k] = A::fma(t, A::rcp(den), d2000);
      } else {
        const V t6 = A::mul(A::mul(t2, t2), t2);
        const V u3 = A::mul(A::mul(u, u), u);
        const V den = A::fma(A::c(-1. / 2000.), t6, u3);
        m[k] = A::fma(A::mul(t6, t), A::rcp(A::neg(den)), d2000);
      }
    }
    r = A::sel(do_map, A::rcp(sum5(m)), r);
#pragma unroll
    for (int k = 0; k < 5; k++) n[k] = A::sel(do_map, m[k], n[k]);
  }
  return r;
}

template <class V, int SIDE>
__device__ __forceinline__ V weno9_edge(const V (&X)[5], const V (&O)[5], V s4, const V (&rk)[5],
                                        typename Arith<V>::B do_map) {
  using A = Arith<V>;
  V n[5];
  const V r = weno9_neg_weights<V, SIDE>(rk, do_map, n);
  V acc = A::mul(n[0], A::fma(odd_of<V, SIDE>(), O[0], X[0]));
#pragma unroll
  for (int k = 1; k < 5; k++) acc = A::fma(n[k], A::fma(odd_of<V, SIDE>(), O[k], X[k]), acc);
  return A::fma(acc, A::mul(r, A::c(pu_weno9::DF_OUT)), s4);
}

// Both edges of one stencil (R float or double) or of two (float2).
template <class V>
__device__ __forceinline__ void weno9_edges(const V (&s)[9], V &qL, V &qR, typename Arith<V>::B do_map,
                                            typename Arith<V>::B imm_L, typename Arith<V>::B imm_R) {
  V X[5], O[5], tv[5], rk[5];
  weno9_windows(s, X, O, tv);
  weno9_rk(tv, imm_L, imm_R, rk);
  qL = weno9_edge<V, 0>(X, O, s[4], rk, do_map);
  qR = weno9_edge<V, 1>(X, O, s[4], rk, do_map);
}

// ---------------------------------------------------------------------------
// FP64.  A division costs about ten FP64 operations, and the form above takes
// twenty per stencil; here the range of FP64 lets products stand in for the
// reciprocals of each group of five,
//   1/b_k : 1/b_j  =  prod_{i != k} b_i : prod_{i != j} b_i,
// (b_k = TV_k^2 + 1e-20 in [1e-20, ~1]; the map_rs denominators in [2e-13, 32];
// products of four stay far inside the range), and the two edges share one
// division where both need one: three divisions per stencil (both edges), two
// for one edge.
// ---------------------------------------------------------------------------
// Every operation is rounded by itself here too (Arith<double>), so that all
// instantiations of the stencil kernels give a stencil the same bits.
// o[k] = product of the other four.
__device__ __forceinline__ void other_products(const double (&b)[5], double (&o)[5]) {
  using A = Arith<double>;
  const double b01 = A::mul(b[0], b[1]), b34 = A::mul(b[3], b[4]);
  const double b012 = A::mul(b01, b[2]), b234 = A::mul(b[2], b34);
  o[0] = A::mul(b[1], b234);
  o[1] = A::mul(b[0], b234);
  o[2] = A::mul(b01, b34);
  o[3] = A::mul(b012, b[4]);
  o[4] = A::mul(b012, b[3]);
}

// The weights up to a common factor, from the TVs:
// P[k] = prod_{i != k} (TV_i^2 + 1e-20) with the normalised TVs.
__device__ __forceinline__ void weno9_products(double (&tv)[5], bool imm_L, bool imm_R, double (&P)[5]) {
  using A = Arith<double>;
  const double tot = sum5(tv);
  const double r = tot > 4.e-20 / pu_weno9::DF_CA ? 1. / tot : 1.;
#pragma unroll
  for (int k = 0; k < 5; k++) tv[k] = A::mul(tv[k], r);
  if (imm_L || imm_R) {
    const double mx = fmax(fmax(fmax(fmax(tv[0], tv[1]), tv[2]), tv[3]), tv[4]);
    if (imm_L) tv[4] = mx;
    if (imm_R) tv[0] = mx;
  }
  double b[5];
#pragma unroll
  for (int k = 0; k < 5; k++) b[k] = A::fma(tv[k], tv[k], 1.e-20);
  other_products(b, P);
}

// Unnormalised weights ideal_k P_k of one edge.
template <bool LEFT>
__device__ __forceinline__ void weno9_raw_weights(const double (&P)[5], double (&w)[5]) {
  using namespace pu_weno9;
#pragma unroll
  for (int k = 0; k < 5; k++) w[k] = Arith<double>::mul(LEFT ? IDEAL_L[k] : IDEAL_R[k], P[k]);
}

// Weighted sum of the windows' edges (num) and sum of the weights (den) of
// one edge from its normalised weights, after map_rs when do_map: the mapped
// weight (d den_k + t_k^7) / den_k times the product of all five den.
template <bool LEFT>
__device__ __forceinline__ void weno9_ratio(const double (&X)[5], const double (&O)[5], double (&w)[5], bool do_map,
                                            double &num, double &den) {
  using namespace pu_weno9;
  using A = Arith<double>;
  den = 1.;
  if (do_map) {
    double q[5], o[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const double dk = LEFT ? IDEAL_L[k] : IDEAL_R[k];
      const double t = A::sub(w[k], dk), t2 = A::mul(t, t), t6 = A::mul(A::mul(t2, t2), t2);
      const double u = A::fma(-w[k], w[k], w[k]), u3 = A::mul(A::mul(u, u), u);
      q[k] = A::fma(2000., u3, t6);
      w[k] = A::fma(dk, q[k], A::mul(t6, t));
    }
    other_products(q, o);
#pragma unroll
    for (int k = 0; k < 5; k++) w[k] = A::mul(w[k], o[k]);
    den = sum5(w);
  }
  num = A::mul(w[0], A::fma(LEFT ? -DF_SO : DF_SO, O[0], X[0]));
#pragma unroll
  for (int k = 1; k < 5; k++) num = A::fma(w[k], A::fma(LEFT ? -DF_SO : DF_SO, O[k], X[k]), num);
}

template <>
__device__ __forceinline__ void weno9_edges<double>(const double (&s)[9], double &qL, double &qR, bool do_map,
                                                    bool imm_L, bool imm_R) {
  using A = Arith<double>;
  double X[5], O[5], tv[5], P[5], wl[5], wr[5];
  weno9_windows(s, X, O, tv);
  weno9_products(tv, imm_L, imm_R, P);
  weno9_raw_weights<true>(P, wl);
  weno9_raw_weights<false>(P, wr);
  const double sl = sum5(wl), sr = sum5(wr), ri = 1. / A::mul(sl, sr), rl = A::mul(ri, sr), rr = A::mul(ri, sl);
#pragma unroll
  for (int k = 0; k < 5; k++) {
    wl[k] = A::mul(wl[k], rl);
    wr[k] = A::mul(wr[k], rr);
  }
  double nl, dl, nr, dr;
  weno9_ratio<true>(X, O, wl, do_map, nl, dl);
  weno9_ratio<false>(X, O, wr, do_map, nr, dr);
  const double r = pu_weno9::DF_OUT / A::mul(dl, dr);
  qL = A::fma(nl, A::mul(r, dr), s[4]);
  qR = A::fma(nr, A::mul(r, dl), s[4]);
}

// The left or the right edge alone, by the two-edge form: the halo cells that
// close a row of faces need the bits their own tile gives that edge, and the
// shared divisions make an edge's last bits depend on both.
template <bool LEFT>
__device__ __forceinline__ double weno9_one_edge(const double (&s)[9], bool do_map, bool imm_L, bool imm_R) {
  double qL, qR;
  weno9_edges(s, qL, qR, do_map, imm_L, imm_R);
  return LEFT ? qL : qR;
}

// The right edge of stencil x and the left edge of stencil y, each
// bit-identical to that edge from weno9_edges: the one edge a tile needs
// from each of the two halo cells that close a row of faces.
__device__ __forceinline__ float2 weno9_outer_edges2(const float2 (&s)[9], bool2 do_map, bool2 imm_L, bool2 imm_R) {
  float2 X[5], O[5], tv[5], rk[5];
  weno9_windows(s, X, O, tv);
  weno9_rk(tv, imm_L, imm_R, rk);
  return weno9_edge<float2, 2>(X, O, s[4], rk, do_map);
}

// Normalised nonlinear weights of the left edge after map_rs, the quantity
// the learned network is trained to reproduce.
template <class R>
__device__ __forceinline__ void weno9_left_weights(const R (&s)[9], R (&w)[5]) {
  R X[5], O[5], tv[5], rk[5], n[5];
  weno9_windows(s, X, O, tv);
  weno9_rk(tv, false, false, rk);
  const R r = weno9_neg_weights<R, 0>(rk, true, n);
#pragma unroll
  for (int k = 0; k < 5; k++) w[k] = n[k] * r;
}

// Edge values from given left-edge and right-edge weights (the last step of
// gll_1 / gll_2, WenoLimiter.h:402-403, 425-426).
template <class R>
__device__ __forceinline__ void edges_from_weights(const R (&s)[9], const R (&wl)[5], const R (&wr)[5], R &qL, R &qR) {
  using namespace pu_weno9;
  R aL = R(0), aR = R(0);
#pragma unroll
  for (int k = 0; k < 5; k++) {
    R dk0 = s[k + 1] - s[k], dk1 = s[k + 2] - s[k + 1], dk2 = s[k + 3] - s[k + 2], dk3 = s[k + 4] - s[k + 3];
    R ll = fma(R(LIN_L[k][3]), dk3, fma(R(LIN_L[k][2]), dk2, fma(R(LIN_L[k][1]), dk1, R(LIN_L[k][0]) * dk0)));
    R lr = fma(R(LIN_R[k][3]), dk3, fma(R(LIN_R[k][2]), dk2, fma(R(LIN_R[k][1]), dk1, R(LIN_R[k][0]) * dk0)));
    aL = fma(wl[k], ll, aL);
    aR = fma(wr[k], lr, aR);
  }
  qL = s[4] + aL;
  qR = s[4] + aR;
}

// Nine-cell linear edges (weno_all == false away from immersed cells,
// dynamics_rk.h:539-545, 584-588).
template <class R>
__device__ __forceinline__ void linear9_edges(const R (&s)[9], R &qL, R &qR) {
  using namespace pu_weno9;
  R l = R(0), r = R(0);
#pragma unroll
  for (int m = 0; m < 8; m++) {
    R dm = s[m + 1] - s[m];
    l = fma(R(S2E_L[m]), dm, l);
    r = fma(R(S2E_R[m]), dm, r);
  }
  qL = s[4] + l;
  qR = s[4] + r;
}

// Zero-derivative extension past the first immersed cell, outward from the
// centre, for a stencil whose centre is not immersed (dynamics_rk.h:478-493).
// imm: bit m set when stencil entry m is immersed.
template <class R>
__device__ __forceinline__ void der0_modify(R (&s)[9], unsigned imm) {
  if (imm == 0u || (imm & 0x10u)) return;
  bool hit = false;
  R v = s[4];
#pragma unroll
  for (int i = 5; i < 9; i++) {
    if (!hit && ((imm >> i) & 1u)) { hit = true; v = s[i - 1]; }
    if (hit) s[i] = v;
  }
  hit = false;
#pragma unroll
  for (int i = 3; i >= 0; i--) {
    if (!hit && ((imm >> i) & 1u)) { hit = true; v = s[i + 1]; }
    if (hit) s[i] = v;
  }
}

}  // namespace pu
