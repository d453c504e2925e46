// The float32 face arithmetic (MUSCL slopes, HLLD) written over lane types: `L1` (one
// value) and `F2` (two values on the packed float32 instructions of sm_100). A face pairs
// what it computes twice: the left and right states' slopes and reconstruction, their fast
// speeds, total pressures and star states; the rest runs on one lane.
//
// Same formulas, region selection and near-degenerate fallback as the float64 templates of
// numerics.cuh (mhd_sweep_pyccel.py:25-48, 51-61, 64-98, 101-145, 148-251; Miyoshi & Kusano
// 2005); the multiply-adds are explicit and every float32 face of every kernel (stage
// kernels, refluxing) runs this code, so a face's flux has the same bits wherever it is
// formed.
#pragma once

#include "lanes.cuh"

namespace wb {

// What bounds these faces is instruction issue, and among the pipes the one that runs
// selects, compares and min / max (half the rate of the multiply-adds): the forms below are
// chosen for few of those. Per face: 57 fewer than selecting every variant (limiter 14, square
// roots 6, first-order fallback 12, star states 10, sign 3, region selection 12). They have the
// bits of the plain selection where no operand or product is subnormal or NaN (a NaN
// difference, of a cell reported as bad, leaves the slope to the other one). B200: a stage of
// the 256^3 box 1.98 ms with those, 1.75 now; of 512 2D instances of 32^2 to 256^2 cells, 0.90
// and 0.81 ms.

// sqrt(x) of a density as x rsqrt(x); x below the smallest normal counts as that, so the root of
// zero is 1e-19.
template <typename V>
__device__ __forceinline__ V lsqrt(V x) {
  const V y = lmax(x, V(kSmallestNormal));
  return lproduct(y, lrsqrt(y));
}

// Half the limited slope of a cell from its backward (a) and forward (b) differences. minmod
// and MC without a product or a sign test: the candidates nearest zero of one sign, the
// other sign's clamp being zero (candidates of both signs clamp to zero twice).
template <int LIM, typename V>
__device__ __forceinline__ V half_slope_l(V a, V b) {
  if (LIM == 3) return V(0.25f) * (a + b);
  if (LIM == 0) return V(0.5f) * (lmax(lmin(a, b), V(0.0f)) + lmin(lmax(a, b), V(0.0f)));
  if (LIM == 1) {
    const V product = a * b;
    return sel(product > V(0.0f), product * linv(a + b), V(0.0f));
  }
  const V quarter = V(0.25f) * (a + b);
  return lmax(lmin3(a, b, quarter), V(0.0f)) + lmin(lmax3(a, b, quarter), V(0.0f));
}

// Fast magnetosonic speed along the normal. The two roots are x rsqrt(x) as it comes: NaN where x
// is zero, negative or below the smallest normal (the discriminant, a fourth power of a speed, is
// that at speeds of 3e-10 in the user's units), and such a face is redone in float64. B200, a step,
// roots floored / by rsqrtf over all of float32 / as here: 256^3 3.98, 4.02 and 3.97 ms, 150 x 97 x
// 75 mixed 1.039, 1.045 and 1.025 ms; 512 planes, two steps 3.75, 3.77 and 3.76 ms.
template <typename V>
__device__ __forceinline__ V fast_speed_l(V rho, V p, V bn, V bt1, V bt2, V gamma) {
  const V ir = linv(rho);
  const V a2 = gamma * p * ir;
  const V bn2 = bn * bn;
  const V b2 = fma(bt1, bt1, fma(bt2, bt2, bn2)) * ir;
  const V s = a2 + b2;
  const V disc = fma(V(-4.0f) * a2 * ir, bn2, s * s);
  const V square = V(0.5f) * (s + lproduct(disc, lrsqrt(disc)));
  return lproduct(square, lrsqrt(square));
}

// Conserved state and normal flux of a normal-frame primitive state; returns p_T.
template <typename V>
__device__ __forceinline__ V side_state_l(const V (&w)[7], V bn, V nbn, V inv_gm1, V (&u)[7], V (&f)[7]) {
  const V rho = w[0], vn = w[1], vt1 = w[2], vt2 = w[3], p = w[4], bt1 = w[5], bt2 = w[6];
  const V magnetic = V(0.5f) * fma(bn, bn, fma(bt1, bt1, bt2 * bt2));
  const V kinetic2 = fma(vn, vn, fma(vt1, vt1, vt2 * vt2));
  const V energy = fma(p, inv_gm1, fma(V(0.5f) * rho, kinetic2, magnetic));
  const V pt = p + magnetic;
  const V vb = fma(vn, bn, fma(vt1, bt1, vt2 * bt2));
  const V mass = rho * vn;
  u[0] = rho;
  u[1] = mass;
  u[2] = rho * vt1;
  u[3] = rho * vt2;
  u[4] = energy;
  u[5] = bt1;
  u[6] = bt2;
  f[0] = mass;
  f[1] = fma(mass, vn, pt - bn * bn);
  f[2] = fma(mass, vt1, nbn * bt1);
  f[3] = fma(mass, vt2, nbn * bt2);
  f[4] = fma(energy + pt, vn, nbn * vb);
  f[5] = fma(bt1, vn, nbn * vt1);
  f[6] = fma(bt2, vn, nbn * vt2);
  return pt;
}

// The wave speeds, S_M, p_T* and both sides' star density, tangential velocity and field,
// and 1 / (S - S_M).
template <typename V>
struct HlldFrontL {
  V sl, sr, ptl, ptr, sm, pts;
  V rsl, vtl1, vtl2, btl1, btl2, inv_sl;
  V rsr, vtr1, vtr2, btr1, btr2, inv_sr;
};

// Star tangential velocity and field of one side; `den` returns d (s - s_M) - B_n^2. No test
// for a vanishing denominator here: a face where it is small is redone in float64.
template <typename V>
__device__ __forceinline__ void star_tangential_l(const V (&w)[7], V bn, V bn2, V s, V d, V sm, V& rho_s, V& vt1,
                                                  V& vt2, V& bt1, V& bt2, V& den, V& inv_ssm) {
  const V vn = w[1];
  const V ssm = s - sm;
  inv_ssm = linv(ssm);
  rho_s = d * inv_ssm;
  den = fma(d, ssm, lneg(bn2));
  const V inv_den = linv(den);
  const V scale = fma(d, s - vn, lneg(bn2)) * inv_den;
  const V shift = bn * (vn - sm) * inv_den;
  vt1 = fma(shift, w[5], w[2]);
  vt2 = fma(shift, w[6], w[3]);
  bt1 = w[5] * scale;
  bt2 = w[6] * scale;
}

// The front half of one face with its left and right sides in the two lanes of F2 (fast
// speeds, total pressures, d = (S - v) rho and the star states of both sides in one packed
// evaluation each); S_M and p_T* on one lane. Where either side's star denominator is near
// zero (relative size below kNearDegenerate32) the front is redone in float64 from the
// float32 inputs.
__device__ __forceinline__ void hlld_front_lr(const float (&L)[7], const float (&Rt)[7], float bn, float gamma,
                                              HlldFrontL<L1>& o) {
  F2 w[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) w[c] = F2(L[c], Rt[c]);
  const L1 vl = L[1], vr = Rt[1];
  const F2 cf2 = fast_speed_l<F2>(w[0], w[4], F2(bn), w[5], w[6], F2(gamma));
  const L1 cf = max_nan(cf2.v.x, cf2.v.y);
  o.sl = lmin(vl, vr) - cf;
  o.sr = lmax(vl, vr) + cf;
  const L1 bn2 = L1(bn) * L1(bn);
  const F2 pt2 = fma(F2(0.5f), fma(w[5], w[5], fma(w[6], w[6], F2(bn2.v))), w[4]);
  o.ptl = pt2.v.x;
  o.ptr = pt2.v.y;
  const F2 s2(o.sl.v, o.sr.v);
  const F2 d2 = (s2 - w[1]) * w[0];
  const L1 dl = d2.v.x, dr = d2.v.y;
  const L1 ndl = lneg(dl);
  const L1 inv_dd = linv(dr - dl);
  o.sm = fma(dr, vr, fma(ndl, vl, o.ptl - o.ptr)) * inv_dd;
  o.pts = fma(dr, o.ptl, fma(ndl, o.ptr, dl * dr * (vr - vl))) * inv_dd;
  F2 rho_s, vt1, vt2, bt1, bt2, den, inv_ssm;
  star_tangential_l<F2>(w, F2(bn), F2(bn2.v), s2, d2, F2(o.sm.v), rho_s, vt1, vt2, bt1, bt2, den, inv_ssm);
  o.rsl = rho_s.v.x, o.rsr = rho_s.v.y;
  o.vtl1 = vt1.v.x, o.vtr1 = vt1.v.y;
  o.vtl2 = vt2.v.x, o.vtr2 = vt2.v.y;
  o.btl1 = bt1.v.x, o.btr1 = bt1.v.y;
  o.btl2 = bt2.v.x, o.btr2 = bt2.v.y;
  o.inv_sl = inv_ssm.v.x, o.inv_sr = inv_ssm.v.y;
  // (written so that a NaN, a zero denominator, also under a negative pressure, and a side without
  // a star state are redone too)
  const float extent = fabsf(inv_ssm.v.x) + fabsf(inv_ssm.v.y) + fabsf(o.sm.v);
  if (!any(!(labs(den) > labs(F2(kNearDegenerate32) * (pt2 + F2(bn2.v))))) && extent < INFINITY) return;
  double Ld[7], Rd[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    Ld[c] = L[c];
    Rd[c] = Rt[c];
  }
  HlldFront<double> d;
  hlld_front<double, MathRefined>(Ld, Rd, double(bn), double(gamma), d);
  o.sl = float(d.sl), o.sr = float(d.sr), o.ptl = float(d.ptl), o.ptr = float(d.ptr);
  o.sm = float(d.sm), o.pts = float(d.pts);
  o.rsl = float(d.rsl), o.vtl1 = float(d.vtl1), o.vtl2 = float(d.vtl2);
  o.btl1 = float(d.btl1), o.btl2 = float(d.btl2), o.inv_sl = linv(o.sl - o.sm);
  o.rsr = float(d.rsr), o.vtr1 = float(d.vtr1), o.vtr2 = float(d.vtr2);
  o.btr1 = float(d.btr1), o.btr2 = float(d.btr2), o.inv_sr = linv(o.sr - o.sm);
  // The tail multiplies what takes no part by zero, so that must be finite: the star states of a
  // supersonic face (cold gas whose fast speed vanishes in the rounding of its velocity has
  // S = S_M and none) and the star density of the side the face does not lie on. Here, in the
  // branch that is rare, and not by a test in the tail: a step of 150 x 97 x 75 mixed 1.046 ms
  // without either, 1.052 with the test, 1.038 here; 256^3 float32 4.03, 4.01 and 3.97.
  const L1 most(3.0e38f);
  o.rsl = lmin(o.rsl, most);
  o.rsr = lmin(o.rsr, most);
  if (o.sl >= L1(0.0f) || o.sr < L1(0.0f)) {
    o.sm = sel(o.sm >= L1(0.0f), L1(1.0f), L1(-1.0f));
    o.rsl = o.rsr = L1(1.0f);
    o.pts = o.inv_sl = o.inv_sr = L1(0.0f);
    o.vtl1 = o.vtl2 = o.btl1 = o.btl2 = o.vtr1 = o.vtr2 = o.btr1 = o.btr2 = L1(0.0f);
  }
}

// The back half of the HLLD flux from its front (straight-line code: the star / double-star
// flux of the side of the contact the face lies on; as hlld_flux in numerics.cuh).
template <typename V>
__device__ __forceinline__ void hlld_tail_l(const V (&L)[7], const V (&Rt)[7], V bn, V inv_gm1,
                                            const HlldFrontL<V>& fr, V (&F)[7]) {
  const V sm = fr.sm;
  const V sql = lsqrt(fr.rsl);
  const V sqr = lsqrt(fr.rsr);
  // the sign of B_n; where it is zero the Alfven waves lie on the contact, and the
  // double-star state, its only use, is not taken
  const V sign = lcopysign(V(1.0f), bn);
  const V inv_sum = linv(sql + sqr);
  const V vt2_1 = fma(sql, fr.vtl1, fma(sqr, fr.vtr1, (fr.btr1 - fr.btl1) * sign)) * inv_sum;
  const V vt2_2 = fma(sql, fr.vtl2, fma(sqr, fr.vtr2, (fr.btr2 - fr.btl2) * sign)) * inv_sum;
  const V cross = sql * sqr * sign;
  const V bt2_1 = fma(sql, fr.btr1, fma(sqr, fr.btl1, cross * (fr.vtr1 - fr.vtl1))) * inv_sum;
  const V bt2_2 = fma(sql, fr.btr2, fma(sqr, fr.btl2, cross * (fr.vtr2 - fr.vtl2))) * inv_sum;
  const V vb2 = fma(sm, bn, fma(vt2_1, bt2_1, vt2_2 * bt2_2));
  // the side of the contact the face lies on (also the upwind side when supersonic)
  const auto left = sm >= V(0.0f);
  V w[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) w[c] = sel(left, L[c], Rt[c]);
  const V s = sel(left, fr.sl, fr.sr);
  const V pt = sel(left, fr.ptl, fr.ptr);
  const V rho_s = sel(left, fr.rsl, fr.rsr);
  const V vt1 = sel(left, fr.vtl1, fr.vtr1);
  const V vt2 = sel(left, fr.vtl2, fr.vtr2);
  const V bt1 = sel(left, fr.btl1, fr.btr1);
  const V bt2 = sel(left, fr.btl2, fr.btr2);
  const V sq = sel(left, sql, sqr);
  const V alfven = labs(bn) * linv(sq);
  const V ss = sel(left, sm - alfven, sm + alfven);
  const auto twice = left ^ (ss >= V(0.0f));
  const auto supersonic = fr.sl >= V(0.0f) | fr.sr < V(0.0f);
  const V sense = sel(left, V(-1.0f), V(1.0f));
  const V nbn = lneg(bn);
  V u[7], f[7];
  side_state_l(w, bn, nbn, inv_gm1, u, f);
  const V vn = w[1];
  const V vb = fma(vn, bn, fma(w[2], w[5], w[3] * w[6]));
  const V vb_s = fma(sm, bn, fma(vt1, bt1, vt2 * bt2));
  const V energy_s =
      fma(s - vn, u[4], fma(fr.pts, sm, fma(bn, vb - vb_s, lneg(pt) * vn))) * sel(left, fr.inv_sl, fr.inv_sr);
  V us[7], ud[7];
  us[0] = rho_s;
  us[1] = rho_s * sm;
  us[2] = rho_s * vt1;
  us[3] = rho_s * vt2;
  us[4] = energy_s;
  us[5] = bt1;
  us[6] = bt2;
  ud[2] = rho_s * vt2_1;
  ud[3] = rho_s * vt2_2;
  ud[4] = fma(sense * sq * sign, vb_s - vb2, energy_s);
  ud[5] = bt2_1;
  ud[6] = bt2_2;
  // f + S (U* - U) + S* (U** - U*), a wave speed the face lies outside of counting as zero.
  // (the front keeps every state that takes no part finite: zero times it is zero)
  const V first = sel(supersonic, V(0.0f), s);
  const V second = sel(!supersonic & twice, ss, V(0.0f));
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    const V star = fma(first, us[c] - u[c], f[c]);
    // the double-star state differs from the star state in rows 2-6 only
    F[c] = c < 2 ? star : fma(second, ud[c] - us[c], star);
  }
}

// ---- float32 entry points of the kernels: one face (L1) ------------------------------------
template <typename V, int N>
__device__ __forceinline__ void to_lanes(const float (&a)[N], V (&b)[N]) {
#pragma unroll
  for (int c = 0; c < N; ++c) b[c] = V(a[c]);
}

template <int N>
__device__ __forceinline__ void from_lanes(const L1 (&a)[N], float (&b)[N]) {
#pragma unroll
  for (int c = 0; c < N; ++c) b[c] = a[c].v;
}

// The float32 HLLD flux of one face: front on the packed lanes, back half on one lane.
__device__ __forceinline__ void hlld_flux(const float (&L)[7], const float (&Rt)[7], float bn, float gamma,
                                          float inv_gm1, float (&F)[7]) {
  HlldFrontL<L1> fr;
  hlld_front_lr(L, Rt, bn, gamma, fr);
  L1 l[7], r[7], f[7];
  to_lanes(L, l);
  to_lanes(Rt, r);
  hlld_tail_l<L1>(l, r, L1(bn), L1(inv_gm1), fr, f);
  from_lanes(f, F);
}

// The left / right states q +- h of a face from the two cells beside it and their half
// slopes, (left, right) on the two lanes of F2. Where a density or pressure is not positive
// the face falls back to first order: its slopes count with the factor `keep` = 0.
__device__ __forceinline__ void face_states(const F2 (&q)[7], const F2 (&h)[7], float (&L)[7], float (&Rt)[7]) {
  const F2 one(1.0f, -1.0f);
  const F2 rho = fma(one, h[0], q[0]), p = fma(one, h[4], q[4]);
  const float least = fminf(fminf(rho.v.x, rho.v.y), fminf(p.v.x, p.v.y));
  const float keep = least > 0.0f ? 1.0f : 0.0f;
  const F2 factor(keep, -keep);
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    const F2 lr = fma(factor, h[c], q[c]);
    L[c] = lr.v.x;
    Rt[c] = lr.v.y;
  }
}

// One face's reconstruction with its left and right states in the two lanes of F2: the
// two limited slopes of each component in one packed evaluation (lane x: the cell below the
// face, lane y: the cell above), the states as one packed FMA. Lane by lane the same
// operations as the one-lane form.
template <int LIM>
__device__ __forceinline__ void reconstruct(const float (&q0)[7], const float (&q1)[7], const float (&q2)[7],
                                            const float (&q3)[7], float (&L)[7], float (&Rt)[7]) {
  F2 q[7], h[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    const F2 a01(q0[c], q1[c]), a12(q1[c], q2[c]), a23(q2[c], q3[c]);
    q[c] = a12;
    h[c] = half_slope_l<LIM>(a12 - a01, a23 - a12);
  }
  face_states(q, h, L, Rt);
}

// The same from half slopes already formed (h1 of q1, h2 of q2).
__device__ __forceinline__ void reconstruct_halves(const float (&q1)[7], const float (&q2)[7], const float (&h1)[7],
                                                   const float (&h2)[7], float (&L)[7], float (&Rt)[7]) {
  F2 q[7], h[7];
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    q[c] = F2(q1[c], q2[c]);
    h[c] = F2(h1[c], h2[c]);
  }
  face_states(q, h, L, Rt);
}

// Half slopes of seven components from their backward (a) and forward (b) differences, two
// components per packed evaluation (lane by lane as half_slope_l<L1>).
template <int LIM>
__device__ __forceinline__ void half_slopes7(const float (&a)[7], const float (&b)[7], float (&out)[7]) {
#pragma unroll
  for (int c = 0; c < 6; c += 2) {
    const F2 s = half_slope_l<LIM>(F2(a[c], a[c + 1]), F2(b[c], b[c + 1]));
    out[c] = s.v.x;
    out[c + 1] = s.v.y;
  }
  out[6] = half_slope_l<LIM>(L1(a[6]), L1(b[6])).v;
}

template <int LIM>
__device__ __forceinline__ float limited_slope(float a, float b) {
  return 2.0f * half_slope_l<LIM>(L1(a), L1(b)).v;
}

}  // namespace wb
