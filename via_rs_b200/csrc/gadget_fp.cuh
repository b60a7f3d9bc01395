// Gadget decomposition in double precision (gadget.cuh restated on exact integer doubles,
// ntt_fp.cuh): for odd moduli and S = B^L < 2^47.
//
// The scaled value is the nearest integer v to c S / Q (there are no ties: Q is odd), and
// its balanced digits only depend on v mod S, so any representative of the coefficient c
// and any v congruent to the scaled value will do.
#pragma once
#include "gadget.cuh"
#include "ntt_fp.cuh"

namespace via {

// One limb, Q S < 8/9 2^53 (a small gadget), |r| <= 9/16 Q: r S is exact, and its product with the
// rounded 1 / Q, within 2^-53 of it in proportion, errs by less than 9/16 S 2^-53 < 1 / (2 Q), its
// distance from a tie. (Not so up to 2^53: Q = 34347294721, S = 509^2, r = 0.537 Q misses.)
__device__ __forceinline__ double fp_scaled(double r, double S, double qinv) {
  return __dadd_rn(__fma_rn(__dmul_rn(r, S), qinv, FP_ROUND), -FP_ROUND);
}

// round((r0 q1 + r1 q0) / Q) for remainders whose quotient lies within 1e-12 of a tie, where
// doubles cannot tell (probability 2^-38; out of line to keep the callers' code small).
static __device__ __noinline__ int fp_round_exact(double r0, double r1, u64 q0, u64 q1) {
  const i128 num = (i128)(i64)r0 * (i128)q1 + (i128)(i64)r1 * (i128)q0;
  const i128 Q = (i128)q0 * q1;
  return 2 * num > Q ? 1 : (2 * num < -Q ? -1 : 0);
}

// Two limbs: c / Q = y0 / q0 + y1 / q1 mod 1 with y_l = c_l (Q / q_l)^-1 mod q_l, and
// S y_l = p_l q_l + r_l exactly. v = p0 + p1 + round(r0 / q0 + r1 / q1).
__device__ __forceinline__ double fp_scaled2(double c0, double c1, const Gadget& g, const DevRing& R) {
  const double q0 = R.t[0].qd, q1 = R.t[1].qd, i0 = R.t[0].qinv, i1 = R.t[1].qinv;
  const double y0 = fp_mulmod(c0, g.ys[0], q0, i0), y1 = fp_mulmod(c1, g.ys[1], q1, i1);
  const double h0 = __dmul_rn(g.dS, y0), h1 = __dmul_rn(g.dS, y1);
  const double l0 = __fma_rn(g.dS, y0, -h0), l1 = __fma_rn(g.dS, y1, -h1);
  const double p0 = __dadd_rn(__fma_rn(h0, i0, FP_ROUND), -FP_ROUND);
  const double p1 = __dadd_rn(__fma_rn(h1, i1, FP_ROUND), -FP_ROUND);
  const double r0 = __dadd_rn(__fma_rn(-p0, q0, h0), l0), r1 = __dadd_rn(__fma_rn(-p1, q1, h1), l1);
  const double s = __fma_rn(r0, i0, __dmul_rn(r1, i1));
  double rnd = __dadd_rn(__dadd_rn(s, FP_ROUND), -FP_ROUND);
  if (fabs(__dadd_rn(s, -rnd)) > 0.5 - 1e-12) rnd = (double)fp_round_exact(r0, r1, R.m[0].q, R.m[1].q);
  return __dadd_rn(__dadd_rn(p0, p1), rnd);
}

// The next balanced digit of v, least significant first, |v| < 2^50: v = d + B v' with
// -B / 2 < d <= B / 2 (an even B's half stays positive: the quarter decides that tie and
// moves no other quotient across one).
__device__ __forceinline__ double fp_next_digit(double& v, const Gadget& g) {
  const double t = __dadd_rn(__fma_rn(__dadd_rn(v, -0.25), g.dBinv, FP_ROUND), -FP_ROUND);
  const double d = __fma_rn(-g.dB, t, v);
  v = t;
  return d;
}

}  // namespace via
