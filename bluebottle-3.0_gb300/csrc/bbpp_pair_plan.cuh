// bbpp_pair_plan.cuh -- the steps that a pair of FP32 iterations takes (bbpp_pair.cu).
#pragma once

#include "bbpp_dev.cuh"

namespace bbpp {
// A pair's steps from the products of its start; d: (r,z), (r,r) - (r,z), (p,w),
// (z,w), (q,w), (z,s), (z,t), (q,t), (s,s'), (s,t'), (t,t') with ' = / dL.  Symmetry
// of L gives the others: (q,s) = (z,t), (p,s) = (z,w), (p,t) = (q,w).
struct PairPlan {
  double a0, b0, a1, b1;
  int steps;   // 1 or 2
  bool anew;   // this pair's search direction is z, not p
  bool fresh;  // the next pair's is
  double rz;   // (r,z) after the steps, by the expansions
};
// The products are FP32 sums (relative errors of some 1e-6), so an expansion is
// known to that part of its largest term: what a step leaves, (r,z) after it, has
// no digits where a step takes nearly all of the residual (a right-hand side of few
// eigenvectors, a mask of isolated cells), and 0 / 0 follows where it takes all.
//   A second step is taken only where each of the two leaves 2^-kStepKeeps of (r,z);
//   else one step, and the next pair's exact sums decide.
//   One step must leave 2^-kBetaKeeps for beta to be used; else p = z next.
//   The exact (r,z) of a pair's start lies within a tenth of what the pair before
//   expected; else p is conjugate to nothing, and this pair takes one step along z
//   (whose products are among the eleven: w = s, q = s / dL).
// Solves of spectral and uniform right-hand sides with 0 to 80% solid cells expect
// (r,z) to 1e-5 or better and take two steps throughout (numpy model at 64^3).
// The tests read high words and a restart selects its products: one thread works here at
// the end of every dots kernel, and an FP64 instruction, taken or not, costs it 16 cycles
// and more (with FP64 compares and a branch of its own for the restart 2 us a pair).
constexpr int kStepKeeps = 5;

__host__ __device__ inline PairPlan pair_plan(const double *d, bool fresh, double expected) {
  const double rz = d[0], zs = d[5], zt = d[6], qt = d[7], ss = d[8], st = d[9], tt = d[10];
  const bool restart = !fresh && !(alike(rz, expected) && hi_word(d[2]) > 0);
  const double pw = restart ? zs : d[2], zw = restart ? zs : d[3], qw = restart ? ss : d[4];
  PairPlan o;
  o.a0 = rz / pw;
  const double a0 = o.a0, rz1 = rz - 2.0 * a0 * zw + a0 * a0 * qw, b0 = rz1 / rz;
  // p1 = z - a0 q + b0 p, w1 = L p1 = s - a0 t + b0 w (not for a restart)
  const double zw1 = zs - 2.0 * a0 * zt + a0 * a0 * qt + b0 * (zw - a0 * qw);  // (z1, w1)
  const double pw1 = zw1 + b0 * (zw - a0 * qw + b0 * pw);                      // (p1, w1)
  const double ww1 = ss + a0 * a0 * tt + b0 * b0 * qw - 2.0 * a0 * st + 2.0 * b0 * (zt - a0 * qt);  // (w1, w1 / dL)
  o.a1 = rz1 / pw1;
  const double rz2 = rz1 - 2.0 * o.a1 * zw1 + o.a1 * o.a1 * ww1;
  o.b1 = rz2 / rz1;
  const bool two = !restart && keeps(rz1, rz, kStepKeeps) && hi_word(pw1) > 0 && keeps(rz2, rz1, kStepKeeps);
  o.steps = two ? 2 : 1;
  o.rz = two ? rz2 : rz1;
  o.fresh = !keeps(rz1, rz, kBetaKeeps);
  o.b0 = o.fresh ? 0.0 : b0;
  o.anew = fresh || restart;
  return o;
}
}  // namespace bbpp
