// backproj_dev.cuh -- geometry of the merged backprojection (k_backproj.cu): where
// the knots of every latitude's spline fall along t for one z.  Plain scalar
// code, compiled by host programs too (PROF_FN, profile_dev.cuh).
#pragma once
#include "profile_dev.cuh"

namespace wrtb {

using wrtp::imax;
using wrtp::imin;

// t in [-kTMax, kTMax] (|t| <= sqrt 2 in the cube) as 32-bit positions.
constexpr double kTMax = 1.4144;
constexpr double kPerT = 1.518e9;  // positions per unit t; 2 kTMax kPerT < 2^32

// One latitude at one z: knot coordinate q(t) = kap t + q0, knots 0 .. ns - 1.
struct Lat {
  double kap, q0;
};
PROF_FN Lat lat_of(double ct, double st, double z, int ns) {
  const double inv_h = 0.5 * (ns - 1);
  Lat l;
  l.kap = st * inv_h;
  l.q0 = (ct * z + 1.0) * inv_h;
  return l;
}
// Position of knot i (any value; outside [0, 2^32) it is off the range).
PROF_FN long long knot_pos(const Lat &l, int i) {
  return wrtp::prof_floor(
      wrtp::prof_mul(wrtp::prof_add(((double)i - l.q0) / l.kap, kTMax), kPerT));
}
// t of knot i from position p0, unrounded: the sums run over many knots, and an
// error in a knot's place grows with the square of the distance from it.
PROF_FN double knot_tau(const Lat &l, int i, long long p0) {
  return wrtp::prof_add(((double)i - l.q0) / l.kap, kTMax) - (double)p0 / kPerT;
}
// Knots that can lie on the range: [*lo, *hi].
PROF_FN void knot_range(const Lat &l, int ns, int *lo, int *hi) {
  const double a = l.q0 - kTMax * l.kap, b = l.q0 + kTMax * l.kap;
  *lo = imax(0, (int)fmax(floor(a), -2e9) - 1);
  *hi = imin(ns - 1, (int)fmin(ceil(b), 2e9) + 1);
}
// Number of knots whose position is below p: the interval at p is that - 1
// (-1: not yet on the line, ns - 1: past its end).
PROF_FN int knots_before(const Lat &l, int ns, long long p) {
  const double q = l.q0 + l.kap * ((double)p / kPerT - kTMax);
  int c = (int)fmin(fmax(ceil(q), 0.0), (double)ns);
  while (c < ns && knot_pos(l, c) < p) ++c;
  while (c > 0 && knot_pos(l, c - 1) >= p) --c;
  return c;
}

}  // namespace wrtb
