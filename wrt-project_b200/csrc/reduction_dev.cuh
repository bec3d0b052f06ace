// reduction_dev.cuh -- positions along a line of the staged reduction
// (k_reduction.cu).  Plain scalar code, compiled by host programs too (PROF_FN,
// profile_dev.cuh).
#pragma once
#include "profile_dev.cuh"

namespace wrtr {

using wrtp::prof_add;
using wrtp::prof_mul;
using wrtp::prof_sub;

// Whether sample k of a line belongs to it (radon_reduction/slicing.c:105-110).
PROF_FN bool on_line(int k, double dtau, double p, double ct, double st) {
  const double tau = prof_mul((double)k, dtau);
  const double z = prof_add(prof_mul(p, ct), prof_mul(tau, st));
  const double s = prof_sub(prof_mul(p, st), prof_mul(tau, ct));
  return !(fabs(prof_add(prof_mul(tau, tau), prof_mul(p, p))) > 1.0) && !(fabs(z) > 1.0) &&
         !(fabs(s) > 1.0);
}

// Samples of a line: [*klo, *khi].
PROF_FN void line_range(int ngrid, double dtau, double p, double ct, double st, int *klo, int *khi) {
  const double r = 1.0 - p * p;
  *khi = -1;
  if (r >= 0.0) *khi = wrtp::imin(2 * ngrid, (int)floor(sqrt(r) / dtau) + 1);
  *klo = -*khi;
  while (*khi >= *klo && !on_line(*khi, dtau, p, ct, st)) --*khi;
  while (*klo <= *khi && !on_line(*klo, dtau, p, ct, st)) ++*klo;
}

// Layer and knot positions of a line's samples in 16.48 fixed point, advanced by one
// addition each.  2^-24 above the exact ones: the fraction, cut to 23 bits, is then
// centred, and a position just below 0 does not leave the first cell.  The steps'
// rounding adds up to at most (2 ngrid + 1) 2^-49 (8200 samples: 2^-36) on top of the
// start's FP64 rounding, far below that.
struct LinePos {
  long long z, s, dz, ds;
};
PROF_FN long long fixed48(double x) {
#ifdef __CUDACC__
  return __double2ll_rn(x * 281474976710656.0);
#else
  return llrint(x * 281474976710656.0);
#endif
}
PROF_FN LinePos line_pos(int ngrid, int ns, double dtau, double p, double ct, double st, int k) {
  const double per_z = 0.5 * (ngrid - 1), per_s = 0.5 * (ns - 1);
  const double tau = (double)k * dtau;
  LinePos l;
  l.z = fixed48((p * ct + tau * st + 1.0) * per_z + 0x1p-24);
  l.s = fixed48((p * st - tau * ct + 1.0) * per_s + 0x1p-24);
  l.dz = fixed48(dtau * st * per_z);
  l.ds = fixed48(-dtau * ct * per_s);
  return l;
}
PROF_FN int cell_of(long long q) { return (int)(q >> 48); }
// The upper 23 bits of the fraction, as the mantissa of a float in [1, 2).
PROF_FN unsigned one_plus_fraction(long long q) {
  return 0x3f800000u | ((unsigned)(q >> 25) & 0x7fffffu);
}

}  // namespace wrtr
