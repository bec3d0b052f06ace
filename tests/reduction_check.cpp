// Host check of the staged reduction's positions (csrc/reduction_dev.cuh): on every
// sample of a line the layer and the knot are within the staged arrays and the
// position is within 2^-23 of the exact one, however many layers the line crosses
// (the kernel reads shared memory at the cell without a check).
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "../wrt-project_b200/csrc/reduction_dev.cuh"

using namespace wrtr;

static int check(int ngrid, int ns, int ntheta, int nshift) {
  const double dtau = (2.0 / (ngrid - 1)) / (2.0);
  double worst = 0.0;
  long long samples = 0;
  for (int it = 0; it < ntheta; ++it) {
    // latitudes from pole to pole, the axis and pi/2 among them
    const double th = M_PI * it / (ntheta - 1), ct = cos(th), st = sin(th);
    for (int is0 = 0; is0 < nshift; is0 += 32) {
      int k0 = 1 << 30;  // a warp's lanes share the first sample
      for (int is = is0; is < std::min(nshift, is0 + 32); ++is) {
        int lo, hi;
        line_range(ngrid, dtau, -1.0 + is * (2.0 / (nshift - 1)), ct, st, &lo, &hi);
        k0 = std::min(k0, lo);
      }
      for (int is = is0; is < std::min(nshift, is0 + 32); ++is) {
        const double p = -1.0 + is * (2.0 / (nshift - 1));
        int lo, hi;
        line_range(ngrid, dtau, p, ct, st, &lo, &hi);
        LinePos at = line_pos(ngrid, ns, dtau, p, ct, st, k0);
        for (int k = k0; k <= hi; ++k, at.z += at.dz, at.s += at.ds) {
          if (k < lo) continue;
          const int iz = cell_of(at.z), i = cell_of(at.s);
          if (iz < 0 || iz > ngrid - 1 || i < 0 || i > ns - 1) {
            std::printf("FAILED: %d layers, %d knots, theta %g, shift %g, sample %d: cell %d, %d\n",
                        ngrid, ns, th, p, k, iz, i);
            return 1;
          }
          const long double tau = (long double)k * dtau;
          const long double z = ((long double)p * ct + tau * st + 1) * (ngrid - 1) / 2;
          const long double s = ((long double)p * st - tau * ct + 1) * (ns - 1) / 2;
          const double fz = (one_plus_fraction(at.z) - 0x3f800000u) * 0x1p-23,
                       fs = (one_plus_fraction(at.s) - 0x3f800000u) * 0x1p-23;
          worst = std::max(worst, (double)fabsl(iz + (long double)fz - z));
          worst = std::max(worst, (double)fabsl(i + (long double)fs - s));
          ++samples;
        }
      }
    }
  }
  if (!samples || worst > 0x1p-23) {
    std::printf("FAILED: %d layers, %d knots: %lld samples, off by %g\n", ngrid, ns, samples, worst);
    return 1;
  }
  return 0;
}

int main() {
  int bad = 0;
  for (int ngrid : {3, 4, 33, 128, 200, 255, 256, 300, 511, 1000, 2000, 4096, 5700})
    bad += check(ngrid, std::max(3, std::min(128, 28000 / ngrid - 2)), 33, 70);
  for (int ns : {300, 2000, 5700}) bad += check(3, ns, 17, 65), bad += check(4, ns, 16, 64);
  if (bad) std::printf("%d checks failed\n", bad);
  else std::printf("ok\n");
  return bad != 0;
}
