// Host check of which unit of t reads a row of the row-sum profiles
// (csrc/profile_dev.cuh): every row lies in exactly one, also where its t is within
// rounding of the border of two (theta = pi/2: all rows of a plane have one t, and at
// many sizes that is a border), and the piece boundaries listed beyond a unit's ends
// are those of its neighbours.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <tuple>
#include <vector>

#include "../wrt-project_b200/csrc/profile_dev.cuh"

using namespace wrtp;

// radon_grid/src/integral.c:10-36, the expressions of the library's direction table
static void direction(double p, double t, double *D) {
  const double nx = sin(t) * cos(p), ny = sin(t) * sin(p), nz = cos(t);
  const double t2 = t + M_PI / 2;
  const double ax = sin(t2) * cos(p), ay = sin(t2) * sin(p), az = cos(t2);
  const double d[9] = {nx, ny, nz, ax, ay, az, ny * az - nz * ay, -(nx * az - nz * ax),
                       nx * ay - ny * ax};
  for (int k = 0; k < 9; ++k) D[k] = d[k];
}

static long long on_border = 0;  // rows within 1e-9 bins of a border

static int rows(int n, bool near, int nshift, int nphi) {
  const double toff = prof_t_off(n, near);
  const int chunks = (int)floor(2 * toff * n / kUnitBins) + 1;
  const double thetas[] = {M_PI / 2, acos(0.0) * 1.0000000000000002, 1.1, 0.3};
  for (int ip = 0; ip < nphi; ++ip) {
    const double phi = 2 * M_PI / nphi * ip;
    for (double theta : thetas) {
      double D[9], B[9];
      direction(phi, theta, D);
      direction(phi, M_PI / 2, B);  // the unit's u: (cos phi, sin phi)
      for (int is = 0; is < nshift; ++is) {
        const double s = -1.0 + is * (2.0 / (nshift - 1));
        for (int i = -n; i < n; ++i) {
          if (s * s + (double)i * i / ((double)n * n) > 1.9) continue;
          int units = 0;
          for (int c = 0; c < chunks; ++c) {
            const Geo g = make_geo(n, near, n, B[7], -B[6], 3.00001, c);
            const RowGeo q = row_geo(D, g);
            const double u = fma((double)i, q.u1, fma(s, q.ub, q.uo));
            if (fabs(u - g.tfirst) < 1e-9) ++on_border;
            // (the kernel looks at rows up to half an edge of bins beyond the ends)
            if (u - g.tfirst > -n && u - g.tfirst < kUnitBins + n)
              units += row_pos(u, g.tfirst) < kUnitEnd;
          }
          if (units != 1) {
            std::printf("FAILED: n %d near %d nshift %d phi %g theta %g s %g row %d in %d units\n",
                        n, near, nshift, phi, theta, s, i, units);
            return 1;
          }
        }
      }
    }
  }
  return 0;
}

static long long listed = 0;

static int ends(int n, bool near, double phi) {
  typedef std::tuple<int, int, int> Id;
  const double toff = prof_t_off(n, near);
  const int chunks = (int)floor(2 * toff * n / kUnitBins) + 1;
  std::vector<Id> last, after;  // of the unit before: next to its end, and beyond it
  for (int c = 0; c < chunks; ++c) {
    const Geo g = make_geo(n, near, 2 * n, cos(phi), sin(phi), 3.00001, c);
    std::vector<Id> first, before, mine, beyond;
    each_boundary(
        g, 0, n, 0, 1,
        [&](unsigned p, int kind, int li, int m) {
          if (p < kBoundary) first.push_back(Id(kind, li, m));
          if (p >= kUnitEnd - kBoundary) mine.push_back(Id(kind, li, m));
        },
        [&](bool a, int kind, int li, int m) { (a ? beyond : before).push_back(Id(kind, li, m)); });
    for (auto *v : {&first, &before, &mine, &beyond}) std::sort(v->begin(), v->end());
    if (c && (after != first || before != last)) {
      std::printf("FAILED: n %d near %d phi %g unit %d: %zu/%zu beyond the end, %zu/%zu before\n",
                  n, near, phi, c, after.size(), first.size(), before.size(), last.size());
      return 1;
    }
    listed += (long long)(beyond.size() + before.size());
    last = mine;
    after = beyond;
  }
  return 0;
}

int main() {
  int bad = 0;
  const int sizes[][3] = {{64, 0, 127}, {64, 1, 65}, {64, 1, 129}, {128, 0, 255}, {128, 1, 129},
                          {96, 0, 191}, {41, 0, 21}, {24, 1, 25}};
  for (auto &z : sizes) bad += rows(z[0], z[1] != 0, z[2], 12);
  for (int n : {24, 64, 65, 128})
    for (bool near : {false, true})
      for (double phi : {0.0, M_PI / 2, M_PI / 4, 0.7, M_PI, 1e-10}) bad += ends(n, near, phi);
  if (!on_border || !listed) {
    std::printf("FAILED: %lld rows on a border, %lld boundaries beyond an end\n", on_border, listed);
    bad = 1;
  }
  if (bad) std::printf("%d checks failed\n", bad);
  else std::printf("ok %lld %lld\n", on_border, listed);
  return bad != 0;
}
