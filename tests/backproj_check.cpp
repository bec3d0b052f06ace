// Host check of the merged backprojection's geometry (csrc/backproj_dev.cuh): the
// pieces of H(t) = sum_theta S_theta(sin theta t + cos theta z), summed up as the
// build kernel sums them, against the splines themselves at random t; the
// interval at a range's start against the knots counted one by one.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../wrt-project_b200/csrc/backproj_dev.cuh"

using namespace wrtb;

static int fail(const char *what, double a, double b) {
  std::printf("FAILED %s: %.17g %.17g\n", what, a, b);
  return 1;
}

struct Knot {
  unsigned pos, id;
};

static int check(int nt, int ns, double z, int nsub_log2, unsigned seed) {
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> N;
  std::vector<std::vector<double>> y(nt), m(nt);
  std::vector<double> ct(nt), st(nt);
  for (int th = 0; th < nt; ++th) {
    const double a = 3.14159265358979 * (th + 0.5) / nt;
    ct[th] = std::cos(a);
    st[th] = std::sin(a);
    y[th].resize(ns);
    m[th].assign(ns, 0.0);
    for (double &v : y[th]) v = N(rng);
    std::vector<double> cp(ns, 0.0);
    for (int i = 1; i + 1 < ns; ++i) {
      cp[i] = 1.0 / (4.0 - (i > 1 ? cp[i - 1] : 0.0));
      m[th][i] = ((y[th][i + 1] - 2 * y[th][i] + y[th][i - 1]) - (i > 1 ? m[th][i - 1] : 0.0)) * cp[i];
    }
    for (int i = ns - 3; i >= 1; --i) m[th][i] -= cp[i] * m[th][i + 1];
  }
  auto cubic = [&](int th, int i, double b, double *c) {  // about b, in knots
    const double y0 = y[th][i], y1 = y[th][i + 1], m0 = m[th][i], m1 = m[th][i + 1];
    const double A = (y1 - y0) - (2 * m0 + m1), B = 3 * m0, C = m1 - m0;
    c[0] = y0 + b * (A + b * (B + b * C));
    c[1] = A + b * (2 * B + 3 * b * C);
    c[2] = B + 3 * b * C;
    c[3] = C;
  };
  std::vector<Knot> k;
  for (int th = 0; th < nt; ++th) {
    const Lat l = lat_of(ct[th], st[th], z, ns);
    int lo, hi, listed = 0, all = 0;
    knot_range(l, ns, &lo, &hi);
    for (int i = 0; i < ns; ++i) {
      const long long p = knot_pos(l, i);
      const bool in = p >= 0 && p < 0x100000000LL;
      all += in;
      if (i < lo || i > hi || !in) continue;
      ++listed;
      k.push_back({(unsigned)p, (unsigned)(th * ns + i) + 1u});
    }
    if (listed != all) return fail("knots in range", listed, all);
  }
  const int nsub = 1 << nsub_log2, shift = 32 - nsub_log2;
  for (int s = 0; s < nsub; ++s) k.push_back({(unsigned)((unsigned long long)s << shift), 0u});
  std::sort(k.begin(), k.end(), [](const Knot &a, const Knot &b) {
    return a.pos != b.pos ? a.pos < b.pos : a.id < b.id;
  });
  std::vector<double> c(4 * k.size());
  double a[4] = {0, 0, 0, 0};
  for (size_t e = 0; e < k.size(); ++e) {
    const unsigned sub = nsub_log2 ? k[e].pos >> shift : 0;
    const long long p0 = (long long)sub << shift;
    double tau = 0.0;
    if (k[e].id) {
      const int th = (k[e].id - 1) / ns, i = (k[e].id - 1) % ns;
      tau = knot_tau(lat_of(ct[th], st[th], z, ns), i, p0);
    }
    if (k[e].id == 0) {  // a new range: from the lines
      a[0] = a[1] = a[2] = a[3] = 0.0;
      const double t0 = (double)p0 / kPerT - kTMax;
      for (int th = 0; th < nt; ++th) {
        const Lat l = lat_of(ct[th], st[th], z, ns);
        const int before = knots_before(l, ns, p0);
        int count = 0;
        for (int i = 0; i < ns; ++i) count += knot_pos(l, i) < p0;
        if (count != before) return fail("knots before", before, count);
        const int i = before - 1;
        if (i < 0 || i > ns - 2) continue;
        double q[4], f = 1;
        cubic(th, i, l.kap * t0 + l.q0 - i, q);
        for (int d = 0; d < 4; ++d, f *= l.kap) a[d] += f * q[d];
      }
    } else {
      const int th = (k[e].id - 1) / ns, i = (k[e].id - 1) % ns;
      const Lat l = lat_of(ct[th], st[th], z, ns);
      const double k3 = l.kap * l.kap * l.kap;
      const std::vector<double> &mm = m[th], &yy = y[th];
      double d = i == 0 ? mm[1] - mm[0] : i == ns - 1 ? -(mm[ns - 1] - mm[ns - 2])
                                                      : (mm[i + 1] - mm[i]) - (mm[i] - mm[i - 1]);
      d *= k3;
      if (i == 0 || i == ns - 1) {
        const double v = i ? -yy[i] : yy[0];
        const double sl = i ? -l.kap * ((yy[i] - yy[i - 1]) + mm[i - 1])
                            : l.kap * ((yy[1] - yy[0]) - mm[1]);
        a[0] += v - sl * tau;
        a[1] += sl;
      }
      a[3] += d;
      a[2] -= 3 * d * tau;
      a[1] += 3 * d * tau * tau;
      a[0] -= d * tau * tau * tau;
    }
    c[4 * e] = a[0] + tau * (a[1] + tau * (a[2] + tau * a[3]));
    c[4 * e + 1] = a[1] + tau * (2 * a[2] + 3 * tau * a[3]);
    c[4 * e + 2] = a[2] + 3 * tau * a[3];
    c[4 * e + 3] = a[3];
  }
  double worst = 0;
  for (int q = 0; q < 4000; ++q) {
    const double t = 1.41421 * (2.0 * (rng() % 1000003) / 1000003.0 - 1.0);
    const unsigned fx = (unsigned)std::floor(t * kPerT + kTMax * kPerT);
    const size_t e = std::upper_bound(k.begin(), k.end(), fx, [](unsigned v, const Knot &b) {
                       return v < b.pos;
                     }) - k.begin();
    if (!e) return fail("no piece before", fx, 0);
    if (fx - k[e - 1].pos <= 2 || (e < k.size() && k[e].pos - fx <= 2)) continue;
    const double d = (double)(fx - k[e - 1].pos) / kPerT;
    const double *p = &c[4 * (e - 1)];
    const double got = p[0] + d * (p[1] + d * (p[2] + d * p[3]));
    double ref = 0;
    for (int th = 0; th < nt; ++th) {
      const Lat l = lat_of(ct[th], st[th], z, ns);
      const double qq = l.kap * t + l.q0;
      if (qq < 0 || qq > ns - 1) continue;
      const int i = std::min((int)qq, ns - 2);
      double v[4];
      cubic(th, i, qq - i, v);
      ref += v[0];
    }
    worst = std::max(worst, std::fabs(got - ref));
  }
  // positions are floored to 1 / kPerT (7e-10), at most 1.3e-7 knots here, and the
  // slope is a few per knot and line: 1e-6 sqrt(nt); the FP64 cubics about a
  // range's start lose (knots per range)^3 roundings
  const double span = 2 * kTMax * 0.5 * (ns - 1) / nsub;
  if (!(worst <= 1e-6 * std::sqrt((double)nt) + 1e-14 * span * span * span * std::sqrt((double)nt * ns))) return fail("H(t)", worst, nt);
  return 0;
}

int main() {
  int bad = 0;
  for (int nt : {1, 2, 7, 32, 96})
    for (int ns : {3, 5, 64, 257, 384})
      for (double z : {0.0, -0.96875, 0.4375, 0.998})
        for (int lg : {0, 3, 6}) bad += check(nt, ns, z, lg, 31 * nt + ns);
  std::printf(bad ? "%d checks failed\n" : "ok\n", bad);
  return bad != 0;
}
