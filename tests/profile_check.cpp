// Host check of the row-sum profiles (csrc/profile_dev.cuh): the pieces of
// G_k(t) = sum_j f_k(t u + j delta v2), summed up as the build role sums them,
// against the sum itself at random t -- every phi class (axis, diagonal,
// generic), both samplers, lattices shorter and longer than the cube, volumes
// that are non-zero up to the cube's faces -- and every index against its
// array.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../wrt-project_b200/csrc/profile_dev.cuh"

using namespace wrtp;

struct Piece {
  unsigned pos;
  unsigned id;
  int kind, li, m;
};

static int fail(const char *what, double a, double b) {
  std::printf("FAILED %s: %.17g %.17g\n", what, a, b);
  return 1;
}

static int check(int n, bool near, int L, double phi, double crop, unsigned seed) {
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> N;
  const double cu = std::cos(phi), su = std::sin(phi);
  std::vector<float> f((size_t)n * n);  // one layer: f[ix][iy]
  const int W = near ? n : n - 1;
  for (int x = 0; x < n; ++x)
    for (int y = 0; y < n; ++y) {
      // the support the crop radius stands for (every node, for crop = 3)
      const double X = -1 + 2.0 * x / (n - 1), Y = -1 + 2.0 * y / (n - 1);
      const double reach = near ? std::sqrt(3.0) * (4.0 / n + 2.0 / (n - 1))
                                : std::sqrt(3.0) * 2.0 / (n - 1);
      const double r = std::sqrt(crop) - reach - 2e-6;
      f[(size_t)x * n + y] = crop >= 3 || X * X + Y * Y <= r * r ? (float)N(rng) : 0.0f;
    }
  const long long elems = (long long)n * n;  // columns
  const double toff = prof_t_off(n, near);
  const int chunks = (int)std::floor(2 * toff * n / kUnitBins) + 1;
  const int sub_bins = std::min(n, kUnitBins), nsub = (kUnitBins + sub_bins - 1) / sub_bins;
  auto node = [&](long long off, int d) {  // off: element offset of layer 0 (k = 0, stride n)
    const long long c = off / n + d;
    if (off % n || c < 0 || c >= elems) {
      std::printf("FAILED: column %lld of %lld\n", c, elems);
      std::exit(1);
    }
    return (double)f[c];
  };
  double worst = 0, size = 0;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const Geo g = make_geo(n, near, L, cu, su, crop, chunk);
    if (near && on_axis(g)) return 0;  // not tabulated
    std::vector<Piece> p;
    each_boundary(g, nsub, sub_bins, 0, 1, [&](unsigned pos, int kind, int li, int m) {
      if (pos >> 20 >= (unsigned)kUnitBins || li > 0xffff || m > 0x1fff) std::exit(2);
      p.push_back({pos, kind == K_NULL ? 0u : ((unsigned)kind << 29 | (unsigned)li << 13 | m) + 1,
                   kind, li, m});
    });
    if ((int)p.size() > unit_cap(n, crop)) return fail("capacity", p.size(), unit_cap(n, crop));
    std::sort(p.begin(), p.end(), [](const Piece &a, const Piece &b) {
      return a.pos != b.pos ? a.pos < b.pos : a.id < b.id;
    });
    std::vector<double> v(p.size()), s(p.size()), c(p.size());
    size_t e = 0;
    for (int sub = 0; sub < nsub; ++sub) {
      const double t0 = (g.tfirst + (double)sub * sub_bins) / n - g.toff;
      const long long b0 = (long long)sub * sub_bins << 20, b1 = (long long)(sub + 1) * sub_bins << 20;
      auto passed = [&](double t) { return pos_of(g, t) < b0; };
      double A0 = 0, A1 = 0, A2 = 0;
      for (int j = g.jlo; j <= g.jhi; ++j) {
        const Line l = make_line(g, j);
        if (!l.ok || !(t0 * t0 + l.jd * l.jd <= g.rc2 + 4 * std::sqrt(g.rc2) + 4) ||
            !passed(l.tin) || passed(l.tout))
          continue;
        const int ix = xcell(g, l.jd, t0, passed), iy = ycell(g, l.jd, t0, passed);
        const long long o = ((long long)ix * n + iy) * n;
        if (near) {
          A0 += node(o, 0);
          continue;
        }
        const double x = g.C + t0 * g.cu - l.jd * g.su - ix, y = g.C + t0 * g.su + l.jd * g.cu - iy;
        const double f00 = node(o, 0), f01 = node(o, 1), f10 = node(o, n), f11 = node(o, n + 1);
        const double dxy = f11 - f01 - f10 + f00;
        A0 += f00 + x * (f10 - f00) + y * (f01 - f00) + x * y * dxy;
        A1 += g.cu * (f10 - f00 + y * dxy) + g.su * (f01 - f00 + x * dxy);
        A2 += g.cu * g.su * dxy;
      }
      for (; e < p.size() && (long long)p[e].pos < b1; ++e) {
        const PieceRec r = make_rec(g, p[e].pos, p[e].kind, p[e].li, p[e].m, sub_bins, near);
        if (r.tau < 0 || r.tau > (double)sub_bins / n) return fail("tau", r.tau, 0);
        if (near) {
          const int st = r.kind == K_X ? n : 1;
          if (r.kind <= K_Y) A0 += r.ca * (node(r.off, 0) - node(r.off, -st));
          else if (r.kind != K_NULL) A0 += (r.kind == K_IN ? 1 : -1) * node(r.off, 0);
        } else if (r.kind <= K_NULL) {
          const int st = r.kind == K_Y ? 1 : n, ot = n + 1 - st;
          const double P = node(r.off, st) - 2 * node(r.off, 0) + node(r.off, -st);
          const double Q = node(r.off, ot + st) - 2 * node(r.off, ot) + node(r.off, ot - st);
          const double ds = r.ca * (P + r.w * (Q - P)), dc = r.cs * (Q - P);
          A2 += dc;
          A1 += ds - 2 * dc * r.tau;
          A0 += r.tau * (dc * r.tau - ds);
        } else {
          const double x = r.w, y = r.w2, sg = r.kind == K_IN ? 1 : -1;
          const double f00 = node(r.off, 0), f01 = node(r.off, 1), f10 = node(r.off, n),
                       f11 = node(r.off, n + 1);
          const double dxy = f11 - f01 - f10 + f00;
          const double ds = sg * (g.cu * (f10 - f00 + y * dxy) + g.su * (f01 - f00 + x * dxy));
          const double dc = sg * g.cu * g.su * dxy;
          A0 += sg * (f00 + x * (f10 - f00) + y * (f01 - f00) + x * y * dxy) +
                r.tau * (dc * r.tau - ds);
          A1 += ds - 2 * dc * r.tau;
          A2 += dc;
        }
        v[e] = A0 + r.tau * (A1 + r.tau * A2);
        s[e] = A1 + 2 * r.tau * A2;
        c[e] = A2;
      }
    }
    if (e != p.size()) return fail("pieces used", e, p.size());
    // ---- values at random t of this unit
    for (int q = 0; q < 60; ++q) {
      const double t = (g.tfirst + kUnitBins * (rng() % 1000003) / 1000003.0) / n - g.toff;
      if (t * t > g.rc2) continue;
      const long long fx = pos_of(g, t);
      if (fx < 0 || fx >= (long long)kUnitBins << 20) continue;
      size_t hi = std::upper_bound(p.begin(), p.end(), (unsigned)fx,
                                   [](unsigned a, const Piece &b) { return a < b.pos; }) - p.begin();
      if (!hi) return fail("no piece before", fx, 0);
      const unsigned near0 = (unsigned)fx - p[hi - 1].pos;
      if (near0 <= 2 || (hi < p.size() && p[hi].pos - fx <= 2)) continue;  // goes exact
      const double dt = near0 / 1048576.0 / n;
      const double got = v[hi - 1] + dt * (s[hi - 1] + dt * c[hi - 1]);
      double ref = 0;
      for (int j = -L; j < L; ++j) {
        const Line l = make_line(g, j);
        const double X = g.C + t * g.cu - l.jd * g.su, Y = g.C + t * g.su + l.jd * g.cu;
        if (!l.ok || X < 0 || Y < 0 || X > W || Y > W) continue;
        const int ix = std::min((int)X, W - 1), iy = std::min((int)Y, W - 1);
        const long long o = ((long long)ix * n + iy) * n;
        if (near) {
          ref += node(o, 0);
          continue;
        }
        const double x = X - ix, y = Y - iy;
        ref += (1 - x) * ((1 - y) * node(o, 0) + y * node(o, 1)) +
               x * ((1 - y) * node(o, n) + y * node(o, n + 1));
      }
      worst = std::max(worst, std::fabs(got - ref));
      size = std::max(size, std::fabs(ref));
    }
  }
  // positions are quantised to 2^-21 bins (half a unit), fractions to FP32:
  // slope ~ sqrt(2n) per cell, so the value's error stays far below 1e-5
  if (!(worst <= 2e-5 * std::max(size, 1.0))) return fail("row sum", worst, size);
  return 0;
}

int main() {
  const double pi = 3.14159265358979323846;
  const double phis[] = {0, pi / 2, pi, 2 * pi / 7, pi / 4, 3 * pi / 4, 5.1, 0.013, pi + 0.4,
                         1.5 * pi - 2e-3};
  int bad = 0;
  for (int n : {8, 9, 24, 33, 64, 101})
    for (bool near : {false, true})
      for (double phi : phis)
        for (int L : {n, 2 * n, n / 2, 3})
          for (double crop : {3.00001, 0.7})
            bad += check(n, near, L, phi, crop, 17 * n + L);
  // the largest edge: capacities and identities
  for (double phi : {pi / 4, 0.7}) bad += check(1024, false, 1024, phi, 3.00001, 5);
  std::printf(bad ? "%d checks failed\n" : "ok\n", bad);
  return bad != 0;
}
