// profile_dev.cuh -- geometry of the row-sum profiles (k_profile.cu): the
// pieces of G_k(t) for one phi.  Plain scalar code: the kernel calls it per
// thread, and a host program can compile it too (PROF_FN).
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define PROF_FN __device__ __forceinline__
#define PROF_HD __host__ __device__
#else
#define PROF_FN inline
#define PROF_HD
#endif

namespace wrtp {

// Separate roundings on the device (a host build does not contract).
#ifdef __CUDACC__
PROF_FN double prof_mul(double a, double b) { return __dmul_rn(a, b); }
PROF_FN double prof_add(double a, double b) { return __dadd_rn(a, b); }
PROF_FN double prof_sub(double a, double b) { return __dsub_rn(a, b); }
PROF_FN long long prof_floor(double a) { return __double2ll_rd(a); }
PROF_FN double prof_ld(const double *p) { return __ldg(p); }
#else
PROF_FN double prof_mul(double a, double b) { return a * b; }
PROF_FN double prof_add(double a, double b) { return a + b; }
PROF_FN double prof_sub(double a, double b) { return a - b; }
PROF_FN long long prof_floor(double a) { return (long long)floor(a); }
PROF_FN double prof_ld(const double *p) { return *p; }
#endif
PROF_FN int imax(int a, int b) { return a > b ? a : b; }
PROF_FN int imin(int a, int b) { return a < b ? a : b; }

constexpr int kUnitBins = 2048;  // bins of t per unit of work
constexpr unsigned kUnitEnd = (unsigned)kUnitBins << 20;  // its length in positions
constexpr unsigned kBoundary = 2;  // 2^-20 bins: rows this near a piece end go exact
// A horizontal axis component below this is a rounding of zero (phi on an
// axis): samples then never cross that axis' cell boundaries.
constexpr double kAxis = 1e-9;

// Offset of t (cells) so that every foot point of the square has t + off > 0.
PROF_HD inline double prof_t_off(int n, bool nearest) {
  return ceil(1.4142136 * 0.5 * (nearest ? n : n - 1)) + 1.0;
}

// Most piece boundaries a unit can hold for data cropped at squared radius
// `crop` (half edges): a length of line crosses at most sqrt 2 boundaries per cell,
// lines are half a cell apart.  Per cell of t that is the chord (at most 2
// sqrt(crop) half edges or the square's diagonal) times 2 sqrt 2, at most 4 n; over
// all t the area (the square's or the disc's).  Every line's first and last
// crossing may round into the unit; sub-range starts count too.
PROF_HD inline int unit_cap(int n, double crop) {
  const double r = sqrt(crop < 2.0 ? crop : 2.0);
  const double strip = 2.8284272 * r * kUnitBins;
  const double disc = 0.7853982 * crop < 1.0 ? 0.7853982 * crop : 1.0;
  const double area = 2.8284272 * disc * ((double)n + 2) * (n + 2);
  const int sub = n < kUnitBins ? n : kUnitBins;
  return (int)(strip < area ? strip : area) + 8 * n + 64 + (kUnitBins + sub - 1) / sub;
}

struct PieceRec {   // one piece boundary, read by whole warps of the build role
  double tau;       // t from the origin of its sub-range, cells
  float w, ca, cs;  // interior crossing: fraction along the line crossed, |c|, c c'
  int off;          // element offset of the crossing's node (or new cell), layer 0
  int kind;         // see below
  float w2;
};
enum { K_X = 0, K_Y = 1, K_NULL = 2, K_IN = 3, K_OUT = 4 };

// Geometry of one (request, phi).
struct Geo {
  int n, W, L;
  double h, C, dl;        // cells per unit length, centre, sample spacing in cells
  double cu, su, icu, isu;
  double rc2;             // crop radius^2, cells^2
  double toff;            // cells
  double tfirst;          // first bin of the unit
  int jlo, jhi;           // lines that can meet the crop disc
};

// crop: squared crop radius (the volume's non-zero nodes and the sampler's
// reach lie inside); c, sn: components of u as the direction table has them.
PROF_FN Geo make_geo(int n, bool nearest, int L, double c, double sn, double crop, int chunk) {
  Geo g;
  g.n = n;
  g.W = nearest ? n : n - 1;
  g.L = L;
  g.h = 0.5 * g.W;
  g.C = 0.5 * g.W;
  g.dl = g.h / n;
  g.cu = fabs(c) < kAxis ? 0.0 : c;
  g.su = fabs(sn) < kAxis ? 0.0 : sn;
  g.icu = g.cu != 0.0 ? 1.0 / g.cu : 0.0;
  g.isu = g.su != 0.0 ? 1.0 / g.su : 0.0;
  g.rc2 = crop * g.h * g.h;
  g.toff = prof_t_off(n, nearest);
  g.tfirst = (double)chunk * kUnitBins;
  const int jm = (int)fmin(sqrt(g.rc2) / g.dl + 1.0, 8.0 * n);
  g.jlo = -L > -jm ? -L : -jm;
  g.jhi = L - 1 < jm ? L - 1 : jm;
  return g;
}

PROF_FN bool on_axis(const Geo &g) { return g.cu == 0.0 || g.su == 0.0; }

// Position of t within the unit in units of 2^-20 bins (monotone in t; may be
// outside [0, kUnitBins << 20)).
PROF_FN long long pos_of(const Geo &g, double t) {
  return prof_floor((fma(t, (double)g.n, g.toff * g.n) - g.tfirst) * 1048576.0);
}

// Line j: the sample's path X = C + t cu - jd su, Y = C + t su + jd cu (cells),
// crossing x line m at tx(m) and y line m at ty(m); inside the cube for t in
// [tin, tout].  Every decision below compares these very values, so a line's
// cells, crossings, entry and exit are consistent whatever the roundings.
struct Line {
  double jd, tin, tout;
  bool ok;
};
PROF_FN double tx_of(const Geo &g, double jd, int m) {
  return prof_mul(prof_add((double)m - g.C, prof_mul(jd, g.su)), g.icu);
}
PROF_FN double ty_of(const Geo &g, double jd, int m) {
  return prof_mul(prof_sub((double)m - g.C, prof_mul(jd, g.cu)), g.isu);
}
// Samples whose constant coordinate (phi on an axis) lies on a cell boundary:
// the reference's rounding decides their cell row by row, so they are left out
// of the tables and evaluated per row (rows role).
PROF_FN bool on_boundary(double q) { return fabs(q - rint(q)) < 1e-7; }

PROF_FN Line make_line(const Geo &g, int j) {
  Line l;
  l.jd = (double)j * g.dl;
  l.tin = -1e30;
  l.tout = 1e30;
  l.ok = true;
  if (g.cu != 0.0) {
    const double a = tx_of(g, l.jd, 0), b = tx_of(g, l.jd, g.W);
    l.tin = fmin(a, b);
    l.tout = fmax(a, b);
  } else {
    const double X = g.C - l.jd * g.su;
    l.ok = X > 0.0 && X < (double)g.W && !on_boundary(X);
  }
  if (g.su != 0.0) {
    const double a = ty_of(g, l.jd, 0), b = ty_of(g, l.jd, g.W);
    l.tin = fmax(l.tin, fmin(a, b));
    l.tout = fmin(l.tout, fmax(a, b));
  } else {
    const double Y = g.C + l.jd * g.cu;
    l.ok &= Y > 0.0 && Y < (double)g.W && !on_boundary(Y);
  }
  l.ok &= l.tin < l.tout;
  return l;
}

// Cell along one axis when the crossings that `passed` accepts are behind the
// sample: line m (1..W-1) is behind when passed(time(m)); q0: estimate.
template <class Time, class Passed>
PROF_FN int cell_of(int W, double q0, double c, Time time, Passed passed) {
  int i = (int)fmin(fmax(floor(q0), 0.0), (double)(W - 1));
  if (c > 0.0) {
    while (i < W - 1 && passed(time(i + 1))) ++i;
    while (i > 0 && !passed(time(i))) --i;
  } else if (c < 0.0) {
    while (i < W - 1 && !passed(time(i + 1))) ++i;
    while (i > 0 && passed(time(i))) --i;
  }
  return i;
}
template <class Passed>
PROF_FN int xcell(const Geo &g, double jd, double t, Passed p) {
  return cell_of(g.W, g.C + t * g.cu - jd * g.su, g.cu,
                 [&](int m) { return tx_of(g, jd, m); }, p);
}
template <class Passed>
PROF_FN int ycell(const Geo &g, double jd, double t, Passed p) {
  return cell_of(g.W, g.C + t * g.su + jd * g.cu, g.su,
                 [&](int m) { return ty_of(g, jd, m); }, p);
}

PROF_FN float clamp01(double x) { return (float)fmin(fmax(x, 0.0), 1.0); }

// Calls f(pos, kind, line index, m) for every piece boundary of the unit, and
// beyond(after, kind, line index, m) for those up to kBoundary before its start
// and after its end (pieces of the units next to it, which a row at this one's end
// may lie on), the tasks dealt to `step` callers (this one is number `first`).
// Tasks 0 .. 3 nl - 1: per line its x crossings, its y crossings, its entry
// and exit; then the sub-range starts.
template <class F, class B>
PROF_FN void each_boundary(const Geo &g, int nsub, int sub_bins, int first, int step, F f,
                           B beyond) {
  const int nl = imax(0, g.jhi - g.jlo + 1);
  const double ta = g.tfirst / g.n - g.toff, tb = (g.tfirst + kUnitBins) / g.n - g.toff;
  const long long end = kUnitEnd, near = kBoundary;
  auto at = [&](long long p, int kind, int li, int m) {
    if (p >= 0 && p < end) f((unsigned)p, kind, li, m);
    else if (p >= -near && p < end + near) beyond(p >= end, kind, li, m);
  };
  for (int k = first; k < 3 * nl + nsub; k += step) {
    if (k >= 3 * nl) {
      const int sub = k - 3 * nl;
      f((unsigned)(sub * sub_bins) << 20, K_NULL, 0, 0);
      continue;
    }
    const int what = k / nl, li = k - what * nl;
    const Line l = make_line(g, g.jlo + li);
    if (!l.ok) continue;
    const double reach = g.rc2 - l.jd * l.jd;
    if (reach < 0.0) continue;
    // boundaries outside the crop disc change nothing: all nodes there are 0
    const double tc = sqrt(reach) + 1e-6;
    if (what == 2) {
#pragma unroll 1
      for (int e = 0; e < 2; ++e) {
        const double t = e ? l.tout : l.tin;
        if (fabs(t) > tc) continue;
        at(pos_of(g, t), e ? K_OUT : K_IN, li, 0);
      }
      continue;
    }
    const double c = what ? g.su : g.cu;
    if (c == 0.0) continue;
    const double a = fmax(fmax(ta - 1.0, l.tin), -tc), b = fmin(fmin(tb + 1.0, l.tout), tc);
    if (a > b) continue;
    const double o = what ? g.C + l.jd * g.cu : g.C - l.jd * g.su;
    const double q0 = o + a * c, q1 = o + b * c;
    const int m0 = imax(1, (int)floor(fmin(q0, q1)) - 1);
    const int m1 = imin(g.W - 1, (int)ceil(fmax(q0, q1)) + 1);
    for (int m = m0; m <= m1; ++m) {
      const double t = what ? ty_of(g, l.jd, m) : tx_of(g, l.jd, m);
      if (!(t > l.tin && t < l.tout) || fabs(t) > tc) continue;
      at(pos_of(g, t), what ? K_Y : K_X, li, m);
    }
  }
}
template <class F>
PROF_FN void each_boundary(const Geo &g, int nsub, int sub_bins, int first, int step, F f) {
  each_boundary(g, nsub, sub_bins, first, step, f, [](bool, int, int, int) {});
}

PROF_FN PieceRec make_rec(const Geo &g, unsigned pos, int kind, int li, int m,
                                             int sub_bins, bool nearest) {
  PieceRec r;
  const int n = g.n;
  const unsigned sub0 = (pos >> 20) / sub_bins * sub_bins;
  r.tau = (double)(pos - (sub0 << 20)) * (1.0 / 1048576.0) / n;
  r.w = r.ca = r.cs = r.w2 = 0.0f;
  r.off = (n + 1) * n;
  r.kind = kind;
  if (kind == K_NULL) return r;
  const double jd = (double)(g.jlo + li) * g.dl;
  if (kind == K_X) {
    const double t = tx_of(g, jd, m);
    const int iy = ycell(g, jd, t, [&](double x) { return x < t; });
    r.w = clamp01(g.C + t * g.su + jd * g.cu - iy);
    r.ca = (float)fabs(g.cu);
    r.cs = (float)(fabs(g.cu) * g.su);
    r.off = (m * n + iy) * n;
    if (nearest) r.ca = g.cu > 0.0 ? 1.0f : -1.0f;
  } else if (kind == K_Y) {
    const double t = ty_of(g, jd, m);
    const int ix = xcell(g, jd, t, [&](double x) { return x <= t; });
    r.w = clamp01(g.C + t * g.cu - jd * g.su - ix);
    r.ca = (float)fabs(g.su);
    r.cs = (float)(fabs(g.su) * g.cu);
    r.off = (ix * n + m) * n;
    if (nearest) r.ca = g.su > 0.0 ? 1.0f : -1.0f;
  } else {
    const Line l = make_line(g, g.jlo + li);
    const double t = kind == K_IN ? l.tin : l.tout;
    const bool in = kind == K_IN;
    const int ix = xcell(g, jd, t, [&](double x) { return in ? x <= t : x < t; });
    const int iy = ycell(g, jd, t, [&](double x) { return in ? x <= t : x < t; });
    r.w = clamp01(g.C + t * g.cu - jd * g.su - ix);
    r.w2 = clamp01(g.C + t * g.su + jd * g.cu - iy);
    r.ca = (float)g.cu;
    r.cs = (float)g.su;
    r.off = (ix * n + iy) * n;
  }
  return r;
}

// Where the rows of one (phi, theta) lie: row i of shift s at bin u = s ub + uo +
// i u1, counted from bin 0 of t for every unit alike, and at z cell s wb + wo + i w1.
struct RowGeo {
  double ub, uo, u1, wb, wo, w1;
};
PROF_FN RowGeo row_geo(const double *D, const Geo &g) {  // D: the direction's nine numbers
  RowGeo q;
  // (roundings spelled out: every kernel has to find the same u)
  q.ub = prof_mul(fma(prof_ld(D), g.cu, prof_mul(prof_ld(D + 1), g.su)), prof_mul(g.h, g.n));
  q.uo = prof_mul(g.toff, g.n);
  q.u1 = prof_mul(fma(prof_ld(D + 3), g.cu, prof_mul(prof_ld(D + 4), g.su)), prof_mul(g.dl, g.n));
  q.wb = prof_ld(D + 2) * g.h;
  q.wo = g.h;
  q.w1 = prof_ld(D + 5) * g.dl;
  return q;
}

// Position of bin u in the unit that starts at bin tfirst, from kUnitEnd up outside
// it.  Rounded down once, in units that all units share (tfirst is a whole number
// and the sum stays within one binade): a row is in exactly one unit, also where its
// u is within rounding of the border of two.  u - tfirst from -kUnitBins up
// to twice that (positions wrap beyond).
PROF_FN unsigned row_pos(double u, double tfirst) {
#ifdef __CUDACC__
  constexpr double kMagicPos = 6442450944.0;  // 1.5 * 2^32: 20 fraction bits
  return (unsigned)__double2loint(__dadd_rd(u, kMagicPos - tfirst));
#else
  return (unsigned)prof_floor((u - tfirst) * 1048576.0);
#endif
}

}  // namespace wrtp
