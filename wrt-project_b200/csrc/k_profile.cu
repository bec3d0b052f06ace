// k_profile.cu -- plane integrals from row-sum profiles.
//
// Every lattice row of a plane (fixed i, running j; radon_grid/src/
// integral.c:43-55) runs along v2 = (-sin phi, cos phi, 0), whatever theta is,
// and its samples sit at j delta along v2 from the foot point t u,
// u = (cos phi, sin phi): t = (s n + i delta v1) . u.  So for one phi all rows
// of all theta, shifts and i are values of ONE function of two variables,
//
//   row(t, z) = (1 - tz) G_k(t) + tz G_{k+1}(t),  k = cell layer of z,
//   G_k(t) = sum_j f_k(t u + j delta v2),
//
// f_k the bilinear interpolation of node layer k (nearest sampler: row(t, z) =
// G_k(t), f_k the cells of layer k).  Along t each sample j moves straight
// through the cells, so G_k is an exact piecewise quadratic (nearest: piecewise
// constant) whose pieces end where some sample crosses a cell boundary: about
// 2.5 n pieces per cell of t, the same for every layer.  The kernel tabulates
// G_k -- one coefficient record per (piece, layer) -- and a row then costs two
// table reads instead of its ~2n samples.  At 128^3 with 64 latitudes, 256
// shifts, a table of 2.8e4 x 128 records serves 4.7e6 rows of ~170 samples.
//
// A step handles as many units of work as the tables' workspace holds, in four
// launches: the pieces of every unit are found and sorted, the tables summed
// up, the rows evaluated, and those that the tables do not decide once more.  A unit
// is one phi (or the pair phi, phi + pi, which share their lines: t -> -t) and one
// range of kUnitBins bins of t.
//
// Coordinates.  t in cells, tb = (t + t_off) * n bins (n bins per cell: 2 to 4
// pieces per bin).  Positions within a unit are fixed point, 12.20 bits.
//
// All requests of one launch sequence have the same sampler.
//
// Exactness.  FP64 positions; piece coefficients summed in FP64 from an origin
// at most one cell away and rounded once to FP32.  A row within 2 * 2^-20 bins
// of a piece boundary (some sample within ~1e-8 cells of a cell boundary, where
// the reference's rounding decides the cell) or with z within 1e-9 cells of a
// node layer is summed sample by sample with the reference's FP64 arithmetic.
// Plane sums are FP64 in an order that the request's sizes fix: bitwise the same
// alone or in any batch.
//
// What bounds it: nothing close to a byte or flop limit any more; the rows
// launch waits for its gathers (random 32-byte reads, mostly from L2: half of a warp's
// cycles, with 22 % of the warps resident; FP64 7 % busy, DRAM 7 %), the build for its
// node loads and its chain of sums.  128^3, 64 x 128 directions x 256
// shifts, lattice [-n, n)^2: 53.7 ms by the staged kernel (lattice samples
// through shared memory), 5.0 ms here; 256^3 BF16, 96 x 192 x 384: 750 and 45
// ms; error against FP64 (doubles, 96^3) 8e-9 (staged 5.1e-8).  Small requests wait for
// the four launches one after another (24^3, 8 x 16 x 32: 109 and 82 us).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "profile_dev.cuh"
#include "wrt_internal.cuh"

namespace {

using wrt::ProfReq;
using wrt::ProfSeg;

constexpr unsigned kAll = 0xffffffffu;
constexpr int kThreads = 256;
constexpr int kSortThreads = 1024;
constexpr int kMaxChunks = 6;  // ranges of t of one phi in a step
constexpr double kMagicInt = 6755399441055744.0;      // 1.5 * 2^52
using namespace wrtp;

__device__ __forceinline__ float crop_of(const ProfReq &r) {
  const float r2 = __uint_as_float(__ldg(r.stats));
  return r.nearest ? wrt::nearest_crop_r2(r2, r.n) : wrt::trilinear_crop_r2(r2, r.n);
}

__device__ __forceinline__ Geo geo_of(const ProfReq &r, int base, int chunk) {
  const double *D = r.dir + 9 * (size_t)base * r.ntheta;
  return make_geo(r.n, r.nearest, r.L, __ldg(D + 7), -__ldg(D + 6), (double)crop_of(r), chunk);
}

__device__ __forceinline__ Geo geo_of_unit(const ProfSeg &s, int unit) {
  return geo_of(s.r, s.base0 + unit % s.nbase, s.chunk + unit / s.nbase);
}

// ------------------------------------------------------------------ sort role
// One block (of 1024 threads: few blocks, on which the whole step waits) finds the
// unit's piece boundaries, counts them per bin, and writes
// them in order of (position, identity): a bin's few entries are ranked by
// counting, so the order does not depend on the atomics.  The identities of
// boundaries just beyond the unit's ends go behind the list, kMaxWindow on each side
// (more are only counted, after start[kUnitBins]).
constexpr int kMaxWindow = 8;  // more boundaries than this at one t: whole row by the warp

__device__ __forceinline__ unsigned boundary_id(int kind, int li, int m) {
  return ((unsigned)kind << 29 | (unsigned)li << 13 | (unsigned)m) + 1u;
}

__device__ void role_sort(const ProfSeg &s, int unit, char *smem) {
  const Geo g = geo_of_unit(s, unit);
  unsigned *pos = s.pos + (size_t)unit * (s.cap + 16);
  unsigned *ids = s.ids + (size_t)unit * (s.cap + 16);
  unsigned *start = s.start + (size_t)unit * (kUnitBins + 8);
  int *cnt = reinterpret_cast<int *>(smem);           // [kUnitBins]
  int *cur = cnt + kUnitBins;                         // [kUnitBins]
  __shared__ int s_warp[kSortThreads / 32], s_beyond[2];
  const int tid = threadIdx.x;
  const bool skip = s.r.nearest && on_axis(g);
  for (int b = tid; b < kUnitBins; b += kSortThreads) cnt[b] = 0;
  if (tid < 2) s_beyond[tid] = 0;
  __syncthreads();
  if (!skip)
    each_boundary(g, s.nsub, s.sub_bins, (int)threadIdx.x, kSortThreads,
                  [&](unsigned p, int, int, int) { atomicAdd(&cnt[p >> 20], 1); });
  __syncthreads();
  // exclusive scan of the bins: kUnitBins / kSortThreads per thread
  constexpr int kPer = kUnitBins / kSortThreads;
  int sum = 0;
#pragma unroll
  for (int q = 0; q < kPer; ++q) sum += cnt[tid * kPer + q];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kAll, incl, o);
    if ((tid & 31) >= o) incl += t;
  }
  if ((tid & 31) == 31) s_warp[tid >> 5] = incl;
  __syncthreads();
  int before = incl - sum;
  for (int w = 0; w < (tid >> 5); ++w) before += s_warp[w];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int b = tid * kPer + q, c = cnt[b];
    start[b] = before;
    cur[b] = before;
    cnt[b] = before;
    before += c;
  }
  int total = 0;
  for (int w = 0; w < kSortThreads / 32; ++w) total += s_warp[w];
  __syncthreads();
  total = min(total, s.cap);  // the capacity bounds every geometry; never exceeded
  if (tid == 0) start[kUnitBins] = total;
  unsigned long long *keys = s.keys + (size_t)unit * s.cap;
  if (!skip)
    each_boundary(g, s.nsub, s.sub_bins, (int)threadIdx.x, kSortThreads,
                  [&](unsigned p, int kind, int li, int m) {
                    const int slot = atomicAdd(&cur[p >> 20], 1);
                    // the sub-range's start precedes everything at its position
                    const unsigned id = kind == K_NULL ? 0u : boundary_id(kind, li, m);
                    if (slot < s.cap) keys[slot] = (unsigned long long)p << 32 | id;
                  },
                  [&](bool after, int kind, int li, int m) {
                    const int slot = atomicAdd(&s_beyond[after], 1);
                    if (slot < kMaxWindow)
                      ids[s.cap + after * kMaxWindow + slot] = boundary_id(kind, li, m);
                  });
  __syncthreads();
  if (tid < 2) {  // in order of identity
    const int m = s_beyond[tid];
    unsigned *list = ids + s.cap + tid * kMaxWindow;
    start[kUnitBins + 1 + tid] = m;
    for (int a = 1; a < min(m, kMaxWindow); ++a)
      for (int b = a; b > 0 && list[b] < list[b - 1]; --b) {
        const unsigned t = list[b];
        list[b] = list[b - 1];
        list[b - 1] = t;
      }
  }
  PieceRec *rec = static_cast<PieceRec *>(s.rec) + (size_t)unit * s.cap;
  for (int e = tid; e < total; e += kSortThreads) {
    const unsigned long long key = keys[e];
    const unsigned p = (unsigned)(key >> 32), id = (unsigned)key;
    const int b = p >> 20;
    const int b0 = cnt[b], b1 = b + 1 < kUnitBins ? cnt[b + 1] : total;
    int rank = 0;
    for (int q = b0; q < min(b1, total); ++q) rank += keys[q] < key;
    const int dst = b0 + rank;
    pos[dst] = p;
    ids[dst] = id;
    const unsigned v = id - 1u;
    rec[dst] = id ? make_rec(g, p, (int)(v >> 29), (int)(v >> 13 & 0xffffu), (int)(v & 0x1fffu),
                             s.sub_bins, s.r.nearest)
                  : make_rec(g, p, K_NULL, 0, 0, s.sub_bins, s.r.nearest);
  }
  // no row is past the unit's end; one next to it is not decided by the table
  if (tid < 16) pos[total + tid] = kUnitEnd;
}

// ----------------------------------------------------------------- build role
__device__ __forceinline__ float ld_node(const float *v, int o) { return __ldg(v + o); }
__device__ __forceinline__ float ld_node(const __nv_bfloat16 *v, int o) {
  return __bfloat162float(__ldg(v + o));
}

// A line inside the cube at a sub-range's start: its cell and fractions.
struct StartLine {
  int off;
  float tx, ty, w;  // w: 1, or 0 for a line that is not there
};

// The quadratic about a sub-range's origin that the build sums up, per layer.
struct Quad {
  double a0, a1, a2;
};

// The sum at a sub-range's start over its lines (cells found once for all
// layers).
template <bool NEAR, typename VT>
__device__ __forceinline__ Quad start_sum(const Geo &g, const StartLine *lines, int nl,
                                          const VT *vol) {
  Quad q = {0.0, 0.0, 0.0};
  const float cu = (float)g.cu, su = (float)g.su, cusu = (float)(g.cu * g.su);
  const int sx = g.n * g.n, sy = g.n;
  // slopes in FP32 over eight lines, FP64 beyond (lines[] is padded with empty ones);
  // values in FP64 at once: where many of them are equal, FP32 sums of eight are all off
  // the same way, and with them every row of the range (24^3 nearest 2.1e-8 from FP64
  // instead of 1.3e-8, 96^3 trilinear 1.6e-8 instead of 8e-9; less than 1 % of the time)
  for (int j0 = 0; j0 < nl; j0 += 8) {
    float sl = 0.0f, cc = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const StartLine l = lines[j0 + j];
      if (NEAR) {
        q.a0 += (double)(l.w * ld_node(vol, l.off));
        continue;
      }
      const float x = l.tx, y = l.ty;
      const float f00 = ld_node(vol, l.off), f01 = ld_node(vol, l.off + sy),
                  f10 = ld_node(vol, l.off + sx), f11 = ld_node(vol, l.off + sx + sy);
      const float dx0 = f10 - f00, dx1 = f11 - f01, dy = f01 - f00, dxy = dx1 - dx0;
      const float fx = fmaf(y, dxy, dx0), fy = fmaf(x, dxy, dy);
      q.a0 += (double)(l.w * fmaf(x, fx, fmaf(y, dy, f00)));
      sl = fmaf(l.w, fmaf(cu, fx, su * fy), sl);
      cc = fmaf(l.w, dxy, cc);
    }
    if (!NEAR) {
      q.a1 += (double)sl;
      q.a2 += (double)(cusu * cc);
    }
  }
  return q;
}

// `count` boundaries from shared memory: each adds its change of value, slope
// and curvature to the quadratic about the sub-range's origin (independent FP64
// additions, no chain through the shifts of origin), and the piece's
// coefficients at its own start are written out.  T: the first piece's record
// of this lane's layer.
template <bool NEAR, typename VT>
__device__ __forceinline__ void add_pieces(const Geo &g, const PieceRec *rec, int count, bool live,
                                           const VT *vol, void *T, Quad *quad) {
  const int n = g.n, sx = n * n, sy = n;
  const float cu = (float)g.cu, su = (float)g.su, cusu = (float)(g.cu * g.su);
  const float kap = (float)(1.0 / 1048576.0 / n), kap2 = kap * kap;
  float4 *T4 = static_cast<float4 *>(T);
  float *T1 = static_cast<float *>(T);
  double A0 = quad->a0, A1 = quad->a1, A2 = quad->a2;
  constexpr int U = NEAR ? 8 : 4;  // boundaries whose loads are in flight together
  for (int e = 0; e < count; e += U) {
    float f[U][NEAR ? 2 : 6];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const PieceRec &r = rec[min(e + u, count - 1)];
      const VT *p = vol + r.off;
      const int kind = r.kind;
      // across the line crossed, and along it (entries and exits: read below)
      const int st = kind > K_NULL ? 0 : kind == K_Y ? sy : sx;
      const int ot = kind > K_NULL ? 0 : sx + sy - st;
      if (NEAR) {
        f[u][0] = ld_node(p, 0);
        f[u][1] = ld_node(p, -st);
      } else {
        f[u][0] = ld_node(p, -st);
        f[u][1] = ld_node(p, 0);
        f[u][2] = ld_node(p, st);
        f[u][3] = ld_node(p, ot - st);
        f[u][4] = ld_node(p, ot);
        f[u][5] = ld_node(p, ot + st);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (e + u >= count) break;
      const PieceRec &r = rec[e + u];
      const int kind = r.kind;
      if (NEAR) {
        if (kind <= K_Y) {
          const double up = (double)f[u][0], dn = (double)f[u][1];
          A0 += r.ca > 0.0f ? up - dn : dn - up;
        } else if (kind != K_NULL) {
          A0 += kind == K_IN ? (double)f[u][0] : -(double)f[u][0];
        }
        if (live) T1[(size_t)(e + u) * n] = (float)A0;
        continue;
      }
      const double tau = r.tau;
      if (kind <= K_NULL) {
        // slope |c| D2, curvature |c| c' (D2' - D2): the second differences of
        // the nodes across the line crossed, at its two ends
        const float P = (f[u][2] - f[u][1]) - (f[u][1] - f[u][0]);
        const float Q = (f[u][5] - f[u][4]) - (f[u][4] - f[u][3]), R = Q - P;
        const double ds = (double)(r.ca * fmaf(r.w, R, P)), dc = (double)(r.cs * R);
        const double t1 = fma(dc, tau, -ds);
        A2 += dc;
        A1 -= fma(dc, tau, t1);
        A0 = fma(tau, t1, A0);
      } else {
        const float x = r.w, y = r.w2;
        const VT *p = vol + r.off;
        const float f00 = ld_node(p, 0), f01 = ld_node(p, sy), f10 = ld_node(p, sx),
                    f11 = ld_node(p, sx + sy);
        const float dx0 = f10 - f00, dx1 = f11 - f01, dy = f01 - f00, dxy = dx1 - dx0;
        const float fx = fmaf(y, dxy, dx0), fy = fmaf(x, dxy, dy);
        const double sg = kind == K_IN ? 1.0 : -1.0;
        const double dv = sg * (double)fmaf(x, fx, fmaf(y, dy, f00));
        const double ds = sg * (double)fmaf(cu, fx, su * fy), dc = sg * (double)(cusu * dxy);
        A2 += dc;
        A1 += fma(-2.0 * dc, tau, ds);
        A0 += fma(tau, fma(dc, tau, -ds), dv);
      }
      if (live)
        T4[(size_t)(e + u) * n] =
            make_float4((float)fma(tau, fma(tau, A2, A1), A0),
                        (float)fma(2.0 * tau, A2, A1) * kap, (float)A2 * kap2, 0.0f);
    }
  }
  quad->a0 = A0;
  quad->a1 = A1;
  quad->a2 = A2;
}

// One block: one sub-range of one unit, a warp per group of 32 layers (blocks
// of up to eight warps; more layers in turn).  The lines at the start and then
// the boundaries, kRecTile at a time, are staged in shared memory for all warps.
constexpr int kRecTile = 128;
template <bool NEAR, typename VT>
__device__ __forceinline__ void role_build(const ProfSeg &s, int blk, const VT *vol, char *smem) {
  const int unit = blk / s.nsub, sub = blk % s.nsub;
  const Geo g = geo_of_unit(s, unit);
  if (NEAR && on_axis(g)) return;
  const int n = g.n, nl = max(0, g.jhi - g.jlo + 1);
  const double t0 = (g.tfirst + (double)sub * s.sub_bins) / n - g.toff;
  const double t1 = t0 + (double)s.sub_bins / n;
  const double tm = t0 > 0.0 ? t0 : (t1 < 0.0 ? -t1 : 0.0);
  const double rr = sqrt(g.rc2) + 1.0;
  if (tm > rr) return;  // outside the crop disc: no row reads it
  PieceRec *tile = reinterpret_cast<PieceRec *>(smem);
  StartLine *lines = reinterpret_cast<StartLine *>(tile + kRecTile);
  const long long b0 = (long long)sub * s.sub_bins << 20;
  auto passed = [&](double t) { return pos_of(g, t) < b0; };
  const int nth = (int)blockDim.x;
  for (int x = threadIdx.x; x < ((nl + 7) & ~7); x += nth) {
    const Line l = make_line(g, g.jlo + x);
    StartLine e = {0, 0.0f, 0.0f, 0.0f};
    // lines beyond the crop disc cross zeros only
    if (x < nl && l.ok && t0 * t0 + l.jd * l.jd <= (rr + 1.0) * (rr + 1.0) && passed(l.tin) &&
        !passed(l.tout)) {
      const int ix = xcell(g, l.jd, t0, passed), iy = ycell(g, l.jd, t0, passed);
      e.off = (ix * n + iy) * n;
      e.tx = (float)(g.C + t0 * g.cu - l.jd * g.su - ix);
      e.ty = (float)(g.C + t0 * g.su + l.jd * g.cu - iy);
      e.w = 1.0f;
    }
    lines[x] = e;
  }
  __syncthreads();
  const unsigned *start = s.start + (size_t)unit * (kUnitBins + 8);
  const int e0 = start[sub * s.sub_bins];
  const int e1 = start[min((sub + 1) * s.sub_bins, kUnitBins)];
  const PieceRec *rec = static_cast<const PieceRec *>(s.rec) + (size_t)unit * s.cap;
  const int lane = threadIdx.x & 31, warps = nth >> 5;
  for (int kg0 = 0; kg0 * 32 < n; kg0 += warps) {
    const int kg = kg0 + (threadIdx.x >> 5);
    // nothing of these layers is read when the whole patch lies outside the
    // crop ball (two cells of margin: rows read layers k and k + 1)
    const double za = kg * 32 - 2.0 - g.C, zb = min(kg * 32 + 33, n + 1) - g.C;
    const double zm = za > 0.0 ? za : (zb < 0.0 ? -zb : 0.0);
    const bool work = kg * 32 < n && tm * tm + zm * zm <= rr * rr;
    const int k = kg * 32 + lane;
    const VT *v = vol + min(k, n - 1);
    Quad q = {0.0, 0.0, 0.0};
    if (work) q = start_sum<NEAR>(g, lines, nl, v);
    for (int e = e0; e < e1; e += kRecTile) {
      const int m = min(kRecTile, e1 - e);
      __syncthreads();
      for (int x = threadIdx.x; x < 2 * m; x += nth)
        reinterpret_cast<int4 *>(tile)[x] = reinterpret_cast<const int4 *>(rec + e)[x];
      __syncthreads();
      if (work)
        add_pieces<NEAR>(g, tile, m, k < n, v,
                         static_cast<char *>(s.table) +
                             (((size_t)unit * s.cap + e) * n + k) * (NEAR ? 4 : 16),
                         &q);
    }
  }
}

// ------------------------------------------------------------------ rows role
// One sample with the reference's arithmetic.
__device__ __noinline__ double exact_at(const ProfReq &r, int d, int is, int i, int j) {
  const double *D = r.dir + 9 * (size_t)d;
  const double s = r.shift[is];
  const double delta = 1.0 / r.n;
  const double di = (double)i, dj = (double)j;
  double p[3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
    p[a] = __dadd_rn(
        __dadd_rn(__dmul_rn(s, D[a]), __dmul_rn(__dmul_rn(delta, D[3 + a]), di)),
        __dmul_rn(__dmul_rn(delta, D[6 + a]), dj));
  if (r.nearest)
    return wrtd::exact_nearest(static_cast<const float *>(r.vol), r.n, p[0], p[1], p[2]);
  return r.storage == WRT_STORAGE_BF16
             ? wrtd::exact_trilinear(static_cast<const __nv_bfloat16 *>(r.vol), r.n, p[0], p[1],
                                     p[2])
             : wrtd::exact_trilinear(static_cast<const float *>(r.vol), r.n, p[0], p[1], p[2]);
}

// The same where every coordinate is at least 1e-9 cells away from a cell
// boundary (and from the faces): plain FP64 interpolation, equal to rounding.
__device__ __noinline__ double sample64(const ProfReq &r, int d, int is, int i, int j) {
  const double *D = r.dir + 9 * (size_t)d;
  const double s = r.shift[is];
  const double delta = 1.0 / r.n;
  const int n = r.n, W = r.nearest ? n : n - 1;
  const double h = 0.5 * W;
  double t[3];
  int c[3];
  bool plain = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double q = (fma(s, D[a], fma(delta * i, D[3 + a], delta * j * D[6 + a])) + 1.0) * h;
    const double fl = floor(q);
    t[a] = q - fl;
    c[a] = (int)fl;
    if (q < -1e-9 || q > W + 1e-9) return 0.0;
    plain &= t[a] > 1e-9 && t[a] < 1.0 - 1e-9 && c[a] >= 0 && c[a] < W;
  }
  if (!plain) return exact_at(r, d, is, i, j);
  const int o = (c[0] * n + c[1]) * n + c[2];
  const float *v = static_cast<const float *>(r.vol);
  const __nv_bfloat16 *b = static_cast<const __nv_bfloat16 *>(r.vol);
  const bool bf = r.storage == WRT_STORAGE_BF16;
  auto f = [&](int x) { return (double)(bf ? ld_node(b, x) : ld_node(v, x)); };
  if (r.nearest) return f(o);
  double e[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int q = o + x * n * n;
    const double a0 = fma(t[2], f(q + 1) - f(q), f(q));
    const double a1 = fma(t[2], f(q + n + 1) - f(q + n), f(q + n));
    e[x] = fma(t[1], a1 - a0, a0);
  }
  return fma(t[0], e[1] - e[0], e[0]);
}

// A whole row by the warp (all lanes call it with the same row): the samples
// that its table holds, i.e. the lattice of the pair's first phi (mirrored: j ->
// -j) without those that no table holds (axis: the multiples of n).
__device__ __noinline__ double exact_row(const ProfReq &r, int d, int is, int i, double crop,
                                         bool axis, bool mirrored) {
  const int lane = threadIdx.x & 31;
  const double s = r.shift[is], di = (double)i / r.n;
  const double rem = crop - s * s - di * di;
  const int jm = rem > 0.0 ? (int)(sqrt(rem) * r.n) + 1 : 0;
  const int lo = max(mirrored ? 1 - r.L : -r.L, -jm), hi = min(mirrored ? r.L : r.L - 1, jm);
  double v = 0.0;
  for (int j = lo + lane; j <= hi; j += 32)
    if (!axis || (j != r.n && j != -r.n && (j != 0 || !(r.n & 1)))) v += sample64(r, d, is, i, j);
  return wrtd::warp_sum(v);
}

// What is missing from the table's value of a row that lies within kBoundary
// of `count` piece boundaries: for each sample they belong to, its value
// by the reference's arithmetic minus the value it has in the table's piece.
__device__ __noinline__ double boundary_terms(const ProfReq &r, const Geo &g, const unsigned *ids,
                                              int count, unsigned fx, double t, int iz, double tz,
                                              int d, int is, int i, bool mirrored) {
  double sum = 0.0;
  const int n = r.n;
  const float *v = static_cast<const float *>(r.vol);
  const __nv_bfloat16 *bv = static_cast<const __nv_bfloat16 *>(r.vol);
  const bool bf = r.storage == WRT_STORAGE_BF16;
  auto f = [&](int x) { return (double)(bf ? ld_node(bv, x) : ld_node(v, x)); };
  for (int q = 0; q < count; ++q) {
    const unsigned id = ids[q];
    if (!id) continue;
    const unsigned line = (id - 1u) >> 13 & 0xffffu;
    bool seen = false;
    for (int x = 0; x < q; ++x) seen |= ids[x] && ((ids[x] - 1u) >> 13 & 0xffffu) == line;
    if (seen) continue;
    const int j = g.jlo + (int)line;
    const Line l = make_line(g, j);
    auto passed = [&](double x) { return pos_of(g, x) <= (long long)fx; };
    double model = 0.0;
    if (l.ok && passed(l.tin) && !passed(l.tout)) {
      const int ix = xcell(g, l.jd, t, passed), iy = ycell(g, l.jd, t, passed);
      const int o = (ix * n + iy) * n + iz;
      if (r.nearest) {
        model = f(o);
      } else {
        const double x = g.C + t * g.cu - l.jd * g.su - ix, y = g.C + t * g.su + l.jd * g.cu - iy;
        double e[2];
        for (int k = 0; k < 2; ++k) {
          const double a = f(o + k), b = f(o + k + n), c = f(o + k + n * n),
                       dd = f(o + k + n * n + n);
          e[k] = a + x * (c - a) + y * (b - a) + x * y * (dd - c - b + a);
        }
        model = fma(tz, e[1] - e[0], e[0]);
      }
    }
    sum += exact_at(r, d, is, i, mirrored ? -j : j) - model;
  }
  return sum;
}

// First piece boundary past fx (binary steps while many share the bin: phis on
// or near an axis, where whole columns of samples cross together).
template <typename S>
__device__ __forceinline__ int find_piece(const unsigned *pos, const S *start, unsigned fx) {
  const int b = fx >> 20;
  int lo = start[b], hi = start[b + 1];
  while (hi - lo > 8) {
    const int m = (lo + hi) >> 1;
    if (pos[m] <= fx) lo = m + 1;
    else hi = m;
  }
  while (lo < hi && pos[lo] <= fx) ++lo;
  return lo;
}

// Where a row lies: position in the unit, z cell and fraction.  layer: within
// 1e-9 cells of a node layer (or rounding to one).
struct RowAt {
  unsigned fx;
  int iz;
  float tz;
  bool in, layer;  // in: in the unit; layer rows are not read from the table
};
__device__ __forceinline__ RowAt row_at(double di, double u0, double u1, double w0, double w1,
                                        double tfirst) {
  RowAt a;
  a.fx = row_pos(fma(di, u1, u0), tfirst);
  const double w = fma(di, w1, w0);
  const double mz = __dadd_rd(w, kMagicInt);
  a.iz = __double2loint(mz);
  a.tz = (float)(w - (mz - kMagicInt));
  a.in = a.fx < kUnitEnd;
  a.layer = a.tz < 1e-9f || a.tz >= 1.0f;
  return a;
}

// The nearest sampler's cell of one coordinate: -1 below the cube, n above.
__device__ __forceinline__ int axis_cell(double x, int n, double width) {
  if (fabs(x) > 1.0) return x < 0.0 ? -1 : n;
  return min((int)__ddiv_rn(__dadd_rn(x, 1.0), width), n - 1);
}

// The nearest sampler's row on a cell face: its samples' z differ by the rounding of
// v2's at most, so where the extremes share a cell by the reference's arithmetic
// (which is monotone), all do.  At theta = pi/2 every other row of a plane is one.
__device__ __noinline__ bool settle_layer(const ProfReq &r, int d, double sh, double di, RowAt *a) {
  const double *D = r.dir + 9 * (size_t)d;
  const double delta = 1.0 / r.n, width = __ddiv_rn(2.0, (double)r.n);
  const double z = __dadd_rn(__dmul_rn(sh, __ldg(D + 2)), __dmul_rn(__dmul_rn(delta, __ldg(D + 5)), di));
  const double c = fabs(__dmul_rn(__dmul_rn(delta, __ldg(D + 8)), (double)r.L));
  const int lo = axis_cell(__dadd_rn(z, -c), r.n, width);
  if (lo != axis_cell(__dadd_rn(z, c), r.n, width)) return false;
  a->iz = lo;
  a->layer = false;
  return true;
}

// Rows lo .. lo + len - 1 of shift sh that can lie in the unit, the cube and the
// crop ball.
__device__ __forceinline__ int row_range(const ProfReq &r, const Geo &g, const RowGeo &w,
                                         double crop, double sh, double u, double w0, int *lo_out) {
  const double rem = crop - sh * sh, u0 = u - g.tfirst;
  *lo_out = 1;
  if (!(rem >= 0.0)) return 0;
  const int im = (int)(sqrt(rem) * r.n);
  int lo = max(-r.L, -im), hi = min(r.L - 1, im);
  if (fabs(w.u1) > 1e-6) {
    const double inv = 1.0 / w.u1;
    const double x = -u0 * inv, y = (kUnitBins - u0) * inv;
    lo = max(lo, (int)fmax(fmin(x, y) - 1.0, -1e9));
    hi = min(hi, (int)fmin(fmax(x, y) + 1.0, 1e9));
  } else if (u0 < -1.0 || u0 > kUnitBins + 1.0) {
    return 0;
  }
  if (fabs(w.w1) > 1e-9) {
    const double inv = 1.0 / w.w1;
    const double x = (-0.5 - w0) * inv, y = (g.W + 0.5 - w0) * inv;
    lo = max(lo, (int)fmax(fmin(x, y) - 1.0, -1e9));
    hi = min(hi, (int)fmin(fmax(x, y) + 1.0, 1e9));
  }
  *lo_out = lo;
  return max(0, hi - lo + 1);
}

// What the table's values of 32 rows (lane: row i, if act) of one plane lack:
// rows on a node layer or on a piece boundary.
__device__ __forceinline__ double slow_rows(const ProfSeg &s, const Geo &g, const RowGeo &q,
                                            int unit, int d, int is, int i, bool act, double u0,
                                            double w0, double crop, bool mirrored) {
  const ProfReq &r = s.r;
  const unsigned *pos = s.pos + (size_t)unit * (s.cap + 16);
  const unsigned *ids = s.ids + (size_t)unit * (s.cap + 16);
  const unsigned *start = s.start + (size_t)unit * (kUnitBins + 8);
  const int total = start[kUnitBins], lane = threadIdx.x & 31, n = r.n;
  RowAt a = row_at((double)i, u0, q.u1, w0, q.w1, g.tfirst);
  act = act && a.in;
  // a settled row is read here, the others' table values the fast pass has added
  const bool settled = r.nearest && act && a.layer && settle_layer(r, d, __ldg(r.shift + is), (double)i, &a);
  bool whole = act && a.layer && a.iz >= -1 && a.iz <= g.W;
  double add = 0.0, val = 0.0;
  if (act && !a.layer && (unsigned)a.iz < (unsigned)g.W) {
    const int e = find_piece(pos, start, a.fx);
    int q0 = e, q1 = e;
    while (q0 > 0 && a.fx - pos[q0 - 1] <= kBoundary && e - q0 <= kMaxWindow) --q0;
    while (q1 < total && pos[q1] - a.fx <= kBoundary && q1 - e <= kMaxWindow) ++q1;
    // the neighbouring units' boundaries next to this one's ends
    const int before = a.fx <= kBoundary ? (int)start[kUnitBins + 1] : 0;
    const int after = kUnitEnd - a.fx <= kBoundary ? (int)start[kUnitBins + 2] : 0;
    const int count = q1 - q0 + before + after;
    if (count > kMaxWindow || settled) {
      const size_t o = ((size_t)unit * s.cap + (e - 1)) * n + a.iz;
      if (r.nearest) {
        val = (double)__ldg(static_cast<const float *>(s.table) + o);
      } else {
        const float4 *c = static_cast<const float4 *>(s.table) + o;
        const float4 x = __ldg(c), y = __ldg(c + 1);
        const float td = (float)(a.fx - pos[e - 1]);
        const float va = fmaf(td, fmaf(td, x.z, x.y), x.x);
        const float vb = fmaf(td, fmaf(td, y.z, y.y), y.x);
        val = (double)fmaf(a.tz, vb - va, va);
      }
    }
    if (count > kMaxWindow) {
      whole = true;
    } else if (count > 0) {
      unsigned win[kMaxWindow];
      int m = 0;
      for (int k = 0; k < before; ++k) win[m++] = ids[s.cap + k];
      for (int k = q0; k < q1; ++k) win[m++] = ids[k];
      for (int k = 0; k < after; ++k) win[m++] = ids[s.cap + kMaxWindow + k];
      const double t = (fma((double)i, q.u1, u0) - q.uo) / n;
      const double w = fma((double)i, q.w1, w0);
      add = boundary_terms(r, g, win, m, a.fx, t, a.iz, w - (double)a.iz, d, is, i, mirrored);
    }
    if (settled) {
      add += val;
      val = 0.0;
    }
  }
  unsigned m = __ballot_sync(kAll, whole);
  while (m) {
    const int src = __ffs(m) - 1;
    m &= m - 1;
    const double v = exact_row(r, d, is, __shfl_sync(kAll, i, src), crop, on_axis(g), mirrored);
    if (lane == src) add = v - val;
  }
  return add;
}

// The planes that the rows role has marked in their units: their rows once more,
// those that need more than the table worked out.  A warp per plane, as a rule for
// one or two such rows; at theta = pi/2, where all rows of a plane have one t and
// can all lie on a boundary and each then takes a warp ~5 us, the block's warps
// share the plane's rows and their sums are added in order (56^3, 11 x 22 x 78:
// 171 us with 8 warps and 32 rows each, 48 us with 16 that take every 16th).
constexpr int kSlowThreads = 512;
// A mark: segment (5 bits), which of its ranges of t (kMaxChunks bits), phi (16), plane (37).
constexpr int kMarkSeg = 59, kMarkChunk = 53, kMarkPhi = 37;
static_assert(kMarkChunk + kMaxChunks <= kMarkSeg, "marks");

template <int S>
__global__ void __launch_bounds__(kSlowThreads)
    profile_slow_kernel(const __grid_constant__ wrt::ProfStep<S> st) {
  __shared__ double s_sum[kSlowThreads / 32];
  const unsigned long long *list = st.list + 1;
  const long long count = (long long)st.list[0];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kW = kSlowThreads / 32;
  for (int pass = 0; pass < 2; ++pass) {
    const bool together = pass == 1;
    const long long first = together ? blockIdx.x : (long long)blockIdx.x * kW + warp;
    const long long step = together ? gridDim.x : (long long)gridDim.x * kW;
    for (long long k = first; k < count; k += step) {
      const unsigned long long item = list[k];
      const ProfSeg &s = st.seg[S == 1 ? 0 : (int)(item >> kMarkSeg)];
      const ProfReq &r = s.r;
      const int phi = (int)(item >> kMarkPhi & 0xffffu);
      const long long plane = (long long)(item & ((1ull << kMarkPhi) - 1));
      const int ndir = r.nphi * r.ntheta;
      const int d = (int)(plane % ndir), is = (int)(plane / ndir);
      if ((fabs(__ldg(r.dir + 9 * (size_t)d + 2)) < 1e-9) != together) continue;  // cos theta
      const double crop = (double)crop_of(r), sh = __ldg(r.shift + is);
      const bool mirrored = d >= (s.base0 + phi + 1) * r.ntheta;
      double sum = 0.0;
      for (int c = 0; c < s.nchunk; ++c) {
        if (!(item >> (kMarkChunk + c) & 1u)) continue;
        const Geo g = geo_of(r, s.base0 + phi, s.chunk + c);
        const RowGeo q = row_geo(r.dir + 9 * (size_t)d, g);
        const double u0 = fma(sh, q.ub, q.uo), w0 = fma(sh, q.wb, q.wo);
        int lo;
        const int len = row_range(r, g, q, crop, sh, u0, w0, &lo);
        const int x0 = together ? warp + kW * lane : lane, dx = together ? kSlowThreads : 32;
        for (int x = x0; x - x0 < len; x += dx)
          sum += slow_rows(s, g, q, c * s.nbase + phi, d, is, lo + x, x < len, u0, w0, crop,
                           mirrored);
      }
      sum = wrtd::warp_sum(sum);
      const double scale = 1.0 / ((double)r.n * r.n);
      if (!together) {
        if (lane == 0) r.out[plane] += sum * scale;
        continue;
      }
      if (lane == 0) s_sum[warp] = sum;
      __syncthreads();
      if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < kW; ++w) v += s_sum[w];
        r.out[plane] += v * scale;
      }
      __syncthreads();
    }
  }
}

// Four rows of one lane, i = di, di + step, ..: no branch between the loads, so
// that the four searches and the four gathers run side by side.  The piece is
// found among the first fifteen past the bin's start by four halving steps; a
// vote sends the warp through more where some lane needs them.  m: rows that
// exist.  Adds the rows' values in order; returns whether some row needs more
// than the table.
template <bool NEAR>
__device__ __forceinline__ bool rows4(const void *table, const unsigned *pos,
                                      const unsigned short *start, int n, int W, double di,
                                      double step, double u0, double u1, double w0, double w1,
                                      double tfirst, int m, double *sum) {
  constexpr int P = 4;
  RowAt a[P];
  int e[P];
  bool ok[P], flag = false;
#pragma unroll
  for (int u = 0; u < P; ++u) {
    a[u] = row_at(di + step * u, u0, u1, w0, w1, tfirst);
    const bool act = u < m && a[u].in;
    flag |= act && a[u].layer;
    ok[u] = act && !a[u].layer && (unsigned)a[u].iz < (unsigned)W;
    if (!ok[u]) {
      a[u].fx = 0;
      a[u].iz = 0;
    }
    e[u] = start[a[u].fx >> 20];
  }
#pragma unroll
  for (int h = 8; h > 0; h >>= 1)
#pragma unroll
    for (int u = 0; u < P; ++u)
      if (pos[e[u] + h - 1] <= a[u].fx) e[u] += h;
  unsigned nx[P], dt[P];
  bool more = false;
#pragma unroll
  for (int u = 0; u < P; ++u) {
    nx[u] = pos[e[u]];
    more |= nx[u] <= a[u].fx;
  }
  if (__any_sync(kAll, more)) {
#pragma unroll
    for (int u = 0; u < P; ++u) {
      if (nx[u] <= a[u].fx) {
        e[u] = find_piece(pos, start, a[u].fx);
        nx[u] = pos[e[u]];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < P; ++u) {
    dt[u] = a[u].fx - pos[e[u] - 1];
    flag |= ok[u] && (dt[u] <= kBoundary || nx[u] - a[u].fx <= kBoundary);
    e[u] = (e[u] - 1) * n + a[u].iz;
  }
  if (NEAR) {
    float v[P];
#pragma unroll
    for (int u = 0; u < P; ++u) v[u] = __ldg(static_cast<const float *>(table) + (unsigned)e[u]);
#pragma unroll
    for (int u = 0; u < P; ++u) *sum += (double)(ok[u] ? v[u] : 0.0f);
  } else {
    float4 p[P], q[P];
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const float4 *c = static_cast<const float4 *>(table) + (unsigned)e[u];
      p[u] = __ldg(c);
      q[u] = __ldg(c + 1);
    }
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const float td = (float)dt[u];
      const float va = fmaf(td, fmaf(td, p[u].z, p[u].y), p[u].x);
      const float vb = fmaf(td, fmaf(td, q[u].z, q[u].y), q[u].x);
      const float v = fmaf(a[u].tz, vb - va, va);
      *sum += (double)(ok[u] ? v : 0.0f);
    }
  }
  return flag;
}

// Lattice samples of a row inside the crop ball (measurement only).
__device__ __noinline__ int row_samples(const ProfReq &r, int is, int i, double u0, double a1,
                                        double tfirst, double crop) {
  if (row_pos(fma((double)i, a1, u0), tfirst) >= kUnitEnd) return 0;
  const double sq = r.shift[is], di = (double)i / r.n;
  const double r2 = crop - sq * sq - di * di;
  const int jm = r2 > 0.0 ? (int)(sqrt(r2) * r.n) : 0;
  return min(r.L - 1, jm) - max(-r.L, -jm) + 1;
}

// One warp per 32 planes (one theta, consecutive shifts).  As a rule each lane walks
// the rows of its own plane (a plane has 4096 / (n |cos theta|) rows in a unit; the
// lanes' counts are nearly equal, no sums across lanes); where that takes more rounds
// (theta near pi/2, where only some planes meet the unit, with all their rows, and
// consecutive rows read neighbouring layers of one piece) the warp takes the planes
// one after another with its lanes on the rows (128^3: 5.7 -> 5.5 ms against a fixed
// 96 rows).  Either way four rows per lane are in flight.  The unit's piece
// positions are in shared memory.  Rows that need more than the table are
// marked for profile_slow_kernel.
template <bool NEAR>
__device__ void role_rows(const ProfSeg &s, int seg, int blk, unsigned long long *list,
                          char *smem) {
  const ProfReq &r = s.r;
  const int phi = blk / s.blk_rows, tile = blk % s.blk_rows, base = s.base0 + phi;
  const int tid = threadIdx.x, lane = tid & 31;
  const int n = r.n, ndir = r.nphi * r.ntheta;
  const double crop = (double)crop_of(r);
  const int sgroups = (r.nshift + 31) / 32;
  const int wi = tile * (kThreads / 32) + (tid >> 5);
  const bool live = wi < sgroups * r.ntheta * (r.paired ? 2 : 1);
  const int half = wi / (sgroups * r.ntheta), ws = wi - half * sgroups * r.ntheta;
  // the thetas nearest pi/2 first: their warps have the most rows to walk
  const int rank = ws / sgroups, is0 = (ws - rank * sgroups) * 32;
  const int it = (r.ntheta - 1) / 2 + (rank & 1 ? (rank + 1) / 2 : -(rank / 2));
  const int np = live ? min(32, r.nshift - is0) : 0;
  const int d = live ? (base + half * (r.nphi / 2)) * r.ntheta + it : 0;
  double mine = 0.0;   // the sum of plane `lane`
  unsigned marks = 0;  // ranges where a row of it is not decided by the table alone
  bool some = false;   // it has rows here
  for (int c = 0; c < s.nchunk; ++c) {
    const Geo g = geo_of(r, base, s.chunk + c);
    if (NEAR && on_axis(g)) return;
    const int unit = c * s.nbase + phi;
    const unsigned *gstart = s.start + (size_t)unit * (kUnitBins + 8);
    const unsigned *gpos = s.pos + (size_t)unit * (s.cap + 16);
    unsigned *pos = reinterpret_cast<unsigned *>(smem);
    const int total = gstart[kUnitBins];
    unsigned short *start = reinterpret_cast<unsigned short *>(pos + s.cap + 16);
    if (c) __syncthreads();
    for (int k = tid; k < total + 16; k += kThreads) pos[k] = gpos[k];
    for (int k = tid; k <= kUnitBins; k += kThreads) start[k] = (unsigned short)gstart[k];
    __syncthreads();
    if (!live) continue;
    const int W = g.W;
    const char *table = static_cast<const char *>(s.table) +
                        (size_t)unit * s.cap * n * (NEAR ? 4 : 16);
    const RowGeo w = row_geo(r.dir + 9 * (size_t)d, g);
    // ---- row ranges, lane = plane
    int lo = 1, len = 0;
    double u0 = 0.0, w0 = 0.0;
    if (lane < np) {
      const double sh = __ldg(r.shift + is0 + lane);
      u0 = fma(sh, w.ub, w.uo);
      w0 = fma(sh, w.wb, w.wo);
      len = row_range(r, g, w, crop, sh, u0, w0, &lo);
    }
    const int most = (int)__reduce_max_sync(kAll, (unsigned)len);
    if (!most) continue;
    some |= len > 0;
    bool flag = false;
    // rounds of four rows per lane, one way and the other
    const int wide = (int)__reduce_add_sync(kAll, (unsigned)((len + 127) >> 7));
    if ((most + 3) >> 2 <= wide) {
      double di = (double)lo;
      for (int x = 0; x < most; x += 4, di += 4.0)
        flag |= rows4<NEAR>(table, pos, start, n, W, di, 1.0, u0, w.u1, w0, w.w1, g.tfirst, len - x,
                            &mine);
    } else {
      for (int p = 0; p < np; ++p) {
        const int lenp = __shfl_sync(kAll, len, p);
        if (!lenp) continue;
        const double up = __shfl_sync(kAll, u0, p), wp = __shfl_sync(kAll, w0, p);
        double di = (double)(__shfl_sync(kAll, lo, p) + lane), acc = 0.0;
        bool mark = false;
        for (int x = lane; x - lane < lenp; x += 128, di += 128.0)
          mark |= rows4<NEAR>(table, pos, start, n, W, di, 32.0, up, w.u1, wp, w.w1, g.tfirst,
                              (lenp - x + 31) >> 5, &acc);
        acc = wrtd::warp_sum(acc);
        mark = __any_sync(kAll, mark);
        if (lane == p) {
          mine += acc;
          flag |= mark;
        }
      }
    }
    marks |= (flag ? 1u : 0u) << c;
    if (r.counter) {
      unsigned long long counted = 0;
      for (int x = 0; x < len; ++x)
        counted += row_samples(r, is0 + lane, lo + x, u0, w.u1, g.tfirst, crop);
      if (counted) atomicAdd(r.counter, counted);
    }
  }
  if (lane >= np) return;
  const unsigned long long plane = (unsigned long long)(is0 + lane) * ndir + d;
  const double v = mine / ((double)n * n);
  if (s.first) r.out[plane] = v;
  else if (some) r.out[plane] += v;
  if (marks)
    list[1 + atomicAdd(list, 1ull)] = (unsigned long long)seg << kMarkSeg |
                                      (unsigned long long)marks << kMarkChunk |
                                      (unsigned long long)phi << kMarkPhi | plane;
}

// Samples that no table holds, one warp per plane (lanes on its rows), added to
// the finished sums: on an axis those with a constant coordinate on a cell
// boundary (j = -n, 0 for odd n, n), and for the second phi of a pair (lattice
// j -> -j) the end sample j = -L in place of j = L.  Only rows whose sample lies
// in the crop ball have any.
__global__ void __launch_bounds__(kThreads) profile_extra_kernel(const ProfReq r) {
  const long long w = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const int ndir = r.nphi * r.ntheta, lane = threadIdx.x & 31;
  if (w >= (long long)ndir * r.nshift) return;
  const int d = (int)(w % ndir), is = (int)(w / ndir), n = r.n;
  const bool mirrored = r.paired && d >= ndir / 2;
  const double *D = r.dir + 9 * (size_t)(d - d % r.ntheta);
  const bool axis = fabs(__ldg(D + 6)) < kAxis || fabs(__ldg(D + 7)) < kAxis;
  const double sh = __ldg(r.shift + is), rem = ((double)crop_of(r) - sh * sh) * n * n;
  const bool ends = mirrored && !(axis && r.L == n) && (double)r.L * r.L <= rem;
  const bool middle = axis && (n & 1) && rem >= 0.0;
  const bool faces = axis && (double)n * n <= rem;
  if ((r.nearest && axis) || (!ends && !middle && !faces)) return;
  const int im = (int)sqrt(rem), lo = max(-r.L, -im), hi = min(r.L - 1, im);
  double v = 0.0;
  for (int i = lo + lane; i <= hi; i += 32) {
    const double left = rem - (double)i * i;
    if (middle) v += exact_at(r, d, is, i, 0);
    if (faces && (double)n * n <= left) {
      if (n <= r.L) v += exact_at(r, d, is, i, -n);
      if (n < r.L) v += exact_at(r, d, is, i, n);
    }
    if (ends && (double)r.L * r.L <= left)
      v += sample64(r, d, is, i, -r.L) - sample64(r, d, is, i, r.L);
  }
  v = wrtd::warp_sum(v);
  if (lane == 0) r.out[(size_t)is * ndir + d] += v / ((double)n * n);
}

template <int S>
__global__ void __launch_bounds__(kSortThreads)
    profile_sort_kernel(const __grid_constant__ wrt::ProfStep<S> st) {
  extern __shared__ __align__(16) char smem[];
  if (blockIdx.x == 0 && threadIdx.x == 0) st.list[0] = 0;
  int b = (int)blockIdx.x;
  for (int k = 0; k < st.n; ++k) {
    const ProfSeg &s = st.seg[k];
    if (b < s.nbase * s.nchunk) return role_sort(s, b, smem);
    b -= s.nbase * s.nchunk;
  }
}

template <bool NEAR, int S>
__global__ void __launch_bounds__(kThreads, 3)
    profile_build_kernel(const __grid_constant__ wrt::ProfStep<S> st) {
  extern __shared__ __align__(16) char smem[];
  int b = (int)blockIdx.x;
  for (int k = 0; k < st.n; ++k) {
    const ProfSeg &s = st.seg[k];
    const int nb = s.nsub * s.nbase * s.nchunk;
    if (b < nb) {
      if (NEAR || s.r.storage != WRT_STORAGE_BF16)
        role_build<NEAR>(s, b, static_cast<const float *>(s.r.vol), smem);
      else
        role_build<NEAR>(s, b, static_cast<const __nv_bfloat16 *>(s.r.vol), smem);
      return;
    }
    b -= nb;
  }
}

template <bool NEAR, int S>
__global__ void __launch_bounds__(kThreads, 3)
    profile_rows_kernel(const __grid_constant__ wrt::ProfStep<S> st) {
  extern __shared__ __align__(16) char smem[];
  int b = (int)blockIdx.x;
  for (int k = 0; k < st.n; ++k) {
    const ProfSeg &s = st.seg[k];
    const int nb = s.blk_rows * s.nbase;
    if (b < nb) return role_rows<NEAR>(s, k, b, st.list, smem);
    b -= nb;
  }
}

// ------------------------------- the nearest sampler's phis on a horizontal axis
// There the lattice runs along a grid axis with every other sample on a cell
// boundary, whatever t is, so that the reference's rounding decides half of the
// cells.  With r the axis that the lattice runs along, the coordinate of sample j
// is fl(e + c_j): c_j = fl(fl(delta v2_r) j) is the same for all planes with one
// v2_r (a phi has two or three: the latitudes round it differently), and
// e = fl(s u_r + ..) is the row's, a few 1e-16.  The cell is monotone in e, so each
// boundary sample has one threshold; thresholds are few (the ties of a few binades),
// and between two of them the row sum depends on the row's other two cells alone.
// So a table [thresholds passed][cell][layer] of each v2_r serves all rows: one
// read each.  128^3, 4 of 128 phis, 64 latitudes, 256 shifts: 0.09 ms for the
// thresholds (four blocks, beside other kernels), 0.08 for the tables, 0.33 for the
// rows, which wait for FP64 divisions and gathers; by the staged kernel, every other
// sample in FP64, 11 ms.
constexpr int kAxisFamilies = 8;  // values of v2_r; rows of others are summed sample by sample
constexpr int kAxisSlots = 96;    // layers of a phi's table
constexpr int kAxisThreads = 128;

struct AxisHead {
  double emax;      // no row's e is beyond
  int run, nfam;    // axis of the lattice (0 or 1)
  int slot0[kAxisFamilies], nrank[kAxisFamilies], nflip[kAxisFamilies];
};
struct AxisJob {
  ProfReq r;
  int phi[4];
  int a0, na, first;  // cells of the fixed axis in the table; nothing added before
  char *head;         // [phi] AxisHead and lists
  size_t head_bytes;
  float *table;       // [phi][slot][na][n]
};
struct AxisLists {
  AxisHead *h;
  double *thr, *step;  // [family][n + 4]: thresholds of samples in order; distinct ones
  int *cell, *rank;    // the cell below; which distinct one
  int *weight;         // [family][n]: samples in a cell below all thresholds
  unsigned char *fam;  // [theta]
};
__host__ __device__ inline size_t axis_head_bytes(int n, int ntheta) {
  return (sizeof(AxisHead) + (size_t)kAxisFamilies * ((n + 4) * 24 + n * 4) + ntheta + 255) &
         ~(size_t)255;
}
__device__ __forceinline__ AxisLists axis_lists(const AxisJob &a, int p) {
  const int n = a.r.n, m = kAxisFamilies * (n + 4);
  AxisLists l;
  l.h = reinterpret_cast<AxisHead *>(a.head + a.head_bytes * p);
  l.thr = reinterpret_cast<double *>(l.h + 1);
  l.step = l.thr + m;
  l.cell = reinterpret_cast<int *>(l.step + m);
  l.rank = l.cell + m;
  l.weight = l.rank + m;
  l.fam = reinterpret_cast<unsigned char *>(l.weight + kAxisFamilies * n);
  return l;
}

// Doubles in order as integers and back.
__device__ __forceinline__ long long order_of(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : -(b & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double of_order(long long k) {
  return k >= 0 ? __longlong_as_double(k) : -__longlong_as_double(-k);
}

// One block per phi: families and their thresholds.
__global__ void __launch_bounds__(kThreads) axis_prepare_kernel(const AxisJob a) {
  const ProfReq &r = a.r;
  const AxisLists l = axis_lists(a, blockIdx.x);
  const double *D = r.dir + 9 * (size_t)a.phi[blockIdx.x] * r.ntheta;
  const int run = fabs(__ldg(D + 6)) < kAxis ? 1 : 0, tid = threadIdx.x, n = r.n;
  const double delta = 1.0 / n, width = __ddiv_rn(2.0, (double)n);
  __shared__ unsigned long long s_max;
  __shared__ int s_pick, s_count;
  if (tid == 0) s_max = 0;
  __syncthreads();
  for (int it = tid; it < r.ntheta; it += kThreads) {
    // |s|, |i delta| <= sqrt(3) inside the cube
    const double e = 1.75 * (fabs(__ldg(D + 9 * it + run)) + fabs(__ldg(D + 9 * it + 3 + run)));
    atomicMax(&s_max, (unsigned long long)__double_as_longlong(e));
    l.fam[it] = 255;
  }
  __syncthreads();
  const double emax = __longlong_as_double((long long)s_max);
  int slots = 0, f = 0;
  for (; f < kAxisFamilies; ++f) {
    if (tid == 0) {
      s_pick = r.ntheta;
      s_count = 0;
    }
    __syncthreads();
    for (int it = tid; it < r.ntheta; it += kThreads)
      if (l.fam[it] == 255) atomicMin(&s_pick, it);
    for (int m = tid; m < n; m += kThreads) l.weight[f * n + m] = 0;
    __syncthreads();
    if (s_pick == r.ntheta) break;
    const double v = __ldg(D + 9 * s_pick + 6 + run), step = __dmul_rn(delta, v);
    for (int it = tid; it < r.ntheta; it += kThreads)
      if (l.fam[it] == 255 && __ldg(D + 9 * it + 6 + run) == v) l.fam[it] = (unsigned char)f;
    double *thr = l.thr + f * (n + 4), *raw = l.step + f * (n + 4);
    int *cell = l.cell + f * (n + 4), *rank = l.rank + f * (n + 4);
    const int jlo = max(-r.L, -n - 2), jhi = min(r.L - 1, n + 2);
    for (int j = jlo + tid; j <= jhi; j += kThreads) {
      const double c = __dmul_rn(step, (double)j);
      const int lo = axis_cell(__dadd_rn(-emax, c), n, width);
      if (lo >= 0 && lo < n) atomicAdd(&l.weight[f * n + lo], 1);
      if (axis_cell(__dadd_rn(emax, c), n, width) == lo) continue;
      long long x = order_of(-emax), y = order_of(emax);  // cell lo at x, not at y
      while (y - x > 1) {
        const long long m = x + (y - x) / 2;
        if (axis_cell(__dadd_rn(of_order(m), c), n, width) == lo) x = m;
        else y = m;
      }
      const int k = atomicAdd(&s_count, 1);
      if (k < n + 4) {
        raw[k] = of_order(y);
        rank[k] = j;
      }
    }
    __syncthreads();
    const int count = min(s_count, n + 4);
    for (int k = tid; k < count; k += kThreads) {
      int pos = 0;
      for (int q = 0; q < count; ++q)
        pos += raw[q] < raw[k] || (raw[q] == raw[k] && rank[q] < rank[k]);
      thr[pos] = raw[k];
      cell[pos] = axis_cell(__dadd_rn(-emax, __dmul_rn(step, (double)rank[k])), n, width);
    }
    __syncthreads();
    if (tid == 0) {
      int ranks = 0;
      for (int k = 0; k < count; ++k) {
        if (!k || thr[k] != thr[k - 1]) raw[ranks++] = thr[k];
        rank[k] = ranks;
      }
      const bool fits = s_count <= n + 4 && slots + ranks + 1 <= kAxisSlots;
      l.h->slot0[f] = fits ? slots : -1;
      l.h->nrank[f] = ranks + 1;
      l.h->nflip[f] = count;
      s_count = fits ? ranks + 1 : 0;
    }
    __syncthreads();
    slots += s_count;
    __syncthreads();
  }
  if (tid == 0) {
    l.h->emax = emax;
    l.h->run = run;
    l.h->nfam = f;
  }
}

// One thread per (cell of the fixed axis, layer): the sum below all thresholds
// from the cells' weights, then threshold by threshold.
__global__ void __launch_bounds__(kAxisThreads) axis_table_kernel(const AxisJob a) {
  const AxisLists l = axis_lists(a, blockIdx.y);
  const int n = a.r.n, groups = (n + kAxisThreads - 1) / kAxisThreads;
  const int ia = blockIdx.x / groups, k = blockIdx.x % groups * kAxisThreads + threadIdx.x;
  if (k >= n) return;
  const size_t step = l.h->run ? n : (size_t)n * n;
  const float *v = static_cast<const float *>(a.r.vol) +
                   (size_t)(a.a0 + ia) * (l.h->run ? (size_t)n * n : n) + k;
  for (int f = 0; f < l.h->nfam; ++f) {
    if (l.h->slot0[f] < 0) continue;
    float *t = a.table + (((size_t)blockIdx.y * kAxisSlots + l.h->slot0[f]) * a.na + ia) * n + k;
    const int *w = l.weight + f * n, *cell = l.cell + f * (n + 4), *rank = l.rank + f * (n + 4);
    double sum = 0.0;
#pragma unroll 8
    for (int m = 0; m < n; ++m) sum += (double)w[m] * (double)__ldg(v + step * m);
    int q = 0;
    for (int h = 0;; ++h) {
      t[(size_t)h * a.na * n] = (float)sum;
      if (h + 1 == l.h->nrank[f]) break;
      for (; q < l.h->nflip[f] && rank[q] == h + 1; ++q) {
        const int c = cell[q];
        const double up = c + 1 < n ? (double)__ldg(v + step * (c + 1)) : 0.0;
        sum += up - (c >= 0 ? (double)__ldg(v + step * c) : 0.0);
      }
    }
  }
}

// One block per plane, threads on its rows.
__global__ void __launch_bounds__(kAxisThreads) axis_rows_kernel(const AxisJob a) {
  const ProfReq &r = a.r;
  const AxisLists l = axis_lists(a, blockIdx.y);
  const int n = r.n, it = blockIdx.x % r.ntheta, is = blockIdx.x / r.ntheta;
  const int d = a.phi[blockIdx.y] * r.ntheta + it, run = l.h->run, fix = 1 - run;
  const double *D = r.dir + 9 * (size_t)d;
  const double s = __ldg(r.shift + is), delta = 1.0 / n, width = __ddiv_rn(2.0, (double)n);
  const double emax = l.h->emax, crop = (double)crop_of(r);
  const double rem = crop - s * s;
  const int im = rem >= 0.0 ? (int)(sqrt(rem) * n) : -1;
  const int lo = max(-r.L, -im), hi = rem >= 0.0 ? min(r.L - 1, im) : lo - 1;
  // what the samples' other two coordinates differ by along the row, at most
  const double cx = fabs(__dmul_rn(__dmul_rn(delta, __ldg(D + 6 + fix)), (double)r.L));
  const double cz = fabs(__dmul_rn(__dmul_rn(delta, __ldg(D + 8)), (double)r.L));
  const double sx = __dmul_rn(s, __ldg(D + fix)), dx = __dmul_rn(delta, __ldg(D + 3 + fix));
  const double se = __dmul_rn(s, __ldg(D + run)), de = __dmul_rn(delta, __ldg(D + 3 + run));
  const double sz = __dmul_rn(s, __ldg(D + 2)), dz = __dmul_rn(delta, __ldg(D + 5));
  const int f = l.fam[it], slot0 = f < kAxisFamilies ? l.h->slot0[f] : -1;
  const int nstep = slot0 >= 0 ? l.h->nrank[f] - 1 : 0;
  const double *step = l.step + (slot0 >= 0 ? f * (n + 4) : 0);
  const float *t = a.table + ((size_t)blockIdx.y * kAxisSlots + max(slot0, 0)) * a.na * n;
  double sum = 0.0;
  unsigned long long counted = 0;
  for (int i0 = lo + (threadIdx.x & ~31); i0 <= hi; i0 += kAxisThreads) {
    const int i = i0 + (threadIdx.x & 31);
    const double di = (double)i;
    const double x = __dadd_rn(sx, __dmul_rn(dx, di)), z = __dadd_rn(sz, __dmul_rn(dz, di));
    const double e = __dadd_rn(se, __dmul_rn(de, di));
    const int ix = axis_cell(__dadd_rn(x, -cx), n, width), iz = axis_cell(__dadd_rn(z, -cz), n, width);
    const int own = min(max(ix, 0), n - 1) - a.a0;
    const bool mine = i <= hi && own >= 0 && own < a.na;
    const bool one = slot0 >= 0 && fabs(e) <= emax && ix == axis_cell(__dadd_rn(x, cx), n, width) &&
                     iz == axis_cell(__dadd_rn(z, cz), n, width);
    if (mine && one && ix >= 0 && ix < n && iz >= 0 && iz < n) {
      int p = 0, q = nstep;  // thresholds at or below e
      while (p < q) {
        const int m = (p + q) >> 1;
        if (step[m] <= e) p = m + 1;
        else q = m;
      }
      sum += (double)__ldg(t + ((size_t)p * a.na + own) * n + iz);
    }
    unsigned m = __ballot_sync(kAll, mine && !one);
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      const double v = exact_row(r, d, is, i0 + src, crop, false, false);
      if ((threadIdx.x & 31) == src) sum += v;
    }
    if (r.counter && a.first && i <= hi) {
      const int jm = (int)(sqrt(fmax(0.0, rem - di * di * delta * delta)) * n);
      counted += min(r.L - 1, jm) - max(-r.L, -jm) + 1;
    }
  }
  if (counted) atomicAdd(r.counter, counted);
  __shared__ double s_sum[kAxisThreads / 32];
  sum = wrtd::warp_sum(sum);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < kAxisThreads / 32; ++w) v += s_sum[w];
    v /= (double)n * n;
    double *o = r.out + ((size_t)is * r.nphi + a.phi[blockIdx.y]) * r.ntheta + it;
    if (a.first) *o = v;
    else if (v != 0.0) *o += v;
  }
}

// ------------------------------------------------------------------ host side
size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

struct UnitBytes {
  size_t table, rec, pos, start, keys, list;
};
UnitBytes unit_bytes(const ProfReq &r, float crop) {
  const int n = r.n;
  const bool nearest = r.nearest != 0;
  const size_t cap = unit_cap(n, crop);
  UnitBytes b;
  b.table = al(cap * n * (nearest ? 4 : 16));
  b.rec = al(cap * sizeof(PieceRec));
  b.pos = al(2 * 4 * (cap + 16));  // positions and identities
  b.start = al(4 * (kUnitBins + 8));
  b.keys = al(8 * cap);
  b.list = 8 * (size_t)r.ntheta * r.nshift * (r.paired ? 2 : 1);
  return b;
}

// The workspace: tables, piece records, positions and identities, sort keys
// (1/256 shares of the whole; a table is n / 2 times its records, so from n =
// 8 up the tables are what fills it).
struct Areas {
  size_t table, rec, place, keys, list;
  explicit Areas(size_t ws) {
    const size_t u = ws / 256 & ~(size_t)255;
    table = 176 * u;
    rec = 32 * u;
    place = 12 * u;
    keys = 6 * u;
    list = 28 * u;
  }
  // the first `units` units beside what is already there
  bool fits(const UnitBytes &b, size_t units, const UnitBytes &had) const {
    return had.table + b.table * units <= table && had.rec + b.rec * units <= rec &&
           had.pos + had.start + (b.pos + b.start) * units <= place &&
           had.keys + b.keys * units <= keys && had.list + b.list * units + 8 <= list;
  }
};

constexpr int kManySegs = 24;
static_assert(kManySegs <= 32, "marks");

// Ranges of t that are computed together: as many as fit half the tables' memory with
// all phis, so that few phis fill the device too (64^3 with 14 x 28 directions 600 ->
// 240 us; 68^3 with 11 x 22 385 -> 230, 78^3 with 23 x 46 850 -> 490), and a phi's
// together in 128 MB.  By the sizes alone, because the order in which a plane's sum
// is added up follows it.
int chunk_group(const ProfReq &r) {
  const double unit = (double)unit_cap(r.n, 3.0) * r.n * (r.nearest ? 4 : 16);
  const int nbase = r.paired ? r.nphi / 2 : r.nphi;
  const double fit = std::min((double)(wrt::kProfTableBytes / 2) / (unit * nbase) + 0.5,
                              (double)((size_t)128 << 20) / unit);
  return std::min(std::max((int)fit, 1), 4);
}

// The ranges of t in which data within the crop bound has rows.
void chunk_range(const ProfReq &r, float crop, int *c0, int *c1) {
  const double h = 0.5 * (r.nearest ? r.n : r.n - 1), toff = prof_t_off(r.n, r.nearest);
  const double tmax = std::min(std::sqrt((double)crop), 1.4142135623730952) * h + 1e-3;
  *c0 = std::max(0, (int)std::floor((toff - tmax) * r.n / kUnitBins));
  *c1 = (int)std::floor((toff + tmax) * r.n / kUnitBins) + 1;
}

// Dynamic shared memory of the build and the rows at the largest edge (70 KB each).
constexpr size_t kMostSmem = 96 * 1024;

template <bool NEAR, int S>
cudaError_t launch_step(wrt_ctx *ctx, cudaStream_t stream, const std::vector<ProfSeg> &segs,
                        unsigned long long *list) {
  static_assert(sizeof(wrt::ProfStep<S>) <= 32000, "kernel parameters");
  static thread_local wrt::ProfStep<S> st;
  st.n = (int)segs.size();
  st.list = list;
  long long sort = 0, build = 0, rows = 0;
  int n = 0, cap = 0;
  for (int k = 0; k < st.n; ++k) {
    st.seg[k] = segs[k];
    cap = std::max(cap, segs[k].cap);
    sort += segs[k].nbase * segs[k].nchunk;
    build += (long long)segs[k].nsub * segs[k].nbase * segs[k].nchunk;
    rows += (long long)segs[k].blk_rows * segs[k].nbase;
    n = std::max(n, segs[k].r.n);
  }
  const size_t sm_build = kRecTile * sizeof(PieceRec) + (size_t)(4 * n + 64) * sizeof(StartLine);
  const int th_build = 32 * std::min(8, (n + 31) / 32);
  const size_t sm_rows = 4 * (size_t)(cap + 16) + 2 * (size_t)(kUnitBins + 8);
  cudaError_t e = cudaSuccess;
  // beyond 48 KB of dynamic shared memory a kernel has to be told
  if (sm_build > 48 * 1024) e = wrt::allow_smem(profile_build_kernel<NEAR, S>, kMostSmem);
  if (e == cudaSuccess && sm_rows > 48 * 1024)
    e = wrt::allow_smem(profile_rows_kernel<NEAR, S>, kMostSmem);
  if (e != cudaSuccess) return e;
  profile_sort_kernel<S><<<(unsigned)sort, kSortThreads, kUnitBins * 8, stream>>>(st);
  profile_build_kernel<NEAR, S><<<(unsigned)build, th_build, sm_build, stream>>>(st);
  profile_rows_kernel<NEAR, S><<<(unsigned)rows, kThreads, sm_rows, stream>>>(st);
  profile_slow_kernel<S><<<ctx->sm_count * 2, kSlowThreads, 0, stream>>>(st);
  ctx->launches += 4;
  return cudaGetLastError();
}

}  // namespace

namespace wrt {

bool profile_covers(int n, int nphi, int ntheta, int nshift) {
  // sizes the fixed-point positions, the piece identities and the parameter
  // ranges hold
  return n >= 8 && n <= 1024 && nphi <= 4096 && (long long)ntheta * nshift <= (1LL << 28) / n;
}

// A phi's tables cost ~2.5 n^2 pieces x n layers whatever is read from them, the
// staged kernel its rows x samples, so what decides is the rows per layer of a
// table, ntheta nshift / n (half that where phi + pi has tables of its own); few phis
// of a large volume leave most of the device idle while they are built.  Against
// the staged kernel on 110 random sizes past the line (n 10 .. 176, 3 .. 64 latitudes,
// 8 .. 256 shifts, 4000 planes up): 0.93 of its speed at worst, 1.05-2.5 times within a
// fifth of the line, 2-4 times at twice; just below it 0.5-1.3 times for n > 100, up
// to 2.5 for n < 60.  Nearest on 86 sizes past the line: 1.03 at worst, 1.3-9 as a
// rule.  Below 4000 planes both are launches; staged and tables by the number of planes,
// trilinear, sizes past the line above: 2000 planes 20^3 66 and 75 us, 24^3 60 and 94;
// 3000: 24^3 94 and 96, 32^3 87 and 100, 40^3 132 and 136; 4000: 24^3 129 and 80, 32^3 124
// and 108, 40^3 115 and 128, 48^3 183 and 177; 5000: 155 and 123 (40^3), 155 and 147 (48^3);
// 10,000: 276 and 93 (32^3), 366 and 187 (64^3).  (Nearest is ahead from 1000 planes up.)
bool profile_route(const wrt_ctx *ctx, int n, int nphi, int ntheta, int nshift) {
  if (!profile_covers(n, nphi, ntheta, nshift)) return false;
  if (ctx->staged_config >= 0) return ctx->staged_config == kNumStagedConfigs - 1;
  // A position is rounded to 2^-20 bins, n bins a cell, and a small volume's rows have
  // few samples: below 15 the error against FP64 passes the staged kernel's (24 phantoms
  // and grids each, trilinear, means: 8^3 1.0e-7 here and 4.5e-8 there, 12^3 5.4 and 4.5,
  // 14^3 4.3 and 4.3, 15^3 3.8 and 4.2, 16^3 3.7 and 3.9, 20^3 2.8 and 3.8).
  if (n < 15) return false;
  const double rows = (double)ntheta * nshift;
  if (rows * nphi < 4000) return false;
  const bool paired = nphi % 2 == 0;
  return rows * (paired ? 1.0 : 0.5) >= n * (7.0 + 0.4 * n / (paired ? nphi / 2 : nphi));
}

// Cells of the fixed axis whose tables are made together, by the sizes alone: a plane's
// sum is added up group by group.  All of them up to n = 512.
static int axis_cells(int n) {
  const size_t cell = 4 * (size_t)kAxisSlots * n * 4;  // of four phis
  return (int)std::min<size_t>(n, std::max<size_t>(1, ((size_t)512 << 20) / cell));
}
static size_t axis_workspace(const ProfReq &r, int nphis) {
  return nphis * (axis_head_bytes(r.n, r.ntheta) + (size_t)kAxisSlots * axis_cells(r.n) * r.n * 4) + 256;
}

// The least workspace a request can be computed in: that of one unit.
size_t profile_workspace_least(const ProfReq &r, float crop) {
  size_t ws = 1 << 20;
  while (!Areas(ws).fits(unit_bytes(r, crop), chunk_group(r), UnitBytes())) ws += ws / 16;
  if (r.nearest) ws = al(ws) + al(axis_workspace(r, 4));
  return ws;
}

// The workspace a set of requests asks for: all units at once, or enough to fill a
// step.
size_t profile_workspace_want(const ProfReq *reqs, const float *crop, int nreq) {
  size_t table = 0, least = 0;
  for (int q = 0; q < nreq; ++q) {
    const ProfReq &r = reqs[q];
    const int nbase = r.paired ? r.nphi / 2 : r.nphi;
    int c0, c1;
    chunk_range(r, crop[q], &c0, &c1);
    const size_t u = unit_bytes(r, crop[q]).table;
    // a lane's share of a single request is whole phis
    table += u * std::min(c1 - c0, chunk_group(r)) * (nreq == 1 ? (nbase + kProfLanes - 1) / kProfLanes * kProfLanes : nbase);
    least = std::max(least, profile_workspace_least(r, crop[q]));
  }
  const size_t ws = std::min(table, kProfTableBytes) / 176 * 256 + (4 << 20);
  // (the tables of the nearest sampler's phis on an axis come first)
  return std::max(least, reqs[0].nearest ? ws + al(axis_workspace(reqs[0], 4)) : ws);
}

static int axis_forward(wrt_ctx *ctx, cudaStream_t stream, const ProfReq &r, const int *phis, int nphis,
                        void *ws) {
  const int cells = axis_cells(r.n);
  AxisJob a = {};
  a.r = r;
  for (int p = 0; p < nphis; ++p) a.phi[p] = phis[p];
  a.head = static_cast<char *>(ws);
  a.head_bytes = axis_head_bytes(r.n, r.ntheta);
  a.table = reinterpret_cast<float *>(a.head + a.head_bytes * nphis);
  axis_prepare_kernel<<<nphis, kThreads, 0, stream>>>(a);
  ctx->launches++;
  const int groups = (r.n + kAxisThreads - 1) / kAxisThreads;
  for (a.a0 = 0; a.a0 < r.n; a.a0 += a.na) {
    a.na = std::min(cells, r.n - a.a0);
    a.first = a.a0 == 0;
    axis_table_kernel<<<dim3(a.na * groups, nphis), kAxisThreads, 0, stream>>>(a);
    axis_rows_kernel<<<dim3(r.ntheta * r.nshift, nphis), kAxisThreads, 0, stream>>>(a);
    ctx->launches += 2;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WRT_OK : cuda_fail(ctx, e, "row sums on an axis");
}

int profile_lanes_init(wrt_ctx *ctx, ProfLanes *l) {
  if (l->fork) return WRT_OK;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < kProfLanes - 1 && e == cudaSuccess; ++k) {
    if (!l->stream[k]) e = cudaStreamCreateWithFlags(&l->stream[k], cudaStreamNonBlocking);
    if (e == cudaSuccess && !l->done[k])
      e = cudaEventCreateWithFlags(&l->done[k], cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&l->fork, cudaEventDisableTiming);
  return e == cudaSuccess ? WRT_OK : cuda_fail(ctx, e, "profile streams");
}

void profile_lanes_release(ProfLanes *l) {
  for (int k = 0; k < kProfLanes - 1; ++k) {
    if (l->stream[k]) cudaStreamDestroy(l->stream[k]);
    if (l->done[k]) cudaEventDestroy(l->done[k]);
  }
  if (l->fork) cudaEventDestroy(l->fork);
  *l = ProfLanes();
}

int profile_forward(wrt_ctx *ctx, cudaStream_t stream, ProfLanes *lanes, const ProfReq *reqs,
                    const float *crop, int nreq, void *ws, size_t ws_bytes, ProfFork fork) {
  if (nreq < 1) return WRT_OK;
  const bool near = reqs[0].nearest != 0;
  // ---- lanes: the launches of a step depend on one another and each ends with
  // a few late blocks, so different phis run on several streams side by side,
  // each with its share of the workspace
  size_t table = 0;
  for (int q = 0; q < nreq; ++q)
    table += unit_bytes(reqs[q], crop[q]).table * (reqs[q].paired ? reqs[q].nphi / 2 : reqs[q].nphi);
  const bool forked = fork == PROF_BESIDE;
  const int most = forked ? kProfLanes - 1 : kProfLanes;
  int nl = table >= kProfLaneBytes ? most : 1;
  for (int q = 0; q < nreq; ++q)  // every request has to fit a lane
    while (nl > 1 && !Areas(ws_bytes / nl & ~(size_t)255)
                          .fits(unit_bytes(reqs[q], crop[q]), chunk_group(reqs[q]), UnitBytes()))
      --nl;
  if (nl > 1 && fork == PROF_ALONE) {
    int st = profile_lanes_init(ctx, lanes);
    if (st) return st;
  }
  // lane l's stream: the caller's is lane 0 unless it has other work
  auto lane_of = [&](int l) {
    return forked ? lanes->stream[l] : l ? lanes->stream[l - 1] : stream;
  };
  const size_t share = ws_bytes / nl & ~(size_t)255;
  const Areas area(share);
  // ---- jobs: groups of phis of one request, dealt to the lanes
  struct Job {
    int req, base0, nbase, c0, c1, c;
  };
  std::vector<std::vector<Job>> jobs(nl);
  std::vector<int> home(nreq);  // the lane of all of a request's jobs, or -1
  size_t dealt = 0;
  for (int q = 0; q < nreq; ++q) {
    const ProfReq &r = reqs[q];
    const UnitBytes b = unit_bytes(r, crop[q]);
    const int nbase = r.paired ? r.nphi / 2 : r.nphi;
    int fit = 1;
    const int group = chunk_group(r);
    while (fit < nbase && fit < 0xffff && area.fits(b, (size_t)group * (fit + 1), UnitBytes())) ++fit;
    int groups = (nbase + fit - 1) / fit;
    if (nreq == 1 && nl > 1 && nbase >= nl) groups = (groups + nl - 1) / nl * nl;
    groups = std::min(groups, nbase);
    home[q] = groups == 1 ? (int)(dealt % nl) : -1;
    for (int k = 0; k < groups; ++k) {
      Job j;
      j.req = q;
      j.base0 = (int)((long long)nbase * k / groups);
      j.nbase = (int)((long long)nbase * (k + 1) / groups) - j.base0;
      chunk_range(r, crop[q], &j.c0, &j.c1);
      j.c = j.c0;
      jobs[dealt++ % nl].push_back(j);
    }
  }
  cudaError_t e = cudaSuccess;
  if (nl > 1 && fork == PROF_ALONE) e = cudaEventRecord(lanes->fork, stream);
  for (int l = forked ? 0 : 1; l < nl && e == cudaSuccess; ++l)
    e = cudaStreamWaitEvent(lane_of(l), lanes->fork, 0);
  // nothing may still use the workspace when a failed call returns
  auto failed = [&](const char *what) {
    for (int l = 0; l < nl; ++l) cudaStreamSynchronize(lane_of(l));
    return cuda_fail(ctx, e, what);
  };
  if (e != cudaSuccess) return failed("profile fork");
  // ---- steps, lane by lane: of every job still open one group of ranges of t (a
  // group adds to the sums of the one before, so they go to different steps), as
  // many jobs as the lane's workspace holds
  std::vector<ProfSeg> out;
  for (bool any = true; any;) {
    any = false;
    for (int l = 0; l < nl; ++l) {
      out.clear();
      UnitBytes had = {};
      char *base = static_cast<char *>(ws) + share * l;
      char *rec = base + area.table, *place = rec + area.rec, *keys = place + area.place;
      unsigned long long *list = reinterpret_cast<unsigned long long *>(keys + area.keys);
      for (Job &j : jobs[l]) {
        if (j.c >= j.c1) continue;
        const ProfReq &r = reqs[j.req];
        const UnitBytes u = unit_bytes(r, crop[j.req]);
        const int group = chunk_group(r), nc = std::min(j.c1, (j.c / group + 1) * group) - j.c;
        if ((int)out.size() >= kManySegs || !area.fits(u, (size_t)j.nbase * nc, had)) break;
        const size_t units = (size_t)j.nbase * nc;
        ProfSeg s = {};
        s.r = r;
        s.chunk = j.c;
        s.nchunk = nc;
        s.base0 = j.base0;
        s.nbase = j.nbase;
        s.first = j.c == j.c0;
        s.cap = unit_cap(r.n, crop[j.req]);
        s.sub_bins = std::min(r.n, kUnitBins);
        s.nsub = (kUnitBins + s.sub_bins - 1) / s.sub_bins;
        const long long warps =
            (long long)r.ntheta * ((r.nshift + 31) / 32) * (r.paired ? 2 : 1);
        s.blk_rows = (int)((warps + kThreads / 32 - 1) / (kThreads / 32));
        s.table = base + had.table;
        s.rec = rec + had.rec;
        s.keys = reinterpret_cast<unsigned long long *>(keys + had.keys);
        s.pos = reinterpret_cast<unsigned *>(place + had.pos + had.start);
        s.ids = s.pos + (size_t)(s.cap + 16) * units;
        s.start = reinterpret_cast<unsigned *>(place + had.pos + had.start + u.pos * units);
        had.table += u.table * units;
        had.rec += u.rec * units;
        had.keys += u.keys * units;
        had.pos += u.pos * units;
        had.start += u.start * units;
        had.list += u.list * units;
        out.push_back(s);
        j.c += nc;
      }
      if (out.empty()) continue;
      any = true;
      const cudaStream_t ls = lane_of(l);
      if (near)
        e = out.size() == 1 ? launch_step<true, 1>(ctx, ls, out, list)
                            : launch_step<true, kManySegs>(ctx, ls, out, list);
      else
        e = out.size() == 1 ? launch_step<false, 1>(ctx, ls, out, list)
                            : launch_step<false, kManySegs>(ctx, ls, out, list);
      if (e != cudaSuccess) return failed("row-sum profile kernels");
    }
  }
  // samples that no table holds: behind the request's last step where that is
  // one lane's, else behind the join
  auto extra = [&](int q, cudaStream_t where) {
    const ProfReq &r = reqs[q];
    // the nearest sampler's phis on an axis are not tabulated at all
    if (r.nearest && !r.paired) return cudaSuccess;
    const double left = (double)crop[q] * r.n * r.n;
    const bool axis = !r.nearest && ((r.n & 1) || (double)r.n * r.n <= left);
    if (!axis && !(r.paired && (double)r.L * r.L <= left)) return cudaSuccess;
    const long long planes = (long long)r.nphi * r.ntheta * r.nshift;
    profile_extra_kernel<<<(unsigned)((planes + kThreads / 32 - 1) / (kThreads / 32)), kThreads, 0,
                           where>>>(r);
    ctx->launches++;
    return cudaGetLastError();
  };
  for (int q = 0; q < nreq && e == cudaSuccess; ++q)
    if (home[q] >= 0) e = extra(q, lane_of(home[q]));
  const cudaStream_t home_stream = lane_of(0);
  for (int l = 1; l < nl && e == cudaSuccess; ++l) {
    const int k = forked ? l : l - 1;
    e = cudaEventRecord(lanes->done[k], lanes->stream[k]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(home_stream, lanes->done[k], 0);
  }
  for (int q = 0; q < nreq && e == cudaSuccess; ++q)
    if (home[q] < 0) e = extra(q, home_stream);
  if (forked && e == cudaSuccess) e = cudaEventRecord(lanes->done[0], home_stream);
  return e == cudaSuccess ? WRT_OK : failed("row-sum profiles");
}

// The phis on an axis beside the others: their first kernel is a few blocks only.  A
// small request's others are on one side stream, a large one's on all lanes.
int profile_forward_nearest(wrt_ctx *ctx, cudaStream_t stream, ProfLanes *lanes, const ProfReq &r,
                            float crop, const int *phis, int nphis, void *ws, size_t ws_bytes) {
  if (!nphis) return profile_forward(ctx, stream, lanes, &r, &crop, 1, ws, ws_bytes);
  int st = profile_lanes_init(ctx, lanes);
  if (st) return st;
  cudaError_t e = cudaEventRecord(lanes->fork, stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "profile fork");
  const size_t part = al(axis_workspace(r, nphis));
  char *rest = static_cast<char *>(ws) + part;
  const bool small = unit_bytes(r, crop).table * (r.paired ? r.nphi / 2 : r.nphi) < kProfLaneBytes;
  if (small) {
    st = profile_forward(ctx, stream, lanes, &r, &crop, 1, rest, ws_bytes - part, PROF_BESIDE);
    if (st) return st;
  }
  st = axis_forward(ctx, stream, r, phis, nphis, ws);
  if (!small)
    return st ? st : profile_forward(ctx, stream, lanes, &r, &crop, 1, rest, ws_bytes - part,
                                     PROF_FORKED);
  e = cudaStreamWaitEvent(stream, lanes->done[0], 0);
  return st || e == cudaSuccess ? st : cuda_fail(ctx, e, "profile join");
}

}  // namespace wrt
