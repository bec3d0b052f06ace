// k_backproj.cu -- the backprojection (radon_inversion/backprojection/C/src/
// integral.c:6-24, interp.c:5-28) from splines merged over the latitudes.
//
// With t = x cos phi + y sin phi a voxel's line coordinate is s = sin theta t +
// cos theta z, so for one longitude and one z the sum over the latitudes
//
//   H(t) = sum_theta w S_theta(sin theta t + cos theta z)
//
// is ONE function of t: a cubic spline whose knots are those of all the
// latitudes, ntheta nshift / 2.. of them on the cube.  Its pieces are summed up
// once (build role: one change of the third derivative per knot) and a voxel
// then costs one table read per longitude instead of one per direction.  The
// knots' places do not depend on the longitude, so one sorted list per z serves
// all of them, and the two directions (phi, theta) and (phi + pi, pi - theta) of
// opposite normals are one line read both ways, so their data are added first
// (even nphi).
//
//   merge:  R[is][phi][theta] -> Y[theta][is][phi < nphi/2], weights applied
//   solve:  natural splines in FP64; m = h^2/6 times the second derivatives, D =
//           the knots' changes of the third derivative in t
//   sort:   per z, the knots' positions in order (bins, ranked by counting)
//   build:  per z and range of t, lanes on longitudes: the cubic about the
//           range's start from the lines directly, then one knot after another,
//           each piece's coefficients at its own start rounded once to FP32
//   (lines: one with a value that is no number has none that is, and a running sum
//           would keep it beyond the line's end, so such lines are listed and zeroed by
//           the solve and their voxels set once the sums are done)
//   gather: threads on voxels of one z, the list's positions in shared memory,
//           one 16-byte record per (voxel, longitude); FP64 sums, every voxel
//           in a fixed order by one thread
//
// A voxel within 2 positions (1.3e-9 in t) of the end of a line, where S jumps to
// zero, is decided by the FP64 position of the direction itself, as in the
// direct kernel (k_spline.cu).  That kernel stays for small direction sets and
// for what has no working memory.
//
// What bounds it: the gather's record loads (one line per lane; L1 at 81 % of its
// throughput on the SMs that a launch keeps busy, more than half of a warp's cycles spent
// waiting), the build's latency.
// 128^3 from 64 x 128 directions x 256 shifts: 15.9 ms by the direct kernel (16
// bytes and ~7 instructions per voxel and direction), 1.77 here; 256^3 from 96 x
// 192 x 384: 237 and 20 ms; error against FP64 (128^3) 6.5e-9 and 4.8e-9.
#include <math.h>

#include <algorithm>
#include <vector>

#include "backproj_dev.cuh"
#include "wrt_internal.cuh"

namespace {

using wrt::BackReq;
using wrt::BackStep;
using namespace wrtb;

constexpr unsigned kAll = 0xffffffffu;
constexpr int kThreads = 256;
constexpr int kSortThreads = 512;
constexpr int kGatherThreads = 512;
constexpr int kVox = 4;  // voxels per thread of the gather
constexpr int kRecTile = 128;
constexpr unsigned kEdge = 2;

enum { K_KNOT = 0, K_NULL = 1, K_IN = 2, K_OUT = 3 };
struct KnotRec {
  double tau;  // t from the range's start
  int off;     // element offset of (theta, knot, longitude 0)
  int kind;    // K_*, theta << 2
};

__device__ __forceinline__ double z_of(int n, int iz) {
  return (-1.0) + (1.0 / n) + iz * (2.0 / n);  // radon3d_ajoint.c:248-250
}

// Y[theta][i][b] = weight x data of direction (b, theta), plus those of the
// opposite direction read backwards; 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(kThreads) back_merge_kernel(const BackReq r) {
  __shared__ double tile[32][33];
  const int i = blockIdx.z, b0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if ((blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) r.lost[0] = 0;
  for (int y = ty; y < 32; y += kThreads / 32) {
    const int b = b0 + y, th = t0 + tx;
    if (b < r.nbase && th < r.ntheta) {
      double v = r.dirw[(size_t)b * r.ntheta + th].w *
                 r.radon[((size_t)i * r.nphi + b) * r.ntheta + th];
      if (r.paired) {
        const int ot = r.ntheta - 1 - th;
        v += r.dirw[(size_t)(b + r.nbase) * r.ntheta + ot].w *
             r.radon[((size_t)(r.ns - 1 - i) * r.nphi + b + r.nbase) * r.ntheta + ot];
      }
      tile[y][tx] = v;
    }
  }
  __syncthreads();
  for (int y = ty; y < 32; y += kThreads / 32) {
    const int th = t0 + y, b = b0 + tx;
    if (b < r.nbase && th < r.ntheta) r.Y[((size_t)th * r.ns + i) * r.nbase + b] = tile[tx][y];
  }
}

// m_{i-1} + 4 m_i + m_{i+1} = y_{i+1} - 2 y_i + y_{i-1} with m_0 = m_{ns-1} = 0
// (elimination factors cp from the host), one thread per line, lanes on
// longitudes; on the way back the changes of the third derivative.  Bound by latency
// (a few warps per SM, two chains of ns steps), so the loads of 16 steps are issued
// together: the compiler cannot move one past the stores (40^3 from 50 x 100 x 220:
// 455 -> 427 us in all, 334 with the lists sorted beside it).
__global__ void __launch_bounds__(64) back_solve_kernel(const BackReq r) {
  const int L = blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= r.ntheta * r.nbase) return;
  const int th = L / r.nbase, b = L % r.nbase, ns = r.ns;
  const size_t st = r.nbase, o = (size_t)th * ns * st + b;
  const double *__restrict__ y = r.Y + o, *__restrict__ cp = r.cp;
  double *__restrict__ m = r.M + o, *__restrict__ D = r.D + o;
  const double kap = r.cs[2 * th + 1] * 0.5 * (ns - 1), k3 = kap * kap * kap;
  constexpr int U = 16;  // elements whose loads are in flight together
  double prev = 0.0, ya = y[0], yb = y[st];
  m[0] = 0.0;
  for (int i0 = 1; i0 + 1 < ns; i0 += U) {
    double v[U], w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u, ns - 2);
      v[u] = y[(i + 1) * st];
      w[u] = cp[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u;
      if (i + 1 >= ns) break;
      prev = ((v[u] - 2.0 * yb + ya) - (i > 1 ? prev : 0.0)) * w[u];
      m[i * st] = prev;
      ya = yb;
      yb = v[u];
    }
  }
  if (!(fabs(prev) < 1e300)) {  // every y enters it
    r.lost[1 + atomicAdd(r.lost, 1)] = L;
    for (int i = 0; i < ns; ++i) r.Y[o + i * st] = m[i * st] = D[i * st] = 0.0;
    return;
  }
  // from the end: mc = m_{i+1}, md = m_{i+2}
  double mc = 0.0, md = 0.0;
  m[(ns - 1) * st] = 0.0;
  for (int i0 = ns - 2; i0 >= 0; i0 -= U) {
    double v[U], w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = max(i0 - u, 1);
      v[u] = m[i * st];
      w[u] = cp[i];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 - u;
      if (i < 0) break;
      const double mi = i ? v[u] - w[u] * mc : 0.0;
      m[i * st] = mi;
      // the knot i + 1: its intervals' cubic coefficients are m_{i+2} - m_{i+1}
      // above and m_{i+1} - m_i below
      D[(i + 1) * st] = (i + 1 == ns - 1 ? -(mc - mi) : (md - mc) - (mc - mi)) * k3;
      md = mc;
      mc = mi;
    }
  }
  D[0] = (md - mc) * k3;
}

// ------------------------------------------------------------------ per z: sort
__global__ void __launch_bounds__(kSortThreads) back_sort_kernel(const BackStep s) {
  extern __shared__ int cnt[];  // [nb]
  __shared__ int s_warp[kSortThreads / 32];
  const BackReq &r = s.r;
  const int zi = blockIdx.x, tid = threadIdx.x, ns = r.ns;
  const double z = z_of(r.n, s.z0 + zi);
  const int nb = s.nb, shift = 32 - s.nb_log2, sub_shift = 32 - s.nsub_log2;
  unsigned *pos = s.pos + (size_t)zi * (s.cap + 16), *ids = s.ids + (size_t)zi * (s.cap + 16);
  unsigned *start = s.start + (size_t)zi * (nb + 8);
  unsigned long long *keys = s.keys + (size_t)zi * s.cap;
  for (int b = tid; b < nb; b += kSortThreads) cnt[b] = 0;
  __syncthreads();
  const int nsub = 1 << s.nsub_log2;
  // a warp per latitude, lanes on its knots; the range starts last
  auto each = [&](auto f) {
    for (int th = tid >> 5; th < r.ntheta; th += kSortThreads / 32) {
      const Lat l = lat_of(r.cs[2 * th], r.cs[2 * th + 1], z, ns);
      int lo, hi;
      knot_range(l, ns, &lo, &hi);
      for (int i = lo + (tid & 31); i <= hi; i += 32) {
        const long long p = knot_pos(l, i);
        if (p >= 0 && p < 0x100000000LL) f((unsigned)p, (unsigned)(th * ns + i) + 1u);
      }
    }
    for (int k = tid; k < nsub; k += kSortThreads) f((unsigned)k << sub_shift, 0u);
  };
  each([&](unsigned p, unsigned) { atomicAdd(&cnt[p >> shift], 1); });
  __syncthreads();
  // exclusive scan of the bins
  const int per = nb / kSortThreads;
  int sum = 0;
  for (int q = 0; q < per; ++q) sum += cnt[tid * per + q];
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kAll, incl, o);
    if ((tid & 31) >= o) incl += t;
  }
  if ((tid & 31) == 31) s_warp[tid >> 5] = incl;
  __syncthreads();
  int before = incl - sum, total = 0;
  for (int w = 0; w < kSortThreads / 32; ++w) {
    if (w < (tid >> 5)) before += s_warp[w];
    total += s_warp[w];
  }
  for (int q = 0; q < per; ++q) {
    const int b = tid * per + q, c = cnt[b];
    start[b] = before;
    cnt[b] = before;
    before += c;
  }
  if (tid == 0) start[nb] = total;
  __syncthreads();
  each([&](unsigned p, unsigned id) {
    const int slot = atomicAdd(&cnt[p >> shift], 1);
    if (slot < s.cap) keys[slot] = (unsigned long long)p << 32 | id;
  });
  __syncthreads();
  total = min(total, s.cap);  // cap = every knot and range start; never exceeded
  KnotRec *rec = static_cast<KnotRec *>(s.rec) + (size_t)zi * s.cap;
  for (int e = tid; e < total; e += kSortThreads) {
    const unsigned long long key = keys[e];
    const unsigned p = (unsigned)(key >> 32), id = (unsigned)key;
    const int b = p >> shift, b0 = start[b], b1 = start[b + 1];
    int rank = 0;
    for (int q = b0; q < min(b1, total); ++q) rank += keys[q] < key;
    const int dst = b0 + rank;
    pos[dst] = p;
    ids[dst] = id;
    KnotRec k;
    const int th = id ? (int)((id - 1u) / ns) : 0, i = id ? (int)((id - 1u) % ns) : 0;
    k.tau = id ? knot_tau(lat_of(r.cs[2 * th], r.cs[2 * th + 1], z, ns), i,
                          (long long)(p >> sub_shift) << sub_shift)
               : 0.0;
    k.off = (th * ns + i) * r.nbase;
    k.kind = (id == 0 ? K_NULL : i == 0 ? K_IN : i == ns - 1 ? K_OUT : K_KNOT) | th << 2;
    rec[dst] = k;
  }
  if (tid < 16) pos[total + tid] = 0xffffffffu;
}

// ----------------------------------------------------------------- per z: build
struct StartLat {  // a latitude's line at a range's start
  double b, kap;   // fraction of the knot interval, knots per t
  double on, k1, k2, k3;  // 1 and kap, kap^2, kap^3, or 0 off the line
  long long off;   // the interval's element offset
};

__global__ void __launch_bounds__(kThreads) back_build_kernel(const BackStep s) {
  extern __shared__ __align__(16) char smem[];
  KnotRec *tile = reinterpret_cast<KnotRec *>(smem);
  StartLat *lats = reinterpret_cast<StartLat *>(tile + kRecTile);
  const BackReq &r = s.r;
  const int nsub = 1 << s.nsub_log2, sub_shift = 32 - s.nsub_log2;
  const int zi = blockIdx.x / nsub, sub = blockIdx.x % nsub;
  const double z = z_of(r.n, s.z0 + zi);
  const int ns = r.ns, B = r.nbase, nth = (int)blockDim.x;
  const long long p0 = (long long)sub << sub_shift;
  const double t0 = (double)p0 / kPerT - kTMax;
  for (int th = threadIdx.x; th < r.ntheta; th += nth) {
    const Lat l = lat_of(r.cs[2 * th], r.cs[2 * th + 1], z, ns);
    const int i = knots_before(l, ns, p0) - 1;
    StartLat a;
    a.kap = l.kap;
    a.b = l.kap * t0 + l.q0 - i;
    a.on = i >= 0 && i <= ns - 2 ? 1.0 : 0.0;
    a.k1 = a.on * l.kap;
    a.k2 = a.k1 * l.kap;
    a.k3 = a.k2 * l.kap;
    a.off = (long long)(th * ns + min(max(i, 0), ns - 2)) * B;
    lats[th] = a;
  }
  __syncthreads();
  const unsigned *start = s.start + (size_t)zi * (s.nb + 8);
  const int per = s.nb >> s.nsub_log2;  // bins per range
  const int e0 = start[sub * per], e1 = start[(sub + 1) * per];
  const KnotRec *rec = static_cast<const KnotRec *>(s.rec) + (size_t)zi * s.cap;
  const int lane = threadIdx.x & 31, warps = nth >> 5;
  const double u1 = 1.0 / kPerT, u2 = u1 * u1, u3 = u2 * u1;
  for (int g0 = 0; g0 * 32 < B; g0 += warps) {
    const int b = (g0 + (threadIdx.x >> 5)) * 32 + lane;
    const bool live = b < B;
    const size_t bc = min(b, B - 1);
    const double *Y = r.Y + bc, *M = r.M + bc, *D = r.D + bc;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll 4
    for (int th = 0; th < r.ntheta; ++th) {
      const StartLat l = lats[th];
      const double y0 = Y[l.off], y1 = Y[l.off + B], m0 = M[l.off], m1 = M[l.off + B];
      const double A = (y1 - y0) - (2.0 * m0 + m1), Bq = 3.0 * m0, C = m1 - m0;
      a0 = fma(l.on, fma(l.b, fma(l.b, fma(l.b, C, Bq), A), y0), a0);
      a1 = fma(l.k1, fma(l.b, fma(3.0 * l.b, C, 2.0 * Bq), A), a1);
      a2 = fma(l.k2, fma(3.0 * l.b, C, Bq), a2);
      a3 = fma(l.k3, C, a3);
    }
    float4 *T = s.table + ((size_t)zi * s.cap) * B + b;
    for (int e = e0; e < e1; e += kRecTile) {
      const int m = min(kRecTile, e1 - e);
      __syncthreads();
      for (int x = threadIdx.x; x < m; x += nth)
        reinterpret_cast<int4 *>(tile)[x] = reinterpret_cast<const int4 *>(rec + e)[x];
      __syncthreads();
      constexpr int U = 8;  // knots whose loads are in flight together
      for (int x = 0; x < m; x += U) {
        double d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) d[u] = __ldg(D + tile[min(x + u, m - 1)].off);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (x + u >= m) break;
          const KnotRec k = tile[x + u];
          const double tau = k.tau;
          const int kind = k.kind & 3;
          const double dd = kind == K_NULL ? 0.0 : d[u];
          if (kind >= K_IN) {
            // a line's first or last knot: value and slope begin or end there
            const double kap = lats[k.kind >> 2].kap;
            const double *y = Y + k.off, *mm = M + k.off;
            const double v = kind == K_IN ? y[0] : -y[0];
            const double sl = kind == K_IN ? kap * ((y[B] - y[0]) - mm[B])
                                           : -kap * ((y[0] - y[-B]) + mm[-B]);
            a0 += fma(-sl, tau, v);
            a1 += sl;
          }
          const double p = dd * tau, q = p * tau;
          a3 += dd;
          a2 = fma(-3.0, p, a2);
          a1 = fma(3.0, q, a1);
          a0 = fma(-q, tau, a0);
          const double t3 = 3.0 * tau * a3;
          const float c0 = (float)fma(tau, fma(tau, fma(tau, a3, a2), a1), a0);
          const float c1 = (float)(fma(tau, fma(2.0, a2, t3), a1) * u1);
          const float c2 = (float)((a2 + t3) * u2);
          const float c3 = (float)(a3 * u3);
          if (live) T[(size_t)(e + x + u) * B] = make_float4(c0, c1, c2, c3);
        }
      }
    }
  }
}

// ---------------------------------------------------------------- per z: gather
// What the table's value lacks for a voxel next to the end of a line: for both
// directions of the merged line, whether the voxel is on the line by the
// direction's own FP64 position.
__device__ __noinline__ double edge_terms(const BackStep &s, int zi, const unsigned *pos, int e,
                                          unsigned fx, int ix, int iy, int b) {
  const BackReq &r = s.r;
  const unsigned *ids = s.ids + (size_t)zi * (s.cap + 16);
  const int total = s.start[(size_t)zi * (s.nb + 8) + s.nb], ns = r.ns;
  const double x = z_of(r.n, ix), y = z_of(r.n, iy), z = z_of(r.n, s.z0 + zi);
  int q0 = e, q1 = e;
  while (q0 > 0 && fx - pos[q0 - 1] <= kEdge) --q0;
  while (q1 < total && pos[q1] - fx <= kEdge) ++q1;
  double sum = 0.0;
  for (int q = q0; q < q1; ++q) {
    const unsigned id = ids[q];
    if (!id) continue;
    const int th = (int)((id - 1u) / ns), i = (int)((id - 1u) % ns);
    if (i != 0 && i != ns - 1) continue;
    bool lost = false;  // not in the table
    for (int k = r.lost[0]; k > 0; --k) lost |= r.lost[k] == th * r.nbase + b;
    if (lost) continue;
    const bool model = (i == 0) == (pos[q] <= fx);
    for (int k = 0; k < (r.paired ? 2 : 1); ++k) {
      const int ph = b + k * r.nbase, t = k ? r.ntheta - 1 - th : th, j = k ? ns - 1 - i : i;
      const double4 g = r.dirw[(size_t)ph * r.ntheta + t];
      const double qk = fma(x, g.x, fma(y, g.y, fma(z, g.z, 0.5 * (ns - 1))));
      const bool on = qk >= 0.0 && qk <= (double)(ns - 1);
      if (on != model)
        sum += (on ? 1.0 : -1.0) * g.w * r.radon[((size_t)j * r.nphi + ph) * r.ntheta + t];
    }
  }
  return sum;
}

__global__ void __launch_bounds__(kGatherThreads, 2) back_gather_kernel(const BackStep s) {
  extern __shared__ __align__(16) char smem[];
  const BackReq &r = s.r;
  const int n = r.n, B = r.nbase, tiles = s.tiles;
  const int zi = blockIdx.x / tiles, tile = blockIdx.x % tiles;
  double2 *dir = reinterpret_cast<double2 *>(smem);             // [B] cos, sin per position
  unsigned *pos = reinterpret_cast<unsigned *>(dir + B);        // [cap + 16]
  unsigned short *start = reinterpret_cast<unsigned short *>(pos + s.cap + 16);
  const int tid = threadIdx.x, shift = 32 - s.nb_log2;
  const unsigned *gstart = s.start + (size_t)zi * (s.nb + 8);
  const unsigned *gpos = s.pos + (size_t)zi * (s.cap + 16);
  const int total = gstart[s.nb];
  for (int k = tid; k < total + 16; k += kGatherThreads) pos[k] = gpos[k];
  for (int k = tid; k < s.nb; k += kGatherThreads) start[k] = (unsigned short)gstart[k];
  for (int k = tid; k < B; k += kGatherThreads) {
    const double *D = r.dir + 9 * (size_t)k * r.ntheta;  // v2 = (-sin phi, cos phi, 0)
    dir[k] = make_double2(D[7] * kPerT, -D[6] * kPerT);
  }
  __syncthreads();
  const float4 *T = s.table + (size_t)zi * s.cap * B;
  const int n2 = n * n;
  for (int v0 = tile * kGatherThreads * kVox; v0 < n2; v0 += tiles * kGatherThreads * kVox) {
    double x[kVox], y[kVox], tot[kVox];
#pragma unroll
    for (int u = 0; u < kVox; ++u) {
      const int v = min(v0 + u * kGatherThreads + tid, n2 - 1);
      x[u] = z_of(n, v / n);
      y[u] = z_of(n, v % n);
      tot[u] = 0.0;
    }
    for (int b = 0; b < B; ++b) {
      const double2 cs = dir[b];
      unsigned fx[kVox], nx[kVox], dt[kVox];
      int e[kVox];
      bool more = false, edge = false;
#pragma unroll
      for (int u = 0; u < kVox; ++u) {
        const double p = fma(x[u], cs.x, fma(y[u], cs.y, kTMax * kPerT));
        fx[u] = (unsigned)__double2loint(__dadd_rd(p, 4503599627370496.0));  // floor, + 2^52
        e[u] = start[fx[u] >> shift];
      }
#pragma unroll
      for (int h = 8; h > 0; h >>= 1)
#pragma unroll
        for (int u = 0; u < kVox; ++u)
          if (pos[e[u] + h - 1] <= fx[u]) e[u] += h;
#pragma unroll
      for (int u = 0; u < kVox; ++u) {
        nx[u] = pos[e[u]];
        more |= nx[u] <= fx[u] && e[u] < total;
      }
      if (more) {
#pragma unroll 1
        for (int u = 0; u < kVox; ++u) {
          int q = u == 0 ? e[0] : u == 1 ? e[1] : u == 2 ? e[2] : e[3];
          const unsigned f = u == 0 ? fx[0] : u == 1 ? fx[1] : u == 2 ? fx[2] : fx[3];
          while (q < total && pos[q] <= f) ++q;
          if (u == 0) e[0] = q;
          else if (u == 1) e[1] = q;
          else if (u == 2) e[2] = q;
          else e[3] = q;
        }
#pragma unroll
        for (int u = 0; u < kVox; ++u) nx[u] = pos[e[u]];
      }
#pragma unroll
      for (int u = 0; u < kVox; ++u) {
        dt[u] = fx[u] - pos[e[u] - 1];
        edge |= dt[u] <= kEdge || nx[u] - fx[u] <= kEdge;
      }
      float4 c[kVox];
#pragma unroll
      for (int u = 0; u < kVox; ++u) c[u] = __ldg(T + (size_t)(unsigned)(e[u] - 1) * B + b);
#pragma unroll
      for (int u = 0; u < kVox; ++u) {
        const float d = (float)dt[u];
        // FP64 at once: two longitudes in FP32 first were 7.5e-9 from FP64 at 128^3 (the
        // direct kernel 6.5e-9, this 4.8e-9) and 1.85 ms instead of 1.77
        tot[u] += (double)fmaf(d, fmaf(d, fmaf(d, c[u].w, c[u].z), c[u].y), c[u].x);
      }
      if (edge) {
#pragma unroll
        for (int u = 0; u < kVox; ++u)
          if (dt[u] <= kEdge || nx[u] - fx[u] <= kEdge) {
            const int v = min(v0 + u * kGatherThreads + tid, n2 - 1);
            tot[u] += edge_terms(s, zi, pos, e[u], fx[u], v / n, v % n, b);
          }
      }
    }
#pragma unroll
    for (int u = 0; u < kVox; ++u) {
      const int v = v0 + u * kGatherThreads + tid;
      if (v < n2) r.out[(size_t)(s.z0 + zi) * n2 + v] = tot[u];
    }
  }
}

// The voxels on the lines that the solve has listed, as a rule none.
__global__ void __launch_bounds__(kThreads) back_lost_kernel(const BackReq r) {
  const int lost = r.lost[0], n = r.n, ns = r.ns;
  if (!lost) return;
  const long long total = (long long)n * n * n;
  for (long long v = blockIdx.x * (long long)kThreads + threadIdx.x; v < total;
       v += (long long)gridDim.x * kThreads) {
    const double z = z_of(n, (int)(v / ((long long)n * n))), x = z_of(n, (int)(v / n % n)),
                 y = z_of(n, (int)(v % n));
    for (int k = 1; k <= lost; ++k) {
      const int th = r.lost[k] / r.nbase, b = r.lost[k] % r.nbase;
      const double4 g = r.dirw[(size_t)b * r.ntheta + th];
      const double q = fma(x, g.x, fma(y, g.y, fma(z, g.z, 0.5 * (ns - 1))));
      if (!(q >= 0.0 && q <= (double)(ns - 1))) continue;
      r.out[v] = __longlong_as_double(0x7ff8000000000000ll);
      break;
    }
  }
}

size_t al(size_t x) { return (x + 255) & ~(size_t)255; }
int log2_up(int x) {
  int k = 0;
  while ((1 << k) < x) ++k;
  return k;
}

struct Plan {
  int cap, nb_log2, nsub_log2, nbase;
  size_t data, lost, table, rec, pos, start, keys;  // data: Y, M, D each; from table on per z
  size_t list() const { return rec + pos + start + keys; }  // of one z plane
};
Plan plan_of(int nphi, int ntheta, int ns) {
  Plan p;
  p.nbase = nphi % 2 == 0 ? nphi / 2 : nphi;
  const int knots = ntheta * ns;
  p.nsub_log2 = std::max(1, log2_up(knots) - 8);  // ~256 knots a range
  p.cap = knots + (1 << p.nsub_log2);
  // at least one bin per thread of the sort and per range
  p.nb_log2 = std::max({log2_up(knots) - 2, 9, p.nsub_log2});
  p.data = al(sizeof(double) * (size_t)knots * p.nbase);
  p.lost = al(sizeof(int) * ((size_t)ntheta * p.nbase + 1));
  p.table = al(16 * (size_t)p.cap * p.nbase);
  p.rec = al(sizeof(KnotRec) * (size_t)p.cap);
  p.pos = al(2 * 4 * (size_t)(p.cap + 16));
  p.start = al(4 * (size_t)((1 << p.nb_log2) + 8));
  p.keys = al(8 * (size_t)p.cap);
  return p;
}
size_t gather_smem(const Plan &p) {
  return 16 * (size_t)p.nbase + 4 * (size_t)(p.cap + 16) + 2 * ((size_t)1 << p.nb_log2);
}
size_t build_smem(int ntheta) {
  return kRecTile * sizeof(KnotRec) + sizeof(StartLat) * (size_t)ntheta;
}
constexpr size_t kMostSmem = 220 * 1024;

}  // namespace

namespace wrt {

bool backproj_covers(int nphi, int ntheta, int ns, int n) {
  const long long knots = (long long)ntheta * ns;
  // the list's positions and the latitudes fit shared memory; larger than the allocation-free
  // path takes, whose volume is the direct kernel's bit for bit.  Measured beyond
  // that (n 16 .. 256, 41 .. 96 latitudes): never slower than the direct kernel,
  // which takes at least 0.43 us per direction, e.g. 33^3 from 64 x 128 x 256 in
  // 3.6 ms against 0.7 here
  if (knots > 50000 || ns < 3 || n > 2048 || (long long)nphi * knots <= 262144) return false;
  if ((long long)nphi * knots > (1LL << 30)) return false;
  return gather_smem(plan_of(nphi, ntheta, ns)) <= kMostSmem && build_smem(ntheta) <= kMostSmem;
}

// Streams of a backprojection with nz z planes in flight, planes on each.
static int lanes_of(int n, int nz) { return nz >= kProfLanes && n >= 2 * kProfLanes ? kProfLanes : 1; }

// The fewest planes in flight that are not slower than the direct kernel.  With few of
// them a round is one long chain, up to 3.2 us a longitude tabulated; the direct kernel
// takes 0.43 us a direction, or 0.93 ps a direction and voxel.  Planes in flight, merged
// and direct: 128^3 from 64 x 128 x 256 1: 26.7 ms, 7: 7.2, 20: 2.0, direct 15.9; 64^3 from
// 33 x 65 x 129 4: 2.5 ms, 13: 1.01, 30: 0.57, direct 0.94; 40^3 from 50 x 100 x 220 2: 2.9,
// 7: 1.5, 18: 0.57, direct 2.2.
static int least_planes(int nphi, int ntheta, int n, int nbase) {
  const double voxels = (double)n * n * n;
  const double direct = (double)nphi * ntheta * std::max(0.43, 0.93e-6 * voxels);
  for (int nz = 1; nz < n; ++nz) {
    const int nl = lanes_of(n, nz), in_flight = std::max(1, nz / nl) * nl;
    if ((n + in_flight - 1) / in_flight * 3.2 * nbase <= 0.9 * direct) return nz;
  }
  return n;
}

// Working memory: the lines' Y, M and D, the sorted lists of every z plane, and
// the tables of the planes in flight.
size_t backproj_workspace(int nphi, int ntheta, int ns, int n, bool least) {
  const Plan p = plan_of(nphi, ntheta, ns);
  const size_t most = std::min<size_t>(n, std::max<size_t>(1, kBackTableBytes / p.table));
  const size_t z = least ? std::min<size_t>(most, least_planes(nphi, ntheta, n, p.nbase)) : most;
  return 3 * p.data + p.lost + n * p.list() + z * p.table + 4096;
}

int backproj_forward(wrt_ctx *ctx, cudaStream_t stream, ProfLanes *lanes, BackReq r, void *ws,
                     size_t ws_bytes) {
  const Plan p = plan_of(r.nphi, r.ntheta, r.ns);
  r.paired = r.nphi % 2 == 0;
  r.nbase = p.nbase;
  char *at = static_cast<char *>(ws);
  r.Y = reinterpret_cast<double *>(at);
  r.M = reinterpret_cast<double *>(at + p.data);
  r.D = reinterpret_cast<double *>(at + 2 * p.data);
  r.lost = reinterpret_cast<int *>(at + 3 * p.data);
  at += 3 * p.data + p.lost;
  cudaError_t e = cudaSuccess;
  // ---- z planes, dealt in groups to the lanes
  char *lists = at;
  at += (size_t)r.n * p.list();
  const size_t left = ws_bytes - (at - static_cast<char *>(ws));
  const int nz = (int)std::max<size_t>(1, std::min<size_t>(r.n, left / p.table));
  const int nl = lanes_of(r.n, nz);
  // nothing may still use the workspace when a failed call returns
  auto failed = [&](cudaError_t err) {
    cudaStreamSynchronize(stream);
    for (int k = 0; nl > 1 && k < kProfLanes - 1; ++k) cudaStreamSynchronize(lanes->stream[k]);
    return cuda_fail(ctx, err, "merged backprojection");
  };
  const size_t sm_sort = 4 * ((size_t)1 << p.nb_log2);
  const size_t sm_build = build_smem(r.ntheta);
  const size_t sm_gather = gather_smem(p);
  if (e == cudaSuccess && sm_sort > 48 * 1024) e = allow_smem(back_sort_kernel, kMostSmem);
  if (e == cudaSuccess && sm_build > 48 * 1024) e = allow_smem(back_build_kernel, kMostSmem);
  if (e == cudaSuccess && sm_gather > 48 * 1024) e = allow_smem(back_gather_kernel, kMostSmem);
  // ---- the lists of all z planes
  BackStep s0 = {};
  s0.r = r;
  s0.cap = p.cap;
  s0.nb_log2 = p.nb_log2;
  s0.nb = 1 << p.nb_log2;
  s0.nsub_log2 = p.nsub_log2;
  s0.tiles = (r.n * r.n + kGatherThreads * kVox - 1) / (kGatherThreads * kVox);
  s0.rec = lists;
  s0.pos = reinterpret_cast<unsigned *>(lists + (size_t)r.n * p.rec);
  s0.ids = s0.pos + (size_t)(p.cap + 16) * r.n;
  s0.start = reinterpret_cast<unsigned *>(lists + (size_t)r.n * (p.rec + p.pos));
  s0.keys = reinterpret_cast<unsigned long long *>(lists + (size_t)r.n * (p.rec + p.pos + p.start));
  if (nl > 1) {
    int st = profile_lanes_init(ctx, lanes);
    if (st) return st;
    // the lists do not depend on the data: beside the splines
    if (e == cudaSuccess) e = cudaEventRecord(lanes->fork, stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(lanes->stream[0], lanes->fork, 0);
  }
  if (e == cudaSuccess) {
    const cudaStream_t ls = nl > 1 ? lanes->stream[0] : stream;
    back_sort_kernel<<<r.n, kSortThreads, sm_sort, ls>>>(s0);
    const dim3 grid((p.nbase + 31) / 32, (r.ntheta + 31) / 32, r.ns);
    back_merge_kernel<<<grid, kThreads, 0, stream>>>(r);
    back_solve_kernel<<<(r.ntheta * p.nbase + 63) / 64, 64, 0, stream>>>(r);
    ctx->launches += 3;
    e = cudaGetLastError();
  }
  if (nl > 1) {
    if (e == cudaSuccess) e = cudaEventRecord(lanes->done[0], lanes->stream[0]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, lanes->done[0], 0);
    if (e == cudaSuccess) e = cudaEventRecord(lanes->fork, stream);
    for (int k = 1; k < nl && e == cudaSuccess; ++k)
      e = cudaStreamWaitEvent(lanes->stream[k - 1], lanes->fork, 0);
  }
  const int per_lane = std::max(1, nz / nl);
  // a whole number of rounds over the lanes, evenly filled
  const int rounds = (r.n + per_lane * nl - 1) / (per_lane * nl);
  const int steps = std::min(r.n, rounds * nl);
  for (int k = 0; k < steps && e == cudaSuccess; ++k) {
    const int l = k % nl;
    BackStep s = s0;
    s.z0 = (int)((long long)r.n * k / steps);
    const int cnt = (int)((long long)r.n * (k + 1) / steps) - s.z0;
    s.table = reinterpret_cast<float4 *>(at + (size_t)l * per_lane * p.table);
    s.rec = static_cast<KnotRec *>(s0.rec) + (size_t)s.z0 * p.cap;
    s.pos += (size_t)s.z0 * (p.cap + 16);
    s.ids += (size_t)s.z0 * (p.cap + 16);
    s.start += (size_t)s.z0 * (s.nb + 8);
    const cudaStream_t ls = l ? lanes->stream[l - 1] : stream;
    const int th = 32 * std::min(8, (p.nbase + 31) / 32);
    back_build_kernel<<<cnt << p.nsub_log2, th, sm_build, ls>>>(s);
    back_gather_kernel<<<cnt * s.tiles, kGatherThreads, sm_gather, ls>>>(s);
    ctx->launches += 2;
    e = cudaGetLastError();
  }
  for (int k = 1; k < nl && e == cudaSuccess; ++k) {
    e = cudaEventRecord(lanes->done[k - 1], lanes->stream[k - 1]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, lanes->done[k - 1], 0);
  }
  if (e == cudaSuccess) {
    back_lost_kernel<<<ctx->sm_count * 2, kThreads, 0, stream>>>(r);
    ctx->launches++;
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? WRT_OK : failed(e);
}

}  // namespace wrt
