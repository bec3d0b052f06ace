// k_reduction.cu -- ray data to Radon data (radon_reduction/slicing.c:5-119), one
// longitude's splines in shared memory.
//
// For one phi a Radon sample is a sum over a line of the (s, z) plane, and all
// its (theta, shift) lines read the same ngrid x nshift_ray spline values and
// curvatures.  A CTA stages those of one phi as (y, m) pairs, m = h^2/6 times the
// natural spline's second derivative (ngrid x ns x 8 bytes: 131 KB at 128 x 128),
// and works through the phi's lines, one thread per line, lanes on consecutive
// shifts.  A sample is then six 8-byte shared loads -- two knots of three layers
// -- and packed FP32 pairs: the quadratic in z combines the layers first (the
// spline is linear in its data), then (a, -ab(1+a)) and (b, -ab(1+b)) weigh the
// (y, m) pairs of the two knots.
//
// Positions along a line advance in 16.48 fixed point (layers, knots): integer
// part = layer or knot, fraction = 23 bits by a mantissa insert; no conversions
// and no FP64 in the loop.  The error is below (2 ngrid + 1) x 2^-49 + 2^-24
// (reduction_dev.cuh; with 32.32 positions the steps' rounding passed 2^-24 from 256
// layers up).  The reference's layer index and knot interval are not reproduced at a layer or
// knot: the interpolant is continuous there (two zero layers and a zero knot
// beyond the ends stand for slicing.c:62-74's zero third value).  Which samples
// belong to a line (tau^2 + p^2 <= 1, slicing.c:110, |z|, |s| <= 1) is decided in
// FP64 with the reference's expressions at the line's ends, the only places where
// they can fail.  Sums: FP32 over two samples, FP64 beyond.
//
// 128 layers x 128 offsets, 64 x 128 directions x 256 shifts: 2.37 ms with three
// 16-byte records per sample gathered through L1 (one request of up to 32 lines
// each), 1.12 ms here (1.04 of it this kernel, at 90 % of the shared-memory
// wavefronts; 1.45 with an odd pitch; every lane at its own line's start: no faster).
// Error against FP64 (doubles, 64 layers x 40 offsets) 7.5e-9, by records 1.2e-8.
#include <algorithm>
#include <vector>

#include "reduction_dev.cuh"
#include "wrt_internal.cuh"

namespace {

using namespace wrtr;

typedef unsigned long long u64;
__device__ __forceinline__ u64 pk(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 lds64(unsigned a) {
  u64 v;
  asm("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}
// m_{i-1} + 4 m_i + m_{i+1} = y_{i+1} - 2 y_i + y_{i-1}, m_0 = m_{ns-1} = 0, one
// thread per line (iz, iphi), element i at [(iz*ns + i)*nphi + iphi]: every access
// of a warp is one row of consecutive phis.  d: forward pass, m: result.
__global__ void __launch_bounds__(128)
    curvature_kernel(const double *__restrict__ rays, int nlines, int nphi, int ns,
                     const double *__restrict__ cp, double *__restrict__ d,
                     float *__restrict__ m) {
  const int L = blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= nlines) return;
  const size_t o = (size_t)(L / nphi) * ns * nphi + L % nphi, st = nphi;
  const double *y = rays + o;
  double prev = 0.0, ya = y[0], yb = y[st];
#pragma unroll 8
  for (int i = 1; i + 1 < ns; ++i) {
    const double yc = y[(i + 1) * st];
    prev = ((yc - 2.0 * yb + ya) - prev) * cp[i];
    d[o + i * st] = prev;
    ya = yb;
    yb = yc;
  }
  m[o] = 0.0f;
  m[o + (ns - 1) * st] = 0.0f;
  prev = 0.0;
#pragma unroll 8
  for (int i = ns - 2; i >= 1; --i) {
    prev = d[o + i * st] - cp[i] * prev;
    m[o + i * st] = (float)prev;
  }
}

struct RedJob {
  const double *rays;   // [iz][is][iphi]
  const float *m;       // the same order
  const double *shift;  // [nshift]
  const double *cs;     // [ntheta][2] cos, sin theta
  double *out;          // [is][iphi][itheta]
  unsigned long long *counter;
  int ngrid, ns, nphi, nshift, ntheta, pitch;
};

template <int T>
__global__ void __launch_bounds__(T, 1) reduction_staged_kernel(const RedJob job) {
  extern __shared__ __align__(16) float2 ym[];  // [ngrid + 2][pitch]
  const int tid = threadIdx.x;
  const int ngrid = job.ngrid, ns = job.ns, pitch = job.pitch;
  const int lines = job.nshift * job.ntheta;
  const int per = (lines + T - 1) / T;  // items per phi
  const long long items = (long long)per * job.nphi;
  // consecutive items per CTA: few changes of phi
  const long long i0 = items * blockIdx.x / gridDim.x, i1 = items * (blockIdx.x + 1) / gridDim.x;
  const unsigned base = (unsigned)__cvta_generic_to_shared(ym);
  const unsigned row = (unsigned)pitch * 8u;
  const double dtau = (2.0 / (ngrid - 1)) / (2.0);  // slicing.c:88
  unsigned long long counted = 0;
  int staged = -1;
  for (long long item = i0; item < i1; ++item) {
    const int ip = (int)(item / per);
    if (ip != staged) {
      __syncthreads();
      for (int k = tid; k < (ngrid + 2) * pitch; k += T) {
        const int iz = k / pitch, i = k - iz * pitch;
        float2 v = make_float2(0.0f, 0.0f);
        if (iz < ngrid && i < ns) {
          const size_t o = ((size_t)iz * ns + i) * job.nphi + ip;
          v = make_float2((float)__ldg(job.rays + o), __ldg(job.m + o));
        }
        ym[k] = v;
      }
      __syncthreads();
      staged = ip;
    }
    const int line0 = (int)(item % per) * T + tid, line = min(line0, lines - 1);
    const int it = line / job.nshift, is = line - it * job.nshift;
    const double p = job.shift[is], ct = job.cs[2 * it], st = job.cs[2 * it + 1];
    int klo, khi;
    line_range(ngrid, dtau, p, ct, st, &klo, &khi);
    // the warp's lanes keep the same tau: their cells then lie half a cell apart
    // along one short line, and neighbours share them
    const int k0 = __reduce_min_sync(0xffffffffu, klo), k1 = __reduce_max_sync(0xffffffffu, khi);
    LinePos at = line_pos(ngrid, ns, dtau, p, ct, st, k0);
    double acc = 0.0;
    // FP64 beyond two samples: beyond eight the error against FP64 was twice as large (64
    // layers x 40 offsets: 1.45e-8 and 7.5e-9; by records and FP64 for every sample 1.2e-8)
    for (int k = k0; k <= k1; k += 2) {
      float part = 0.0f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bool on = k + j >= klo && k + j <= khi;
        const int iz = on ? cell_of(at.z) : 0, i = on ? cell_of(at.s) : 0;
        const float f = __uint_as_float(one_plus_fraction(at.z)) - 1.0f,
                    b = __uint_as_float(one_plus_fraction(at.s)) - 1.0f;
        at.z += at.dz;
        at.s += at.ds;
        const unsigned a0 = base + (unsigned)iz * row + (unsigned)i * 8u;
        const unsigned a1 = a0 + row, a2 = a1 + row;
        const u64 l00 = lds64(a0), l01 = lds64(a0 + 8), l10 = lds64(a1), l11 = lds64(a1 + 8),
                  l20 = lds64(a2), l21 = lds64(a2 + 8);
        // quadratic through the three layers (slicing.c:62-74)
        const float g = 2.0f - f, e = f - 1.0f;
        const float w1 = f * g, w0 = -0.5f * e * g, w2 = 0.5f * f * e;
        const u64 W0 = pk(w0, w0), W1 = pk(w1, w1), W2 = pk(w2, w2);
        const u64 A = fma2(W2, l20, fma2(W1, l10, mul2(W0, l00)));
        const u64 B = fma2(W2, l21, fma2(W1, l11, mul2(W0, l01)));
        const float a = 1.0f - b, t = -a * b;
        const u64 v = fma2(pk(b, fmaf(t, b, t)), B, mul2(pk(a, fmaf(t, a, t)), A));
        float x, y;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
        part += on ? x + y : 0.0f;
      }
      acc += (double)part;
    }
    if (line0 >= lines) continue;
    if (khi >= klo) counted += khi - klo + 1;
    job.out[((size_t)is * job.nphi + ip) * job.ntheta + it] = acc * dtau;
  }
  if (job.counter && counted) atomicAdd(job.counter, counted);
}

// Row pitch in pairs: a zero knot after the last, and 4 mod 16.  Sixteen lanes read
// cells along a short line of the (z, s) grid in any direction; with 16 bank
// pairs two cells (dz, ds) apart collide when pitch dz + ds = 0 mod 16, and pitch
// 4 keeps colliding cells at least 4 apart whatever the direction (an odd pitch of
// 129 = 1 mod 16 collides along ds = -dz: 4.2 wavefronts per load, 1.45 ms).
// Where that does not fit, any odd one.
constexpr size_t kMostSmem = 225 * 1024;
size_t bytes_of(int ngrid, int pitch) { return sizeof(float2) * (size_t)(ngrid + 2) * pitch; }
int pitch_of(int ngrid, int ns) {
  int p = ns + 1;
  while (p % 16 != 4) ++p;
  return bytes_of(ngrid, p) <= kMostSmem ? p : (ns + 1) | 1;
}
size_t smem_of(int ngrid, int ns) { return bytes_of(ngrid, pitch_of(ngrid, ns)); }

}  // namespace

namespace wrt {

// One phi's splines fit a CTA's shared memory (sizes alone decide).
bool reduction_covers(int ngrid, int ns_ray) { return smem_of(ngrid, ns_ray) <= kMostSmem; }

int reduction_staged(wrt_ctx *ctx, cudaStream_t stream, const double *rays, int ngrid, int ns_ray,
                     int nphi, const double *shift, int nshift, const double *cs, int ntheta,
                     const double *cp, double *scratch, float *m, unsigned long long *counter,
                     double *out) {
  const int nlines = ngrid * nphi;
  curvature_kernel<<<(nlines + 127) / 128, 128, 0, stream>>>(rays, nlines, nphi, ns_ray, cp,
                                                             scratch, m);
  RedJob j = {rays, m, shift, cs, out, counter, ngrid, ns_ray, nphi, nshift, ntheta,
              pitch_of(ngrid, ns_ray)};
  const size_t smem = smem_of(ngrid, ns_ray);
  // one CTA of 1024 threads per SM, or several of 512 where their tiles fit
  const bool big = smem > 110 * 1024;
  const int threads = big ? 1024 : 512;
  const int per_sm = big ? 1 : std::min(4, (int)(224 * 1024 / (smem + 1024)));
  const long long lines = (long long)nshift * ntheta;
  const long long items = (lines + threads - 1) / threads * nphi;
  const unsigned grid = (unsigned)std::min<long long>(items, (long long)ctx->sm_count * per_sm);
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024)
    e = big ? allow_smem(reduction_staged_kernel<1024>, kMostSmem)
            : allow_smem(reduction_staged_kernel<512>, kMostSmem);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "reduction kernel attribute");
  if (big)
    reduction_staged_kernel<1024><<<grid, 1024, smem, stream>>>(j);
  else
    reduction_staged_kernel<512><<<grid, 512, smem, stream>>>(j);
  ctx->launches += 2;
  return check_launch(ctx, "reduction_staged_kernel");
}

}  // namespace wrt
