// k_ray.cu -- layer-by-layer ray integrals (ray_grid/src/integral.c:11-50).
//
// Two kernels.  In a rotated layer frame one lane per ray (ray_dev.cuh).  On the
// reference's z-slices all slices of one (shift, phi) run through the same (x, y)
// points, and the sampler is linear in z between node layers, so the slices
// kernel sums
//   G_k = sum_j f_k(x_j, y_j)
// over the node layers k and interpolates G once per slice: a warp takes one
// (shift, phi), works out 32 sample points at a time (one per lane, FP64, the
// reference's own cell and fraction where a coordinate is within 1e-9 cells of a
// cell boundary), and then every lane adds the four weighted columns of a point
// for its own four layers -- one 16-byte load per column and lane where the
// volume's rows allow it (n a multiple of 4), no cell arithmetic per sample.
#include "ray_dev.cuh"

namespace {

// A warp takes a tile of kShiftLanes consecutive shifts x 32 / kShiftLanes
// consecutive angles of one layer.  The rays of one shift at neighbouring angles
// have the same chord through the crop ball.  Measured at 128^3 (128 layers x 128
// shifts x 128 angles): 0.60 ms with 2 x 16 (0.82 with 32 x 1, 0.63 with 4 x 8).
// Each ray is the same computation whichever lane takes it.
constexpr int kShiftLanes = 2;

__global__ void __launch_bounds__(256) ray_kernel(wrt::RayJob job, float guard) {
  constexpr int kS = kShiftLanes, kA = 32 / kS;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = (int)(t & 31);
  const long long tile = t >> 5;
  const long long ts_n = (job.nshift + kS - 1) / kS, tp_n = (job.nphi + kA - 1) / kA;
  const long long iz = tile / (ts_n * tp_n), rem = tile % (ts_n * tp_n);
  const long long is = (rem % ts_n) * kS + lane % kS, ip = (rem / ts_n) * kA + lane / kS;
  if (iz >= job.nslices || is >= job.nshift || ip >= job.nphi) return;
  wrtd::ray_one(job, (iz * job.nphi + ip) * job.nshift + is, guard);
}

constexpr int kWarps = 8;    // consecutive shifts of one angle: neighbouring lines share columns
constexpr int kSlots = 128;  // layers per warp, four per lane

// Cell and fraction of one coordinate, cube_trilinear_interp's
// (radon_grid/src/interp.c:32-53): its own arithmetic next to a cell boundary,
// where rounding decides them, else the reciprocal's (equal to rounding).
__device__ __forceinline__ void cell_of(double x, int n, int *i, double *c) {
  const double x1 = __dadd_rn(x, 1.0), q = x1 * (0.5 * (n - 1)), fl = floor(q);
  *i = (int)fl;
  *c = q - fl;
  if (*c < 1e-9 || *c > 1.0 - 1e-9) {
    const double delta = __ddiv_rn(2.0, (double)(n - 1));
    *i = (int)__ddiv_rn(x1, delta);
    *c = __ddiv_rn(wrtd::exact_rem(x1, delta), delta);
    if (*i == n - 1) {
      *i -= 1;
      *c = 1.0;
    }
  }
}

// The layers the slots of a warp stand for: all node layers, kSlots at a time
// from `base` (slices: those whose cell lies in [base, base + step)), or, when
// there are few slices, the two layers of each slice (pairs).
template <bool VEC>
__global__ void __launch_bounds__(32 * kWarps)
    ray_slices_kernel(wrt::RayJob job, int groups, int step, int pairs) {
  __shared__ float4 s_w[kWarps][32];
  // columns, as a volume may have more than 2^31 nodes (their 64-bit offsets here: 228
  // us at 128^3 instead of 223)
  __shared__ int s_col[kWarps][32];
  __shared__ double s_g[kWarps][kSlots];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = job.n;
  const int ts = (job.nshift + kWarps - 1) / kWarps;
  const int ip = (int)(blockIdx.x / (ts * groups)), rest = (int)(blockIdx.x % (ts * groups));
  const int is0 = rest / groups * kWarps, base = rest % groups * step;
  const int is = is0 + warp;
  const double delta = (2.0 / (n - 1)) / (2.0);                       // integral.c:32
  const double dz = 2.0 / (job.nslices - 1);                          // ray_grid.c:244
  auto slice_cell = [&](int iz, int *zc, double *cz) {
    const double z = __dadd_rn(-1.0, __dmul_rn((double)iz, dz));      // ray_grid.c:247
    if (!(fabs(z) <= 1.0)) {
      *zc = -1;
      return;
    }
    cell_of(z, n, zc, cz);
  };
  // this lane's layers
  int layer[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int slot = VEC ? 4 * lane + r : lane + 32 * r;
    if (pairs) {
      const int iz = (base + slot) >> 1;
      int zc = 0;
      double cz;
      if (iz < job.nslices) slice_cell(iz, &zc, &cz);
      layer[r] = max(zc, 0) + (slot & 1);
    } else {
      // past the last layer: any other (its sums are not used); vector loads
      // keep their four layers together, inside the row and aligned
      layer[r] = VEC ? min(base + 4 * lane, n - 4) + r : min(base + slot, n - 1);
    }
  }
  double g[4] = {0.0, 0.0, 0.0, 0.0};
  if (is < job.nshift) {
    const double *T = job.trig + 4 * ip;
    const double s = job.shift[is];
    const double p0x = __dmul_rn(s, T[0]), p0y = __dmul_rn(s, T[1]);
    const double ax = __dmul_rn(delta, T[2]), ay = __dmul_rn(delta, T[3]);
    double crop_r2 = 3.0 + 1e-9;
    if (job.r2bits) {
      const double r = sqrt((double)__uint_as_float(__ldg(job.r2bits))) + job.margin;
      crop_r2 = fmin(r * r, crop_r2);
    }
    const double rem = crop_r2 - s * s;
    int klo = 1, khi = 0;
    if (rem >= 0.0) {
      const int km = (int)floor(sqrt(rem) / delta) + 1;
      klo = max(-2 * n, -km);
      khi = min(2 * n, km);
      if (!(wrtd::clip_axis(p0x, ax, klo, khi) && wrtd::clip_axis(p0y, ay, klo, khi))) khi = klo - 1;
    }
    // exactly the samples inside: their coordinates are monotone in k
    auto inside = [&](int k) {
      return fabs(__dadd_rn(p0x, __dmul_rn(ax, (double)k))) <= 1.0 &&
             fabs(__dadd_rn(p0y, __dmul_rn(ay, (double)k))) <= 1.0;
    };
    while (klo <= khi && !inside(klo)) ++klo;
    while (klo <= khi && !inside(khi)) --khi;
    int taken = 0;
    for (int k0 = klo; k0 <= khi; k0 += 32) {
      const int k = k0 + lane;
      const double x = __dadd_rn(p0x, __dmul_rn(ax, (double)k));
      const double y = __dadd_rn(p0y, __dmul_rn(ay, (double)k));
      float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
      int col = 0;
      if (k <= khi) {
        int ix, iy;
        double cx, cy;
        cell_of(x, n, &ix, &cx);
        cell_of(y, n, &iy, &cy);
        w = make_float4((float)((1.0 - cx) * (1.0 - cy)), (float)((1.0 - cx) * cy),
                        (float)(cx * (1.0 - cy)), (float)(cx * cy));
        col = ix * n + iy;
        ++taken;
      }
      __syncwarp();
      s_w[warp][lane] = w;
      s_col[warp][lane] = col;
      __syncwarp();
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      const int m = min(32, khi - k0 + 1);
#pragma unroll 4
      for (int j = 0; j < m; ++j) {
        const float4 c = s_w[warp][j];
        const float *v = job.vol + (size_t)s_col[warp][j] * n;
        if (VEC) {
          const float *q = v + layer[0];
          const float4 f0 = __ldg(reinterpret_cast<const float4 *>(q));
          const float4 f1 = __ldg(reinterpret_cast<const float4 *>(q + n));
          const float4 f2 = __ldg(reinterpret_cast<const float4 *>(q + (size_t)n * n));
          const float4 f3 = __ldg(reinterpret_cast<const float4 *>(q + (size_t)n * n + n));
          a[0] = fmaf(c.w, f3.x, fmaf(c.z, f2.x, fmaf(c.y, f1.x, fmaf(c.x, f0.x, a[0]))));
          a[1] = fmaf(c.w, f3.y, fmaf(c.z, f2.y, fmaf(c.y, f1.y, fmaf(c.x, f0.y, a[1]))));
          a[2] = fmaf(c.w, f3.z, fmaf(c.z, f2.z, fmaf(c.y, f1.z, fmaf(c.x, f0.z, a[2]))));
          a[3] = fmaf(c.w, f3.w, fmaf(c.z, f2.w, fmaf(c.y, f1.w, fmaf(c.x, f0.w, a[3]))));
        } else {
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float *q = v + layer[r];
            a[r] = fmaf(c.x, __ldg(q), a[r]);
            a[r] = fmaf(c.y, __ldg(q + n), a[r]);
            a[r] = fmaf(c.z, __ldg(q + (size_t)n * n), a[r]);
            a[r] = fmaf(c.w, __ldg(q + (size_t)n * n + n), a[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) g[r] += (double)a[r];
    }
    if (job.counter && base == 0) {
      for (int o = 16; o > 0; o >>= 1) taken += __shfl_xor_sync(0xffffffffu, taken, o);
      if (lane == 0 && taken)
        atomicAdd(job.counter, (unsigned long long)taken * (unsigned long long)job.nslices);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) s_g[warp][VEC ? 4 * lane + r : lane + 32 * r] = g[r];
  __syncthreads();
  // ---- slices: kWarps consecutive shifts each
  const int iz0 = pairs ? base >> 1 : 0, iz1 = pairs ? min(job.nslices, iz0 + kSlots / 2) : job.nslices;
  for (int t = tid; t < (iz1 - iz0) * kWarps; t += 32 * kWarps) {
    const int iz = iz0 + t / kWarps, w = t % kWarps;
    int zc = 0;
    double cz = 0.0;
    slice_cell(iz, &zc, &cz);
    double v = 0.0;
    if (zc >= 0) {
      const int slot = pairs ? 2 * (iz - iz0) : zc - base;
      if (!pairs && (slot < 0 || slot >= step)) continue;  // another group's
      v = fma(cz, s_g[w][slot + 1] - s_g[w][slot], s_g[w][slot]);
    } else if (base) {
      continue;
    }
    if (is0 + w < job.nshift)
      job.out[((long long)iz * job.nshift + is0 + w) * job.nphi + ip] = v * delta;
  }
}

}  // namespace

namespace wrt {

int ray_forward(wrt_ctx *ctx, cudaStream_t stream, const RayJob &job) {
  const long long nrays = (long long)job.nslices * job.nshift * job.nphi;
  if (nrays == 0) return WRT_OK;
  ctx->launches++;
  if (!job.has_frame) {
    const int n = job.n;
    // few slices: their own layers two by two; else all of them, in groups that
    // overlap by a layer (by four where rows are read 16 bytes at a time)
    const int pairs = 2 * job.nslices < n ? 1 : 0;
    const bool vec = !pairs && n % 4 == 0;
    const int step = pairs ? kSlots : vec ? kSlots - 4 : kSlots - 1;
    const int groups = pairs ? (2 * job.nslices + kSlots - 1) / kSlots
                             : n <= kSlots ? 1 : (n - 1 + step - 1) / step;
    const long long blocks = (long long)job.nphi * ((job.nshift + kWarps - 1) / kWarps) * groups;
    if (blocks > 0x7fffffffLL) return fail(ctx, WRT_ERR_INVALID_ARGUMENT, "too many rays");
    const int cells = groups == 1 && !pairs ? kSlots - 1 : step;
    if (vec)
      ray_slices_kernel<true><<<(unsigned)blocks, 32 * kWarps, 0, stream>>>(job, groups, cells, pairs);
    else
      ray_slices_kernel<false><<<(unsigned)blocks, 32 * kWarps, 0, stream>>>(job, groups, cells, pairs);
    return check_launch(ctx, "ray_slices_kernel");
  }
  // one warp per tile
  const int kS = kShiftLanes, kA = 32 / kS;
  const long long tiles =
      (long long)job.nslices * ((job.nshift + kS - 1) / kS) * ((job.nphi + kA - 1) / kA);
  const long long blocks = (tiles + 7) / 8;
  if (blocks > 0x7fffffffLL) return fail(ctx, WRT_ERR_INVALID_ARGUMENT, "too many rays");
  ray_kernel<<<(unsigned)blocks, 256, 0, stream>>>(job, wrtd::ray_guard(job.n));
  return check_launch(ctx, "ray_kernel");
}

}  // namespace wrt
