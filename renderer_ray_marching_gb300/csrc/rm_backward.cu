// rm_backward.cu -- gradient of an image loss through each pixel's first hit.
//
// The reference has no gradient path.  The differentiable model fixed here:
//   colour(p) = colour[hit(p)]                          (float32 RGB)
//   depth(p)  = entry distance of ray p into the sphere (c_hit, r_hit)
// with hit(p) the index stored by the forward pass, held constant.  The
// marcher's own depth stops within MIN_DIST (1e-3) of the union of the
// nearest spheres, so it differs from this analytic surrogate by less than
// MIN_DIST plus one step; the surrogate is what is differentiated.
//
// Per pixel the kernel recomputes the ray exactly as the forward did and
// evaluates the gradient of t = (b - sqrt(disc)) / a, with a = |d|^2,
// b = d.(c - o) and disc = a r^2 - |q|^2 for q = d x (c - o) (Lagrange's
// identity for b^2 - a (|c - o|^2 - r^2)):
//   dt/dc = (d - (d x q) / sqrt(disc)) / a,   dt/dr = -r / sqrt(disc).
// It scales by the incoming dL/ddepth and accumulates into float32 per-point
// gradients.  A warp's pixels are neighbours in a row; runs of them that share
// a hit point are summed in registers first, so each run costs one atomic per
// channel.
//
// Arithmetic.  A millimetre-scale discriminant of metre-scale operands needs
// more than float32.  sm_103a has one FP64 unit for 64 FP32 lanes, and in
// FP64 this kernel was bound by it: 1.44 ms for 16 views of 1067x690, now
// 0.27 (issue-bound, 72% of the slots, 650 instructions per 32 pixels).  Here
// every value is an unevaluated sum of two floats (about 48 bits, T. J.
// Dekker's double-length arithmetic with fma products), and the cancellation
// is taken out of the formula instead: q is as small as the ray's distance
// from the centre, so disc = a r^2 - |q|^2 is off by 2^-45 |q| |c - o|, where
// b^2 - a (...) in FP64 is off by 2^-52 b^2.  That is less for spheres
// narrower than 2^-7 of their distance; the silhouettes of wider ones keep
// FP64.  So do coordinates, radii or incoming gradients outside the range
// where floats hold such products (a product of an infinity is one; its low
// part would be NaN).
#include "rm_internal.h"

namespace rm {

struct BackArgs {
  const ViewDev* views;
  const int64_t* pix_base;   // per view, first pixel of the view; [n] = total
  int nviews;
  int64_t total;
  int64_t n;                 // points in the cloud
  const float* dl_drgb;      // 3 floats per pixel
  const float* dl_ddepth;    // 1 float per pixel
  const int32_t* hit;        // cloud index per pixel, -1 = miss
  const float4* pos;         // cloud order
  const float* radius;       // cloud order, clamped
  float* g_rgb;              // 3 floats per point
  float* g_xyz;              // 3 floats per point
  float* g_radius;           // 1 float per point
};

__device__ __forceinline__ int view_of_pixel(const int64_t* base, int n, int64_t p) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= p) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------- two floats
// hi + lo with |lo| <= ulp(hi) / 2 after a sum.
struct Two {
  float hi, lo;
};
__device__ __forceinline__ Two quick_two(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return Two{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ Two two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return Two{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Two two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return Two{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ Two neg(Two a) { return Two{-a.hi, -a.lo}; }
// error 2^-47 (|a| + |b|)
__device__ __forceinline__ Two add(Two a, Two b) {
  const Two s = two_sum(a.hi, b.hi);
  return quick_two(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
// products, not normalised: |lo| <= 2 ulp(hi)
__device__ __forceinline__ Two mul(Two a, float b) {
  const Two p = two_prod(a.hi, b);
  return Two{p.hi, __fmaf_rn(a.lo, b, p.lo)};
}
__device__ __forceinline__ Two mul(Two a, Two b) {
  const Two p = two_prod(a.hi, b.hi);
  return Two{p.hi, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo))};
}
__device__ __forceinline__ float rounded(Two a) { return __fadd_rn(a.hi, a.lo); }
// 1 / sqrt(a) and 1 / a: a float start and one Newton step
__device__ __forceinline__ Two inv_sqrt(Two a) {
  const float y = rsqrtf(a.hi);
  const Two e = add(Two{1.0f, 0.0f}, neg(mul(a, two_prod(y, y))));
  return quick_two(y, __fmul_rn(__fmul_rn(0.5f, y), e.hi));
}
__device__ __forceinline__ Two inv(Two a) {
  const float y = __frcp_rn(a.hi);
  const Two e = add(Two{1.0f, 0.0f}, neg(mul(a, y)));
  return quick_two(y, __fmul_rn(y, e.hi));
}

// Gradient of the entry distance, times `ld`: out[0..2] by the centre, [3] by
// the radius.  oc: from the ray's origin to the centre.
__device__ __forceinline__ void entry_gradient(const Ray& r, const float4& c, float rad, float ld, float* out) {
  const float d[3] = {r.dx, r.dy, r.dz};
  const Two oc[3] = {two_sum(c.x, -r.ox), two_sum(c.y, -r.oy), two_sum(c.z, -r.oz)};
  const float far = fmaxf(fmaxf(fabsf(oc[0].hi), fabsf(oc[1].hi)), fabsf(oc[2].hi));
  const float up = fabsf(ld);
  Two aa = two_prod(d[0], d[0]);
  aa = add(aa, two_prod(d[1], d[1]));
  aa = add(aa, two_prod(d[2], d[2]));
  // (a ray of a matrix with a fourth row can be far from unit length; NaN and
  // infinities fail these tests)
  if (far < 1048576.0f && rad < 1048576.0f && (rad >= 1e-9f || rad == 0.0f) && up < 1e25f &&
      (up > 1e-25f || up == 0.0f) && aa.hi > 0.25f) {
    Two q[3], n[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int j = (i + 1) % 3, k = (i + 2) % 3;
      q[i] = add(mul(oc[k], d[j]), neg(mul(oc[j], d[k])));
    }
    Two disc = mul(aa, two_prod(rad, rad));
#pragma unroll
    for (int i = 0; i < 3; ++i) disc = add(disc, neg(mul(q[i], q[i])));
    // For a wide sphere near its silhouette FP64's disc is the better one (see
    // above), and the root lets the error through; two floats are kept where
    // it stays below 2^-24 of the result all the same.
    const float across = fmaxf(fmaxf(fabsf(q[0].hi), fabsf(q[1].hi)), fabsf(q[2].hi));
    if (across <= 0x1p-7f * far || fabsf(disc.hi) >= 0x1p-20f * across * far) {
      const Two ia = mul(inv(aa), ld);
      if (disc.hi > 0.0f) {
        const Two is = inv_sqrt(disc);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int j = (i + 1) % 3, k = (i + 2) % 3;
          n[i] = add(mul(q[k], d[j]), neg(mul(q[j], d[k])));
          out[i] = rounded(mul(add(Two{d[i], 0.0f}, neg(mul(n[i], is))), ia));
        }
        out[3] = -rounded(mul(is, two_prod(rad, ld)));
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) out[i] = rounded(mul(ia, d[i]));
        out[3] = 0.0f;
      }
      return;
    }
  }
  const double d0 = r.dx, d1 = r.dy, d2 = r.dz, rr = rad;
  const double oc0 = (double)c.x - (double)r.ox, oc1 = (double)c.y - (double)r.oy, oc2 = (double)c.z - (double)r.oz;
  const double a2 = d0 * d0 + d1 * d1 + d2 * d2, b = d0 * oc0 + d1 * oc1 + d2 * oc2;
  const double disc = b * b - a2 * (oc0 * oc0 + oc1 * oc1 + oc2 * oc2 - rr * rr);
  const double ia = 1.0 / a2, is = disc > 0.0 ? 1.0 / sqrt(disc) : 0.0;
  const bool in = disc > 0.0;
  out[0] = (float)((double)ld * ((in ? d0 - (b * d0 - a2 * oc0) * is : d0) * ia));
  out[1] = (float)((double)ld * ((in ? d1 - (b * d1 - a2 * oc1) * is : d1) * ia));
  out[2] = (float)((double)ld * ((in ? d2 - (b * d2 - a2 * oc2) * is : d2) * ia));
  out[3] = (float)((double)ld * (in ? -rr * is : 0.0));
}

__global__ void __launch_bounds__(256) k_backward(BackArgs a) {
  const unsigned FULL = 0xffffffffu;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  // uniform trip count across the warp so every lane reaches the shuffles
  int64_t warp_first = first - (threadIdx.x & 31);
  for (int64_t wbase = warp_first; wbase < a.total; wbase += stride) {
    int64_t p = wbase + (threadIdx.x & 31);
    int32_t h = -1;
    const int v0 = view_of_pixel(a.pix_base, a.nviews, wbase);  // the warp's first pixel's, same for all lanes
    float g[7] = {0, 0, 0, 0, 0, 0, 0};
    if (p < a.total) {
      h = __ldg(a.hit + p);
      if (h >= a.n) h = -1;  // caller-supplied index outside the cloud: ignored
      if (h >= 0) {
        int v = v0;
        while (p >= a.pix_base[v + 1]) ++v;
        const ViewDev& V = a.views[v];
        const int local = (int)(p - a.pix_base[v]);  // a view has fewer than 2^31 pixels
        const Ray r = make_ray(V.m, V.width, V.height, V.pane, local % V.width, local / V.width);
        entry_gradient(r, __ldg(a.pos + h), __ldg(a.radius + h), __ldg(a.dl_ddepth + p), g + 3);
        g[0] = __ldg(a.dl_drgb + 3 * p + 0);
        g[1] = __ldg(a.dl_drgb + 3 * p + 1);
        g[2] = __ldg(a.dl_drgb + 3 * p + 2);
      }
    }
    // sums over runs of equal hits, in the run's first lane
    const int lane = threadIdx.x & 31;
    const int32_t before = __shfl_up_sync(FULL, h, 1);
    const unsigned heads = __ballot_sync(FULL, lane == 0 || h != before);
    const unsigned above = heads >> lane >> 1;
    const int last = above ? lane + __ffs(above) - 1 : 31;  // of the lane's run
    const int longest = __reduce_max_sync(FULL, last - lane);
    for (int off = 1; off <= longest; off *= 2) {
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        const float o = __shfl_down_sync(FULL, g[k], off);
        if (lane + off <= last) g[k] += o;
      }
    }
    bool write = h >= 0 && ((heads >> lane) & 1u);
    // Interleaved runs of few points (two points pixel by pixel: 13.3 ms for 8
    // views of 1067x690, bound by atomics on two places, now 0.88; ten points
    // at random 5.3, now 1.4): where a point has two runs or more on average,
    // its runs are summed as well.  Looked for in warps of 16 runs or more,
    // and in those of 8 or more where a run in four repeats the one before the
    // last: two thirds of an image's warps have 8 (16 views of 1M points took
    // 4% longer with all of them looked at, and no longer like this).
    bool mixed = __popc(heads) >= 16;
    if (!mixed && __popc(heads) >= 8) {
      // the hit before the previous run: handed on from run to run
      const unsigned below = heads & ((1u << lane) - 1u);
      const int32_t h2 = __shfl_sync(FULL, before, below ? 31 - __clz(below) : 0);
      mixed = 4 * __popc(__ballot_sync(FULL, write && below && h == h2)) >= __popc(heads);
    }
    if (mixed) {
      const unsigned runs = __ballot_sync(FULL, write);
      const unsigned same = __match_any_sync(FULL, write ? h : -2 - lane);
      unsigned first = __ballot_sync(FULL, write && lane == __ffs(same) - 1);
      if (2 * __popc(first) <= __popc(runs)) {
        write = write && ((first >> lane) & 1u);
        for (; first; first &= first - 1u) {
          const int src = __ffs(first) - 1;
          const bool in = (__shfl_sync(FULL, same, src) >> lane) & 1u;
#pragma unroll
          for (int k = 0; k < 7; ++k) {
            float t = in ? g[k] : 0.0f;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(FULL, t, off);
            if (lane == src) g[k] = t;
          }
        }
      }
    }
    if (write) {
      atomicAdd(a.g_rgb + 3 * (int64_t)h + 0, g[0]);
      atomicAdd(a.g_rgb + 3 * (int64_t)h + 1, g[1]);
      atomicAdd(a.g_rgb + 3 * (int64_t)h + 2, g[2]);
      atomicAdd(a.g_xyz + 3 * (int64_t)h + 0, g[3]);
      atomicAdd(a.g_xyz + 3 * (int64_t)h + 1, g[4]);
      atomicAdd(a.g_xyz + 3 * (int64_t)h + 2, g[5]);
      atomicAdd(a.g_radius + h, g[6]);
    }
  }
}

void launch_backward(Ctx& c, const ViewDev* views_dev, int n, int64_t total_pixels,
                     const int64_t* pix_base, const float* dl_drgb, const float* dl_ddepth,
                     const int32_t* hit, float* g_rgb, float* g_xyz, float* g_radius) {
  BackArgs a;
  a.views = views_dev;
  a.pix_base = pix_base;
  a.nviews = n;
  a.total = total_pixels;
  a.n = c.n;
  a.dl_drgb = dl_drgb;
  a.dl_ddepth = dl_ddepth;
  a.hit = hit;
  a.pos = c.pos.ptr<float4>();
  a.radius = c.radii_clamped.ptr<float>();
  a.g_rgb = g_rgb;
  a.g_xyz = g_xyz;
  a.g_radius = g_radius;
  int64_t blocks = (total_pixels + 255) / 256;
  int64_t cap = (int64_t)c.sm_count * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  k_backward<<<(unsigned)blocks, 256, 0, c.stream>>>(a);
}

}  // namespace rm
