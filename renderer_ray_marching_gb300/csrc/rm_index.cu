// rm_index.cu -- device-built spatial index replacing the FLANN CUDA kd-tree
// (third_party/flann/algorithms/kdtree_cuda_builder.h:483-599, which sorts
// x, y and z separately and syncs with the host once per tree level).
//
// Build, all on the device with no host round trip between passes:
//   1. bounds:   of the cloud, kept when it was packed (+ a non-finite flag);
//   2. keys:     32-bit Hilbert-curve key of each point's cubic cell;
//   3. sort:     LSD radix sort of (key, cloud index), 4 passes of 8 bits,
//                stable warp-level ranking by digit votes;
//   4. blocks:   1024 consecutive points per CTA, split by medians down to
//                leaves of `leaf` points; packed float4 records (x, y, z,
//                radius), colours and cloud indices in that order, and the
//                boxes of the leaves and of the nodes inside the block;
//   5. tree:     an implicit 4-ary tree over the leaves whose nodes store
//                their four children's boxes as one 128-byte group (min
//                x/y/z, max x/y/z as float4 lanes); the levels above the
//                blocks are built bottom-up, five per launch.  Groups two
//                and more levels below an empty node are never read, and
//                not written.
// The kNN answers do not depend on the build order: searches are exact with
// (d2, cloud index) ordering, so only speed depends on the layout.
#include "rm_internal.h"

#include <algorithm>
#include <cstring>

namespace rm {

// ---------------------------------------------------------------- points
// Points as float4: x, y, z and the packed colour in .w; and the cloud's
// bounds on the way: bounds[0..2] lower (complemented) and [3..5] upper corner
// as ordered_bits, [6] nonzero if a coordinate is not finite; all zero before.
constexpr int PACK_THREADS = 256;
__global__ void __launch_bounds__(PACK_THREADS)
k_pack(const float* __restrict__ xyz, int stride, const uint8_t* __restrict__ rgb, int64_t n,
       float4* __restrict__ pos, uint32_t* __restrict__ bounds) {
  float lo[3] = {INFINITY, INFINITY, INFINITY};
  float hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  bool bad = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float* p = xyz + i * stride;
    const float c[3] = {p[0], p[1], p[2]};
    uint32_t u = 0xffffffu;
    if (rgb) u = (uint32_t)rgb[3 * i] | ((uint32_t)rgb[3 * i + 1] << 8) | ((uint32_t)rgb[3 * i + 2] << 16);
    pos[i] = make_float4(c[0], c[1], c[2], __uint_as_float(u));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      bad |= !isfinite(c[a]);
      lo[a] = fminf(lo[a], c[a]);
      hi[a] = fmaxf(hi[a], c[a]);
    }
  }
  __shared__ uint32_t sh[6][PACK_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint32_t l = __reduce_max_sync(0xffffffffu, ~ordered_bits(lo[a]));
    const uint32_t h = __reduce_max_sync(0xffffffffu, ordered_bits(hi[a]));
    if (lane == 0) {
      sh[a][warp] = l;
      sh[3 + a][warp] = h;
    }
  }
  const int any_bad = __syncthreads_or(bad);
  if (threadIdx.x < 6) {
    uint32_t v = sh[threadIdx.x][0];
    for (int w = 1; w < PACK_THREADS / 32; ++w) v = max(v, sh[threadIdx.x][w]);
    atomicMax(bounds + threadIdx.x, v);
  }
  if (any_bad && threadIdx.x == 0) atomicOr(bounds + 6, 1u);
}

// ---------------------------------------------------------------- curve keys
// Every third bit of a 30-bit word, bit 0 first.
__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// Position of cell (x, y, z), CURVE_BITS bits each, along a Hilbert curve:
// the reflections and rotations are undone from the top bit down, then the
// digits are Gray-coded (J. Skilling, "Programming the Hilbert curve", AIP
// Conf. Proc. 707, 2004).  The curve never jumps, so a run of consecutive
// points is one connected patch, where a Morton run is cut at every
// power-of-two face.  Of the 33 bits of position the lowest is dropped.
constexpr int CURVE_BITS = 11;
__device__ __forceinline__ uint32_t curve_key(uint32_t x, uint32_t y, uint32_t z) {
#pragma unroll
  for (int b = CURVE_BITS - 1; b > 0; --b) {
    const uint32_t low = (1u << b) - 1u;
    if ((x >> b) & 1u) x ^= low;
    const uint32_t ty = (x ^ y) & low;
    const bool ry = (y >> b) & 1u;
    x ^= ry ? low : ty;
    y ^= ry ? 0u : ty;
    const uint32_t tz = (x ^ z) & low;
    const bool rz = (z >> b) & 1u;
    x ^= rz ? low : tz;
    z ^= rz ? 0u : tz;
  }
  y ^= x;
  z ^= y;
  uint32_t f = 0;
#pragma unroll
  for (int b = CURVE_BITS - 1; b > 0; --b)
    if ((z >> b) & 1u) f ^= (1u << b) - 1u;
  x ^= f;
  y ^= f;
  z ^= f;
  const uint32_t top = (spread10(x >> 1) << 2) | (spread10(y >> 1) << 1) | spread10(z >> 1);
  return (top << 2) | ((x & 1u) << 1) | (y & 1u);
}

// Cells of the curve's grid: cubes, 2^CURVE_BITS along the longest side of
// the cloud's body (grid_of); points outside that fall in the cells at its
// border.
struct CurveGrid {
  float lo[3], sc;
  __device__ __forceinline__ void cell(const float4& p, uint32_t (&q)[3]) const {
    const float c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a)
      q[a] = (uint32_t)fminf(fmaxf((c[a] - lo[a]) * sc, 0.0f), (float)((1 << CURVE_BITS) - 1));
  }
};

// The body: the bounds, less what lies BODY spans beyond the middle of 1024
// sampled points.  One point 20 km above a room would make the cells as wide
// as the room, every block a random sample of it, and every search a walk
// through most of the tree (1M points: radii 187 ms and a batch of four
// 640x480 views 1426, against 0.25 and 6.9 ms without the point).  The span
// is the longest side of the box between the medians of 32 group minima and
// maxima, 32 samples each (2% and 98% of the points); at 33 spans the cells
// are still 1/62 of it.  Every CTA computes it, all with the same result: an
// index build takes 0.3 us more at 100k points, 6 at 2M, 12 at 20M, and a
// launch of its own as much.
constexpr int GRID_THREADS = 256;
constexpr float BODY = 16.0f;
__device__ __forceinline__ CurveGrid grid_of(const float4* __restrict__ pos, int64_t n, const uint32_t* __restrict__ bounds) {
  __shared__ uint32_t group[6][32];
  __shared__ float mid[6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < 1024 / GRID_THREADS; ++r) {
    // places spread evenly by the golden ratio, those of a group too
    const uint32_t h = (uint32_t)(r * GRID_THREADS + threadIdx.x) * 2654435769u;
    const float4 p = __ldg(pos + (int64_t)(((uint64_t)h * (uint64_t)n) >> 32));
    const float c[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t lo = __reduce_min_sync(0xffffffffu, ordered_bits(c[a]));
      const uint32_t hi = __reduce_max_sync(0xffffffffu, ordered_bits(c[a]));
      if (lane == 0) {
        group[a][r * (GRID_THREADS / 32) + warp] = lo;
        group[3 + a][r * (GRID_THREADS / 32) + warp] = hi;
      }
    }
  }
  __syncthreads();
  if (warp < 6) {
    const uint32_t v = group[warp][lane];
    int rank = 0;
    for (int j = 0; j < 32; ++j) {
      const uint32_t o = group[warp][j];
      rank += o < v || (o == v && j < lane);
    }
    if (rank == 16) mid[warp] = from_ordered(v);
  }
  __syncthreads();
  const float span = fmaxf(fmaxf(mid[3] - mid[0], mid[4] - mid[1]), mid[5] - mid[2]);
  const float reach = span > 0.0f ? BODY * span : INFINITY;  // nearly all points at one place: the bounds
  CurveGrid g;
  float side = 1e-30f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float lo = from_ordered(~bounds[a]), hi = from_ordered(bounds[3 + a]);
    g.lo[a] = fmaxf(lo, mid[a] - reach);
    side = fmaxf(side, fminf(hi, mid[3 + a] + reach) - g.lo[a]);
  }
  g.sc = (float)((1 << CURVE_BITS) - 1) / side;
  return g;
}

// Points per coarse cell (2^g along a side), for the keys below: of every 256
// points 32 are counted.
__global__ void __launch_bounds__(GRID_THREADS)
k_coarse_count(const float4* __restrict__ pos, int64_t n, const uint32_t* __restrict__ bounds, int g,
               uint32_t* __restrict__ count, CurveGrid* __restrict__ grid_out) {
  const CurveGrid grid = grid_of(pos, n, bounds);
  if (blockIdx.x == 0 && threadIdx.x == 0) *grid_out = grid;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = (t >> 5) * 256 + (t & 31);
    if (i >= n) break;
    uint32_t q[3];
    grid.cell(pos[i], q);
    atomicAdd(count + ((((q[0] >> (CURVE_BITS - g)) << g) + (q[1] >> (CURVE_BITS - g))) << g) + (q[2] >> (CURVE_BITS - g)), 1u);
  }
}

// Curve keys, with the strays of a surface kept at their surface.  Where a
// surface lies along a face of the coarse grid, its outermost points fall in
// cells that hold little else; the curve visits those in another part of the
// cloud, and they make leaves tens of centimetres wide that every search
// nearby has to look into.  A point whose coarse cell holds under an eighth
// of the points of the cell beyond a near face (at most a quarter cell away)
// takes its key from that cell's edge.
__global__ void k_curve_keys(const float4* __restrict__ pos, int64_t n, const CurveGrid* __restrict__ grid_in, int g,
                             const uint32_t* __restrict__ count, uint32_t* __restrict__ keys) {
  const CurveGrid grid = *grid_in;
  const int sh = CURVE_BITS - g;
  const uint32_t quarter = 1u << sh >> 2, in = (1u << sh) - 1u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t q[3];
    grid.cell(pos[i], q);
    const uint32_t own = ((((q[0] >> sh) << g) + (q[1] >> sh)) << g) + (q[2] >> sh);
    uint32_t most = 8u * __ldg(count + own) + 8u, to = 0;
    int axis = -1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t step = a == 0 ? 1u << (2 * g) : a == 1 ? 1u << g : 1u;
      const uint32_t off = q[a] & in, cell = q[a] >> sh;
      const bool down = off < quarter && cell > 0, up = off > in - quarter && cell + 1 < (1u << g);
      if (down || up) {
        const uint32_t c = __ldg(count + (down ? own - step : own + step));
        if (c > most) {
          most = c;
          axis = a;
          to = down ? (cell << sh) - 1u : (cell + 1u) << sh;
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (axis == a) q[a] = to;
    keys[i] = curve_key(q[0], q[1], q[2]);
  }
}

// ---------------------------------------------------------------- radix sort
// Tile = SORT_THREADS threads x SORT_ITEMS keys; warp w owns the contiguous
// run [w*32*SORT_ITEMS, (w+1)*32*SORT_ITEMS) of its tile, processed in
// rounds of 32 consecutive keys, so ranks follow input order (stable).
//
// Bound by HBM: a pass reads and writes 16 bytes per point (and its counts
// read 4).  A tile is put in digit order in shared memory first and goes out
// in runs of one digit, so that stores fill whole sectors; written from
// registers in input order a pass took 0.30 ms at 20M points and 2.3 ms at
// 100M, now 0.11 and 0.49 (3.3 TB/s).  Tiles of 8192 measured 0.52 ms at 100M,
// votes of __match_any_sync instead of one per bit 0.60.  The first pass
// takes each key's index from its position.
constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 16;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int RADIX = 256;
// Up to this many tiles the scatter sums the counts itself: 2 launches a pass
// instead of 5, 66 -> 43 us for the whole sort at 100k points.
constexpr int64_t SORT_OWN_SCAN = 64;

__global__ void __launch_bounds__(SORT_THREADS)
k_sort_hist(const uint32_t* __restrict__ keys, int64_t n, int shift, int64_t ntiles,
            uint32_t* __restrict__ counts) {
  __shared__ uint32_t hist[RADIX];
  for (int d = threadIdx.x; d < RADIX; d += blockDim.x) hist[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * SORT_TILE;
  if (base + SORT_TILE <= n) {
    const uint4* k4 = reinterpret_cast<const uint4*>(keys + base);  // tiles start on 32 KB
    uint4 v[SORT_ITEMS / 4];
#pragma unroll
    for (int r = 0; r < SORT_ITEMS / 4; ++r) v[r] = __ldg(k4 + r * SORT_THREADS + threadIdx.x);
#pragma unroll
    for (int r = 0; r < SORT_ITEMS / 4; ++r) {
      atomicAdd(&hist[(v[r].x >> shift) & (RADIX - 1)], 1u);
      atomicAdd(&hist[(v[r].y >> shift) & (RADIX - 1)], 1u);
      atomicAdd(&hist[(v[r].z >> shift) & (RADIX - 1)], 1u);
      atomicAdd(&hist[(v[r].w >> shift) & (RADIX - 1)], 1u);
    }
  } else {
    for (int64_t i = base + threadIdx.x; i < n; i += SORT_THREADS)
      atomicAdd(&hist[(keys[i] >> shift) & (RADIX - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RADIX; d += blockDim.x)
    counts[(int64_t)d * ntiles + blockIdx.x] = hist[d];
}

// Exclusive scan of `len` uint32 in place, block level: each block scans
// SCAN_TILE elements and writes its total.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s += y;
    }
    warp_sums[lane] = s;
  }
  __syncthreads();
  uint32_t prefix = warp > 0 ? warp_sums[warp - 1] : 0u;
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return prefix + x - v;
}

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_tiles(uint32_t* __restrict__ data, int64_t len, uint32_t* __restrict__ tile_sums) {
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
  uint32_t v[SCAN_ITEMS];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    v[k] = (base + k < len) ? data[base + k] : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(s, &total);
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    if (base + k < len) data[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Single block: exclusive scan of the tile sums (any length).
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_sums(uint32_t* __restrict__ sums, int64_t len) {
  uint32_t carry = 0;
  for (int64_t start = 0; start < len; start += SCAN_THREADS) {
    int64_t i = start + threadIdx.x;
    uint32_t v = i < len ? sums[i] : 0u;
    uint32_t total;
    uint32_t ex = block_exclusive_scan(v, &total);
    if (i < len) sums[i] = carry + ex;
    carry += total;
  }
}

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_add(uint32_t* __restrict__ data, int64_t len, const uint32_t* __restrict__ tile_sums) {
  uint32_t add = tile_sums[blockIdx.x];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_THREADS) {
    int64_t i = base + k;
    if (i < len) data[i] += add;
  }
}

// Exclusive prefix over RADIX digit counts, one per thread.
__device__ __forceinline__ uint32_t digit_prefix(uint32_t v, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += warp_sums[w];
  return before + x - v;
}

struct SortSmem {
  uint32_t cnt[SORT_WARPS][RADIX];  // per warp: keys of each digit, then the warp's first place
  uint32_t base[RADIX];             // global place of the tile's first key of a digit, less its local place
  uint32_t sums[RADIX / 32];
  uint32_t key[SORT_TILE], val[SORT_TILE];
};

// FIRST: the values are the positions.  SCANNED: `offsets` holds the scanned
// counts; else the counts themselves, and every CTA sums what precedes it.
template <bool FIRST, bool SCANNED>
__global__ void __launch_bounds__(SORT_THREADS, 4)
k_sort_scatter(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
               int64_t n, int shift, int64_t ntiles, const uint32_t* __restrict__ offsets,
               uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  SortSmem& sm = *reinterpret_cast<SortSmem*>(sort_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = lane; d < RADIX; d += 32) sm.cnt[warp][d] = 0;
  __syncwarp();
  const uint32_t lt_mask = (1u << lane) - 1u;
  const int64_t tile = (int64_t)blockIdx.x * SORT_TILE;
  const int64_t wbase = tile + (int64_t)warp * 32 * SORT_ITEMS;
  uint32_t key[SORT_ITEMS], rank[SORT_ITEMS / 2];  // ranks in 16 bits
#pragma unroll
  for (int r = 0; r < SORT_ITEMS; ++r) {
    const int64_t i = wbase + r * 32 + lane;
    key[r] = i < n ? __ldcs(keys_in + i) : 0u;
  }
#pragma unroll
  for (int r = 0; r < SORT_ITEMS; ++r) {
    const bool valid = wbase + r * 32 + lane < n;
    const uint32_t dig = (key[r] >> shift) & (RADIX - 1);
    // lanes with the same digit, one vote per bit
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint32_t v = __ballot_sync(0xffffffffu, (dig >> b) & 1u);
      peers &= (dig >> b) & 1u ? v : ~v;
    }
    const uint32_t before = __popc(peers & lt_mask);
    const uint32_t prev = valid ? sm.cnt[warp][dig] : 0u;
    __syncwarp();
    if (valid && before == 0) sm.cnt[warp][dig] = prev + __popc(peers);
    __syncwarp();
    if (r & 1) rank[r / 2] |= (prev + before) << 16;
    else rank[r / 2] = prev + before;
  }
  __syncthreads();
  // places within the tile: digits in order, and within a digit the warps
  static_assert(SORT_THREADS == RADIX, "one digit per thread");
  uint32_t total = 0;
  const int d = threadIdx.x;
#pragma unroll
  for (int w = 0; w < SORT_WARPS; ++w) total += sm.cnt[w][d];
  const uint32_t first = digit_prefix(total, sm.sums);
  uint32_t place = 0;
  if (!SCANNED) {
    uint32_t mine = 0, all = 0;
    for (int64_t t = 0; t < ntiles; ++t) {
      const uint32_t v = __ldg(offsets + (int64_t)d * ntiles + t);
      all += v;
      mine += t < (int64_t)blockIdx.x ? v : 0u;
    }
    __syncthreads();  // sums are read again
    place = digit_prefix(all, sm.sums) + mine;
  } else {
    place = offsets[(int64_t)d * ntiles + blockIdx.x];
  }
  {
    sm.base[d] = place - first;
    uint32_t run = first;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) {
      const uint32_t c = sm.cnt[w][d];
      sm.cnt[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < SORT_ITEMS; ++r) {
    const int64_t i = wbase + r * 32 + lane;
    if (i < n) {
      const uint32_t at = sm.cnt[warp][(key[r] >> shift) & (RADIX - 1)] + (r & 1 ? rank[r / 2] >> 16 : rank[r / 2] & 0xffffu);
      sm.key[at] = key[r];
      sm.val[at] = FIRST ? (uint32_t)i : __ldcs(vals_in + i);
    }
  }
  __syncthreads();
  const int m = (int)min((int64_t)SORT_TILE, n - tile);
  for (int j = threadIdx.x; j < m; j += SORT_THREADS) {
    const uint32_t k = sm.key[j];
    const uint32_t dst = sm.base[(k >> shift) & (RADIX - 1)] + (uint32_t)j;
    keys_out[dst] = k;
    vals_out[dst] = sm.val[j];
  }
}

// ---------------------------------------------------------------- blocks
struct Box {
  float lo[3], hi[3];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = INFINITY;
      hi[a] = -INFINITY;
    }
  }
  __device__ __forceinline__ void add(const float4& p) {
    lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
    hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
  }
  // union over the lanes that differ in bit `off`
  __device__ __forceinline__ void merge_lane(int off) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], off));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], off));
    }
  }
};

// Boxes of sibling-ordered nodes in shared memory, [component][node].
template <int COUNT>
struct BoxTable {
  float v[6][COUNT];
  __device__ __forceinline__ void put(int i, const Box& b) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[a][i] = b.lo[a];
      v[3 + a][i] = b.hi[a];
    }
  }
  __device__ __forceinline__ void get(int i, Box& b) const {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = v[a][i];
      b.hi[a] = v[3 + a][i];
    }
  }
};

// Writes the boxes 0 .. count-1 of T (a multiple of 4), which are the nodes
// first, first + 1, ... of level lvl + 1, as whole groups of level lvl, with
// coalesced 16-byte stores.  Nodes past the level's last slot are dropped.
template <int COUNT>
__device__ __forceinline__ void write_groups(const BoxTable<COUNT>& T, int count, int lvl, int64_t first,
                                             float4* __restrict__ groups) {
  const int64_t g0 = first >> 2;
  const int64_t room = (1ll << (2 * lvl)) - g0;
  for (int w = threadIdx.x; w < count / 4 * GROUP_F4; w += blockDim.x) {
    const int g = w / GROUP_F4, f = w % GROUP_F4;
    if (g >= room) break;
    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (f < 6) o = make_float4(T.v[f][4 * g], T.v[f][4 * g + 1], T.v[f][4 * g + 2], T.v[f][4 * g + 3]);
    groups[(size_t)GROUP_F4 * (size_t)(group_offset(lvl) + g0 + g) + f] = o;
  }
}

// Union of sibling boxes 4i .. 4i+3 of A into box i of B.
template <int CA, int CB>
__device__ __forceinline__ void union4(const BoxTable<CA>& A, BoxTable<CB>& B, int i) {
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const float* a = &A.v[c][4 * i];
    B.v[c][i] = c < 3 ? fminf(fminf(a[0], a[1]), fminf(a[2], a[3])) : fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3]));
  }
}

// Block of consecutive curve-ordered points whose leaves are laid out
// together: 4 points per thread, thread t holding positions 4t .. 4t+3.
constexpr int BLK_THREADS = 256;
constexpr int BLK = 4 * BLK_THREADS;

// Compare-exchange stage of a bitonic sort over the block, stride J inside
// runs of K; every run of S is sorted ascending on its own.
template <int S, int K, int J>
__device__ __forceinline__ void bitonic_stage(uint32_t (&k)[4], uint4* ex) {
  const int t = threadIdx.x;
  uint32_t o[4];
  if constexpr (J >= 128) {
    __syncthreads();
    ex[t] = make_uint4(k[0], k[1], k[2], k[3]);
    __syncthreads();
    const uint4 v = ex[t ^ (J / 4)];
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  } else if constexpr (J >= 4) {
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = __shfl_xor_sync(0xffffffffu, k[r], J / 4);
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = k[r ^ J];
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = 4 * t + r;
    const bool low = (i & J) == 0, up = K == S || (i & K) == 0;
    k[r] = low == up ? min(k[r], o[r]) : max(k[r], o[r]);
  }
}
template <int S, int K, int J>
__device__ __forceinline__ void bitonic_merge(uint32_t (&k)[4], uint4* ex) {
  bitonic_stage<S, K, J>(k, ex);
  if constexpr (J > 1) bitonic_merge<S, K, J / 2>(k, ex);
}
template <int S, int K>
__device__ __forceinline__ void bitonic_sort(uint32_t (&k)[4], uint4* ex) {
  bitonic_merge<S, K, K / 2>(k, ex);
  if constexpr (K < S) bitonic_sort<S, 2 * K>(k, ex);
}

// One median split: every run of S positions is sorted along the longest
// side of its own bounding box, so that its two halves are the two sides of
// the median.  A word is (coordinate in 22 bits of the run's box, slot);
// slots past the block's m points sort last.
template <int S, int LEAF>
__device__ __forceinline__ void split_runs(uint32_t (&k)[4], const float4* __restrict__ P, int m,
                                           uint4* ex, BoxTable<BLK_THREADS / 32>& wbox) {
  const int t = threadIdx.x;
  Box b;
  b.clear();
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if ((int)k[r] < m) b.add(P[k[r]]);
#pragma unroll
  for (int off = 1; off < 32 && off < S / 4; off *= 2) b.merge_lane(off);
  if (S > 128) {
    __syncthreads();
    if ((t & 31) == 0) wbox.put(t >> 5, b);
    __syncthreads();
    const int w0 = (t >> 5) & ~(S / 128 - 1);
    wbox.get(w0, b);
#pragma unroll
    for (int w = 1; w < S / 128; ++w) {
      Box o;
      wbox.get(w0 + w, o);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        b.lo[a] = fminf(b.lo[a], o.lo[a]);
        b.hi[a] = fmaxf(b.hi[a], o.hi[a]);
      }
    }
  }
  const float ex0 = b.hi[0] - b.lo[0], ex1 = b.hi[1] - b.lo[1], ex2 = b.hi[2] - b.lo[2];
  const int ax = ex0 >= ex1 && ex0 >= ex2 ? 0 : ex1 >= ex2 ? 1 : 2;
  const float lo = ax == 0 ? b.lo[0] : ax == 1 ? b.lo[1] : b.lo[2];
  const float len = fmaxf(fmaxf(ex0, ex1), fmaxf(ex2, 1e-30f));
  const float sc = 4194302.0f / len;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    uint32_t q = 4194303u;
    if ((int)k[r] < m) {
      const float4 p = P[k[r]];
      const float c = ax == 0 ? p.x : ax == 1 ? p.y : p.z;
      q = (uint32_t)fminf(fmaxf((c - lo) * sc, 0.0f), 4194302.0f);
    }
    k[r] |= q << 10;
  }
  bitonic_sort<S, 2>(k, ex);
#pragma unroll
  for (int r = 0; r < 4; ++r) k[r] &= 1023u;
  if constexpr (S / 2 > LEAF) split_runs<S / 2, LEAF>(k, P, m, ex, wbox);
}

// Leaves, records and the tree's lowest levels, one CTA per 1024 consecutive
// points in curve order.  The curve alone makes poor leaves: a run of 16 is
// a ragged patch whose box overlaps its neighbours', and inside one curve
// cell the points are in no order at all.  Here the CTA splits its points by
// medians down to the leaf size (a k-d order in shared memory), so leaves
// are compact, equal in count and nearly disjoint.  Then it writes the
// records, colours and permutation in that order, and the groups of the
// three (leaf 32: two) levels above the leaves that lie inside the block.
//
// Bound by the random 16-byte gather of the points (2.1 GB of DRAM reads at
// 20M points, 107 bytes a point) and by the sorting networks' instructions:
// 0.94 ms at 20M points, where the gather alone in curve order, with the leaf
// boxes and a launch per level, took 1.48.  Without a register cap two CTAs
// fit on an SM and it took 1.15; three to six CTAs measured the same.  What
// it buys at 20M points, against a Morton order: 50 instead of 74 node
// expansions and 17.5 instead of 25.4 leaves per step of the marcher's warps
// (24 views: 313 -> 240 ms).
template <int LEAF>
__global__ void __launch_bounds__(BLK_THREADS, 3)
k_blocks(const float4* __restrict__ pos, const float* __restrict__ radii, const uint32_t* __restrict__ order,
         int64_t n, int depth, float4* __restrict__ rec, uint32_t* __restrict__ col, int32_t* __restrict__ perm,
         float4* __restrict__ groups) {
  __shared__ float4 P[BLK];
  __shared__ uint32_t I[BLK];
  __shared__ uint4 E[BLK_THREADS];
  __shared__ BoxTable<BLK_THREADS / 32> wbox;
  constexpr int C0 = BLK / LEAF, C1 = C0 / 4, C2 = C1 / 4;
  __shared__ BoxTable<C0> B0;
  __shared__ BoxTable<C1> B1;
  __shared__ BoxTable<C2> B2;
  const int t = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.x * BLK;
  const int m = (int)max((int64_t)0, min((int64_t)BLK, n - base));
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int s = t + r * BLK_THREADS;
    if (s < m) {
      const uint32_t i = __ldg(order + base + s);
      I[s] = i;
      P[s] = __ldg(pos + i);
    }
  }
  __syncthreads();
  uint32_t k[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) k[r] = 4u * t + r;
  split_runs<BLK, LEAF>(k, P, m, E, wbox);
  // leaf boxes: LEAF / 4 threads hold a leaf
  Box b;
  b.clear();
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if ((int)k[r] < m) b.add(P[k[r]]);
#pragma unroll
  for (int off = 1; off < LEAF / 4; off *= 2) b.merge_lane(off);
  if ((4 * t) % LEAF == 0) B0.put(4 * t / LEAF, b);
  __syncthreads();
  E[t] = make_uint4(k[0], k[1], k[2], k[3]);
  if (t < C1) union4(B0, B1, t);
  __syncthreads();
  if (t < C2) union4(B1, B2, t);
  const uint32_t* slot = reinterpret_cast<const uint32_t*>(E);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int j = t + r * BLK_THREADS;
    if (j < m) {  // the slots past m sorted last
      const uint32_t s = slot[j];
      const float4 p = P[s];
      const uint32_t i = I[s];
      rec[base + j] = make_float4(p.x, p.y, p.z, radii ? __ldg(radii + i) : 0.0f);
      col[base + j] = __float_as_uint(p.w);
      perm[base + j] = (int32_t)i;
    }
  }
  __syncthreads();
  const int64_t first = (int64_t)blockIdx.x * C0;  // first leaf slot
  write_groups(B0, C0, depth - 1, first, groups);
  if (depth >= 2) write_groups(B1, C1, depth - 2, first / 4, groups);
  if (C2 >= 4 && depth >= 3) write_groups(B2, C2, depth - 3, first / 16, groups);
}
// levels of groups that k_blocks writes (C2 of leaf 32 is two boxes, half a group)
static int block_levels(int leaf) { return leaf == 32 ? 2 : 3; }

// Levels above: a CTA takes 1024 nodes of level lvl (of which `count` exist),
// unions each one's children and writes the groups of the levels lvl - 1 to
// lvl - 5 that they fill.
__global__ void __launch_bounds__(BLK_THREADS)
k_levels_up(int lvl, int64_t count, float4* __restrict__ groups) {
  __shared__ BoxTable<1024> B0;
  __shared__ BoxTable<256> B1;
  __shared__ BoxTable<64> B2;
  __shared__ BoxTable<16> B3;
  __shared__ BoxTable<4> B4;
  const int t = threadIdx.x;
  const int64_t first = (int64_t)blockIdx.x * 1024;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t j = first + t + r * BLK_THREADS;
    Box b;
    b.clear();
    if (j < count) {
      const float4* g = groups + (size_t)GROUP_F4 * (size_t)(group_offset(lvl) + j);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float4 l = g[a], h = g[3 + a];
        b.lo[a] = fminf(fminf(l.x, l.y), fminf(l.z, l.w));
        b.hi[a] = fmaxf(fmaxf(h.x, h.y), fmaxf(h.z, h.w));
      }
    }
    B0.put(t + r * BLK_THREADS, b);
  }
  __syncthreads();
  if (t < 256) union4(B0, B1, t);
  __syncthreads();
  if (t < 64) union4(B1, B2, t);
  __syncthreads();
  if (t < 16) union4(B2, B3, t);
  __syncthreads();
  if (t < 4) union4(B3, B4, t);
  __syncthreads();
  write_groups(B0, 1024, lvl - 1, first, groups);
  if (lvl >= 2) write_groups(B1, 256, lvl - 2, first / 4, groups);
  if (lvl >= 3) write_groups(B2, 64, lvl - 3, first / 16, groups);
  if (lvl >= 4) write_groups(B3, 16, lvl - 4, first / 64, groups);
  if (lvl >= 5) write_groups(B4, 4, lvl - 5, first / 256, groups);
}

__global__ void k_set_radius(float4* __restrict__ rec, const int32_t* __restrict__ perm,
                             const float* __restrict__ radii_clamped, int64_t n) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n;
       s += (int64_t)gridDim.x * blockDim.x)
    rec[s].w = radii_clamped[perm[s]];
}

__global__ void k_clamp_radii(const float* __restrict__ in, int64_t n, float max_radius,
                              float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float r = in[i];
    // main.cu:144-149
    out[i] = (max_radius > 0.0f && r > max_radius) ? max_radius : r;
  }
}

// Maximum radius (for the culling bound); radii are >= 0 so the float bit
// pattern orders like an unsigned integer.
__global__ void k_max_radius(const float* __restrict__ r, int64_t n, unsigned int* __restrict__ out) {
  float m = 0.0f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, r[i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

// ---------------------------------------------------------------- host side
static int grid_for(int64_t n, int threads, int max_blocks = 152 * 32) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (int)b;
}

void launch_pack(Ctx& c, const float* xyz, int stride, const uint8_t* rgb, int64_t n) {
  uint32_t* bounds = c.scalars.ptr<uint32_t>();
  CK(cudaMemsetAsync(bounds, 0, 7 * 4, c.stream));
  k_pack<<<grid_for(n, PACK_THREADS), PACK_THREADS, 0, c.stream>>>(xyz, stride, rgb, n, c.pos.ptr<float4>(), bounds);
}

void launch_clamp_radii_only(Ctx& c, const float* in, float max_radius) {
  k_clamp_radii<<<grid_for(c.n, 256), 256, 0, c.stream>>>(in, c.n, max_radius,
                                                            c.radii_clamped.ptr<float>());
}

void launch_set_radius(Ctx& c) {
  k_set_radius<<<grid_for(c.n, 256), 256, 0, c.stream>>>(c.rec.ptr<float4>(), c.perm.ptr<int32_t>(),
                                                          c.radii_clamped.ptr<float>(), c.n);
}

void launch_clamp_radii(Ctx& c, const float* in, float max_radius) {
  launch_clamp_radii_only(c, in, max_radius);
  launch_set_radius(c);
  refresh_max_radius(c);
}

void launch_max_radius(Ctx& c) {
  unsigned int* mr = c.scalars.ptr<unsigned int>() + 8;
  CK(cudaMemsetAsync(mr, 0, sizeof(unsigned int), c.stream));
  k_max_radius<<<grid_for(c.n, 256, 1024), 256, 0, c.stream>>>(c.radii_clamped.ptr<float>(), c.n, mr);
}

void set_max_radius(Ctx& c, unsigned bits) {
  float r;
  memcpy(&r, &bits, sizeof(r));
  c.max_r = (r < INFINITY) ? r : INFINITY;
}

void refresh_max_radius(Ctx& c) {
  launch_max_radius(c);
  unsigned int bits = 0;
  CK(cudaMemcpyAsync(&bits, c.scalars.ptr<unsigned int>() + 8, sizeof(bits), cudaMemcpyDeviceToHost, c.stream));
  CK(cudaStreamSynchronize(c.stream));
  set_max_radius(c, bits);
}

// Builds the index from c.pos / c.rgb.  Returns false (with c.err set) on
// invalid input.
bool build_index(Ctx& c) {
  const int64_t n = c.n;
  cudaStream_t st = c.stream;
  uint32_t* bounds = c.scalars.ptr<uint32_t>();
  // keys
  // Coarse cells of about 500 points where points lie on surfaces (about
  // 2.5 cells across occupied per cell of a face), half a block of the tree.
  int g = 1;
  while (g < 8 && n > (int64_t)1280 << (2 * g + 1)) ++g;
  c.half = std::max((n + 63) / 64 * 64, (int64_t)1 << (3 * g));  // halves start on 256 bytes
  c.keys.reserve((size_t)c.half * 8);
  c.vals.reserve((size_t)c.half * 8);
  uint32_t* coarse = c.key(1);  // counted in the sort's second buffer
  CK(cudaMemsetAsync(coarse, 0, (size_t)4 << (3 * g), st));
  CurveGrid* grid = reinterpret_cast<CurveGrid*>(c.scalars.ptr<uint32_t>() + 64);
  k_coarse_count<<<grid_for((n + 7) / 8, GRID_THREADS, c.sm_count * 8), GRID_THREADS, 0, st>>>(
      c.pos.ptr<float4>(), n, bounds, g, coarse, grid);
  k_curve_keys<<<grid_for(n, 256), 256, 0, st>>>(c.pos.ptr<float4>(), n, grid, g, coarse, c.key(0));
  // radix sort, 32-bit keys: shifts 0, 8, 16, 24
  int64_t ntiles = (n + SORT_TILE - 1) / SORT_TILE;
  int64_t clen = ntiles * RADIX;
  int64_t nscan = (clen + SCAN_TILE - 1) / SCAN_TILE;
  c.sort_counts.reserve((size_t)clen * 4);
  c.scan_sums.reserve((size_t)(nscan + 1) * 4 + 1024);  // also the buckets' cursors (rm_radii.cu)
  int cur = 0;
  for (int shift = 0; shift < 32; shift += 8) {
    uint32_t* cnt = c.sort_counts.ptr<uint32_t>();
    k_sort_hist<<<(unsigned)ntiles, SORT_THREADS, 0, st>>>(c.key(cur), n, shift, ntiles, cnt);
    const bool scanned = ntiles > SORT_OWN_SCAN;
    if (scanned) {
      k_scan_tiles<<<(unsigned)nscan, SCAN_THREADS, 0, st>>>(cnt, clen, c.scan_sums.ptr<uint32_t>());
      k_scan_sums<<<1, SCAN_THREADS, 0, st>>>(c.scan_sums.ptr<uint32_t>(), nscan);
      k_scan_add<<<(unsigned)nscan, SCAN_THREADS, 0, st>>>(cnt, clen, c.scan_sums.ptr<uint32_t>());
    }
    auto scatter = [&](auto kern) {
      CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem)));
      kern<<<(unsigned)ntiles, SORT_THREADS, sizeof(SortSmem), st>>>(
          c.key(cur), c.val(cur), n, shift, ntiles, cnt,
          c.key(cur ^ 1), c.val(cur ^ 1));
    };
    if (scanned) {
      if (shift == 0) scatter(k_sort_scatter<true, true>);
      else scatter(k_sort_scatter<false, true>);
    } else {
      if (shift == 0) scatter(k_sort_scatter<true, false>);
      else scatter(k_sort_scatter<false, false>);
    }
    cur ^= 1;
  }
  // leaves and tree
  c.rec.reserve((size_t)n * sizeof(float4));
  c.col.reserve((size_t)n * 4);
  c.perm.reserve((size_t)n * 4);
  const int leaf = c.cfg.leaf_size;
  const int64_t nleaves = (n + leaf - 1) / leaf;
  int depth = 1;
  while ((1ll << (2 * depth)) < nleaves) ++depth;
  if (depth > MAX_LEVELS) {
    c.err = "cloud too large for the index depth limit";
    return false;
  }
  c.groups.reserve((size_t)group_offset(depth) * GROUP_F4 * sizeof(float4));
  // Siblings of a real node are written down to the next two levels even
  // where they are empty: the one-query walks read two levels at a time.  So
  // blocks, and nodes above, are taken in fours.
  const unsigned nblocks = (unsigned)((n + BLK - 1) / BLK + 3) / 4 * 4;
  auto blocks = [&](auto kern) {
    kern<<<nblocks, BLK_THREADS, 0, st>>>(c.pos.ptr<float4>(), c.have_radii ? c.radii_clamped.ptr<float>() : nullptr,
                                          c.val(cur), n, depth, c.rec.ptr<float4>(),
                                          c.col.ptr<uint32_t>(), c.perm.ptr<int32_t>(), c.groups.ptr<float4>());
  };
  if (leaf == 8) blocks(k_blocks<8>);
  else if (leaf == 16) blocks(k_blocks<16>);
  else blocks(k_blocks<32>);
  // groups of the levels above, five per launch
  const int done = block_levels(leaf);
  int64_t count = (int64_t)nblocks * (BLK / leaf) >> (2 * done);
  for (int lvl = depth - done; lvl >= 1; lvl -= 5) {
    const unsigned g = (unsigned)((count + 1023) / 1024 + 3) / 4 * 4;
    k_levels_up<<<g, BLK_THREADS, 0, st>>>(lvl, count, c.groups.ptr<float4>());
    count = g;
  }
  c.depth = depth;
  c.nleaves = nleaves;
  CK(cudaGetLastError());
  if (c.have_radii) launch_max_radius(c);
  // bounds, the non-finite flag and the largest radius in one read (an index
  // over non-finite points is built but not used)
  uint32_t hb[9];
  CK(cudaMemcpyAsync(hb, bounds, sizeof(hb), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (hb[6] != 0) {
    c.err = "cloud contains non-finite coordinates";
    return false;
  }
  for (int a = 0; a < 6; ++a) {
    const uint32_t u = from_ordered_bits(a < 3 ? ~hb[a] : hb[a]);
    memcpy(&c.bounds[a], &u, sizeof(u));
  }
  if (c.have_radii) set_max_radius(c, hb[8]);
  c.have_index = true;
  return true;
}

}  // namespace rm
