// rm_radii.cu -- exact nearest-neighbour radii and the general kNN query.
//
// Replaces the reference's radii precompute (main.cu:107-113): FLANN
// nearestKernel with k = 2 (kdtree_cuda_3d_index.cu:132-154, one thread per
// query, result arrays in global memory), followed by a host loop doing 2N
// synchronous device_reference copies for sqrt, and a separate clamp pass
// (main.cu:144-149).  Here one kernel does the search and the sqrt for nearly
// every point, in index order, so the queries of a warp are spatial
// neighbours; the few that it leaves over are searched one per warp, and
// short passes write the results in cloud order and clamp.
#include "rm_internal.h"

#include <algorithm>

namespace rm {

__global__ void __launch_bounds__(128)
k_radii(IndexDev ix, float max_radius, float* __restrict__ radii_out, int32_t* __restrict__ nn_out,
        float* __restrict__ radii_clamped, unsigned long long* __restrict__ err) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < ix.n;
       s += (int64_t)gridDim.x * blockDim.x) {
    float4 q = __ldg(ix.rec + s);
    KList<2> L;
    klist_init<2>(L);
    if (!knn_search(ix, q.x, q.y, q.z, L)) atomicAdd(err, 1ull);
    // sqrt of the second entry (main.cu:111); +inf when the cloud has one point
    float r = __fsqrt_rn(L.d[1]);
    int32_t i = __ldg(ix.perm + s);
    if (radii_out) radii_out[i] = r;
    if (nn_out) nn_out[i] = L.s[1] >= 0 ? __ldg(ix.perm + L.s[1]) : -1;
    radii_clamped[i] = (max_radius > 0.0f && r > max_radius) ? max_radius : r;
  }
}

// Region form: a warp takes 32 or 64 consecutive records (one compact piece
// of the median-split order) as one or two chunks of 32 queries.
//
//   1. Seed: every lane measures the other 31 points of its query's chunk,
//      which bounds all of the chunk's searches by the largest distance W.
//   2. One walk for the region: eight pending nodes are expanded at a time,
//      one child per lane, and each child's box is tested against the
//      chunks' boxes grown by W.  Leaves that any chunk may need go
//      onto a list with the mask of those chunks.
//      A chunk that straddles a gap (two surfaces, a stray point) has a box
//      far wider than its searches; such a chunk's children are tested again
//      against every query's own bound before they are kept.
//   3. Scan: per chunk, a listed leaf that lies within some lane's own bound
//      is staged in shared memory and measured by all lanes.  A full list is
//      scanned in mid-walk, which also tightens the W of the rest.
//
// The box-to-box distance is the same fma chain over per-axis gaps as
// d2_box, and each gap is at most that of any query in the chunk, so a
// needed leaf is never missed.
//
// Issue-bound (79% of the issue slots at 20M points).  One walk of the tree
// per 32 queries, with every lane testing its own query against every box,
// spent most of its instructions on the descent (59 expansions and 23 leaves
// per warp in curve order).  Here an expansion tests 32 boxes at once, and
// per chunk about 19 listed leaves are tested and 11 measured, four points at
// a time (d2_point4: 3.6 -> 2.7 ms at 20M).  8.5 -> 2.9 ms at 20M points, 61 ->
// 16 ms at 100M of uneven density, 76 -> 60 us at 100k, with the handed-over
// queries and the order of the records (k_blocks in rm_index.cu).
//
// Memory traffic.  Warps take their regions from a global counter in sorted
// order, so all resident warps work inside one window of a few MB that
// stays in L2.  Results go out in sorted order with coalesced stores;
// k_to_cloud, or k_to_buckets and k_from_buckets, and k_split move them to
// cloud order afterwards.
constexpr int RADII_WARPS = 4;
// Chunks per region.  Two share the descent, but make half as many, longer
// regions: 1 against 2 chunks measured 0.12 / 0.19 ms at 500k points (search
// and handed-over queries), 0.61 / 0.65 at 4M, 1.15 / 1.20 at 8M, 2.87 / 2.85
// at 20M and 8.6 / 8.4 at 60M.
constexpr int64_t RADII_SMALL = 12 << 20;
constexpr int REGION_STACK = 512;  // depth-first, one node at a time, needs 3 entries per level beyond the last 64
constexpr int REGION_LIST = 96;
// scans of a full list before a region gives up its walk
template <int CHUNKS>
constexpr int REGION_SCANS = CHUNKS == 1 ? 1 : 6;
// In squared lengths, a chunk on a surface is about 55 times as wide as its
// largest search; well above that its box says little (REGION_WIDE).  The
// squared distances to the nearest neighbour on an even surface are
// exponentially distributed: one in 10^7 is over 24 medians (REGION_LOST is
// wider, a search costs its query as much as 25 others).
constexpr float REGION_WIDE = 1024.0f, REGION_LOST = 64.0f;
static_assert(REGION_STACK > 64 + 3 * MAX_LEVELS, "region stack too small");

struct alignas(16) ListedLeaf {
  float box[6];
  uint32_t leaf, chunks;  // number, mask of the chunks that may need it
};
template <int CHUNKS>
struct RegionSmem {
  ListedLeaf list[REGION_LIST];
  alignas(16) float x[32], y[32], z[32];         // staged leaf
  alignas(16) float qx[32 * CHUNKS], qy[32 * CHUNKS], qz[32 * CHUNKS];  // queries
  float d[32 * CHUNKS];                          // nearest other point so far (Nearest); d = -1: no query
  int32_t s[32 * CHUNKS], s2[32 * CHUNKS];
  alignas(16) float chunk[CHUNKS][8];            // box, largest d
  uint32_t stack[REGION_STACK];
};

// Nearest other point of a query: (d, s) and s2, the point of the next
// higher cloud index at the same distance d (-1: none).
struct Nearest {
  float d;
  int32_t s, s2;
  // a candidate with dd <= d; the query itself and points met before are skipped
  __device__ __forceinline__ void consider(float dd, int32_t ss, int32_t self, const int32_t* __restrict__ perm) {
    if (ss == self || ss == s || ss == s2) return;
    if (dd < d) {
      d = dd;
      s = ss;
      s2 = -1;
    } else if (s >= 0) {  // equal distances: lower cloud indices first
      const int32_t i = __ldg(perm + ss);
      if (i < __ldg(perm + s)) {
        s2 = s;
        s = ss;
      } else if (s2 < 0 || i < __ldg(perm + s2)) {
        s2 = ss;
      }
    }
  }
  // cloud index of the second entry of the self-inclusive list, -1: none
  __device__ __forceinline__ int32_t second(int64_t self, const int32_t* __restrict__ perm) const {
    int32_t nn = s >= 0 ? __ldg(perm + s) : -1;
    if (d == 0.0f) {  // coincident points: the second of (self, nearest, next) by cloud index
      const int32_t i = __ldg(perm + self);
      if (nn < i) nn = s2 >= 0 ? min(i, __ldg(perm + s2)) : i;
    }
    return nn;
  }
};

// d2_point of four points given as coordinate arrays (paired arithmetic, the
// same bits); the query twice per register pair.
__device__ __forceinline__ void d2_point4(const float* x, const float* y, const float* z, unsigned long long qx2,
                                          unsigned long long qy2, unsigned long long qz2, float (&d)[4]) {
  const float4 X = *reinterpret_cast<const float4*>(x), Y = *reinterpret_cast<const float4*>(y),
               Z = *reinterpret_cast<const float4*>(z);
  const unsigned long long x0 = f2_sub(f2_pack(X.x, X.y), qx2), x1 = f2_sub(f2_pack(X.z, X.w), qx2);
  const unsigned long long y0 = f2_sub(f2_pack(Y.x, Y.y), qy2), y1 = f2_sub(f2_pack(Y.z, Y.w), qy2);
  const unsigned long long z0 = f2_sub(f2_pack(Z.x, Z.y), qz2), z1 = f2_sub(f2_pack(Z.z, Z.w), qz2);
  f2_unpack(f2_fma(z0, z0, f2_fma(x0, x0, f2_mul(y0, y0))), d[0], d[1]);
  f2_unpack(f2_fma(z1, z1, f2_fma(x1, x1, f2_mul(y1, y1))), d[2], d[3]);
}

// Queries left to searches of their own (k_radii_hard): sorted positions.
struct HardList {
  uint32_t* pos;              // room for every point
  unsigned long long* count;
};
__device__ __forceinline__ void hand_over(bool mine, uint32_t s, const HardList& hard) {
  const unsigned m = __ballot_sync(0xffffffffu, mine);
  if (m == 0) return;
  const int lane = threadIdx.x & 31;
  unsigned long long at = 0;
  if (lane == 0) at = atomicAdd(hard.count, (unsigned long long)__popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (mine) hard.pos[at + __popc(m & ((1u << lane) - 1u))] = s;
}

// Scans the listed leaves for every chunk that may need them and refreshes
// the chunks' W.
template <int CHUNKS>
__device__ void region_scan(const IndexDev& ix, RegionSmem<CHUNKS>& sm, int64_t base, int listed) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int c = 0; c < CHUNKS; ++c) {
    const float qx = sm.qx[32 * c + lane], qy = sm.qy[32 * c + lane], qz = sm.qz[32 * c + lane];
    const unsigned long long qx2 = f2_pack(qx, qx), qy2 = f2_pack(qy, qy), qz2 = f2_pack(qz, qz);
    Nearest N{sm.d[32 * c + lane], sm.s[32 * c + lane], sm.s2[32 * c + lane]};
    const int32_t self = (int32_t)(base + 32 * c + lane);
    for (int e = 0; e < listed; ++e) {
      const float4 lo = *reinterpret_cast<const float4*>(sm.list[e].box);
      const uint4 hi = *reinterpret_cast<const uint4*>(sm.list[e].box + 4);
      if (!((hi.w >> c) & 1u)) continue;
      const float m = d2_box(lo.x, lo.y, lo.z, lo.w, __uint_as_float(hi.x), __uint_as_float(hi.y), qx, qy, qz);
      if (!__ballot_sync(FULL, m <= N.d)) continue;
      const int64_t start = (int64_t)hi.z * ix.leaf;
      const int cnt = (int)min((int64_t)ix.leaf, ix.n - start);
      __syncwarp();
      const float none = __int_as_float(0x7fffffff);  // NaN, past the leaf's end: within no bound
      const float4 r = lane < cnt ? __ldg(ix.rec + start + lane) : make_float4(none, none, none, none);
      sm.x[lane] = r.x;
      sm.y[lane] = r.y;
      sm.z[lane] = r.z;
      __syncwarp();
      for (int k = 0; k < cnt; k += 4) {
        float d[4];
        d2_point4(sm.x + k, sm.y + k, sm.z + k, qx2, qy2, qz2, d);
        if (fminf(fminf(d[0], d[1]), fminf(d[2], d[3])) <= N.d) {
          // rare: 11 of 170 points are within the bound of any lane
#pragma unroll 1
          for (int j = 0; j < 4; ++j) {
            if (d[0] <= N.d) N.consider(d[0], (int32_t)start + k + j, self, ix.perm);
            d[0] = d[1];
            d[1] = d[2];
            d[2] = d[3];
          }
        }
      }
    }
    sm.d[32 * c + lane] = N.d;
    sm.s[32 * c + lane] = N.s;
    sm.s2[32 * c + lane] = N.s2;
    // distances are >= 0 (or -1 for no query): ordered like signed integers
    const int w = __reduce_max_sync(FULL, __float_as_int(N.d));
    if (lane == 0) sm.chunk[c][6] = __int_as_float(w);
  }
  __syncwarp();
}

template <int CHUNKS>
__global__ void __launch_bounds__(32 * RADII_WARPS)
k_radii_region(IndexDev ix, float* __restrict__ r_sorted, int32_t* __restrict__ nn_sorted,
               unsigned long long* __restrict__ next, HardList hard) {
  constexpr int REGION = 32 * CHUNKS;
  __shared__ RegionSmem<CHUNKS> smem[RADII_WARPS];
  const unsigned FULL = 0xffffffffu;
  const float INF = __int_as_float(0x7f800000);
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  RegionSmem<CHUNKS>& sm = smem[threadIdx.x >> 5];
  const uint32_t last_first = (uint32_t)group_offset(ix.depth - 1);  // first group of level depth-1
  while (true) {
    unsigned long long region = 0;
    if (lane == 0) region = atomicAdd(next, 1ull);
    const int64_t base = (int64_t)__shfl_sync(FULL, region, 0) * REGION;
    if (base >= ix.n) break;
    // seed
    unsigned wide = 0;  // chunks whose box is far wider than their searches
    for (int c = 0; c < CHUNKS; ++c) {
      const int64_t s = base + 32 * c + lane;
      const bool active = s < ix.n;
      const float4 q = active ? __ldg(ix.rec + s) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float none = __int_as_float(0x7fffffff);  // a place without a query is near to none
      sm.qx[32 * c + lane] = active ? q.x : none;
      sm.qy[32 * c + lane] = active ? q.y : none;
      sm.qz[32 * c + lane] = active ? q.z : none;
      __syncwarp();
      const int cnt = (int)max((int64_t)0, min((int64_t)32, ix.n - (base + 32 * c)));
      const unsigned long long qx2 = f2_pack(q.x, q.x), qy2 = f2_pack(q.y, q.y), qz2 = f2_pack(q.z, q.z);
      float d = INF;
      int at = -1;
      bool tie = false;
#pragma unroll 2
      for (int k = 0; k < 32; k += 4) {
        float dd[4];
        d2_point4(sm.qx + 32 * c + k, sm.qy + 32 * c + k, sm.qz + 32 * c + k, qx2, qy2, qz2, dd);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (k + j == lane) dd[j] = INF;
          const bool less = dd[j] < d;
          tie = !less && (tie || dd[j] == d);
          at = less ? k + j : at;
          d = less ? dd[j] : d;
        }
      }
      Nearest N{d, at >= 0 ? (int32_t)(base + 32 * c) + at : -1, -1};
      if (tie && at >= 0)  // equal nearest distances in the chunk: order them by cloud index
        for (int k = 0; k < cnt; ++k) {
          const float dd = d2_point(make_float4(sm.qx[32 * c + k], sm.qy[32 * c + k], sm.qz[32 * c + k], 0.0f), q.x, q.y, q.z);
          if (dd == d) N.consider(dd, (int32_t)(base + 32 * c) + k, (int32_t)s, ix.perm);
        }
      if (active && cnt < 32 && base + 32 * c >= 32)  // a short last chunk: a bound from the chunk before it
        for (int k = 1; k <= 32; ++k) {
          const int64_t p = base + 32 * c - k;
          const float dd = d2_point(__ldg(ix.rec + p), q.x, q.y, q.z);
          if (dd <= N.d) N.consider(dd, (int32_t)p, (int32_t)s, ix.perm);
        }
      // A query far from the rest of its chunk (alone on its side of a gap):
      // the chunk tells little about it, and it would widen the chunk's
      // box, so it gets a search of its own.  The rest is judged by the
      // median of the queries that do not coincide with another point (to
      // rounding): beside repeated points every other one would seem far
      // (16M points, 60% of them repeated: 17.0 ms against 2.9).
      const float ulp = fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z)) * 0x1p-22f;
      const int same = __popc(__ballot_sync(FULL, active && N.d <= ulp * ulp));
      float med = active ? N.d : INF;  // by a sort across the lanes
#pragma unroll
      for (int size = 2; size <= 32; size *= 2)
#pragma unroll
        for (int j = size / 2; j > 0; j /= 2) {
          const float o = __shfl_xor_sync(FULL, med, j);
          med = ((lane & j) == 0) == ((lane & size) == 0) ? fminf(med, o) : fmaxf(med, o);
        }
      med = __shfl_sync(FULL, med, min(same + max(cnt - same - 1, 0) / 2, 31));
      const bool lost = active && N.d < INF && N.d > REGION_LOST * med;
      hand_over(lost, (uint32_t)s, hard);
      const bool here = active && !lost;
      const float lim[6] = {q.x, q.y, q.z, q.x, q.y, q.z};
#pragma unroll
      for (int f = 0; f < 6; ++f) {
        const uint32_t o = ordered_bits(here ? lim[f] : f < 3 ? INF : -INF);
        const float v = from_ordered(f < 3 ? __reduce_min_sync(FULL, o) : __reduce_max_sync(FULL, o));
        if (lane == 0) sm.chunk[c][f] = v;
      }
      __syncwarp();
      const float* cb = sm.chunk[c];
      const float ex = cb[3] - cb[0], ey = cb[4] - cb[1], ez = cb[5] - cb[2];
      const float diag2 = ex * ex + ey * ey + ez * ez;
      sm.d[32 * c + lane] = here ? N.d : -1.0f;
      sm.s[32 * c + lane] = N.s;
      sm.s2[32 * c + lane] = N.s2;
      const int w = __reduce_max_sync(FULL, __float_as_int(here ? N.d : -1.0f));
      if (lane == 0) sm.chunk[c][6] = __int_as_float(w);
      if (diag2 > REGION_WIDE * __int_as_float(w)) wide |= 1u << c;
    }
    if (lane == 0) sm.stack[0] = 0;
    __syncwarp();
    // walk
    int sp = 1, listed = 0, scans = 0;
    while (sp > 0) {
      if (listed > REGION_LIST - 32) {
        if (++scans > REGION_SCANS<CHUNKS>) {
          // The chunks' bounds are loose as a whole (points strewn over a
          // dense surface of other blocks): a search for every query
          // instead.  Only coincident points stay: their bound of 0 is as
          // tight as a search's.
          bool stay = false;
          for (int c = 0; c < CHUNKS; ++c) {
            const float d = sm.d[32 * c + lane];
            hand_over(d > 0.0f, (uint32_t)(base + 32 * c + lane), hard);
            if (d > 0.0f) sm.d[32 * c + lane] = -1.0f;
            const bool some = __ballot_sync(FULL, d == 0.0f) != 0;
            if (lane == 0) sm.chunk[c][6] = some ? 0.0f : -1.0f;
            stay |= some;
          }
          __syncwarp();
          if (!stay) {
            listed = 0;
            break;
          }
        }
        region_scan(ix, sm, base, listed);
        listed = 0;
      }
      const int take = sp < REGION_STACK - 64 - 3 * MAX_LEVELS ? min(sp, 8) : 1;
      const int slot = lane >> 2, ch = lane & 3;
      uint32_t G = 0, need = 0;
      float b[6] = {};
      if (slot < take) {
        G = sm.stack[sp - 1 - slot];
        const float* g = reinterpret_cast<const float*>(ix.groups + (size_t)GROUP_F4 * G) + ch;
#pragma unroll
        for (int f = 0; f < 6; ++f) b[f] = __ldg(g + 4 * f);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
          const float4 u = *reinterpret_cast<const float4*>(sm.chunk[c]), v = *reinterpret_cast<const float4*>(sm.chunk[c] + 4);
          const float gx = fmaxf(fmaxf(__fsub_rn(b[0], u.w), __fsub_rn(u.x, b[3])), 0.0f);
          const float gy = fmaxf(fmaxf(__fsub_rn(b[1], v.x), __fsub_rn(u.y, b[4])), 0.0f);
          const float gz = fmaxf(fmaxf(__fsub_rn(b[2], v.y), __fsub_rn(u.z, b[5])), 0.0f);
          const float m = __fmaf_rn(gz, gz, __fmaf_rn(gx, gx, __fmul_rn(gy, gy)));
          need |= m <= fminf(v.z, FLT_BIG) ? 1u << c : 0u;  // empty boxes, at +inf, never
        }
      }
      for (unsigned todo = __ballot_sync(FULL, need & wide); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        float o[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) o[f] = __shfl_sync(FULL, b[f], src);
        for (unsigned cs = __shfl_sync(FULL, need & wide, src); cs; cs &= cs - 1u) {
          const int c = __ffs(cs) - 1;
          const float m = d2_box(o[0], o[1], o[2], o[3], o[4], o[5], sm.qx[32 * c + lane], sm.qy[32 * c + lane],
                                 sm.qz[32 * c + lane]);
          if (!__ballot_sync(FULL, m <= sm.d[32 * c + lane]) && lane == src) need &= ~(1u << c);
        }
      }
      sp -= take;
      const bool bottom = G >= last_first;
      const uint32_t leaf = (G - last_first) * 4u + ch;
      if (bottom && need) {
        // the chunk's own leaves were measured by the seed
        const uint64_t own = (uint64_t)leaf * (uint32_t)ix.leaf - (uint64_t)base;
        if (own < REGION) need &= ~(1u << (own / 32));
      }
      const unsigned inner = __ballot_sync(FULL, need && !bottom), leaves = __ballot_sync(FULL, need && bottom);
      __syncwarp();  // every lane has read its stack entry
      if (need) {
        if (!bottom) {
          sm.stack[sp + __popc(inner & lt)] = 4u * G + 1u + ch;
        } else {
          const int e = listed + __popc(leaves & lt);
          *reinterpret_cast<float4*>(sm.list[e].box) = make_float4(b[0], b[1], b[2], b[3]);
          *reinterpret_cast<uint4*>(sm.list[e].box + 4) =
              make_uint4(__float_as_uint(b[4]), __float_as_uint(b[5]), leaf, need);
        }
      }
      sp += __popc(inner);
      listed += __popc(leaves);
      __syncwarp();
    }
    region_scan(ix, sm, base, listed);
    for (int c = 0; c < CHUNKS; ++c) {
      const int64_t s = base + 32 * c + lane;
      const float d = sm.d[32 * c + lane];
      if (d < 0.0f) continue;  // no query, or handed over
      const int32_t p = sm.s[32 * c + lane], p2 = sm.s2[32 * c + lane];
      // sqrt of the second entry of the self-inclusive list (main.cu:111);
      // +inf when the cloud has one point
      r_sorted[s] = __fsqrt_rn(d);
      nn_sorted[s] = Nearest{d, p, p2}.second(s, ix.perm);
    }
    __syncwarp();
  }
}

// The queries that the regions handed over, one per warp.
__global__ void __launch_bounds__(32 * RADII_WARPS)
k_radii_hard(IndexDev ix, HardList hard, float* __restrict__ r_sorted, int32_t* __restrict__ nn_sorted) {
  __shared__ WarpPool pools[RADII_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long count = *hard.count;
  for (unsigned long long t = blockIdx.x * RADII_WARPS + warp; t < count; t += (unsigned long long)gridDim.x * RADII_WARPS) {
    const int32_t self = (int32_t)hard.pos[t];
    const float4 q = __ldg(ix.rec + self);
    // its three nearest hold the two nearest others, and itself (unless three
    // other points coincide with it)
    WarpList<true> L;
    L.clear(__int_as_float(0x7f800000));
    warp_knn(ix, q.x, q.y, q.z, 3, L, pools[warp]);
    const int a = __shfl_sync(0xffffffffu, L.s, 0) == self ? 1 : 0;
    const int b = __shfl_sync(0xffffffffu, L.s, a + 1) == self ? a + 2 : a + 1;
    const float da = L.dist(a), db = L.dist(b);
    const int32_t sa = __shfl_sync(0xffffffffu, L.s, a), sb = __shfl_sync(0xffffffffu, L.s, b);
    if (lane == 0) {
      r_sorted[self] = __fsqrt_rn(da);
      nn_sorted[self] = Nearest{da, sa, db == da ? sb : -1}.second(self, ix.perm);
    }
    __syncwarp();
  }
}

// Sorted-order results to cloud order (main.cu:110-113 leaves them in PLY
// order).  Scattered stores cost an L2 request per point and array whatever
// their size, so radius and neighbour go as one 8-byte pair; k_split then
// streams the pairs apart into the caller's arrays and the context's clamped
// radii, and the records get theirs in sorted order.
//
// Direct form: one scattering pass.  While the pairs fit in L2 their sectors
// fill up there.
__device__ __forceinline__ float clamp_radius(float r, float max_radius) {  // main.cu:144-149
  return (max_radius > 0.0f && r > max_radius) ? max_radius : r;
}
__device__ __forceinline__ void set_record(float4* __restrict__ rec, int64_t s, float r) {
  float4 p = rec[s];  // whole records rewritten: full-sector stores
  p.w = r;
  rec[s] = p;
}
__global__ void k_to_cloud(const float* __restrict__ r_sorted, const int32_t* __restrict__ nn_sorted,
                           const int32_t* __restrict__ perm, int64_t n, float max_radius, float4* __restrict__ rec,
                           int2* __restrict__ pairs) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
    const float r = __ldcs(r_sorted + s);
    pairs[__ldcs(perm + s)] = make_int2(__float_as_int(r), __ldcs(nn_sorted + s));
    set_record(rec, s, clamp_radius(r, max_radius));
  }
}

// Bucket form, for pairs beyond L2, where nearly every scattered store costs
// a sector read and written in DRAM.  First the pairs are brought into
// BUCKETS ranges of cloud indices: a tile is put in bucket order in shared
// memory and goes out in runs, each tile taking its places in a bucket from
// that bucket's cursor (the order inside a bucket does not matter).  A bucket
// covers 2^shift cloud indices, exactly as many as it has places.  Then a
// second pass scatters bucket by bucket, a few MB at a time.
//
// Bound by the scattered stores' L2 requests (95 G/s).  Direct and bucket
// form without k_split: 53 and 87 us at 4M points, 131 and 182 at 8M, 643 and
// 423 at 20M, 4.4 and 2.1 ms at 100M; three scattering passes of 4-byte
// values took 0.70 ms at 20M and 11.0 ms at 100M where this, with k_split,
// takes 0.49 and 2.4.
constexpr int BUCKETS = 256;
constexpr int BUCKET_THREADS = 256;
constexpr int BUCKET_ITEMS = 16;
constexpr int BUCKET_TILE = BUCKET_THREADS * BUCKET_ITEMS;
constexpr int64_t BUCKET_MIN = 12 << 20;  // points from which the bucket form is taken
struct BucketSmem {
  uint32_t cnt[BUCKETS], first[BUCKETS], base[BUCKETS];
  uint32_t sums[BUCKETS / 32];
  int32_t i[BUCKET_TILE];
  int2 pair[BUCKET_TILE];
};
__global__ void __launch_bounds__(BUCKET_THREADS, 4)
k_to_buckets(const float* __restrict__ r_sorted, const int32_t* __restrict__ nn_sorted,
             const int32_t* __restrict__ perm, int64_t n, int shift, float max_radius, float4* __restrict__ rec,
             uint32_t* __restrict__ cursor, int32_t* __restrict__ to_i, int2* __restrict__ to_pair) {
  extern __shared__ __align__(16) unsigned char bucket_smem[];
  BucketSmem& sm = *reinterpret_cast<BucketSmem*>(bucket_smem);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  sm.cnt[t] = 0;
  __syncthreads();
  const int64_t tile = (int64_t)blockIdx.x * BUCKET_TILE;
  int32_t idx[BUCKET_ITEMS];
  uint32_t rank[BUCKET_ITEMS];
#pragma unroll
  for (int k = 0; k < BUCKET_ITEMS; ++k) {
    const int64_t s = tile + k * BUCKET_THREADS + t;
    idx[k] = s < n ? __ldcs(perm + s) : -1;
  }
#pragma unroll
  for (int k = 0; k < BUCKET_ITEMS; ++k)
    if (idx[k] >= 0) rank[k] = atomicAdd(&sm.cnt[idx[k] >> shift], 1u);
  __syncthreads();
  const uint32_t c = sm.cnt[t];
  uint32_t x = c;  // exclusive prefix over the buckets, one per thread
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) sm.sums[warp] = x;
  __syncthreads();
  uint32_t first = x - c;
  for (int w = 0; w < warp; ++w) first += sm.sums[w];
  sm.first[t] = first;
  sm.base[t] = c ? ((uint32_t)t << shift) + atomicAdd(cursor + t, c) - first : 0u;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < BUCKET_ITEMS; ++k) {
    if (idx[k] < 0) continue;
    const int64_t s = tile + k * BUCKET_THREADS + t;
    const float r = __ldcs(r_sorted + s);
    set_record(rec, s, clamp_radius(r, max_radius));
    const uint32_t at = sm.first[idx[k] >> shift] + rank[k];
    sm.i[at] = idx[k];
    sm.pair[at] = make_int2(__float_as_int(r), __ldcs(nn_sorted + s));
  }
  __syncthreads();
  const int count = (int)min((int64_t)BUCKET_TILE, n - tile);
  for (int j = t; j < count; j += BUCKET_THREADS) {
    const int32_t i = sm.i[j];
    const uint32_t at = sm.base[i >> shift] + (uint32_t)j;
    to_i[at] = i;
    to_pair[at] = sm.pair[j];
  }
}
// One tile per CTA, so that the resident CTAs work on adjacent tiles.
__global__ void __launch_bounds__(BUCKET_THREADS)
k_from_buckets(const int32_t* __restrict__ from_i, const int2* __restrict__ from_pair, int64_t n,
               int2* __restrict__ pairs) {
  const int64_t tile = (int64_t)blockIdx.x * BUCKET_TILE;
#pragma unroll 8
  for (int k = 0; k < BUCKET_ITEMS; ++k) {
    const int64_t j = tile + k * BUCKET_THREADS + threadIdx.x;
    if (j < n) pairs[__ldcs(from_i + j)] = __ldcs(from_pair + j);
  }
}

// Pairs to the caller's arrays (either may be null) and the context's clamped
// radii; `largest` gets the bits of the largest of those (they are >= 0).
__global__ void k_split(const int2* __restrict__ pairs, int64_t n, float max_radius, float* __restrict__ radius,
                        int32_t* __restrict__ nn, float* __restrict__ clamped, unsigned* __restrict__ largest) {
  float m = 0.0f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int2 p = __ldcs(pairs + i);
    const float r = __int_as_float(p.x), c = clamp_radius(r, max_radius);
    if (radius) radius[i] = r;
    if (nn) nn[i] = p.y;
    clamped[i] = c;
    m = fmaxf(m, c);
  }
  __shared__ unsigned most;
  if (threadIdx.x == 0) most = 0;
  __syncthreads();
  atomicMax(&most, __float_as_uint(m));
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(largest, most);
}

// General k-NN (k <= 32): one query per warp, the k nearest in the warp's
// lanes (warp_knn).  Where queries come in any order, 32 of them in one
// warp share nothing: one query per lane, with its list in that lane's
// registers, took 27.3 ms for 500k unsorted queries (k = 10, 2M points, in
// divergent walks) where this takes 1.25, and 570 us for 1000 queries (k = 1,
// 100k points, the latency of the longest walk) where this takes 32.
// Issue-bound for many queries, latency-bound for few (about 8 expansions and
// 5 batches of leaves, one after the other).
//
// REST: only the queries that k_knn_lanes marked are left.
constexpr int KNN_WARPS = 4;
constexpr int32_t KNN_LEFT = -2;
template <bool REST>
__global__ void __launch_bounds__(32 * KNN_WARPS)
k_knn(IndexDev ix, const float* __restrict__ q, int stride, int64_t m, int k,
      int32_t* __restrict__ idx_out, float* __restrict__ d2_out) {
  __shared__ WarpPool pools[KNN_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t step = (int64_t)gridDim.x * KNN_WARPS;
  const auto search = [&](int64_t t) {
    const float* p = q + t * stride;
    WarpList<false> L;
    L.clear(__int_as_float(0x7f800000));
    warp_knn(ix, __ldg(p), __ldg(p + 1), __ldg(p + 2), k, L, pools[warp]);
    if (lane < k) {
      idx_out[t * k + lane] = L.index();
      d2_out[t * k + lane] = __uint_as_float((unsigned)(L.key >> 32));
    }
    __syncwarp();
  };
  if (REST) {
    // 32 of the warp's queries looked at together
    for (int64_t t0 = blockIdx.x * (int64_t)KNN_WARPS + warp; t0 < m; t0 += 32 * step) {
      const int64_t mine = t0 + lane * step;
      unsigned left = __ballot_sync(0xffffffffu, mine < m && idx_out[mine * k] == KNN_LEFT);
      for (; left; left &= left - 1u) search(t0 + (__ffs(left) - 1) * step);
    }
  } else {
    for (int64_t t = blockIdx.x * (int64_t)KNN_WARPS + warp; t < m; t += step) search(t);
  }
}

// k of 1 and 2 where one query per lane is the better one: 32 consecutive
// queries that are close together walk the same nodes, and in a small tree any
// queries do.  The warp searches for the first query's 8 nearest points; if
// the box of the 32 is not larger than 8 times the distance of the 8th (2, 4,
// 6 and 11 measured: the gain levels off at 8), every lane walks for its own
// query, bounded by its distances to those points.  Other queries are left to
// k_knn (`all`: they walk alone all the same).
//
// GB300, k of 1, one query per warp -> this: 3M queries in spatial order,
// 20k points 3.18 -> 0.44 ms, 200k points 4.25 -> 0.76; a grid of 2.25M
// queries in its own order, 20k points 3.31 -> 1.55.  1M queries in any order,
// 100 points 0.45 -> 0.11 ms, 1000 points 0.66 -> 0.18.  (Unbounded walks of
// lanes took 1.30, 2.78, 2.71, 0.17 and 0.50.)
template <int K>
__global__ void __launch_bounds__(32 * KNN_WARPS)
k_knn_lanes(IndexDev ix, const float* __restrict__ q, int stride, int64_t m, float far2, bool all,
            int32_t* __restrict__ idx_out, float* __restrict__ d2_out) {
  __shared__ WarpPool pools[KNN_WARPS];
  constexpr int NEAR = 8;
  const unsigned FULL = 0xffffffffu;
  const float INF = __int_as_float(0x7f800000);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t t0 = (blockIdx.x * (int64_t)KNN_WARPS + warp) * 32; t0 < m; t0 += (int64_t)gridDim.x * KNN_WARPS * 32) {
    const int64_t t = t0 + lane;
    const bool mine = t < m;
    const float* p = q + (mine ? t : t0) * stride;
    const float c[3] = {__ldg(p), __ldg(p + 1), __ldg(p + 2)};
    float diag2 = 0.0f;  // of the queries' box; not a number if one of them is not finite
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t o = ordered_bits(c[a]);
      const float e = __fsub_rn(from_ordered(__reduce_max_sync(FULL, o)), from_ordered(__reduce_min_sync(FULL, o)));
      diag2 = __fmaf_rn(e, e, diag2);
    }
    KList<K> N;
    klist_init<K>(N);
    bool near = diag2 <= far2;
    if (near) {
      WarpList<true> L;
      L.clear(INF);
      warp_knn(ix, __shfl_sync(FULL, c[0], 0), __shfl_sync(FULL, c[1], 0), __shfl_sync(FULL, c[2], 0), NEAR, L,
               pools[warp]);
      near = diag2 <= 64.0f * L.dist(NEAR - 1);
      // the K smallest of the lane's distances to the 8 points; placeholders
      // one ulp above the K-th, as in KSet::restart
      float b[2] = {INF, INF};
#pragma unroll
      for (int j = 0; j < NEAR; ++j) {
        const int32_t s = __shfl_sync(FULL, L.s, j);
        if (s < 0) continue;
        const float d = d2_point(__ldg(ix.rec + s), c[0], c[1], c[2]);
        b[1] = fminf(b[1], fmaxf(b[0], d));
        b[0] = fminf(b[0], d);
      }
#pragma unroll
      for (int j = 0; j < K; ++j) N.d[j] = b[K - 1] < INF ? __uint_as_float(__float_as_uint(b[K - 1]) + 1u) : INF;
    }
    if (near || all) {
      if (mine) {
        knn_search(ix, c[0], c[1], c[2], N);
#pragma unroll
        for (int j = 0; j < K; ++j) {
          idx_out[t * K + j] = N.s[j] >= 0 ? __ldg(ix.perm + N.s[j]) : -1;
          d2_out[t * K + j] = N.s[j] >= 0 ? N.d[j] : INF;
        }
      }
    } else if (mine) {
      idx_out[t * K] = KNN_LEFT;
    }
    __syncwarp();
  }
}

static int blocks_for(const Ctx& c, int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  int64_t cap = (int64_t)c.sm_count * 64;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// Radii of every point: search, then cloud-order outputs, the context's
// clamped radii, the records' radius lanes and the largest radius (on the
// device, for set_max_radius).
void launch_radii(Ctx& c, float max_radius, float* radii_out, int32_t* nn_out) {
  unsigned long long* err = c.scalars.ptr<unsigned long long>() + 8;
  if (c.launch.search == 1) {
    // sorted-order results in the radix sort's key buffers (N x 4 B each,
    // free once the index is built)
    float* r_sorted = reinterpret_cast<float*>(c.key(0));
    int32_t* nn_sorted = reinterpret_cast<int32_t*>(c.key(1));
    // scalars, cleared by the caller: [4] largest radius, [5] region counter,
    // [6] handed-over queries (positions in the sort's value buffer, free like
    // its key buffers)
    unsigned long long* next = c.scalars.ptr<unsigned long long>() + 5;
    const HardList hard{c.val(0), next + 1};
    auto go = [&](auto kern, int chunks) {
      int per_sm = 0;
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * RADII_WARPS, 0));
      const int64_t regions = (c.n + 32 * chunks - 1) / (32 * chunks);
      int64_t grid = (int64_t)c.sm_count * (per_sm > 0 ? per_sm : 1);
      const int64_t need = (regions + RADII_WARPS - 1) / RADII_WARPS;
      if (grid > need) grid = need;
      kern<<<(unsigned)grid, 32 * RADII_WARPS, 0, c.stream>>>(c.index(), r_sorted, nn_sorted, next, hard);
    };
    if (c.n < RADII_SMALL) go(k_radii_region<1>, 1);
    else go(k_radii_region<2>, 2);
    k_radii_hard<<<(unsigned)(c.sm_count * 8), 32 * RADII_WARPS, 0, c.stream>>>(c.index(), hard, r_sorted, nn_sorted);
    const int32_t* perm = c.perm.ptr<int32_t>();
    float4* rec = c.rec.ptr<float4>();
    int2* pairs = reinterpret_cast<int2*>(c.val(0));
    if (c.n < BUCKET_MIN) {
      k_to_cloud<<<blocks_for(c, c.n, 256), 256, 0, c.stream>>>(r_sorted, nn_sorted, perm, c.n, max_radius, rec, pairs);
    } else {
      int shift = 0;
      while ((c.n - 1) >> shift >= BUCKETS) ++shift;
      uint32_t* cursor = c.scan_sums.ptr<uint32_t>();
      CK(cudaMemsetAsync(cursor, 0, BUCKETS * 4, c.stream));
      c.bucket_i.reserve((size_t)c.n * 4);
      int32_t* to_i = c.bucket_i.ptr<int32_t>();
      CK(cudaFuncSetAttribute(k_to_buckets, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BucketSmem)));
      const unsigned tiles = (unsigned)((c.n + BUCKET_TILE - 1) / BUCKET_TILE);
      k_to_buckets<<<tiles, BUCKET_THREADS, sizeof(BucketSmem), c.stream>>>(r_sorted, nn_sorted, perm, c.n, shift,
                                                                          max_radius, rec, cursor, to_i, pairs);
      int2* apart = pairs;
      pairs = reinterpret_cast<int2*>(c.key(0));  // the sorted results have been read
      k_from_buckets<<<tiles, BUCKET_THREADS, 0, c.stream>>>(to_i, apart, c.n, pairs);
    }
    unsigned* largest = c.scalars.ptr<unsigned>() + 8;
    k_split<<<std::min(blocks_for(c, c.n, 256), c.sm_count * 8), 256, 0, c.stream>>>(pairs, c.n, max_radius, radii_out, nn_out,
                                                           c.radii_clamped.ptr<float>(), largest);
  } else {
    k_radii<<<blocks_for(c, c.n, 128), 128, 0, c.stream>>>(c.index(), max_radius, radii_out, nn_out,
                                                           c.radii_clamped.ptr<float>(), err);
    launch_set_radius(c);
    launch_max_radius(c);
  }
}

void launch_knn(Ctx& c, const float* q, int stride, int64_t m, int k, int32_t* idx, float* d2) {
  const auto grid = [&](int64_t warps) {
    return (unsigned)std::min((warps + KNN_WARPS - 1) / KNN_WARPS, (int64_t)c.sm_count * 64);
  };
  // One query per lane.  Small trees: a walk's cost grows with the leaves it
  // scans point by point, and one query per warp gets better above about
  // 5000 points at leaf 8, 2000 at 16, 1300 at 32.  Many queries for each
  // point: below about 4, 32 queries in spatial order span too many points,
  // and one query per warp is as fast as unbounded walks of lanes were.
  // Queries in any order pay 2 to 3% for the look at their boxes (1M on 20k
  // points 1.11 -> 1.14 ms).
  const bool small = m >= 65536 && c.n * c.cfg.leaf_size <= 40000;
  const bool dense = m >= 262144 && m >= 4 * c.n;
  if (k <= 2 && (small || dense)) {
    float far2 = 0.0f;  // an eighth of the cloud's diagonal, squared lengths: no 32 queries farther apart are near
    for (int a = 0; a < 3; ++a) far2 += (c.bounds[3 + a] - c.bounds[a]) * (c.bounds[3 + a] - c.bounds[a]);
    const auto lanes = [&](auto kern) {
      kern<<<grid((m + 31) / 32), 32 * KNN_WARPS, 0, c.stream>>>(c.index(), q, stride, m, far2 / 8.0f, small, idx, d2);
    };
    if (k == 1) lanes(k_knn_lanes<1>);
    else lanes(k_knn_lanes<2>);
    if (small) return;
    k_knn<true><<<grid(m), 32 * KNN_WARPS, 0, c.stream>>>(c.index(), q, stride, m, k, idx, d2);
    return;
  }
  k_knn<false><<<grid(m), 32 * KNN_WARPS, 0, c.stream>>>(c.index(), q, stride, m, k, idx, d2);
}

}  // namespace rm
