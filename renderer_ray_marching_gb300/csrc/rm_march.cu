// rm_march.cu -- the sphere-tracing marcher (replaces the reference's
// render kernel, src/ray_marching.cu:63-91, and its per-step FLANN query,
// :202-292).
//
// Work unit: one warp marches the rays of a screen tile (tile_w x tile_h
// pixels, 32 rays; with rays_per_lane > 1 an item is rays_per_lane such
// tiles stacked vertically and a lane whose ray ends takes the item's next
// pixel).  Each distance step is an exact 10-NN of every lane's step
// position, found by a warp packet traversal:
//
//   1. seed: every lane re-measures its previous step's 10 points at the new
//      position; the largest of those distances bounds the new 10th distance
//      (they are valid candidates), so its set restarts with that finite
//      bound (KSet::restart);
//   2. the warp walks the tree once, as a unit (packet_knn_bf): a node is
//      expanded when its box lies within the current 10th distance of ANY
//      active lane (one OR-reduction of 4-bit child votes), children are
//      visited nearest-first for a leading lane, and pending nodes wait in a
//      priority queue keyed by the leading lane's box distance;
//   3. a leaf's records are staged once for the whole warp (broadcast
//      loads) and every lane updates its own sorted set, so all lanes'
//      bounds tighten while the walk goes on.
// Neighbouring rays need nearly the same leaves (at surfaces, and in open
// space where the 10 nearest of every lane cluster around the same foot
// point), so the warp pays for the union of their searches once instead of
// serialising 32 divergent walks.  Search mode 0 keeps one independent walk
// per lane.  Then the step value min(sqrtf(d2) - r) and the reference's
// termination tests (MIN_DIST hit, far plane, MAX_STEPS).
//
// Plain form (rm_render): one warp per 8x4 tile, four warps per CTA.
// Batched form (rm_render_batch): a persistent kernel whose warps pull items
// of any view from one global counter; the whole launch is a CUDA graph.
// Both are templated on the CTAs per SM their register cap is sized for
// (4 to 8, regs_for_ctas); the kernel is latency-bound, so resident warps matter and
// the per-item view and the statistics live in shared memory (WarpSmem).
//
// Culling.  The reference's view-frustum test is a no-op (is_inside,
// src/ray_marching.cu:231-258, returns true); its effective culling is the
// near-plane start and the far-plane stop.  Here each ray additionally gets
// an exact exit bound: let E be the box of all sphere centres grown by
// (max radius + MIN_DIST + slack).  Every step position beyond the ray's
// exit from E is farther than max radius + MIN_DIST from every centre, so
// every later distance value exceeds MIN_DIST (and is positive, so t keeps
// growing): the reference would march on to the far plane or the step cap
// and report a miss.  Stopping at the exit therefore never changes an
// output, it only skips work.  The slack (2e-3 m plus 1e-6 of the scene
// scale) covers float rounding of positions and distances.
#include "rm_internal.h"

#include <cmath>
#include <cstring>
#include <type_traits>

namespace rm {

struct ClipBox {
  float lo[3], hi[3];
};

// Exit parameter of the ray from box E (-inf if the ray never meets E).
__device__ __forceinline__ float clip_exit(const Ray& r, const ClipBox& e) {
  float o[3] = {r.ox, r.oy, r.oz}, d[3] = {r.dx, r.dy, r.dz};
  float tmin = -INFINITY, tmax = INFINITY;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (d[a] != 0.0f) {
      float inv = 1.0f / d[a];
      float t1 = (e.lo[a] - o[a]) * inv, t2 = (e.hi[a] - o[a]) * inv;
      tmin = fmaxf(tmin, fminf(t1, t2));
      tmax = fminf(tmax, fmaxf(t1, t2));
    } else if (o[a] < e.lo[a] || o[a] > e.hi[a]) {
      tmax = -INFINITY;
    }
  }
  if (!(tmin <= tmax)) return -INFINITY;
  // outward slack for the rounding of the slab divisions
  return tmax + fabsf(tmax) * 1e-5f + 1e-3f;
}

constexpr int WARPS_PER_CTA = 4;

// Register cap of a marcher instance sized for `ctas` resident CTAs per SM:
// the SM's 65,536 registers shared by ctas x 128 threads, rounded down to the
// allocation granule of 8 (4 -> 128, 5 -> 96, 6 -> 80, 7 -> 72, 8 -> 64).
// The kernels take it as __maxnreg__ rather than as the minimum-blocks
// argument of __launch_bounds__: both give ptxas the same register count,
// but it then spills different values, and on the 20M-point batched
// workload (32 views, leaf 16) the capped form measured 54.7 Mrays/s at 64
// and at 72 registers against 48.2 for __launch_bounds__(128, 8).  The
// marcher is latency-bound, so the extra resident warps are worth the
// spills (72 registers: 200 B of spill stores per thread).
constexpr int regs_for_ctas(int ctas) { return (65536 / (ctas * 32 * WARPS_PER_CTA)) / 8 * 8; }

struct MarchParams {
  ClipBox clip;
  int few;          // rays left at which a late item hands them to the tail kernel
  unsigned budget;  // expansions and leaves after which any item does
  int search;  // 1: warp packet traversal, 0: one walk per lane
};

// View as seen by the marcher (kept per warp in shared memory).
struct ViewArgs {
  float m[16];
  int32_t width, height;
  float pane;
  float4* rgbd;
  int32_t* hit;
  float* depth;
  int32_t* steps;
};

// counters: [0] steps, [1] rays, [2] hits, [3] search errors,
//           [4] packet lane-steps, [5] per-lane lane-steps, [6] leaves scanned by packets,
//           [7] nodes expanded by packets, [8] warp steps, [9] warp steps split in two packets
//           (no longer split: always 0), [10] queue entries moved to the overflow stack,
//           [11] packet walks that fell back to depth-first order
enum { C_STEPS, C_RAYS, C_HITS, C_BAD, C_COOP, C_SOLO, C_LEAVES, C_NODES, C_WSTEPS, C_SPLIT, C_SPILL, C_DFS,
       C_N,
       C_TAIL = 15 };  // rays handed to the tail kernel; [14] how many of them it has taken

// Per-warp shared state.  The view of the current item, the statistics and
// each lane's ray live here rather than in registers: they are read or bumped
// at a ray's start and end, or once per step (the ray's origin, direction and
// t before the walk, t and the step count after it), and every register the
// walk does not have to hold lets more warps stay resident (the marcher is
// bound by instruction latency, so resident warps are what hides it; parking
// the ray here cut the 64-register instance's spills from 314 to 204 B and
// gained 1%).
struct RayLanes {
  float ox[32], oy[32], oz[32], dx[32], dy[32], dz[32];
  float t[32], t_stop[32], t_far[32];
  int32_t nsteps[32], pix[32];
};
struct WarpSmem {
  PacketQueue ps;
  ViewArgs v;                   // warp-uniform; written by lane 0 per item
  unsigned long long cnt[C_N];  // this warp's statistics
  RayLanes ray;
};

__device__ __forceinline__ void write_result(const IndexDev& ix, const ViewArgs& v, int64_t pix, int32_t s,
                                             float depth, int32_t steps, unsigned long long* cnt) {
  atomicAdd(cnt + C_STEPS, (unsigned long long)steps);
  atomicAdd(cnt + C_RAYS, 1ull);
  if (s >= 0) atomicAdd(cnt + C_HITS, 1ull);
  if (s >= 0) {
    // colour with the depth in .w (src/ray_marching.cu:85-89); uint8 / 255.0f
    // as the PLY loader does (src/pointcloud.cpp:55)
    const uint32_t u = __ldg(ix.col + s);
    const float4 c = make_float4(__fdiv_rn((float)(u & 255u), 255.0f), __fdiv_rn((float)((u >> 8) & 255u), 255.0f),
                                 __fdiv_rn((float)((u >> 16) & 255u), 255.0f), depth);
    if (v.rgbd) v.rgbd[pix] = c;
    if (v.hit) v.hit[pix] = __ldg(ix.perm + s);
    if (v.depth) v.depth[pix] = depth;
  } else {
    if (v.rgbd) v.rgbd[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // BACKGROUND_COLOR
    if (v.hit) v.hit[pix] = -1;
    if (v.depth) v.depth[pix] = 0.0f;
  }
  if (v.steps) v.steps[pix] = steps;
}

// A ray that leaves its packet: where it is, and the 10 nearest points of its
// last step (-1: none yet), which bound the next one's search.
struct alignas(64) TailRay {
  int32_t view, pix;
  float t;
  int32_t nsteps;
  int32_t seed[KNN];
  int32_t unused[2];
};
static_assert(sizeof(TailRay) == 64, "one record per half line");

// Rays handed to the tail kernel.  `cap` records; `count` may run past it
// (rays without a record stay with their warp).
struct TailList {
  TailRay* rays;
  unsigned long long* count;
  int64_t cap;
};

// Marches one ray to its end with the whole warp searching for it.  All
// lanes pass the same ray; lane j < KNN holds its seed j.  Same steps as a
// packet's: the same search, the same order of the tests.  3 to 4 ns per step
// with all warps busy, against 0.6 to 0.7 of a packet with 18 to 23 lanes;
// but its step takes 4 us where a packet's takes 40.
__device__ __forceinline__ void march_one(const IndexDev& ix, const ClipBox& clip, WarpSmem& sm, int32_t pix, float t,
                                          int32_t nsteps, int32_t seed) {
  const unsigned FULL = 0xffffffffu;
  const float INF = __int_as_float(0x7f800000);
  const int lane = threadIdx.x & 31;
  const ViewArgs& v = sm.v;
  const Ray r = make_ray(v.m, v.width, v.height, v.pane, pix % v.width, pix / v.width);
  const float t_stop = clip_exit(r, clip);
  const int32_t first = nsteps;
  int32_t hit = -1;
  bool fin = false;
  while (!fin && !(t > t_stop)) {  // past the exit bound: a miss
    const float px = __fmaf_rn(r.dx, t, r.ox), py = __fmaf_rn(r.dy, t, r.oy), pz = __fmaf_rn(r.dz, t, r.oz);
    // bound as in KSet::restart: one ulp above the seeds' largest distance
    float d = 0.0f;
    if (lane < KNN && seed >= 0) d = d2_point(__ldg(ix.rec + seed), px, py, pz);
    const bool full = __ballot_sync(FULL, lane < KNN && seed >= 0) == (1u << KNN) - 1u;
    const float w = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(d)));
    WarpList<true> L;
    L.clear(full && w < INF ? __uint_as_float(__float_as_uint(w) + 1u) : INF);
    warp_knn(ix, px, py, pz, KNN, L, sm.ps.pool);
    // the smallest sqrtf(d2) - r; the list is in (d2, cloud index) order, so
    // the first lane that holds it is the reference's choice
    seed = lane < KNN ? L.s : -1;
    float val = INF;
    if (seed >= 0) val = __fsub_rn(__fsqrt_rn(__uint_as_float((unsigned)(L.key >> 32))), __ldg(&ix.rec[seed].w));
    float best = val == val ? val : INF;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = fminf(best, __shfl_xor_sync(FULL, best, off));
    const unsigned at = __ballot_sync(FULL, seed >= 0 && val == best);
    const int32_t s = at ? __shfl_sync(FULL, seed, __ffs(at) - 1) : -1;
    ++nsteps;
    t = __fadd_rn(t, best);
    if (best < MIN_DIST) {  // src/ray_marching.cu:219-222
      fin = true;
      hit = s;
    } else {
      fin = t > r.t_far || nsteps >= MAX_STEPS;
    }
  }
  if (lane == 0) {
    write_result(ix, v, pix, hit, hit >= 0 ? t : 0.0f, nsteps, sm.cnt);
    sm.cnt[C_SOLO] += (unsigned long long)(nsteps - first);
  }
  __syncwarp();
}

// Marches every ray of one item (origin x0, y0; tile_w x tile_h*rpl pixels)
// of view v.  All 32 lanes call it.  SEARCH: 1 packet traversal, 0 per lane.
//
// Rays that leave the item.  A walk costs about the same for 5 lanes as for
// 30 (it is the union of their searches, and its steps follow one another),
// and the rays that graze an edge go on for tens of steps: with 6 or fewer
// lanes left are 37% of the warp steps but 5% of the ray steps at 2M points.
// Single items (rays far from everything, or spread over several surfaces)
// took 11.5 of the 11.6 ms of a 1067x690 view whose median warp was done after
// 6.6, and 32 of the 53 ms of 65 small views.  So where there is a `tail` list, an item that has used
// up its budget of expansions and leaves, and a late item with a few rays
// left, hands its rays over; k_march_tail spreads them over all warps.
template <int SEARCH>
__device__ void march_item(const IndexDev& ix, int x0, int y0, int tile_w, int tile_h, int rpl,
                           const MarchParams& mp, WarpSmem& sm, int view, const TailList* tail, bool late) {
  const ViewArgs& v = sm.v;
  RayLanes& R = sm.ray;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int item_rays = tile_w * tile_h * rpl;
  int next = 0;
  unsigned work = 0;
  bool has = false;
  KSet L;
  L.clear();
  while (true) {
    // hand unclaimed pixels of the item to lanes without a ray
    unsigned need = __ballot_sync(FULL, !has);
    while (need && next < item_rays) {
      int idx = next + __popc(need & lt);
      if (!has && idx < item_rays) {
        int x = x0 + idx % tile_w;
        int y = y0 + idx / tile_w;
        if (x < v.width && y < v.height) {
          has = true;
          const Ray r = make_ray(v.m, v.width, v.height, v.pane, x, y);
          R.pix[lane] = y * v.width + x;
          R.ox[lane] = r.ox; R.oy[lane] = r.oy; R.oz[lane] = r.oz;
          R.dx[lane] = r.dx; R.dy[lane] = r.dy; R.dz[lane] = r.dz;
          R.t_stop[lane] = clip_exit(r, mp.clip);
          R.t_far[lane] = r.t_far;
          R.t[lane] = r.t_near;
          R.nsteps[lane] = 0;
          L.clear();
        }
      }
      next += __popc(need);
      need = __ballot_sync(FULL, !has);
    }
    const unsigned alive = __ballot_sync(FULL, has);
    if (alive == 0) break;
    if (SEARCH == 1 && tail && next >= item_rays && ((late && __popc(alive) <= mp.few) || work > mp.budget)) {
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(tail->count, (unsigned long long)__popc(alive));
      at = __shfl_sync(FULL, at, 0) + __popc(alive & lt);
      if (has && (int64_t)at < tail->cap) {
        TailRay& o = tail->rays[at];
        o.view = view;
        o.pix = R.pix[lane];
        o.t = R.t[lane];
        o.nsteps = R.nsteps[lane];
#pragma unroll
        for (int j = 0; j < KNN; ++j) o.seed[j] = L.s[j];
        has = false;
      }
      if (__ballot_sync(FULL, has) == 0) break;
      tail = nullptr;  // the list is full: the rest stays
    }

    float t = R.t[lane];
    bool stepping = has && !(t > R.t_stop[lane]);  // past the exit bound: a miss (culled)
    if (has && !stepping) {
      write_result(ix, v, R.pix[lane], -1, 0.0f, R.nsteps[lane], sm.cnt);
      has = false;
    }
    float px = __fmaf_rn(R.dx[lane], t, R.ox[lane]);
    float py = __fmaf_rn(R.dy[lane], t, R.oy[lane]);
    float pz = __fmaf_rn(R.dz[lane], t, R.oz[lane]);
    if (stepping) L.restart(ix, px, py, pz);
    if (SEARCH == 1) {
      // One packet: every stepping lane walks with the warp.  (A split into
      // a tight and a loose packet helped the depth-first walk; with the
      // best-first order loose lanes no longer steer the walk and the split
      // measured 2% slower.)
      unsigned lv = 0, nd = 0;
      if (!packet_knn_bf(ix, stepping, px, py, pz, L, sm.ps, lv, nd) && stepping) atomicAdd(sm.cnt + C_BAD, 1ull);
      const unsigned any_step = __ballot_sync(FULL, stepping);  // every lane votes
      work += nd + lv;
      if (lane == 0) {
        sm.cnt[C_LEAVES] += lv;
        sm.cnt[C_NODES] += nd;
        sm.cnt[C_WSTEPS] += any_step ? 1 : 0;
      }
    } else if (stepping) {
      if (!knn_search(ix, px, py, pz, L)) atomicAdd(sm.cnt + C_BAD, 1ull);
    }
    if (stepping) {
      int32_t s;
      L.order(ix.perm);
      float step = L.step_value(ix, &s);
      const int nsteps = R.nsteps[lane] + 1;
      R.nsteps[lane] = nsteps;
      t = __fadd_rn(R.t[lane], step);
      R.t[lane] = t;
      bool fin = false;
      int32_t hs = -1;
      float hd = 0.0f;
      if (step < MIN_DIST) {  // src/ray_marching.cu:219-222
        fin = true;
        hs = s;
        hd = t;
      } else if (t > R.t_far[lane] || nsteps >= MAX_STEPS) {
        fin = true;
      }
      if (fin) {
        write_result(ix, v, R.pix[lane], hs, hd, nsteps, sm.cnt);
        has = false;
      }
    }
  }
}

__device__ __forceinline__ void clear_counters(WarpSmem& sm) {
  const int lane = threadIdx.x & 31;
  if (lane < C_N) sm.cnt[lane] = 0ull;
  if (lane == 0) {
    sm.ps.n_spill = 0;
    sm.ps.n_dfs = 0;
  }
  __syncwarp();
}

// Adds the warp's statistics to the launch's counters.  Lane-steps are the
// rays' step counts, counted at a ray's end; those of march_one and of the
// per-lane mode are reported as steps of single rays, the others as packet
// steps.
template <int SEARCH>
__device__ __forceinline__ void flush_counters(WarpSmem& sm, unsigned long long* counters) {
  __syncwarp();
  const int lane = threadIdx.x & 31;
  if (lane < C_N) {
    unsigned long long v = lane == C_COOP ? (SEARCH == 1 ? sm.cnt[C_STEPS] - sm.cnt[C_SOLO] : 0ull)
                         : lane == C_SOLO ? (SEARCH == 1 ? sm.cnt[C_SOLO] : sm.cnt[C_STEPS])
                         : lane == C_SPILL ? (unsigned long long)sm.ps.n_spill
                         : lane == C_DFS ? (unsigned long long)sm.ps.n_dfs
                         : sm.cnt[lane];
    if (v) atomicAdd(counters + lane, v);
  }
}


struct PlainArgs {
  float m[16];
  int32_t width, height;
  float fov;
  float4* rgbd;
  int32_t* hit;
  float* depth;
  int32_t* steps;
};

__device__ __forceinline__ void load_view(ViewArgs& v, const PlainArgs& a) {
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v.m[k] = a.m[k];
    v.width = a.width;
    v.height = a.height;
    v.pane = view_pane(a.width, a.fov);
    v.rgbd = a.rgbd;
    v.hit = a.hit;
    v.depth = a.depth;
    v.steps = a.steps;
  }
  __syncwarp();
}
__device__ __forceinline__ void load_view(ViewArgs& v, const ViewDev& V) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the previous item's readers of v are done
  if (lane < 16) v.m[lane] = V.m[lane];
  if (lane == 0) {
    v.width = V.width;
    v.height = V.height;
    v.pane = V.pane;
    v.rgbd = V.rgbd;
    v.hit = V.hit;
    v.depth = V.depth;
    v.steps = V.steps;
  }
  __syncwarp();
}

// One warp per 8x4 tile.
template <int SEARCH>
__device__ __forceinline__ void plain_body(const IndexDev& ix, const PlainArgs& a, const MarchParams& mp,
                                           unsigned long long* __restrict__ counters, const TailList& tail) {
  __shared__ WarpSmem smem[WARPS_PER_CTA];
  const int warp = threadIdx.x >> 5;
  int tiles_x = (a.width + 7) / 8;
  int tile = blockIdx.x * WARPS_PER_CTA + warp;
  int tiles = tiles_x * ((a.height + 3) / 4);
  WarpSmem& sm = smem[warp];
  clear_counters(sm);
  if (tile < tiles) {
    load_view(sm.v, a);
    march_item<SEARCH>(ix, (tile % tiles_x) * 8, (tile / tiles_x) * 4, 8, 4, 1, mp, sm, 0, tail.cap > 0 ? &tail : nullptr, true);
  }
  flush_counters<SEARCH>(sm, counters);
}

// Packet-walk instances, MINB: the CTAs per SM their register cap is sized
// for (the launch's ctas_per_sm picks the instance).  The per-lane walk keeps
// the minimum-blocks form, under which it measured faster (20.0 against
// 17.2 Mrays/s with __maxnreg__ at the same 90 registers).
template <int MINB>
__global__ void __launch_bounds__(32 * WARPS_PER_CTA) __maxnreg__(regs_for_ctas(MINB))
k_march_plain(IndexDev ix, PlainArgs a, MarchParams mp, unsigned long long* __restrict__ counters, TailList tail) {
  plain_body<1>(ix, a, mp, counters, tail);
}
__global__ void __launch_bounds__(32 * WARPS_PER_CTA, 4)
k_march_plain_lane(IndexDev ix, PlainArgs a, MarchParams mp, unsigned long long* __restrict__ counters, TailList tail) {
  plain_body<0>(ix, a, mp, counters, tail);
}

// ---------------------------------------------------------------- batched
__global__ void k_prepare_views(ViewDev* __restrict__ views, int n) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) views[v].pane = view_pane(views[v].width, views[v].fov);
}

__global__ void k_view_pane(const rm_view* __restrict__ views, int n, float* __restrict__ out) {
  int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) out[v] = view_pane(views[v].width, views[v].fov);
}

struct BatchArgs {
  const ViewDev* views;
  int nviews;
  int64_t total_items;
  int64_t late_items;       // items at the queue's end that count as late
  int tile_w, tile_h, rpl;  // item = tile_w x (tile_h * rpl) pixels
};

__device__ __forceinline__ int find_view(const ViewDev* views, int n, int64_t item) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (views[mid].tile_base <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <int SEARCH>
__device__ __forceinline__ void batch_body(const IndexDev& ix, const BatchArgs& a, const MarchParams& mp,
                                           unsigned long long* __restrict__ queue,
                                           unsigned long long* __restrict__ counters, const TailList& tail) {
  __shared__ WarpSmem smem[WARPS_PER_CTA];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpSmem& sm = smem[warp];
  clear_counters(sm);
  while (true) {
    unsigned long long it = 0;
    if (lane == 0) it = atomicAdd(queue, 1ull);
    it = __shfl_sync(0xffffffffu, it, 0);
    if ((int64_t)it >= a.total_items) break;
    int iv = find_view(a.views, a.nviews, (int64_t)it);
    const ViewDev& V = a.views[iv];
    int64_t local = (int64_t)it - V.tile_base;
    load_view(sm.v, V);
    int x0 = (int)(local % V.tiles_x) * a.tile_w;
    int y0 = (int)(local / V.tiles_x) * (a.tile_h * a.rpl);
    const bool late = (int64_t)it + a.late_items >= a.total_items;
    march_item<SEARCH>(ix, x0, y0, a.tile_w, a.tile_h, a.rpl, mp, sm, iv, tail.cap > 0 ? &tail : nullptr, late);
  }
  flush_counters<SEARCH>(sm, counters);
}

template <int MINB>
__global__ void __launch_bounds__(32 * WARPS_PER_CTA) __maxnreg__(regs_for_ctas(MINB))
k_march_batch(IndexDev ix, BatchArgs a, MarchParams mp, unsigned long long* __restrict__ queue,
              unsigned long long* __restrict__ counters, TailList tail) {
  batch_body<1>(ix, a, mp, queue, counters, tail);
}
__global__ void __launch_bounds__(32 * WARPS_PER_CTA, 4)
k_march_batch_lane(IndexDev ix, BatchArgs a, MarchParams mp, unsigned long long* __restrict__ queue,
                   unsigned long long* __restrict__ counters, TailList tail) {
  batch_body<0>(ix, a, mp, queue, counters, tail);
}

// The rays that left their items, one per warp, taken in the list's order.
// VIEWS: the view table, or the plain form's one view.
template <class VIEWS>
__global__ void __launch_bounds__(32 * WARPS_PER_CTA, 8)
k_march_tail(IndexDev ix, VIEWS views, ClipBox clip, unsigned long long* __restrict__ counters, TailList tail) {
  __shared__ WarpSmem smem[WARPS_PER_CTA];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpSmem& sm = smem[warp];
  const unsigned long long count = min(*tail.count, (unsigned long long)tail.cap);
  if ((unsigned long long)blockIdx.x * WARPS_PER_CTA + warp >= count) return;  // no more warps than rays
  clear_counters(sm);
  if constexpr (std::is_same<VIEWS, PlainArgs>::value) load_view(sm.v, views);
  while (true) {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(tail.count - 1, 1ull);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= count) break;
    const TailRay& o = tail.rays[t];
    if constexpr (!std::is_same<VIEWS, PlainArgs>::value) load_view(sm.v, views[o.view]);
    march_one(ix, clip, sm, o.pix, o.t, o.nsteps, lane < KNN ? o.seed[lane] : -1);
  }
  flush_counters<1>(sm, counters);
}

// ---------------------------------------------------------------- host side
// Box E of the culling argument above; max_r = +inf disables culling.
static ClipBox clip_box(const Ctx& c, float max_r) {
  ClipBox e;
  if (!(max_r < INFINITY)) {
    for (int a = 0; a < 3; ++a) {
      e.lo[a] = -INFINITY;
      e.hi[a] = INFINITY;
    }
    return e;
  }
  float scale = 0.0f;
  for (int a = 0; a < 6; ++a) scale = fmaxf(scale, fabsf(c.bounds[a]));
  float m = max_r + MIN_DIST + 2e-3f + 1e-6f * (scale + ZFAR * 16.0f);
  for (int a = 0; a < 3; ++a) {
    e.lo[a] = c.bounds[a] - m;
    e.hi[a] = c.bounds[3 + a] + m;
  }
  return e;
}

static TailList tail_list(const Ctx& c, unsigned long long* counters) {
  return TailList{c.tail.ptr<TailRay>(), counters + C_TAIL, (int64_t)(c.tail.cap / sizeof(TailRay))};
}

// Which rays leave their packets.  `few`: a late item's last rays (of 2, 4, 6,
// 8, 12 the fastest for one 1067x690 view at 2M points; 6.9 -> 6.6 ms by
// itself).  The budget counts node expansions and leaves of an item (about
// 1000 at 2M points, 1400 at 20M); a ray costs the tail kernel about four
// times its share of a full packet, so the budget is the larger the more
// items a warp has to work off anyway, and with them the time in which a
// slow one is hidden, and larger for a deeper tree, whose every walk opens
// more nodes: the factor 20 + 90 * depth is 650 at 100k points and 1010 at
// 20M.  Measured optima: 200 at 0.12 items per resident warp (160x120
// pixels), 600 at 0.5, 900 at 2, 1000 at 5 (1067x690), 1400 at 17 (65 small
// views), 4000 to 6000 at 160 (24 views at 20M points); with a factor of 1010
// instead of 650 for every tree, one view at 20M points took 3.60 instead of
// 4.17 ms, but 20 small views at 100k 5.51 instead of 5.28.  It is the rule for
// items of one ray per lane and 8 CTAs per SM: longer items (rays_per_lane)
// hand over more of their rays, 14% of the steps at 4 against 2 to 3%.  Times
// without -> with the tail kernel when it was added: 160x120 at 100k points
// 1.73 -> 0.65 ms, 320x240 at 2M 3.2 -> 1.4, 1067x690 at 2M 6.9 -> 5.6, 65
// small views at 1M 47.7 -> 33.9, 24 views at 20M 334 -> 316.
constexpr int FEW = 6;
static unsigned tail_budget(const Ctx& c, int64_t items) {
  const double per_warp = (double)items / ((double)c.sm_count * 8 * WARPS_PER_CTA);
  return (unsigned)fmax(200.0, (20.0 + 90.0 * c.depth) * pow(per_warp, 0.38));  // depth 7 at 100k points, 11 at 20M
}

// 524,288 rays: 6 of every tile of a 1920x1080 view, and more.  When they are
// used up, rays stay with their items.  Reserved with the radii, since a
// render call may be under stream capture; where there is no memory for it,
// renders go without.
void reserve_tail(Ctx& c) {
  try {
    c.tail.reserve((size_t)1 << 25);
  } catch (const OomError&) {
  }
}

static MarchParams march_params(const Ctx& c, int64_t items) {
  MarchParams mp;
  mp.clip = clip_box(c, c.max_r);
  mp.search = c.launch.search;
  mp.few = FEW;
  mp.budget = tail_budget(c, items);
  return mp;
}

void launch_view_pane(Ctx& c, const rm_view* views_dev, int n, float* pane_out) {
  k_view_pane<<<(n + 127) / 128, 128, 0, c.stream>>>(views_dev, n, pane_out);
}

void launch_render_plain(Ctx& c, const rm_view& v, float4* rgbd, int32_t* hit, float* depth,
                         int32_t* steps, unsigned long long* counters) {
  PlainArgs a;
  memcpy(a.m, v.cam2world, sizeof(a.m));
  a.width = v.width;
  a.height = v.height;
  a.fov = v.fov;
  a.rgbd = rgbd;
  a.hit = hit;
  a.depth = depth;
  a.steps = steps;
  int64_t tiles = (int64_t)((v.width + 7) / 8) * ((v.height + 3) / 4);
  unsigned grid = (unsigned)((tiles + WARPS_PER_CTA - 1) / WARPS_PER_CTA);
  MarchParams mp = march_params(c, tiles);
  const TailList tail = tail_list(c, counters);
  auto go = [&](auto kern) { kern<<<grid, 32 * WARPS_PER_CTA, 0, c.stream>>>(c.index(), a, mp, counters, tail); };
  const int cps = c.launch.ctas_per_sm;
  if (mp.search == 1) {
    if (cps >= 8) go(k_march_plain<8>);
    else if (cps >= 7) go(k_march_plain<7>);
    else if (cps >= 6) go(k_march_plain<6>);
    else if (cps >= 5) go(k_march_plain<5>);
    else go(k_march_plain<4>);
    if (tail.cap > 0)
      k_march_tail<<<(unsigned)(c.sm_count * 8), 32 * WARPS_PER_CTA, 0, c.stream>>>(c.index(), a, mp.clip, counters, tail);
  } else {
    go(k_march_plain_lane);
  }
}

void launch_prepare_views(Ctx& c, ViewDev* views_dev, int n) {
  k_prepare_views<<<(n + 127) / 128, 128, 0, c.stream>>>(views_dev, n);
}

// `queue` is the work-queue counter the launch's warps pull items from (zero
// before the launch): the context's own for rm_render_batch, the static
// scratch's for the allocation-free entry point, which has no list of tail
// rays either (with_tail false: every warp ends its own rays).
void launch_render_batch(Ctx& c, ViewDev* views_dev, int n, int64_t total_items, const rm_launch& L,
                         unsigned long long* queue, unsigned long long* counters, bool with_tail) {
  BatchArgs a;
  a.views = views_dev;
  a.nviews = n;
  a.total_items = total_items;
  a.tile_w = L.tile_w;
  a.tile_h = L.tile_h;
  a.rpl = L.rays_per_lane;
  int grid = c.sm_count * (L.ctas_per_sm > 0 ? L.ctas_per_sm : 4);
  a.late_items = (int64_t)grid * WARPS_PER_CTA * 2;
  MarchParams mp = march_params(c, total_items);
  TailList tail = tail_list(c, counters);
  if (!with_tail) tail.cap = 0;
  auto go = [&](auto kern) {
    kern<<<grid, 32 * WARPS_PER_CTA, 0, c.stream>>>(c.index(), a, mp, queue, counters, tail);
  };
  const int cps = L.ctas_per_sm;
  if (mp.search == 1) {
    if (cps >= 8) go(k_march_batch<8>);
    else if (cps >= 7) go(k_march_batch<7>);
    else if (cps >= 6) go(k_march_batch<6>);
    else if (cps >= 5) go(k_march_batch<5>);
    else go(k_march_batch<4>);
    if (tail.cap > 0)
      k_march_tail<<<(unsigned)(c.sm_count * 8), 32 * WARPS_PER_CTA, 0, c.stream>>>(c.index(), (const ViewDev*)views_dev,
                                                                                    mp.clip, counters, tail);
  } else {
    go(k_march_batch_lane);
  }
}

}  // namespace rm
