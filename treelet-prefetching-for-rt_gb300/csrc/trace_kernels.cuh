// Traversal kernels.
//
//   trace_plain_kernel    traceRay order (vulkan_ray_tracing.cc:2309-3076)
//   trace_treelet_kernel  traceRayWithTreelets order (vulkan_ray_tracing.cc:1522-2307);
//                         with STAGED = true, node reads that fall in a treelet
//                         in shared memory are served from there: one pinned for
//                         the launch, or one that the warp's lanes voted for (the
//                         treelet-prefetch decision of shader.cc:3419-3441 with
//                         heuristic ALWAYS) and copied into one of its slots.  Both
//                         are copied with cp.async.bulk.  Staging changes
//                         where a node's bytes come from, never which nodes a
//                         ray visits or in which order.
//
// One thread walks one ray, with its stack(s) in local memory.  Each thread
// keeps the reference's visit order exactly; FP32 arithmetic keeps the
// reference's operation order and is compiled without FMA contraction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/treelet_rt.h"
#include "device_nodes.cuh"
#include "format.h"
#include "rtmath.h"

namespace rtk {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kTop = 2u, kLeaf = 1u;  // stack entry = unit << 2 | top | leaf

// Device counters, all uint64.
enum Stat { ST_NODE_BYTES = 0, ST_STAGED_BYTES, ST_SMEM_READS, ST_GMEM_READS, ST_STAGINGS, ST_COUNT };
// Status word bits set by kernels (device-wide, not per ray).
constexpr uint32_t kStatusTimeout = 1u;

// What a walk needs of one scene.
struct SceneView {
  const uint4* blob;      // headers, leaves and instance leaves
  const uint4* walk;      // walk nodes (walk_node.h); the same array unless a unit has both uses
  const uint4* raw;       // the blob as uploaded
  const uint2* meta;      // per unit: x = treelet root unit, y = dense << 10 | slot
  const uint16_t* route;  // per unit: routing bits of the treelet-ordered walk (treelets.h)
  uint32_t n_units;
};

// The walks' copy of the blob: units marked in `internal` as walk nodes
// (walk_node.h), the others as they are; without marks every unit is taken as
// an internal node.
__global__ void __launch_bounds__(256) walk_nodes_kernel(const uint4* __restrict__ blob,
                                                         const uint32_t* __restrict__ internal,
                                                         const uint16_t* __restrict__ route, uint32_t n_units,
                                                         uint4* __restrict__ walk) {
  const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n_units) return;
  uint32_t raw[16], node[16];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 x = __ldcs(blob + (uint64_t)u * 4 + q);
    raw[4 * q] = x.x, raw[4 * q + 1] = x.y, raw[4 * q + 2] = x.z, raw[4 * q + 3] = x.w;
  }
  rtw::walk_node(raw, u, n_units, route ? route[u] : 0u, node);
  const bool keep = internal && !((internal[u >> 5] >> (u & 31u)) & 1u);
#pragma unroll
  for (int q = 0; q < 16; ++q) node[q] = keep ? raw[q] : node[q];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    walk[(uint64_t)u * 4 + q] = make_uint4(node[4 * q], node[4 * q + 1], node[4 * q + 2], node[4 * q + 3]);
}

struct TraceArgs {
  const uint4* blob;
  const uint4* walk;
  const uint4* raw;
  uint32_t n_units;
  // several scenes in one launch: rays [item_begin[k], item_begin[k+1]) use
  // scenes[item_scene[k]]; n_items == 0 means every ray uses blob / meta
  const SceneView* scenes;
  const uint32_t* item_begin;
  const uint32_t* item_scene;
  uint32_t n_items;
  const rt_ray* rays;
  const uint32_t* flags;
  uint32_t default_flags;
  uint32_t n;
  rt_hit* hits;
  uint32_t* rows;              // traced: n rows of `cap` entries, visits or (rows_tl) treelet ids, or null
  uint32_t rows_tl;
  uint32_t cap;
  uint32_t* ids;               // rows of treelet ids beside the visits', or null (trace_group_kernel writes them)
  const uint2* meta;           // per unit: x = treelet root unit, y = dense << 10 | slot
  const uint16_t* route;       // per unit: routing bits of the treelet-ordered walk
  const uint4* pin_image;      // staged: pinned-treelet records (pinned.h), copied to shared memory per CTA
  uint32_t pin_bytes;          // its size (multiple of 128), 0 = nothing pinned
  uint32_t pin_root;           // record of the TLAS root node, 0 = not pinned
  const uint4* images;         // staged image store
  const unsigned long long* image_off;  // per dense treelet, n_treelets + 1
  uint32_t n_treelets;
  unsigned long long* stats;   // ST_COUNT counters
  uint32_t* status;            // kStatus* bits
  uint32_t slots;              // staged treelet slots per CTA
  uint32_t slot_bytes;         // bytes per slot (multiple of 128)
  uint32_t epoch;              // node visits per ray between votes
  uint32_t* queue;             // next ray to hand out (persistent kernels; zeroed per launch)
  uint32_t refill;             // idle lanes of a warp that trigger a refill
  uint32_t min_votes;          // lanes that must want a treelet before a warp stages it
  const uint32_t* hint;        // staged: predicted next treelet per (treelet, direction octant), or null
  uint32_t wait_tries;         // staged: probes of the wait for the pinned image before staging stops
  uint32_t tbuf_off;           // byte offset of the trace staging area in dynamic shared
                               // memory (128-aligned base), kNone: trace entries go straight to the rows
  uint32_t ss_off;             // plain walk with SHORT: byte offset of the short stacks, likewise
};

// Access traces.  A walk writes one row per ray: the visits, or the treelet
// ids when only they are asked for.  With both asked for the treelet ids are
// filled in from the visits afterwards (trace_treelet_ids_kernel): looked up
// in the walk each cost a dependent load, a second scattered store and L1
// room.
//
// Staging.  A lane writing its ray's row one 4-byte entry at a time leaves
// partly written 32-byte sectors that L2 fills from DRAM and writes back again
// and again (4.5x the entries' bytes written, as many read, on bounce rays).
// Instead each lane keeps its ray's next 8 entries in its warp's 1 KiB staging
// area ([entry 0..7][lane] words: lanes hit distinct banks) and writes
// them as one whole, aligned sector.  Used when the row capacity is a multiple
// of 8 and the rows start on 32-byte boundaries; the last partial sector is
// written when the ray ends.
constexpr uint32_t kTraceBufWarpBytes = 1024;

extern __shared__ __align__(128) uint8_t rt_dyn_smem[];

// The calling lane's entry 0 of its warp's staging area.
__device__ __forceinline__ uint32_t* trace_buf(uint32_t off) {
  uint8_t* base = rt_dyn_smem + ((128u - ((uint32_t)__cvta_generic_to_shared(rt_dyn_smem) & 127u)) & 127u);
  return reinterpret_cast<uint32_t*>(base + off + (threadIdx.x >> 5) * kTraceBufWarpBytes) + (threadIdx.x & 31u);
}

// Starts a pushed node on its way to L1: a walk waits for its nodes more than
// for anything else once its instructions are few, and a pushed node stays on
// the stack for a while before its visit.  GB300, us without / with: 2M-triangle
// terrain, 49K bounce rays plain 441 / 386, treelet order 521 / 424, staged 571 /
// 463; 2M rays 2124 / 2059, 2683 / 2607, 2997 / 2852; 1M-triangle blobs, 1M bounce
// rays 764 / 662, 941 / 741, 1016 / 772.  2M any-hit rays in treelet order lose
// 1.7% (1636 / 1664).  (A prefetch into L2 only was slower than none.)  A child
// outside the blob is within the array's padding (rtw::kPadUnits).
__device__ __forceinline__ void touch_node(const uint4* walk, uint32_t unit) {
  __shared__ uint32_t scratch;
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(&scratch);
  rtd::touch_l1(s, walk + (uint64_t)unit * 4);
  rtd::touch_l1(s, walk + (uint64_t)unit * 4 + 2);
}

// Records entry n (< capacity) of ray r's row.
__device__ __forceinline__ void trace_put(const TraceArgs& a, uint32_t r, uint32_t n, uint32_t x) {
  if (a.tbuf_off == kNone) {
    a.rows[(uint64_t)r * a.cap + n] = x;
    return;
  }
  uint32_t* b = trace_buf(a.tbuf_off);
  const uint32_t j = n & 7u;
  b[j * 32] = x;
  if (j == 7u) {
    uint4* d = reinterpret_cast<uint4*>(a.rows + (uint64_t)r * a.cap + (n - 7u));
    __stcs(d, make_uint4(b[0], b[32], b[64], b[96]));
    __stcs(d + 1, make_uint4(b[128], b[160], b[192], x));
  }
}

// Writes the staged entries of a ray's last partial sector; m = entries
// recorded (at most the capacity).  A row shorter than kIdsSkip is whole in the
// staging area: its treelet ids are written too.
constexpr uint32_t kIdsSkip = 8;
__device__ __forceinline__ void trace_drain(const TraceArgs& a, uint32_t r, uint32_t m, const uint2* meta) {
  const uint32_t k = m & 7u;
  if (a.tbuf_off == kNone || k == 0) return;
  const uint32_t* b = trace_buf(a.tbuf_off);
  const uint64_t at = (uint64_t)r * a.cap + (m - k);
  for (uint32_t j = 0; j < k; ++j) a.rows[at + j] = b[j * 32];
  if (a.ids && m < kIdsSkip)
    for (uint32_t j = 0; j < k; ++j) a.ids[at + j] = __ldg(&meta[b[j * 32] >> 3].x);
}

// The treelet id of every recorded visit: reads and writes the rows in order,
// the scattered part is the 8-byte table entry.  WIDE: eight lanes take a row,
// four entries each (rows that start on 16-byte boundaries), so that a warp has
// up to 128 table reads on their way; with one warp per row and one entry a
// lane the pass was bound by two dependent loads (282 us for 1M bounce rays' 63M
// entries on a GB300; WIDE 208, by then bound by L2 sectors; eight lanes a row
// without WIDE are 4-11% faster for rows of a few entries, 3-5% slower for long
// ones).  Rows shorter than `skip` have their ids already (trace_drain).  WIDE reads
// a row's count one row ahead: 1M rays of 1M-triangle blobs, both traces, in treelet
// order 728 / 710 us, 810,000 of 2,000-triangle blobs, nearly all of which miss, with
// the skip 166 / 142.
template <bool WIDE>
__global__ void __launch_bounds__(256) trace_treelet_ids_kernel(const uint32_t* __restrict__ visits,
                                                                const rt_hit* __restrict__ hits,
                                                                const uint2* __restrict__ meta, uint32_t n,
                                                                uint32_t cap, uint32_t skip,
                                                                uint32_t* __restrict__ treelets) {
  constexpr uint32_t kLanes = WIDE ? 8u : 32u, kEach = WIDE ? 4u : 1u;
  const uint32_t lane = threadIdx.x % kLanes;
  const uint64_t rows = (uint64_t)gridDim.x * blockDim.x / kLanes;
  uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  uint32_t next = r < n ? min(hits[r].n_visits, cap) : 0u;
  for (; r < n; r += rows) {
    const uint32_t m = WIDE ? next : min(hits[r].n_visits, cap);
    if (WIDE && r + rows < n) next = min(hits[r + rows].n_visits, cap);
    if (m < skip) continue;
    const uint64_t row = r * cap;
#pragma unroll 2
    for (uint32_t j = lane * kEach; j < m; j += kLanes * kEach) {
      if (WIDE && j + 4 <= m) {
        const uint4 x = __ldcs(reinterpret_cast<const uint4*>(visits + row + j));
        __stcs(reinterpret_cast<uint4*>(treelets + row + j),
               make_uint4(__ldg(&meta[x.x >> 3].x), __ldg(&meta[x.y >> 3].x), __ldg(&meta[x.z >> 3].x),
                          __ldg(&meta[x.w >> 3].x)));
      } else {
        for (uint32_t k = j; k < min(j + kEach, m); ++k) treelets[row + k] = __ldg(&meta[visits[row + k] >> 3].x);
      }
    }
  }
}

__device__ __forceinline__ void load_ray(const rt_ray* rays, uint32_t r, rtm::V3& o, float& tmin, rtm::V3& d,
                                         float& tmax) {
  const float4* p = reinterpret_cast<const float4*>(rays + r);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  o = rtm::v3(a.x, a.y, a.z);
  tmin = a.w;
  d = rtm::v3(b.x, b.y, b.z);
  tmax = b.w;
}

// The scene ray r walks.  MULTI = false compiles a launch over one scene,
// whose tables are the launch arguments themselves.
template <bool MULTI>
__device__ __forceinline__ SceneView scene_of(const TraceArgs& a, uint32_t r) {
  if (!MULTI || a.n_items == 0) return SceneView{a.blob, a.walk, a.raw, a.meta, a.route, a.n_units};
  uint32_t lo = 0, hi = a.n_items;  // last item with item_begin <= r
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(a.item_begin + mid) <= r) lo = mid;
    else hi = mid;
  }
  const SceneView* s = a.scenes + __ldg(a.item_scene + lo);
  SceneView v;
  v.blob = reinterpret_cast<const uint4*>(__ldg(reinterpret_cast<const unsigned long long*>(&s->blob)));
  v.walk = reinterpret_cast<const uint4*>(__ldg(reinterpret_cast<const unsigned long long*>(&s->walk)));
  v.raw = reinterpret_cast<const uint4*>(__ldg(reinterpret_cast<const unsigned long long*>(&s->raw)));
  v.meta = reinterpret_cast<const uint2*>(__ldg(reinterpret_cast<const unsigned long long*>(&s->meta)));
  v.route = reinterpret_cast<const uint16_t*>(__ldg(reinterpret_cast<const unsigned long long*>(&s->route)));
  v.n_units = __ldg(&s->n_units);
  return v;
}

// Hit record from the closest leaf / instance (vulkan_ray_tracing.cc:2990-3028).
__device__ __forceinline__ void write_hit(const TraceArgs& a, const SceneView& v, uint32_t r, bool hit, float min_thit, rtm::V3 O,
                                          rtm::V3 D, float tmin, float tmax, uint32_t c_leaf, uint32_t c_inst,
                                          float c_tobj, uint32_t n_visits, uint32_t status) {
  rt_hit h;
  h.hit_geometry = 0;
  h.geometry_index = 0;
  h.primitive_index = 0;
  h.instance_index = 0;
  h.world_min_thit = 0.0f;
  h.barycentric[0] = h.barycentric[1] = h.barycentric[2] = 0.0f;
  h.intersection_point[0] = h.intersection_point[1] = h.intersection_point[2] = 0.0f;
  h.closest_leaf = 0;
  h.closest_instance = 0;
  h.reserved = 0;
  if (hit) {
    rtd::Node64 q;
    rtd::load64(v.blob + (uint64_t)c_leaf * 4, q);
    rtd::Instance in;
    rtd::load_instance(v.blob + (uint64_t)c_inst * 4, in);
    const rtm::ObjRay orr = rtm::make_transformed_ray(in.w2o, O, D, tmin, tmax);
    h.hit_geometry = 1;
    h.geometry_index = rtf::geometry_index_of(q.w[1]);
    h.primitive_index = q.w[2];
    h.instance_index = in.instance_id;
    h.world_min_thit = min_thit;
    h.intersection_point[0] = O.x + D.x * min_thit;
    h.intersection_point[1] = O.y + D.y * min_thit;
    h.intersection_point[2] = O.z + D.z * min_thit;
    const rtm::V3 p = rtm::v3(orr.o.x + orr.d.x * c_tobj, orr.o.y + orr.d.y * c_tobj, orr.o.z + orr.d.z * c_tobj);
    const rtm::V3 v0 = rtm::v3(__uint_as_float(q.w[4]), __uint_as_float(q.w[5]), __uint_as_float(q.w[6]));
    const rtm::V3 v1 = rtm::v3(__uint_as_float(q.w[7]), __uint_as_float(q.w[8]), __uint_as_float(q.w[9]));
    const rtm::V3 v2 = rtm::v3(__uint_as_float(q.w[10]), __uint_as_float(q.w[11]), __uint_as_float(q.w[12]));
    const rtm::V3 b = rtm::barycentric(p, v0, v1, v2);
    h.barycentric[0] = b.x;
    h.barycentric[1] = b.y;
    h.barycentric[2] = b.z;
    h.closest_leaf = c_leaf;
    h.closest_instance = c_inst;
  }
  h.n_visits = n_visits;
  h.status = status | (a.cap && n_visits > a.cap ? RT_RAY_TRACE_OVERFLOW : 0u);
  a.hits[r] = h;
}

// The ray a walk tests nodes with: the world ray at top-level nodes (unit
// kNone, mult 1), an instance's object ray (make_transformed_ray) in its BLAS.
// A walk keeps one of them in registers and changes it when the next node
// needs the other, instead of holding both and selecting per node.  The
// interval is the world ray's times mult in either case (mult = 1 is exact).
struct RayCtx {
  uint32_t unit;
  rtm::V3 o, d, idir;
  float mult;
  bool fast;  // the box test may tell planes apart by the direction's sign
};

__device__ __forceinline__ void enter_instance(const rtd::Instance& in, uint32_t unit, rtm::V3 O, rtm::V3 D, float tmin,
                                               float tmax, RayCtx& c) {
  const rtm::ObjRay r = rtm::make_transformed_ray(in.w2o, O, D, tmin, tmax);
  c.unit = unit;
  c.o = r.o;
  c.d = r.d;
  c.mult = r.mult;
  c.idir = rtm::calculate_idir(r.d);
  c.fast = rtd::finite_ray(r.o, r.d, r.tmin, r.tmax);
}

// Flags of a walk, above the RT_RAY_* status bits of its hit record.
constexpr uint32_t kRayTerminate = 0x100u, kRayOpaque = 0x200u, kRayWorldFast = 0x400u, kRayStatusMask = 0xffu;

// Node bytes a ray reads: 64 per transaction, but 128 for an instance leaf and
// 8 for a leaf descriptor.  A walk counts transactions per ray and, per
// thread, the difference in units of 8 bytes.
constexpr int kInstanceExtra = 8, kDescriptorExtra = -7;

// Adds v summed over the calling warp's active lanes with one atomic.
__device__ __forceinline__ void add_warp_total(unsigned long long* dst, uint32_t v) {
  const uint32_t mask = __activemask();
  const uint32_t sum = __reduce_add_sync(mask, v);
  if ((threadIdx.x & 31u) == (uint32_t)(__ffs(mask) - 1)) atomicAdd(dst, (unsigned long long)sum);
}

// The same for 64-bit values; all 32 lanes must call it.
__device__ __forceinline__ void add_warp_total64(unsigned long long* dst, unsigned long long v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  if ((threadIdx.x & 31u) == 0) atomicAdd(dst, v);
}

// One turn of a warp's lanes (all 32 call it; `have`: the lane walks a ray).
// A lane's next node is an internal node, a primitive leaf, or an entry: an
// instance leaf, or a node of another instance than the one whose ray the
// lane holds.  The three kinds cost about 300, 150 and 250 instructions, and
// most nodes are internal; a warp that visits one node of every lane per turn
// spends half its issue slots on leaves and entries with few lanes active.
// So internal nodes are visited again and again while at least
// kInternalShare / 16 of the walking lanes are at one; leaf and entry lanes
// wait, and are then visited together.  Every ray's own visit order is
// unchanged.  A lane whose ray is over gets have = false, ended = true; the
// turn ends early once `spare` lanes have no ray.  With warp slots `left` counts
// the warp's visits down, and the turn is broken off when it reaches 0: the
// warp votes, and goes on where it was.
// Measured on a GB300 (2M-triangle terrain, 1M-triangle blobs; ms): one visit of
// every lane per turn 3.23 for 2M bounce rays plain, 3.12 for 1M traced bounce
// rays in treelet order, 1.86 for 2M any-hit rays; share 4 3.57 / 3.07 / 2.34,
// 8 2.98 / 2.83 / 1.88, 11 2.86 / 2.84 / 1.72, 12 2.90 / 2.88 / 1.71,
// 13 2.97 / 2.94 / 1.72, 16 3.49 / 3.30 / 2.04.  Letting entries wait for more
// lanes, or running only the larger of leaves and entries, changed nothing
// (2.88-2.90 / 2.85-2.88 / 1.74).
constexpr int kInternalShare = 11;

template <class W, class Lookup>
__device__ __forceinline__ void warp_turn(const TraceArgs& a, W& w, uint32_t r, bool& have, bool& ended, int spare,
                                          const Lookup& lookup, uint32_t& left) {
  for (;;) {
    if (have && !w.pop(a)) {
      have = false;
      ended = true;
    }
    const bool in = have && w.at_internal();
    const int m = __popc(__ballot_sync(0xffffffffu, in)), busy = __popc(__ballot_sync(0xffffffffu, have));
    if (m == 0 || 16 * m < kInternalShare * busy || 32 - busy >= spare) break;
    if (in) w.internal(a, r, lookup);
    if (Lookup::kSlots && --left == 0) return;
  }
  if (have && w.at_leaf()) w.leaf(a, r, lookup);
  else if (have && w.at_entry()) w.entry(a, r, lookup);
  if (Lookup::kSlots) --left;
}

struct NoLookup {
  static constexpr bool kSlots = false;
  __device__ __forceinline__ uint32_t operator()(uint32_t, uint32_t, const uint2*) const { return 0u; }
};

// Finds a ray for every idle lane of the warp (one atomic per refill) and
// runs the lanes' walkers turn by turn.  A lane that finishes
// its ray gets a new one as soon as `refill` lanes of its warp are idle, so
// warps stay full while rays of very different lengths finish (persistent
// threads with dynamic ray fetch).  Every ray's own visit order is unchanged.
// Hit records are written at the refill, by all lanes that finished since the
// last one together: a record costs about as many instructions as a node
// visit (two matrix products, nine divisions), and written by one or two
// lanes at the end of each ray's last step it cost 6-10% of the launch (GB300,
// 2M-triangle terrain: 2M bounce rays plain 4.58 -> 4.25 ms, 2M primary rays
// staged 3.56 -> 3.29 ms; any-hit rays in treelet order 2.35 -> 2.13 ms).
template <class W>
__device__ __forceinline__ void run_persistent(const TraceArgs& a, W& w, unsigned long long& bytes_out) {
  const uint32_t lane = threadIdx.x & 31u;
  bool have = false, ended = false, exhausted = false;  // ended: a finished ray whose record is not written yet
  uint32_t r = 0;
  unsigned long long bytes = 0;
  uint32_t left = 0;
  for (;;) {
    const uint32_t need = __ballot_sync(0xffffffffu, !have);
    if (need == 0xffffffffu || (!exhausted && __popc(need) >= (int)a.refill)) {
      if (ended) {
        w.finish(a, r);
        bytes += 64ull * w.n_tx;
        ended = false;
      }
      if (exhausted) break;  // every lane is idle
      const int leader = __ffs(need) - 1;
      uint32_t base = 0;
      if ((int)lane == leader) base = atomicAdd(a.queue, (uint32_t)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (base + (uint32_t)__popc(need) >= a.n) exhausted = true;
      if (!have) {
        const uint32_t rr = base + (uint32_t)__popc(need & ((1u << lane) - 1u));
        if (rr < a.n) {
          r = rr;
          w.init(a, r);
          have = true;
        }
      }
    }
    warp_turn(a, w, r, have, ended, exhausted ? 33 : (int)a.refill, NoLookup(), left);
  }
  bytes_out = bytes + (unsigned long long)(8ll * w.extra);
}

// ----------------------------------------------------------------- plain

// A ray's traceRay walk (vulkan_ray_tracing.cc:2309-3076) as a sequence of
// node visits.  One LIFO stack of unit << 2 | top | leaf entries; `e` is the
// entry visited next once popped: the first hit internal child (:2570-2578)
// or the stack's top, 0 for none yet (no entry is 0: unit 0 is the TLAS
// header); leaves and further children are pushed.  A top-level instance leaf is followed by
// its whole BLAS before the next top-level entry (:2602-2679), so a
// bottom-level entry always belongs to the instance entered last.
// The warp-synchronous short stack (SHORT): entries 0..kShortStack-1 of each
// ray's stack in its warp's shared memory, entry k of the warp's 32 rays in
// one 128-byte row (lane l in bank l, so a warp's pushes and pops at any mix
// of depths never conflict), the deeper entries in the local-memory stack.
constexpr int kShortStack = 16;
constexpr uint32_t kShortStackWarpBytes = kShortStack * 32 * 4;

// Entries past CAP that a visit may write before its depth is checked: a
// node's children are pushed without a check each.
constexpr int kStackPad = 8;
// Words after the stack entries: what a step rarely needs stays in local
// memory (the stack array is indexed at run time, so the compiler leaves all
// of it there), so that the walk's registers hold the ray it tests with.
constexpr int kPlainCold = 12;

// TRACED = false compiles the walk of a launch without traces (no trace
// code at all); TRACED = true writes the rows.  SHORT keeps the bottom of the
// stack in shared memory (rt_tuning.short_stack).
template <int CAP, bool MULTI, bool TRACED, bool SHORT = false>
struct PlainWalker {
  RayCtx cx;
  float tmin, tmax, min_thit;
  uint32_t e, flags;
  int sp;
  uint32_t n_tx;  // the ray's transactions
  int extra;      // the thread's byte difference (kInstanceExtra)
  uint32_t* stk;  // CAP + kStackPad + kPlainCold words, a local array of the kernel
  SceneView v;

  // The next node to visit into e; false when the walk is over.
  __device__ __forceinline__ bool pop(const TraceArgs& a) {
    if (e) return true;
    if (sp == 0) return false;
    e = *slot(a, --sp);
    return true;
  }
  // a bottom-level entry always belongs to the instance entered last
  __device__ __forceinline__ bool at_internal() const { return !(e & kLeaf); }
  __device__ __forceinline__ bool at_leaf() const { return (e & (kLeaf | kTop)) == kLeaf; }
  __device__ __forceinline__ bool at_entry() const { return (e & (kLeaf | kTop)) == (kLeaf | kTop); }

  // ---- the cold words
  __device__ __forceinline__ uint32_t& cold(int k) const { return stk[CAP + kStackPad + k]; }
  __device__ __forceinline__ rtm::V3 cold3(int k) const {
    return rtm::v3(__uint_as_float(cold(k)), __uint_as_float(cold(k + 1)), __uint_as_float(cold(k + 2)));
  }
  __device__ __forceinline__ void set_cold3(int k, rtm::V3 x) {
    cold(k) = __float_as_uint(x.x);
    cold(k + 1) = __float_as_uint(x.y);
    cold(k + 2) = __float_as_uint(x.z);
  }
  __device__ __forceinline__ rtm::V3 world_d() const { return cold3(0); }
  __device__ __forceinline__ rtm::V3 world_o() const { return cold3(3); }
  __device__ __forceinline__ rtm::V3 world_idir() const { return cold3(6); }
  __device__ __forceinline__ void set_hit(uint32_t leaf, uint32_t inst, float tobj) {
    cold(9) = leaf;
    cold(10) = inst;
    cold(11) = __float_as_uint(tobj);
  }

  // entry i of the stack (the short stack's rows for i < kShortStack)
  __device__ __forceinline__ uint32_t* slot(const TraceArgs& a, int i) {
    if (SHORT && i < kShortStack) {
      uint8_t* base = rt_dyn_smem + ((128u - ((uint32_t)__cvta_generic_to_shared(rt_dyn_smem) & 127u)) & 127u);
      return reinterpret_cast<uint32_t*>(base + a.ss_off + (threadIdx.x >> 5) * kShortStackWarpBytes) +
             i * 32 + (threadIdx.x & 31u);
    }
    return stk + i;
  }

  __device__ __forceinline__ void record(const TraceArgs& a, uint32_t r, uint32_t unit, uint32_t type) {
    if (TRACED && n_tx < a.cap) trace_put(a, r, n_tx, a.rows_tl ? v.meta[unit].x : rtf::pack_visit(unit, type));
    n_tx++;
  }

  __device__ __forceinline__ void init(const TraceArgs& a, uint32_t r) {
    v = scene_of<MULTI>(a, r);
    rtm::V3 O, D;
    load_ray(a.rays, r, O, tmin, D, tmax);
    const uint32_t f = a.flags ? a.flags[r] : a.default_flags;
    flags = (f & rtf::RAY_FLAG_TERMINATE_ON_FIRST_HIT ? kRayTerminate : 0u) | (f & rtf::RAY_FLAG_OPAQUE ? kRayOpaque : 0u);
    n_tx = 0;
    sp = 0;
    e = 0;
    min_thit = tmax;
    const rtm::V3 id = rtm::calculate_idir(D);
    set_cold3(0, D);
    set_cold3(3, O);
    set_cold3(6, id);
    set_hit(0, 0, 0.0f);
    if (rtd::finite_ray(O, D, tmin, tmax)) flags |= kRayWorldFast;
    world();
    record(a, r, 0, rtf::TX_STRUCTURE);
    const uint4 h0 = __ldg(v.blob), h1 = __ldg(v.blob + 1);
    const uint64_t root_off = (uint64_t)h0.x | ((uint64_t)h0.y << 32);
    const rtm::V3 bmin = rtm::v3(__uint_as_float(h0.z), __uint_as_float(h0.w), __uint_as_float(h1.x));
    const rtm::V3 bmax = rtm::v3(__uint_as_float(h1.y), __uint_as_float(h1.z), __uint_as_float(h1.w));
    float th;
    if (rtm::ray_box_test(bmin, bmax, id, O, tmin, tmax, th)) e = ((uint32_t)(root_off >> 6) << 2) | kTop;
  }

  // The world ray as the ray tested with (its direction is not: only
  // bottom-level leaves and instance entries read one).
  __device__ __forceinline__ void world() {
    cx.unit = kNone;
    cx.o = world_o();
    cx.idir = world_idir();
    cx.mult = 1.0f;
    cx.fast = (flags & kRayWorldFast) != 0;
  }

  __device__ __forceinline__ void stop(uint32_t bits) {
    flags |= bits;
    sp = 0;
    e = 0;
  }

  // The entry's unit, and 64 bytes of its node in `from` (the walk nodes or
  // the blob); false (and the ray stopped) when it lies outside the blob.
  __device__ __forceinline__ bool load(const uint4* from, uint32_t& unit, uint32_t units, rtd::Node64& q) {
    unit = e >> 2;
    if (unit + units > v.n_units) {
      stop(RT_RAY_BAD_NODE);
      return false;
    }
    rtd::load64(from + (uint64_t)unit * 4, q);
    return true;
  }

  template <class Lookup>
  __device__ __forceinline__ void internal(const TraceArgs& a, uint32_t r, const Lookup&) {
    uint32_t unit;
    rtd::Node64 nd;
    if (!load(v.walk, unit, 1, nd)) return;
    // the stack's top, read while the node is on its way: 40% of the visits
    // end with it as the next entry (2M bounce rays 2.71 against 2.81 ms on a
    // GB300; the treelet walk, with two stacks to choose from, gained nothing)
    const uint32_t below = sp > 0 ? *slot(a, sp - 1) : 0u;
    const uint32_t level = e & kTop;
    record(a, r, unit, rtf::TX_INTERNAL);
    if (level && cx.unit != kNone) world();
    const float t0 = tmin * cx.mult, t1 = tmax * cx.mult, cull = min_thit * cx.mult;
    uint32_t hit = cx.fast && !(nd.w[5] & rtw::kExact)
                       ? rtd::hit_children(nd, cx.o, cx.idir, t0, t1, cull)
                       : rtd::hit_children_exact(v.raw + (uint64_t)unit * 4, cx.o, cx.idir, t0, t1, cull);
    // the first hit internal child is visited next; the other hit children
    // are pushed in order (1.2 hits a visit, so a loop over the bits is
    // shorter than six predicated pushes: 2.81 against 2.92 ms for 2M bounce
    // rays on a GB300)
    auto entry_of = [&](int i) {
      return ((nd.w[3] + ((nd.w[6] >> (4 * i)) & 15u)) << 2) | level | ((nd.w[5] >> (i + rtw::kLeafShift)) & kLeaf);
    };
    const uint32_t inner = hit & nd.w[5];
    e = 0;
    if (inner) {
      const int i = __ffs(inner) - 1;
      e = entry_of(i);
      hit &= ~(1u << i);
      // its visit waits for the warp's leaves and entries when those are due
      // (GB300, us without / with: 49K bounce rays of the 2M-triangle terrain 390 /
      // 334, 262K 686 / 653, 2M 2095 / 2062; 1M-triangle blobs 349 / 294, 468 / 416,
      // 689 / 663; the benchmark's 2M bounce rays 2717 / 2747)
      touch_node(v.walk, e >> 2);
    }
    uint32_t last = 0;
#pragma unroll 1
    for (; hit; hit &= hit - 1u) {
      last = entry_of(__ffs(hit) - 1);
      *slot(a, sp++) = last;
      touch_node(v.walk, last >> 2);
    }
    const bool deep = sp > CAP;
    if (!e && sp > 0) {
      e = last ? last : below;
      --sp;
    }
    if (deep) stop(RT_RAY_STACK_OVERFLOW);
  }

  template <class Lookup>
  __device__ __forceinline__ void leaf(const TraceArgs& a, uint32_t r, const Lookup&) {
    uint32_t unit;
    rtd::Node64 q;
    if (!load(v.blob, unit, 1, q)) return;
    e = 0;
    record(a, r, unit, rtf::TX_LEAF_DESC);
    extra += kDescriptorExtra;
    uint32_t type = rtf::TX_PROCEDURAL_LEAF;
    if (rtf::leaf_type_of(q.w[1]) == 0) {
      const rtm::V3 v0 = rtm::v3(__uint_as_float(q.w[4]), __uint_as_float(q.w[5]), __uint_as_float(q.w[6]));
      const rtm::V3 v1 = rtm::v3(__uint_as_float(q.w[7]), __uint_as_float(q.w[8]), __uint_as_float(q.w[9]));
      const rtm::V3 v2 = rtm::v3(__uint_as_float(q.w[10]), __uint_as_float(q.w[11]), __uint_as_float(q.w[12]));
      float t = 0.0f;
      type = rtf::TX_QUAD_LEAF;
      if (rtm::ray_triangle_test(v0, v1, v2, cx.o, cx.d, t)) {
        const float wt = t / cx.mult;
        if (tmin <= wt && wt <= tmax) {  // :2843-2859
          if ((flags & kRayOpaque) && wt < min_thit) min_thit = wt;
          set_hit(unit, cx.unit, t);
          if (flags & kRayTerminate) sp = 0;
          type = rtf::TX_QUAD_LEAF_HIT;
        }
      }
    } else {
      flags |= RT_RAY_HIT_PROCEDURAL;
    }
    record(a, r, unit, type);
  }

  // an instance leaf
  template <class Lookup>
  __device__ __forceinline__ void entry(const TraceArgs& a, uint32_t r, const Lookup&) {
    uint32_t unit;
    rtd::Node64 q;
    if (!load(v.blob, unit, 2, q)) return;
    record(a, r, unit, rtf::TX_INSTANCE_LEAF);
    extra += kInstanceExtra;
    rtd::Instance in;
    rtd::instance_from(q, v.blob + (uint64_t)unit * 4, 0, in);
    const uint64_t hdr = (uint64_t)unit * 64 + in.bvh_address;
    if ((hdr & 63) || hdr / 64 >= v.n_units) return stop(RT_RAY_BAD_NODE);
    const uint4 h0 = __ldg(v.blob + (hdr >> 4));
    const uint64_t broot = hdr + ((uint64_t)h0.x | ((uint64_t)h0.y << 32));
    enter_instance(in, unit, world_o(), world_d(), tmin, tmax, cx);
    if (sp < CAP) e = (uint32_t)(broot >> 6) << 2;
    else stop(RT_RAY_STACK_OVERFLOW);
    record(a, r, (uint32_t)(hdr >> 6), rtf::TX_STRUCTURE);
  }

  __device__ __forceinline__ void finish(const TraceArgs& a, uint32_t r) {
    const bool bad = flags & (RT_RAY_STACK_OVERFLOW | RT_RAY_BAD_NODE);
    if (TRACED) trace_drain(a, r, min(n_tx, a.cap), v.meta);
    write_hit(a, v, r, !bad && (min_thit < tmax), min_thit, world_o(), world_d(), tmin, tmax, cold(9), cold(10),
              __uint_as_float(cold(11)), n_tx, flags & kRayStatusMask);
  }
};

// Four 256-thread CTAs per SM, 64 registers: with one ray context in
// registers and the rest in the stack's cold words, 2M bounce rays of the
// 2M-triangle terrain take 2.70 ms on a GB300 (56 registers 2.73, 72 2.80; when
// the node test took more registers, 48 were 9% and 85 4% slower than 64).
// With both the world ray and the object ray live the walk took 90 registers,
// and did best with all its fields left in local memory at 48: 4.27 ms, bound
// by those loads.
constexpr int kPlainMinBlocks = 4;
template <int CAP, bool MULTI, bool TRACED, bool SHORT = false>
__global__ void __launch_bounds__(256, kPlainMinBlocks) trace_plain_kernel(TraceArgs a) {
  uint32_t stack[CAP + kStackPad + kPlainCold];
  PlainWalker<CAP, MULTI, TRACED, SHORT> w;
  w.stk = stack;
  w.extra = 0;
  unsigned long long bytes = 0;
  run_persistent(a, w, bytes);
  rtd::touch_l1_done();
  if (a.stats) add_warp_total64(a.stats + ST_NODE_BYTES, bytes);
}

}  // namespace rtk
