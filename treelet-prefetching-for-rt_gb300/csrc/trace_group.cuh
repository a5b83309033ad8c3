// The walks for small launches: eight lanes walk one ray.
//
// With one ray per lane a launch of a few thousand rays leaves most of the
// GPU idle, and its time is the longest warp's: 32 divergent rays, each visit
// a chain of several hundred instructions.  Here lane j of a ray's eight tests
// child j of a node (lanes 6 and 7 help with leaves only), the hit children
// go onto the ray's stack in shared memory in one store, and up to eight
// consecutive leaves on the stack's top are tested at once; what the ray's
// state says is computed by all its lanes alike.  The visits, their order and
// every value are those of PlainWalker and Walker.  A warp holds `rpw` rays
// (1, 2 or 4): with one, no ray waits for another's branch.
#pragma once
#include <type_traits>

#include "trace_treelet.cuh"

namespace rtk {

constexpr uint32_t kGroup = 8;          // lanes of a ray
constexpr uint32_t kGroupThreads = 128;

// Shared-memory bytes of one ray's stack (entries past the depth: RT stacks
// are checked once per visit, as the walkers').
__host__ __device__ constexpr uint32_t group_stack_bytes(bool treelet, uint32_t depth) {
  return (depth + (uint32_t)kStackPad) * (treelet ? 16u : 4u) + 16u;
}


// One ray's walk over its eight lanes.
template <bool TREELET, bool TRACED>
struct GroupWalk {
  using Entry = std::conditional_t<TREELET, unsigned long long, uint32_t>;
  static constexpr uint32_t kShift = TREELET ? kEShift : 2u;
  const TraceArgs& a;
  const SceneView v;
  const uint32_t j, mask;  // lane within the group, the group's lanes
  const int depth;
  Entry* const cu;  // the stack (plain), the current-treelet stack
  Entry* const ot;  // the other-treelet stack
  const uint32_t scratch;  // touch_l1's word
  uint32_t r;
  rtm::V3 O, D, I;  // the world ray
  RayCtx cx;
  float tmin, tmax, min_thit, c_tobj;
  uint32_t flags, c_leaf, c_inst, n_tx;
  int extra, ncu, not_;
  Entry e;        // the entry visited next, 0 = none popped
  bool from_cu;   // the stack it came from

  __device__ __forceinline__ uint32_t ballot(bool p) const {
    return (__ballot_sync(mask, p) >> (threadIdx.x & 24u)) & 0xffu;
  }
  template <class T>
  __device__ __forceinline__ T from_lane(T x, int l) const {
    return __shfl_sync(mask, x, l, kGroup);
  }
  __device__ __forceinline__ void put(uint32_t at, uint32_t unit, uint32_t type) const {
    if (TRACED && at < a.cap)
      a.rows[(uint64_t)r * a.cap + at] = a.rows_tl ? v.meta[unit].x : rtf::pack_visit(unit, type);
  }
  __device__ __forceinline__ void record(uint32_t unit, uint32_t type) {
    if (j == 0) put(n_tx, unit, type);
    n_tx++;
  }
  __device__ __forceinline__ void clear() {
    e = 0;
    ncu = not_ = 0;
  }
  __device__ __forceinline__ void stop(uint32_t bits) {
    flags |= bits;
    clear();
  }
  __device__ __forceinline__ void world() {
    cx.unit = kNone;
    cx.o = O;
    cx.idir = I;
    cx.mult = 1.0f;
    cx.fast = (flags & kRayWorldFast) != 0;
  }
  __device__ __forceinline__ uint32_t inst() const { return TREELET ? (uint32_t)((unsigned long long)e >> 32) : 0u; }
  static __device__ __forceinline__ Entry make(uint32_t code, uint32_t in) {
    if constexpr (TREELET) return (unsigned long long)code | ((unsigned long long)in << 32);
    else return code;
  }

  __device__ __forceinline__ void init(uint32_t ray) {
    r = ray;
    load_ray(a.rays, r, O, tmin, D, tmax);
    const uint32_t f = a.flags ? a.flags[r] : a.default_flags;
    flags = (f & rtf::RAY_FLAG_TERMINATE_ON_FIRST_HIT ? kRayTerminate : 0u) | (f & rtf::RAY_FLAG_OPAQUE ? kRayOpaque : 0u);
    n_tx = 0;
    extra = 0;
    clear();
    min_thit = tmax;
    c_leaf = c_inst = 0;
    c_tobj = 0.0f;
    I = rtm::calculate_idir(D);
    if (rtd::finite_ray(O, D, tmin, tmax)) flags |= kRayWorldFast;
    world();
    record(0, rtf::TX_STRUCTURE);
    const uint4 h0 = __ldg(v.blob), h1 = __ldg(v.blob + 1);
    const uint64_t root_off = (uint64_t)h0.x | ((uint64_t)h0.y << 32);
    const rtm::V3 bmin = rtm::v3(__uint_as_float(h0.z), __uint_as_float(h0.w), __uint_as_float(h1.x));
    const rtm::V3 bmax = rtm::v3(__uint_as_float(h1.y), __uint_as_float(h1.z), __uint_as_float(h1.w));
    float th;
    if (rtm::ray_box_test(bmin, bmax, I, O, tmin, tmax, th)) {
      const uint32_t code = ((uint32_t)(root_off >> 6) << kShift) | kTop;
      e = make(code, 0);
      if constexpr (TREELET) {  // current_treelet_root starts as the TLAS header, unit 0 (:1707)
        const uint32_t unit = code >> kShift;
        from_cu = (unit < v.n_units ? __ldg(&v.meta[unit].x) : kNone) == 0u;
      }
    }
  }

  // The stack's top into e when nothing is popped; false when the walk is over.
  __device__ __forceinline__ bool pop() {
    if (e) return true;
    if constexpr (TREELET) {
      if ((ncu | not_) == 0) return false;
      from_cu = ncu > 0;
      e = from_cu ? cu[ncu - 1] : ot[not_ - 1];
      ncu -= from_cu ? 1 : 0;
      not_ -= from_cu ? 0 : 1;
    } else {
      if (ncu == 0) return false;
      e = cu[--ncu];
    }
    return true;
  }

  // Lane j's slab test of child j.
  __device__ __forceinline__ bool hit_child(uint32_t unit, const uint4 q0, const uint4 q1, float t0, float t1,
                                            float cull) const {
    const uint32_t c = min(j, 5u);
    if (cx.fast && !(q1.y & rtw::kExact)) {
      const uint8_t* b = reinterpret_cast<const uint8_t*>(v.walk + (uint64_t)unit * 4) + c;
      const uint32_t hi = c < 4u ? 36u : 30u;  // child c's upper bound, axis x (walk_node.h)
      const float s[3] = {__uint_as_float((q1.x << 23) & 0x7f800000u), __uint_as_float((q1.x << 15) & 0x7f800000u),
                          __uint_as_float((q1.x << 7) & 0x7f800000u)};
      const float org[3] = {__uint_as_float(q0.x), __uint_as_float(q0.y), __uint_as_float(q0.z)};
      const float o[3] = {cx.o.x, cx.o.y, cx.o.z}, id[3] = {cx.idir.x, cx.idir.y, cx.idir.z};
      float lo[3], up[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lo[k] = (__fmaf_rn((float)__ldg(b + 28 + 12 * k), s[k], org[k]) - o[k]) * id[k];
        up[k] = (__fmaf_rn((float)__ldg(b + hi + 12 * k), s[k], org[k]) - o[k]) * id[k];
      }
      const float tn = fmaxf(rtd::max3(fminf(lo[0], up[0]), fminf(lo[1], up[1]), fminf(lo[2], up[2])), t0);
      const float tf = fminf(rtd::min3(fmaxf(lo[0], up[0]), fmaxf(lo[1], up[1]), fmaxf(lo[2], up[2])), t1);
      return tn <= tf && !(tn >= cull);
    }
    return rtd::hit_children_exact(v.raw + (uint64_t)unit * 4, cx.o, cx.idir, t0, t1, cull, c, c + 1u) != 0;
  }

  __device__ __forceinline__ void internal() {
    const uint32_t code = (uint32_t)e, unit = code >> kShift, in = inst(), level = code & kTop;
    if (unit >= v.n_units) return stop(RT_RAY_BAD_NODE);
    const uint4 q0 = __ldg(v.walk + (uint64_t)unit * 4), q1 = __ldg(v.walk + (uint64_t)unit * 4 + 1);
    record(unit, rtf::TX_INTERNAL);
    if (level && cx.unit != kNone) world();
    const uint32_t valid = (q1.y | (q1.y >> rtw::kLeafShift)) & rtw::kChildMask;
    const bool h = hit_child(unit, q0, q1, tmin * cx.mult, tmax * cx.mult, min_thit * cx.mult);
    uint32_t hit = ballot(h) & valid;
    // hit children start on their way to L1 while the ray is elsewhere
    if ((hit >> j) & 1u) {
      const uint4* const child = v.walk + (uint64_t)(q0.w + ((q1.z >> (4 * j)) & 15u)) * 4;
      rtd::touch_l1(scratch, child);
      rtd::touch_l1(scratch, child + 2);
    }
    auto entry_of = [&](uint32_t i) {
      const uint32_t c = q0.w + ((q1.z >> (4 * i)) & 15u);
      return make((c << kShift) | level | ((q1.y >> (i + rtw::kLeafShift)) & kLeaf), in);
    };
    const uint32_t below = (1u << j) - 1u;
    e = 0;
    if constexpr (TREELET) {
      const uint32_t same = q1.y >> (from_cu ? rtw::kSameShift : rtw::kOtherShift);
      const uint32_t to_cu = hit & same, to_ot = hit & ~same;
      if ((hit >> j) & 1u) {
        if ((to_cu >> j) & 1u) cu[ncu + __popc(to_cu & below)] = entry_of(j);
        else ot[not_ + __popc(to_ot & below)] = entry_of(j);
      }
      ncu += __popc(to_cu);
      not_ += __popc(to_ot);
      __syncwarp(mask);
      if (ncu > depth + 1 || not_ > depth) return stop(RT_RAY_STACK_OVERFLOW);
      if (to_cu) {  // the entry just put on top
        e = entry_of(31u - __clz(to_cu));
        from_cu = true;
        --ncu;
      }
    } else {
      const uint32_t inner = hit & q1.y;  // the first hit internal child is visited next
      if (inner) {
        const uint32_t i = __ffs(inner) - 1;
        e = entry_of(i);
        hit &= ~(1u << i);
      }
      if ((hit >> j) & 1u) cu[ncu + __popc(hit & below)] = entry_of(j);
      ncu += __popc(hit);
      __syncwarp(mask);
      if (ncu > depth) return stop(RT_RAY_STACK_OVERFLOW);
      if (!e && hit) {
        e = entry_of(31u - __clz(hit));
        --ncu;
      }
    }
  }

  // Leaf e and the leaves right below it on its stack (same instance): lane j
  // tests the j-th; their results are applied in stack order.
  __device__ __forceinline__ void leaves() {
    Entry x = e;
    const int top = TREELET ? (from_cu ? ncu : not_) : ncu;
    bool ok = j == 0;
    if (j > 0 && top >= (int)j) {
      x = (TREELET && !from_cu) ? ot[top - (int)j] : cu[top - (int)j];
      ok = ((uint32_t)x & (kLeaf | kTop)) == kLeaf;
      if constexpr (TREELET) ok = ok && (uint32_t)(x >> 32) == cx.unit;
    }
    const uint32_t unit = (uint32_t)x >> kShift;
    int k = __ffs(~ballot(ok && unit < v.n_units)) - 1;  // leaves of this batch
    if (k == 0) return stop(RT_RAY_BAD_NODE);
    rtd::Node64 q;
    bool quad = false, hit = false;
    float t = 0.0f, wt = 0.0f;
    if ((int)j < k) {
      rtd::load64(v.blob + (uint64_t)unit * 4, 0, q);
      quad = rtf::leaf_type_of(q.w[1]) == 0;
      if (quad) {
        const rtm::V3 v0 = rtm::v3(__uint_as_float(q.w[4]), __uint_as_float(q.w[5]), __uint_as_float(q.w[6]));
        const rtm::V3 v1 = rtm::v3(__uint_as_float(q.w[7]), __uint_as_float(q.w[8]), __uint_as_float(q.w[9]));
        const rtm::V3 v2 = rtm::v3(__uint_as_float(q.w[10]), __uint_as_float(q.w[11]), __uint_as_float(q.w[12]));
        if (rtm::ray_triangle_test(v0, v1, v2, cx.o, cx.d, t)) {
          wt = t / cx.mult;
          hit = tmin <= wt && wt <= tmax && (!TREELET || wt < min_thit);
        }
      }
    }
    const uint32_t cand = ballot(hit);
    uint32_t accepted = 0;
    for (uint32_t m = cand; m; m &= m - 1u) {
      const int l = __ffs(m) - 1;
      const float w = from_lane(wt, l);
      const bool closer = w < min_thit;
      if (TREELET && !closer) continue;  // :2127-2141
      if (closer && (TREELET || (flags & kRayOpaque))) min_thit = w;  // :2843-2859
      c_leaf = from_lane(unit, l);
      c_tobj = from_lane(t, l);
      c_inst = cx.unit;
      accepted |= 1u << l;
      if (flags & kRayTerminate) {
        k = l + 1;
        break;
      }
    }
    if (ballot((int)j < k && !quad)) flags |= RT_RAY_HIT_PROCEDURAL;
    if ((int)j < k) {
      put(n_tx + 2 * j, unit, rtf::TX_LEAF_DESC);
      put(n_tx + 2 * j + 1, unit,
          !quad ? rtf::TX_PROCEDURAL_LEAF : ((accepted >> j) & 1u ? rtf::TX_QUAD_LEAF_HIT : rtf::TX_QUAD_LEAF));
    }
    n_tx += 2 * k;
    extra += kDescriptorExtra * k;
    e = 0;
    if (TREELET && !from_cu) not_ -= k - 1;
    else ncu -= k - 1;
    if (accepted && (flags & kRayTerminate)) clear();
  }

  // The ray context for e: an instance leaf enters its own instance, a BLAS
  // node's instance is entered again and the node stays to be visited.
  __device__ __forceinline__ void entry() {
    const uint32_t code = (uint32_t)e;
    const bool top = code & kTop;
    const uint32_t unit = top ? code >> kShift : inst();
    if (top && unit + 2 > v.n_units) return stop(RT_RAY_BAD_NODE);
    rtd::Instance in;
    rtd::load_instance(v.blob + (uint64_t)unit * 4, 0, in);
    enter_instance(in, unit, O, D, tmin, tmax, cx);
    if (!top) return;
    record(unit, rtf::TX_INSTANCE_LEAF);
    extra += kInstanceExtra;
    const uint64_t hdr = (uint64_t)unit * 64 + in.bvh_address;
    if ((hdr & 63) || hdr / 64 >= v.n_units) return stop(RT_RAY_BAD_NODE);
    const uint4 h0 = __ldg(v.blob + (hdr >> 4));
    const uint64_t broot = hdr + ((uint64_t)h0.x | ((uint64_t)h0.y << 32));
    record((uint32_t)(hdr >> 6), rtf::TX_STRUCTURE);
    const uint32_t next = (uint32_t)(broot >> 6) << kShift;
    if constexpr (TREELET) {
      // visited next from the stack its route bit names: cu is popped first,
      // and ot only when cu is empty
      const bool same = (__ldg(v.route + unit) >> (kRouteInst + (from_cu ? 0u : 1u))) & 1u;
      if (same ? ncu + 1 > depth + 1 : not_ + 1 > depth) return stop(RT_RAY_STACK_OVERFLOW);
      e = make(next, unit);
      if (same || ncu == 0) {
        from_cu = same;
      } else {
        if (j == 0) ot[not_] = e;
        ++not_;
        __syncwarp(mask);
        e = 0;
      }
    } else {
      if (ncu >= depth) return stop(RT_RAY_STACK_OVERFLOW);
      e = next;
    }
  }

  __device__ __forceinline__ void run(uint32_t ray) {
    init(ray);
    while (pop()) {
      const uint32_t code = (uint32_t)e;
      const bool leaf = code & kLeaf, top = code & kTop;
      if (top ? leaf : (TREELET && inst() != cx.unit)) entry();
      else if (leaf) leaves();
      else internal();
    }
    if (j == 0) {
      const bool bad = flags & (RT_RAY_STACK_OVERFLOW | RT_RAY_BAD_NODE);
      write_hit(a, v, r, !bad && (min_thit < tmax), min_thit, O, D, tmin, tmax, c_leaf, c_inst, c_tobj, n_tx,
                flags & kRayStatusMask);
    }
  }
};

// rays r = group index, + groups of the launch, ...; dynamic shared memory:
// group_stack_bytes per group of the CTA.
template <bool TREELET, bool TRACED>
__global__ void __launch_bounds__(kGroupThreads) trace_group_kernel(TraceArgs a, uint32_t depth, uint32_t rpw) {
  using W = GroupWalk<TREELET, TRACED>;
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  const uint32_t lane = threadIdx.x & 31u, g = lane / kGroup, warps = blockDim.x / 32u;
  if (g >= rpw) return;
  const uint32_t slot = (threadIdx.x >> 5) * rpw + g;
  typename W::Entry* stack = reinterpret_cast<typename W::Entry*>(dyn_smem + slot * group_stack_bytes(TREELET, depth));
  W w{a,    scene_of<false>(a, 0), lane % kGroup, 0xffu << (g * kGroup), (int)depth, stack, stack + depth + kStackPad,
      smem_u32(dyn_smem) + (slot + 1) * group_stack_bytes(TREELET, depth) - 16u};
  unsigned long long bytes = 0;
  for (uint32_t r = blockIdx.x * warps * rpw + slot; r < a.n; r += gridDim.x * warps * rpw) {
    w.run(r);
    bytes += 64ull * w.n_tx + (unsigned long long)(8ll * w.extra);
    __syncwarp(w.mask);
  }
  rtd::touch_l1_done();
  if (a.stats && lane % kGroup == 0 && bytes) atomicAdd(a.stats + ST_NODE_BYTES, bytes);
}

}  // namespace rtk
