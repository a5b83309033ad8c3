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
// (1, 2 or 4): with one, no ray waits for another's branch.  STAGED reads
// pinned treelets' nodes from the CTA's copy of the pinned image, as
// trace_staged_kernel does.
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
template <bool TREELET, bool TRACED, bool STAGED>
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
  const uint32_t pin_base, pin_root;  // STAGED: shared address of the pinned records, the TLAS root's record (0: none)
  uint32_t r;
  rtm::V3 O, D, I;  // the world ray
  RayCtx cx;
  float tmin, tmax, min_thit, c_tobj;
  uint32_t flags, c_leaf, c_inst, n_tx;
  int extra, ncu, not_;
  Entry e;        // the entry visited next, 0 = none popped
  bool from_cu;   // the stack it came from
  uint32_t smem_reads, gmem_reads;

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
  static __device__ __forceinline__ bool pinned(uint32_t code) { return STAGED && (code & kEPin); }
  // A node's address: its pinned record, else unit `unit` of `from`.  `unit`
  // is read from the record of a pinned node.
  __device__ __forceinline__ const uint4* locate(uint32_t code, const uint4* from, uint32_t& unit) const {
    if (pinned(code)) {
      const uint32_t saddr = pin_base + (code >> kShift) * 16u;
      unit = rtd::ld_shared_u32(saddr + ((code & kLeaf) ? 0u : rtp::IN_UNIT));
      return reinterpret_cast<const uint4*>(__cvta_shared_to_generic(saddr));
    }
    unit = code >> kShift;
    return from + (uint64_t)unit * 4;
  }
  static __device__ __forceinline__ uint4 ld16(const uint4* p) { return STAGED ? *p : __ldg(p); }
  static __device__ __forceinline__ uint8_t ld1(const uint8_t* p) { return STAGED ? *p : __ldg(p); }
  __device__ __forceinline__ void count_reads(uint32_t shared, uint32_t all) {
    if (STAGED) {
      smem_reads += shared;
      gmem_reads += all - shared;
    }
  }
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
      e = make(STAGED && pin_root ? ((pin_root << kShift) | kEPin | kTop) : code, 0);
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
  __device__ __forceinline__ bool hit_child(const uint4* src, uint32_t unit, const uint4 q0, const uint4 q1, float t0,
                                            float t1, float cull) const {
    const uint32_t c = min(j, 5u);
    if (cx.fast && !(q1.y & rtw::kExact)) {
      const uint8_t* b = reinterpret_cast<const uint8_t*>(src) + c;
      const uint32_t hi = c < 4u ? 36u : 30u;  // child c's upper bound, axis x (walk_node.h)
      const float s[3] = {__uint_as_float((q1.x << 23) & 0x7f800000u), __uint_as_float((q1.x << 15) & 0x7f800000u),
                          __uint_as_float((q1.x << 7) & 0x7f800000u)};
      const float org[3] = {__uint_as_float(q0.x), __uint_as_float(q0.y), __uint_as_float(q0.z)};
      const float o[3] = {cx.o.x, cx.o.y, cx.o.z}, id[3] = {cx.idir.x, cx.idir.y, cx.idir.z};
      float lo[3], up[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lo[k] = (__fmaf_rn((float)ld1(b + 28 + 12 * k), s[k], org[k]) - o[k]) * id[k];
        up[k] = (__fmaf_rn((float)ld1(b + hi + 12 * k), s[k], org[k]) - o[k]) * id[k];
      }
      const float tn = fmaxf(rtd::max3(fminf(lo[0], up[0]), fminf(lo[1], up[1]), fminf(lo[2], up[2])), t0);
      const float tf = fminf(rtd::min3(fmaxf(lo[0], up[0]), fmaxf(lo[1], up[1]), fmaxf(lo[2], up[2])), t1);
      return tn <= tf && !(tn >= cull);
    }
    return rtd::hit_children_exact(v.raw + (uint64_t)unit * 4, cx.o, cx.idir, t0, t1, cull, c, c + 1u) != 0;
  }

  __device__ __forceinline__ void internal() {
    const uint32_t code = (uint32_t)e, in = inst(), level = code & kTop;
    uint32_t unit;
    const uint4* src = locate(code, v.walk, unit);
    if (!pinned(code) && unit >= v.n_units) return stop(RT_RAY_BAD_NODE);
    const uint4 q0 = ld16(src), q1 = ld16(src + 1);
    uint32_t so = 0;  // a pinned parent names its pinned children's records: lane j's child
    if (pinned(code)) so = rtd::ld_shared_u16(pin_base + (code >> kShift) * 16u + rtp::IN_CHILD_SOFF + 2u * min(j, 5u));
    count_reads(pinned(code) ? 1u : 0u, 1u);
    record(unit, rtf::TX_INTERNAL);
    if (level && cx.unit != kNone) world();
    const uint32_t valid = (q1.y | (q1.y >> rtw::kLeafShift)) & rtw::kChildMask;
    const bool h = hit_child(src, unit, q0, q1, tmin * cx.mult, tmax * cx.mult, min_thit * cx.mult);
    uint32_t hit = ballot(h) & valid;
    // hit children start on their way to L1 while the ray is elsewhere (touch_node)
    if ((hit >> j) & 1u && !so) {
      const uint4* const child = v.walk + (uint64_t)(q0.w + ((q1.z >> (4 * j)) & 15u)) * 4;
      rtd::touch_l1(scratch, child);
      rtd::touch_l1(scratch, child + 2);
    }
    auto entry_of = [&](uint32_t i, uint32_t so_i) {
      const uint32_t c = q0.w + ((q1.z >> (4 * i)) & 15u);
      const uint32_t at = STAGED && so_i ? ((so_i << kShift) | kEPin) : c << kShift;
      return make(at | level | ((q1.y >> (i + rtw::kLeafShift)) & kLeaf), in);
    };
    auto entry_for_all = [&](uint32_t i) { return entry_of(i, STAGED ? from_lane(so, (int)i) : 0u); };
    const uint32_t below = (1u << j) - 1u;
    e = 0;
    if constexpr (TREELET) {
      const uint32_t same = q1.y >> (from_cu ? rtw::kSameShift : rtw::kOtherShift);
      const uint32_t to_cu = hit & same, to_ot = hit & ~same;
      if ((hit >> j) & 1u) {
        if ((to_cu >> j) & 1u) cu[ncu + __popc(to_cu & below)] = entry_of(j, so);
        else ot[not_ + __popc(to_ot & below)] = entry_of(j, so);
      }
      ncu += __popc(to_cu);
      not_ += __popc(to_ot);
      __syncwarp(mask);
      if (ncu > depth + 1 || not_ > depth) return stop(RT_RAY_STACK_OVERFLOW);
      if (to_cu) {  // the entry just put on top
        e = entry_for_all(31u - __clz(to_cu));
        from_cu = true;
        --ncu;
      }
    } else {
      const uint32_t inner = hit & q1.y;  // the first hit internal child is visited next
      if (inner) {
        const uint32_t i = __ffs(inner) - 1;
        e = entry_for_all(i);
        hit &= ~(1u << i);
      }
      if ((hit >> j) & 1u) cu[ncu + __popc(hit & below)] = entry_of(j, so);
      ncu += __popc(hit);
      __syncwarp(mask);
      if (ncu > depth) return stop(RT_RAY_STACK_OVERFLOW);
      if (!e && hit) {
        e = entry_for_all(31u - __clz(hit));
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
    uint32_t unit = 0;
    const uint4* src = v.blob;
    if (ok) src = locate((uint32_t)x, v.blob, unit);
    int k = __ffs(~ballot(ok && (pinned((uint32_t)x) || unit < v.n_units))) - 1;  // leaves of this batch
    if (k == 0) return stop(RT_RAY_BAD_NODE);
    rtd::Node64 q;
    bool quad = false, hit = false;
    float t = 0.0f, wt = 0.0f;
    if ((int)j < k) {
      if (STAGED) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint4 y = src[w];
          q.w[4 * w] = y.x, q.w[4 * w + 1] = y.y, q.w[4 * w + 2] = y.z, q.w[4 * w + 3] = y.w;
        }
      } else {
        rtd::load64(src, q);
      }
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
    if (STAGED) count_reads(__popc(ballot((int)j < k && pinned((uint32_t)x))), (uint32_t)k);
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
    const bool rec = top && pinned(code);  // a pinned record: decoded rows, units and route bits
    uint32_t unit = inst();
    const uint4* src = v.blob;
    if (top) {
      src = locate(code, v.blob, unit);
      if (!rec && unit + 2 > v.n_units) return stop(RT_RAY_BAD_NODE);
      count_reads(rec ? 1u : 0u, 1u);
    }
    rtd::Instance in;
    uint4 head = make_uint4(0, 0, 0, 0);
    if (rec) {
      head = src[0];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint4 y = src[rtp::IL_W2O / 16 + k];
        const uint32_t w[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) in.w2o.m[(4 * k + q) / 3][(4 * k + q) % 3] = __uint_as_float(w[q]);
      }
    } else {
      rtd::load_instance(v.blob + (uint64_t)unit * 4, in);
    }
    enter_instance(in, unit, O, D, tmin, tmax, cx);
    if (!top) return;
    record(unit, rtf::TX_INSTANCE_LEAF);
    extra += kInstanceExtra;
    uint32_t hdr_unit = head.y, next = 0;
    if (rec) {
      const uint32_t so = head.w >> 16;
      next = so ? ((so << kShift) | kEPin) : head.z << kShift;
    } else {
      const uint64_t hdr = (uint64_t)unit * 64 + in.bvh_address;
      if ((hdr & 63) || hdr / 64 >= v.n_units) return stop(RT_RAY_BAD_NODE);
      const uint4 h0 = __ldg(v.blob + (hdr >> 4));
      const uint64_t broot = hdr + ((uint64_t)h0.x | ((uint64_t)h0.y << 32));
      hdr_unit = (uint32_t)(hdr >> 6);
      next = (uint32_t)(broot >> 6) << kShift;
    }
    record(hdr_unit, rtf::TX_STRUCTURE);
    if constexpr (TREELET) {
      // visited next from the stack its route bit names: cu is popped first,
      // and ot only when cu is empty
      const uint32_t route = rec ? head.w & 0xffffu : __ldg(v.route + unit);
      const bool same = (route >> (kRouteInst + (from_cu ? 0u : 1u))) & 1u;
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
    if (TRACED && a.ids) {  // the ids of the ray's visits, read back from its row
      __syncwarp(mask);
      const uint32_t m = min(n_tx, a.cap);
      const uint64_t row = (uint64_t)r * a.cap;
#pragma unroll 4
      for (uint32_t k = j; k < m; k += kGroup) a.ids[row + k] = __ldg(&v.meta[a.rows[row + k] >> 3].x);
    }
    if (j == 0) {
      const bool bad = flags & (RT_RAY_STACK_OVERFLOW | RT_RAY_BAD_NODE);
      write_hit(a, v, r, !bad && (min_thit < tmax), min_thit, O, D, tmin, tmax, c_leaf, c_inst, c_tobj, n_tx,
                flags & kRayStatusMask);
    }
  }
};

// rays r = group index, + groups of the launch, ...; dynamic shared memory:
// the pinned image (STAGED), then group_stack_bytes per group of the CTA.
template <bool TREELET, bool TRACED, bool STAGED = false>
__global__ void __launch_bounds__(kGroupThreads) trace_group_kernel(TraceArgs a, uint32_t depth, uint32_t rpw) {
  using W = GroupWalk<TREELET, TRACED, STAGED>;
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  __shared__ uint64_t pin_bar;
  __shared__ uint32_t pin_ok;
  uint8_t* const smem0 = dyn_smem + ((128u - (smem_u32(dyn_smem) & 127u)) & 127u);
  if (STAGED) {  // as trace_staged_kernel
    if (threadIdx.x == 0) {
      pin_ok = 0;
      if (a.pin_bytes) {
        mbar_init(&pin_bar, 1);
        mbar_expect_tx(&pin_bar, a.pin_bytes);
        for (uint32_t off = 0; off < a.pin_bytes; off += kPinChunk)
          bulk_copy_g2s(smem0 + off, reinterpret_cast<const uint8_t*>(a.pin_image) + off,
                        min(kPinChunk, a.pin_bytes - off), &pin_bar);
        pin_ok = mbar_wait(&pin_bar, 0, a.wait_tries) ? 1u : 0u;
        if (!pin_ok) atomicOr(a.status, kStatusTimeout);
      }
    }
    __syncthreads();
  }
  const uint32_t lane = threadIdx.x & 31u, g = lane / kGroup, warps = blockDim.x / 32u;
  if (g >= rpw) return;
  const uint32_t slot = (threadIdx.x >> 5) * rpw + g;
  uint8_t* const mine = smem0 + (STAGED ? a.pin_bytes : 0u) + slot * group_stack_bytes(TREELET, depth);
  typename W::Entry* stack = reinterpret_cast<typename W::Entry*>(mine);
  W w{a,
      scene_of<false>(a, 0),
      lane % kGroup,
      0xffu << (g * kGroup),
      (int)depth,
      stack,
      stack + depth + kStackPad,
      smem_u32(mine) + group_stack_bytes(TREELET, depth) - 16u,
      STAGED && pin_ok ? smem_u32(smem0) : 0u,
      STAGED && pin_ok ? a.pin_root : 0u};
  w.smem_reads = w.gmem_reads = 0;
  unsigned long long bytes = 0;
  for (uint32_t r = blockIdx.x * warps * rpw + slot; r < a.n; r += gridDim.x * warps * rpw) {
    w.run(r);
    bytes += 64ull * w.n_tx + (unsigned long long)(8ll * w.extra);
    __syncwarp(w.mask);
  }
  rtd::touch_l1_done();
  // a pinned image still in flight must land before the CTA's shared memory goes away
  if (STAGED && threadIdx.x == 0 && a.pin_bytes && !pin_ok) {
    if (!mbar_wait(&pin_bar, 0, kWaitTries)) atomicOr(a.status, kStatusTimeout);
  }
  if (a.stats && lane % kGroup == 0 && bytes) {
    atomicAdd(a.stats + ST_NODE_BYTES, bytes);
    if (STAGED) {
      atomicAdd(a.stats + ST_SMEM_READS, (unsigned long long)w.smem_reads);
      atomicAdd(a.stats + ST_GMEM_READS, (unsigned long long)w.gmem_reads);
    }
  }
  if (STAGED && a.stats && threadIdx.x == 0 && pin_ok && blockIdx.x == 0) {
    // the pinned image counts once as staged bytes (copied by every CTA)
    atomicAdd(a.stats + ST_STAGED_BYTES, (unsigned long long)a.pin_bytes * gridDim.x);
    atomicAdd(a.stats + ST_STAGINGS, (unsigned long long)gridDim.x);
  }
}

}  // namespace rtk
