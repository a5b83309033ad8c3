// Treelet-ordered traversal (traceRayWithTreelets, vulkan_ray_tracing.cc:1522-2307)
// and its shared-memory staged variant.
#pragma once
#include "pinned.h"
#include "trace_kernels.cuh"

namespace rtk {

constexpr uint32_t kSlotBitsDev = 10;
// Stack entry of the treelet-ordered walk, low word:
//   unit << 3 | top | leaf          node in global memory
//   soff << 3 | kEPin | top | leaf  node held as a pinned record in shared memory
// high word: the instance leaf a bottom-level node belongs to.
constexpr uint32_t kEShift = 3, kEPin = 4;
constexpr uint32_t kRouteOther = 6, kRouteInst = 12;  // route bits (treelets.h)

// A ray's treelet-ordered walk.  Two LIFO stacks as in the reference
// (push_front / pop_front on std::list, :1708-1709): `cu` holds nodes of the
// current treelet, `ot` the rest (:1821-1856).  Both live in one local array
// (cu first, then ot), so that a push goes to either with one predicated
// store instead of a branch per child.  Which stack a child goes to
// is read from the per-node route bits (treelets.h): a node popped from `cu`
// is in the current treelet, and a node popped from `ot` becomes the current
// treelet root, so the reference's addrToTreeletID comparison is fixed per
// node and precomputed.  The staged location of a node (dense treelet << 10 |
// 64-byte slot in that treelet's image) is read from the node table when a
// warp has a staged slot; pinned nodes are named by their record.
//
// Fields a step rarely needs live in the tail of the stack array, in local
// memory, instead of registers (kColdWords 64-bit words): the world ray, read
// when the walk comes back to a top-level node or enters an instance, and the
// closest hit.  The trace rows are found from the ray index, which the
// kernel's loop holds anyway.
constexpr int kColdWords = 6;

// SLAB = true keeps the other-treelet stack in a per-ray slab of global
// memory (`ot`, CAP entries) instead of the local array, so that a ray can
// stop between treelets and go on later in another thread: the treelet-queued
// walk (trace_queued.cuh).  The local array then holds only the current
// stack and the cold tail.
// TRACED = false compiles the walk of a launch without traces (no trace code
// at all), TOUCH = false one that fetches no pushed node ahead (touch_node).
template <int CAP, bool STAGED, bool MULTI, bool SLAB = false, bool TRACED = true, bool TOUCH = true>
struct Walker {
  // local array: cu, ot (unless SLAB), each with room for the entries a visit
  // may push before its depths are checked, then the cold words
  static constexpr int kOt = CAP + kStackPad, kCold = SLAB ? kOt : kOt + CAP + kStackPad;
  static constexpr int kWords = kCold + kColdWords;
  RayCtx cx;
  float tmin, tmax, min_thit;
  uint32_t flags;
  unsigned long long* stk;  // kWords entries, a local array of the kernel
  unsigned long long* ot;   // SLAB: the ray's other-treelet stack in global memory
  int ncu, not_;            // entries on cu and on ot
  // The entry popped (`popped` != 0) and visited next, or the top of `cu` when
  // the previous node visit pushed it, kept in a register instead of a
  // local-memory round trip (0 = none; no stack entry is 0, a blob's unit 0 is
  // its TLAS header).
  unsigned long long e;
  uint32_t popped;  // 0 no, else 1 + which route bits apply: kPopCu from cu, kPopOt from ot (:1748-1754)
  static constexpr uint32_t kPopCu = 1u, kPopOt = 2u;
  uint32_t n_tx;  // the ray's transactions
  int extra;      // the thread's byte difference (kInstanceExtra)
  SceneView v;
  uint32_t smem_reads, gmem_reads;  // the thread's node reads (staged walks)
  uint32_t pin_base;  // shared address of the pinned records, 0 = none
  uint32_t pin_root;  // record of the TLAS root node, 0 = not pinned

  __device__ __forceinline__ bool active() const { return (ncu | not_) != 0; }

  __device__ __forceinline__ void clear() {
    e = 0;
    popped = 0;
    ncu = not_ = 0;
  }

  // The next node to visit into e; false when the walk is over.
  __device__ __forceinline__ bool pop(const TraceArgs&) {
    if (popped) return true;
    if ((ncu | not_) == 0) return false;
    const bool from_cu = ncu > 0;
    if (!e) e = SLAB ? (from_cu ? stk[ncu - 1] : ot[not_ - 1]) : stk[from_cu ? ncu - 1 : kOt + not_ - 1];
    ncu -= from_cu ? 1 : 0;
    not_ -= from_cu ? 0 : 1;
    popped = from_cu ? kPopCu : kPopOt;
    return true;
  }
  // Kinds of the popped entry: a bottom-level node of another instance than
  // the one whose ray is held is an entry first.
  __device__ __forceinline__ bool other_inst() const {
    return !((uint32_t)e & kTop) && (uint32_t)(e >> 32) != cx.unit;
  }
  __device__ __forceinline__ bool at_internal() const { return !((uint32_t)e & kLeaf) && !other_inst(); }
  __device__ __forceinline__ bool at_leaf() const { return ((uint32_t)e & (kLeaf | kTop)) == kLeaf && !other_inst(); }
  __device__ __forceinline__ bool at_entry() const {
    return ((uint32_t)e & (kLeaf | kTop)) == (kLeaf | kTop) || other_inst();
  }

  // ---- the cold words
  __device__ __forceinline__ unsigned long long& cold(int k) const { return stk[kCold + k]; }
  // ---- entry i of the other-treelet stack
  __device__ __forceinline__ unsigned long long& ot_at(int i) const { return SLAB ? ot[i] : stk[kOt + i]; }
  static __device__ __forceinline__ unsigned long long pack(float a, float b) {
    return (unsigned long long)__float_as_uint(a) | ((unsigned long long)__float_as_uint(b) << 32);
  }
  static __device__ __forceinline__ float lo(unsigned long long w) { return __uint_as_float((uint32_t)w); }
  static __device__ __forceinline__ float hi(unsigned long long w) { return __uint_as_float((uint32_t)(w >> 32)); }
  __device__ __forceinline__ void set_world(rtm::V3 o, rtm::V3 d, rtm::V3 id) {
    cold(0) = pack(d.x, d.y);
    reinterpret_cast<uint32_t*>(&cold(1))[0] = __float_as_uint(d.z);
    cold(3) = pack(o.x, o.y);
    cold(4) = pack(o.z, id.x);
    cold(5) = pack(id.y, id.z);
  }
  __device__ __forceinline__ rtm::V3 dir() const {
    const unsigned long long a = cold(0), b = cold(1);
    return rtm::v3(lo(a), hi(a), lo(b));
  }
  __device__ __forceinline__ rtm::V3 world_o() const {
    const unsigned long long a = cold(3), b = cold(4);
    return rtm::v3(lo(a), hi(a), lo(b));
  }
  __device__ __forceinline__ rtm::V3 world_idir() const {
    const unsigned long long b = cold(4), c = cold(5);
    return rtm::v3(hi(b), lo(c), hi(c));
  }
  // the closest hit: word 2 its leaf and instance, the high half of word 1 its object-space t
  __device__ __forceinline__ void set_hit(uint32_t leaf, uint32_t inst, float tobj) {
    cold(2) = (unsigned long long)leaf | ((unsigned long long)inst << 32);
    reinterpret_cast<uint32_t*>(&cold(1))[1] = __float_as_uint(tobj);
  }
  // The world ray as the ray tested with (RayCtx).
  __device__ __forceinline__ void world() {
    cx.unit = kNone;
    cx.o = world_o();
    cx.idir = world_idir();
    cx.mult = 1.0f;
    cx.fast = (flags & kRayWorldFast) != 0;
  }
  // one visit of the trace (the reference's MemoryTransactionRecord)
  __device__ __forceinline__ void record(const TraceArgs& a, uint32_t r, uint32_t unit, uint32_t type) {
    if (TRACED && n_tx < a.cap) trace_put(a, r, n_tx, a.rows_tl ? v.meta[unit].x : rtf::pack_visit(unit, type));
    n_tx++;
  }

  // Staged location (dense treelet << 10 | slot) of the node the ray visits
  // next, i.e. its first pending access; kNone for a pinned node.
  __device__ __forceinline__ uint32_t next_loc() const {
    unsigned long long x = e;  // popped, or the cached top of cu
    if (!x) {
      if (ncu > 0) x = stk[ncu - 1];
      else if (not_ > 0) x = ot_at(not_ - 1);
      else return kNone;
    }
    if ((uint32_t)x & kEPin) return kNone;
    const uint32_t unit = (uint32_t)x >> kEShift;
    return unit < v.n_units ? __ldg(reinterpret_cast<const uint32_t*>(v.meta) + 2ull * unit + 1) : kNone;
  }

  // Pushes an entry onto cu (same treelet; it becomes e too) or ot.  Depths
  // are checked once per visit (too_deep); a slab has no room past CAP, so an
  // entry beyond it is not written (the ray is flagged and its stacks cleared).
  __device__ __forceinline__ void push(bool same, uint32_t code, uint32_t inst) {
    const unsigned long long x = (unsigned long long)code | ((unsigned long long)inst << 32);
    if (SLAB) {
      if (same || not_ < CAP) *(same ? stk + ncu : ot + not_) = x;
    } else {
      stk[same ? ncu : kOt + not_] = x;
    }
    ncu += same ? 1 : 0;
    not_ += same ? 0 : 1;
    e = same ? x : e;
  }
  // CAP entries per stack, one more on cu for the entry held in e
  __device__ __forceinline__ bool too_deep() const { return ncu > CAP + 1 || not_ > CAP; }

  __device__ __forceinline__ void bad_node() {
    flags |= RT_RAY_BAD_NODE;
    clear();
  }

  __device__ __forceinline__ void init(const TraceArgs& a, uint32_t r) {
    v = scene_of<MULTI>(a, r);
    rtm::V3 o, D;
    load_ray(a.rays, r, o, tmin, D, tmax);
    const uint32_t f = a.flags ? a.flags[r] : a.default_flags;
    flags = f & rtf::RAY_FLAG_TERMINATE_ON_FIRST_HIT ? kRayTerminate : 0u;
    n_tx = 0;
    clear();
    min_thit = tmax;
    const rtm::V3 id = rtm::calculate_idir(D);
    set_world(o, D, id);
    set_hit(0, 0, 0.0f);
    if (rtd::finite_ray(o, D, tmin, tmax)) flags |= kRayWorldFast;
    world();
    record(a, r, 0, rtf::TX_STRUCTURE);
    const uint4 h0 = __ldg(v.blob), h1 = __ldg(v.blob + 1);
    const uint64_t root_off = (uint64_t)h0.x | ((uint64_t)h0.y << 32);
    const rtm::V3 bmin = rtm::v3(__uint_as_float(h0.z), __uint_as_float(h0.w), __uint_as_float(h1.x));
    const rtm::V3 bmax = rtm::v3(__uint_as_float(h1.y), __uint_as_float(h1.z), __uint_as_float(h1.w));
    float th;
    if (rtm::ray_box_test(bmin, bmax, id, o, tmin, tmax, th)) {
      // current_treelet_root starts as the TLAS header, unit 0 (:1707)
      const uint32_t code = ((uint32_t)(root_off >> 6) << kEShift) | kTop;
      const uint32_t unit = code >> kEShift;
      const uint32_t root = unit < v.n_units ? __ldg(&v.meta[unit].x) : kNone;
      push(root == 0u, pin_root ? ((pin_root << kEShift) | kEPin | kTop) : code, 0);
    }
  }

  // ---- the treelet-queued walk (SLAB): a ray's state between two treelets,
  // 64 bytes: the ray (origin, tmin, direction, tmax), then min_thit, status
  // (bit 31: terminate on first hit), transactions, a spare word, the
  // closest leaf, its instance, its object-space t, and the other-treelet
  // stack's size.  The current-treelet stack is empty between treelets.
  static constexpr uint32_t kTerminateBit = 0x80000000u;

  __device__ __forceinline__ void save_ray(uint4* st) const {
    const rtm::V3 o = world_o(), d = dir();
    st[0] = make_uint4(__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), __float_as_uint(tmin));
    st[1] = make_uint4(__float_as_uint(d.x), __float_as_uint(d.y), __float_as_uint(d.z), __float_as_uint(tmax));
  }

  __device__ __forceinline__ void suspend(uint4* st) const {
    const unsigned long long h = cold(2);
    st[2] = make_uint4(__float_as_uint(min_thit),
                       (flags & kRayStatusMask) | ((flags & kRayTerminate) ? kTerminateBit : 0u), n_tx, 0u);
    st[3] = make_uint4((uint32_t)h, (uint32_t)(h >> 32), (uint32_t)(cold(1) >> 32), (uint32_t)not_);
  }

  __device__ __forceinline__ void resume(const TraceArgs& a, uint32_t r, const uint4* st) {
    v = scene_of<MULTI>(a, r);
    const uint4 q0 = st[0], q1 = st[1], q2 = st[2], q3 = st[3];
    const rtm::V3 o = rtm::v3(__uint_as_float(q0.x), __uint_as_float(q0.y), __uint_as_float(q0.z));
    const rtm::V3 D = rtm::v3(__uint_as_float(q1.x), __uint_as_float(q1.y), __uint_as_float(q1.z));
    tmin = __uint_as_float(q0.w);
    tmax = __uint_as_float(q1.w);
    min_thit = __uint_as_float(q2.x);
    flags = (q2.y & kRayStatusMask) | ((q2.y & kTerminateBit) ? kRayTerminate : 0u);
    n_tx = q2.z;
    set_world(o, D, rtm::calculate_idir(D));
    set_hit(q3.x, q3.y, __uint_as_float(q3.z));
    clear();
    not_ = (int)q3.w;
    if (rtd::finite_ray(o, D, tmin, tmax)) flags |= kRayWorldFast;
    world();
  }

  // True while the walk is inside its current treelet: the next pop would
  // come from the current-treelet stack.
  __device__ __forceinline__ bool in_treelet() const { return ncu > 0; }

  // Where a popped node is: its unit, and the address of its pinned record or
  // staged copy in shared memory (`lookup(unit, units, meta)`: a node of so
  // many units that lies whole in a warp slot), 0 when it is read from `from`
  // (the walk nodes or the blob).
  // Loads its first 64 bytes (or the whole pinned record of an instance leaf).
  // False, and the ray stopped, when it lies outside the blob.
  template <class Lookup>
  __device__ __forceinline__ bool load(const uint4* from, uint32_t code, uint32_t units, const Lookup& lookup,
                                       uint32_t& unit, uint32_t& saddr, rtd::Node64& nd) {
    saddr = 0;
    if (STAGED && (code & kEPin)) {
      saddr = pin_base + (code >> kEShift) * 16u;
      unit = rtd::ld_shared_u32(saddr + ((code & kLeaf) ? 0u : rtp::IN_UNIT));
      ++smem_reads;
    } else {
      unit = code >> kEShift;
      if (unit + units > v.n_units) {
        bad_node();
        return false;
      }
      if (STAGED) {
        saddr = lookup(unit, units, v.meta);
        if (saddr) ++smem_reads;
        else ++gmem_reads;
      }
    }
    const uint4* src = from + (uint64_t)unit * 4;
    if (STAGED) {
      // one generic load for lanes reading shared memory and lanes reading
      // global memory, instead of both load paths for a mixed warp
      if (saddr) src = reinterpret_cast<const uint4*>(__cvta_shared_to_generic(saddr));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint4 w = src[k];
        nd.w[4 * k + 0] = w.x;
        nd.w[4 * k + 1] = w.y;
        nd.w[4 * k + 2] = w.z;
        nd.w[4 * k + 3] = w.w;
      }
    } else {
      rtd::load64(src, nd);
    }
    return true;
  }

  // internal node, top (:1758-1869) or bottom (:1954-2070)
  template <class Lookup>
  __device__ __forceinline__ void internal(const TraceArgs& a, uint32_t r, const Lookup& lookup) {
    const uint32_t code = (uint32_t)e, inst = (uint32_t)(e >> 32), level = code & kTop;
    // which route bits apply
    const uint32_t shift = popped == kPopCu ? rtw::kSameShift : rtw::kOtherShift;
    const bool pinned = STAGED && (code & kEPin);
    uint32_t unit, saddr;
    rtd::Node64 nd;
    if (!load(v.walk, code, 1, lookup, unit, saddr, nd)) return;
    if (STAGED && Lookup::kSlots && saddr && !pinned) {  // a warp slot holds the blob's bytes
      uint32_t raw[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) raw[k] = nd.w[k];
      rtw::walk_node(raw, unit, v.n_units, __ldg(v.route + unit), nd.w);
    }
    e = 0;
    popped = 0;
    if (level && cx.unit != kNone) world();
    record(a, r, unit, rtf::TX_INTERNAL);
    const float t0 = tmin * cx.mult, t1 = tmax * cx.mult, cull = min_thit * cx.mult;
    uint32_t hit = cx.fast && !(nd.w[5] & rtw::kExact)
                       ? rtd::hit_children(nd, cx.o, cx.idir, t0, t1, cull)
                       : rtd::hit_children_exact(v.raw + (uint64_t)unit * 4, cx.o, cx.idir, t0, t1, cull);
    // 1.2 hits a visit: a loop over the bits is shorter than six predicated
    // pushes (2M any-hit rays 1.64 against 1.70 ms on a GB300)
#pragma unroll 1
    for (; hit; hit &= hit - 1u) {
      const int i = __ffs(hit) - 1;
      const uint32_t lf = (nd.w[5] >> (i + rtw::kLeafShift)) & kLeaf;
      uint32_t so = 0;  // a pinned parent names its pinned children's records
      if (pinned) so = rtd::ld_shared_u16(saddr + rtp::IN_CHILD_SOFF + 2u * i);
      const uint32_t c = nd.w[3] + ((nd.w[6] >> (4 * i)) & 15u);
      push((nd.w[5] >> (shift + i)) & 1u, (so ? (so << kEShift) | kEPin : c << kEShift) | level | lf, inst);
      if (TOUCH && !so) touch_node(v.walk, c);
    }
    check_depth();
  }

  // primitive leaf (:2071-2196)
  template <class Lookup>
  __device__ __forceinline__ void leaf(const TraceArgs& a, uint32_t r, const Lookup& lookup) {
    uint32_t unit, saddr;
    rtd::Node64 q;
    if (!load(v.blob, (uint32_t)e, 1, lookup, unit, saddr, q)) return;
    e = 0;
    popped = 0;
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
        if (tmin <= wt && wt <= tmax && wt < min_thit) {  // :2127-2141
          min_thit = wt;
          set_hit(unit, cx.unit, t);
          type = rtf::TX_QUAD_LEAF_HIT;
          if (flags & kRayTerminate) clear();
        }
      }
    } else {
      flags |= RT_RAY_HIT_PROCEDURAL;
    }
    record(a, r, unit, type);
  }

  // The ray context for the popped entry: an instance leaf (:1870-1953)
  // enters its own instance; a BLAS node's instance is entered again when the
  // walk comes back to it from another instance's nodes or from the TLAS
  // (make_transformed_ray is deterministic, so recomputing gives the
  // reference's stored objectRay), and the node itself stays popped.
  template <class Lookup>
  __device__ __forceinline__ void entry(const TraceArgs& a, uint32_t r, const Lookup& lookup) {
    const uint32_t code = (uint32_t)e;
    const bool top = code & kTop, pinned = STAGED && (code & kEPin);
    rtd::Instance in;
    rtd::Node64 nd;
    uint32_t unit = (uint32_t)(e >> 32), saddr = 0;
    if (top) {
      if (!load(v.blob, code, 2, lookup, unit, saddr, nd)) return;
      if (pinned) {
#pragma unroll
        for (int k = 0; k < 12; ++k) in.w2o.m[k / 3][k % 3] = __uint_as_float(nd.w[rtp::IL_W2O / 4 + k]);
      } else {
        rtd::instance_from(nd, v.blob + (uint64_t)unit * 4, saddr, in);
      }
    } else {
      rtd::load_instance(v.blob + (uint64_t)unit * 4, in);
    }
    enter_instance(in, unit, world_o(), dir(), tmin, tmax, cx);
    if (!top) return;
    const uint32_t rsh = popped - kPopCu;
    e = 0;
    popped = 0;
    record(a, r, unit, rtf::TX_INSTANCE_LEAF);
    extra += kInstanceExtra;
    uint32_t hdr_unit, broot_unit, broot_soff = 0, rbits;
    if (pinned) {  // the 64-byte record: units, route bits, BLAS root record, rows
      hdr_unit = nd.w[rtp::IL_HDR_UNIT / 4];
      broot_unit = nd.w[rtp::IL_BROOT_UNIT / 4];
      rbits = nd.w[rtp::IL_ROUTE / 4] & 0xffffu;
      broot_soff = nd.w[rtp::IL_ROUTE / 4] >> 16;
    } else {
      rbits = __ldg(v.route + unit);
      const uint64_t hdr = (uint64_t)unit * 64 + in.bvh_address;
      if ((hdr & 63) || hdr / 64 >= v.n_units) return bad_node();
      hdr_unit = (uint32_t)(hdr >> 6);
      const uint4 h0 = __ldg(v.blob + (hdr >> 4));
      const uint64_t broot = hdr + ((uint64_t)h0.x | ((uint64_t)h0.y << 32));
      broot_unit = (uint32_t)(broot >> 6);
    }
    record(a, r, hdr_unit, rtf::TX_STRUCTURE);
    const uint32_t cc = broot_soff ? ((broot_soff << kEShift) | kEPin) : (broot_unit << kEShift);
    push((rbits >> (kRouteInst + rsh)) & 1u, cc, unit);
    check_depth();
  }

  __device__ __forceinline__ void check_depth() {
    if (too_deep()) {
      flags |= RT_RAY_STACK_OVERFLOW;
      clear();
    }
  }

  // One node visit (the caller checks active() first).
  template <class Lookup>
  __device__ __forceinline__ void step(const TraceArgs& a, uint32_t r, const Lookup& lookup) {
    pop(a);
    if (at_entry()) {
      const bool top = (uint32_t)e & kTop;
      entry(a, r, lookup);
      if (top) return;
    }
    if ((uint32_t)e & kLeaf) leaf(a, r, lookup);
    else internal(a, r, lookup);
  }

  __device__ __forceinline__ void finish(const TraceArgs& a, uint32_t r) {
    const bool bad = flags & (RT_RAY_STACK_OVERFLOW | RT_RAY_BAD_NODE);
    const unsigned long long h = cold(2);
    if (TRACED) trace_drain(a, r, min(n_tx, a.cap), v.meta);
    write_hit(a, v, r, !bad && (min_thit < tmax), min_thit, world_o(), dir(), tmin, tmax, (uint32_t)h,
              (uint32_t)(h >> 32), hi(cold(1)), n_tx, flags & kRayStatusMask);
  }
};

// The walker's stacks are a separate local array so that its fields stay in
// registers (stacks inside it would leave every field in local memory).
// 72 registers: seven 128-thread CTAs per SM.  GB300, ms for 1M traced bounce
// rays / 2M any-hit rays: 2.36 / 1.64; 64 registers (eight CTAs) 2.44 / 1.64,
// 56 2.51 / 1.67, 85 2.49 / 1.76.  A batch's walk, which looks its scene up per
// ray, spills at 72: 48 scenes in one launch 0.69 ms, at 80 0.65.
constexpr int kTreeletRegs = 72, kTreeletBatchRegs = 80;

template <int CAP, bool MULTI, bool TRACED>
__global__ void __maxnreg__(MULTI ? kTreeletBatchRegs : kTreeletRegs) trace_treelet_kernel(TraceArgs a) {
  using W = Walker<CAP, false, MULTI, false, TRACED>;
  unsigned long long stack[W::kWords];
  W w;
  w.stk = stack;
  w.extra = 0;
  w.pin_base = 0;
  w.pin_root = 0;
  unsigned long long bytes = 0;
  run_persistent(a, w, bytes);
  rtd::touch_l1_done();
  if (a.stats) add_warp_total64(a.stats + ST_NODE_BYTES, bytes);
}

// ------------------------------------------------------------------ staged

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// One non-blocking probe of the phase with the given parity.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait for the phase with the given parity; false if it gave up.
// The first of the max_tries probes does not block (test_wait), the others
// may suspend the thread for a while each (try_wait).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t max_tries) {
  const uint32_t addr = smem_u32(bar);
  if (max_tries == 0) return false;
  if (mbar_test(bar, parity)) return true;
  for (uint32_t i = 1; i < max_tries; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Global -> shared bulk copy completing on `bar`.  The fence orders this
// thread's earlier generic-proxy accesses before the async-proxy writes.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// A lookup of nodes staged in warp slots (Walker::load).
template <class F>
struct SlotLookup {
  static constexpr bool kSlots = true;
  F f;
  __device__ __forceinline__ uint32_t operator()(uint32_t unit, uint32_t units, const uint2* meta) const {
    return f(unit, units, meta);
  }
};
template <class F>
__device__ __forceinline__ SlotLookup<F> slot_lookup(F f) {
  return SlotLookup<F>{f};
}

constexpr int kMaxSlots = 8;  // slots per warp
constexpr uint32_t kWaitTries = 1u << 22;
// 256-thread CTAs per SM: three at 80 registers; four at 64 spill 96 bytes.  GB300,
// us, three / four:
//                                     131,769    313,600    1,000,000    2,097,152
//   2M-tri terrain, primary                      530 / 565  1122 / 1170  2152 / 2158
//   the same, bounce                             865 / 949  2021 / 2041  3886 / 3845
//   131K-tri terrain, bounce          601 / 675  827 / 899  1939 / 1961
//   1M-tri blobs, bounce                                    797 / 856    1002 / 1055
//   2,000-tri cube and plane, bounce  87 / 115   105 / 123  (810,000 rays: 164 / 177)
// and traced: 1M bounce rays of the 2M-triangle terrain 2423 / 2528.  With one slot a
// warp: 2,013 bounce rays of the terrain 581 / 641, 307,200 primary rays 713 / 826, of the
// blobs 527 / 548, 2M primary rays of the terrain 2848 / 3229.  Large launches of any-hit
// rays, which end early and are taken at once, run four (kStagedAnyHitRays).
constexpr int kStagedMaxThreads = 256;
constexpr int kStagedMinBlocks = 3, kStagedAnyHitMinBlocks = 4;
constexpr uint32_t kPinChunk = 32768;  // bytes per bulk copy of the pinned image

// Per-warp staging state in shared memory.
struct WarpStage {
  uint64_t bar;
  uint32_t resident[kMaxSlots];  // dense treelet id per slot, or kNone
  uint32_t units[kMaxSlots];     // 64-byte units of that treelet held in the slot
  uint32_t pending_slot, pending_id, pending_units, phase, victim, disabled;
};

// Whether the calling warp's 32 rays, just taken, leave one point within a
// narrow cone of the first (kCone: cosine squared, 3 degrees), as a camera's
// neighbouring rays do.  GB300, 1M primary rays staged, tiles of 8 x 4 pixels a
// warp, us waiting / refilling (kTogetherRays), for frames whose tiles are ever
// narrower:
//                    32 x 32      64 x 64      128 x 128    192 x 192    256 x 256    512 x 512    1024 x 1024
//   2M-tri terrain   2033 / 1682  1813 / 1644  1607 / 1616  1489 / 1562  1460 / 1557  1319 / 1461  1166 / 1314
//   1M-tri blobs     932 / 651    782 / 640    697 / 636    654 / 620    652 / 624    623 / 613    596 / 602
// A 192 x 192 frame's tile is 2.6 degrees across, a 128 x 128 frame's 3.9: from there on
// waiting gains more on the one than it loses on the other.  The same camera's rays in
// random order 2603 / 1758 and 1566 / 679.
constexpr float kCone = 0.9973f;

__device__ __forceinline__ bool rays_together(rtm::V3 o, rtm::V3 d) {
  const float ox = __shfl_sync(0xffffffffu, o.x, 0), oy = __shfl_sync(0xffffffffu, o.y, 0);
  const float oz = __shfl_sync(0xffffffffu, o.z, 0), dx = __shfl_sync(0xffffffffu, d.x, 0);
  const float dy = __shfl_sync(0xffffffffu, d.y, 0), dz = __shfl_sync(0xffffffffu, d.z, 0);
  const float dot = d.x * dx + d.y * dy + d.z * dz;
  const float len = (d.x * d.x + d.y * d.y + d.z * d.z) * (dx * dx + dy * dy + dz * dz);
  return __all_sync(0xffffffffu, o.x == ox && o.y == oy && o.z == oz && dot > 0.0f && dot * dot >= kCone * len);
}

// Rays from which on a staged launch waits for the last ray of a warp whose rays
// are together, to take 32 neighbours again: neighbours walk the same nodes, and a
// ray taken alone walks beside rays that are far ahead.  GB300, primary rays,
// waiting / refilling at 8 idle lanes, us: 2M-triangle terrain 537,600 rays 711 / 752,
// 1M 1166 / 1314, 2M (two a pixel) 2230 / 2567, 4M 4360 / 5068; traced 1473 / 1622 at
// 1M; 1M-triangle blobs 433 / 428, 596 / 602, 937 / 949, 1676 / 1677.  At 307,200
// rays, three per lane of the chip, the warps' uneven ends cost what it gains (terrain
// 501 / 516, blobs 354 / 339).  Bounce rays: 2101 / 2086 us at 1M, 3920 / 3899 at 2M.  The unstaged treelet
// walk gains as much on such rays but pays 0.4% on all others for the check,
// and the plain walk gains nothing (1036 / 1025): neither does it.
constexpr uint32_t kTogetherRays = 1u << 19;

// The staged walk.  Persistent warps with ray refill (as run_persistent).
//
// Pinned treelets: at launch each CTA copies the pinned image (the treelets
// most rays visit, decoded into records, pinned.h) into shared memory with
// cp.async.bulk and keeps it for the whole launch; every node read that names
// a record is served from it.
//
// Warp slots: every `epoch` visits (of all its lanes that are at a node of the
// kind visited, one step each) a warp votes: each lane names the treelet of its
// next access, __match_any_sync counts equal names, and the most popular treelet
// that is not resident (ties to the lowest treelet, i.e. the lowest root address,
// as the RT unit's decision in shader.cc:3424-3441) is copied with cp.async.bulk
// into the warp's least recently filled slot, provided at least `min_votes` lanes
// want it.  A slot holds the first
// slot_bytes of the treelet's image (the whole image when it fits).  Node
// reads that fall in a resident slot are served from shared memory.  A slot
// is read only by its own warp; __syncwarp orders the slot's reads before it
// is refilled.  SLOTS = false compiles the warp slots out (a.slots == 0).
template <int CAP, bool SLOTS, bool TRACED, int MIN_BLOCKS = kStagedMinBlocks>
__global__ void __launch_bounds__(kStagedMaxThreads, MIN_BLOCKS) trace_staged_kernel(TraceArgs a) {
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  __shared__ WarpStage ws[kStagedMaxThreads / 32];
  __shared__ uint64_t pin_bar;
  __shared__ uint32_t pin_ok;
  uint8_t* const smem0 = dyn_smem + ((128u - (smem_u32(dyn_smem) & 127u)) & 127u);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t slots = a.slots;
  uint8_t* const my_slots = smem0 + a.pin_bytes + (size_t)warp * slots * a.slot_bytes;
  const uint32_t slot_base = smem_u32(my_slots);
  WarpStage& st = ws[warp];
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
  if (lane == 0) {
    mbar_init(&st.bar, 1);
    for (int s = 0; s < kMaxSlots; ++s) {
      st.resident[s] = kNone;
      st.units[s] = 0;
    }
    st.pending_slot = kNone;
    st.pending_id = kNone;
    st.pending_units = 0;
    st.phase = 0;
    st.victim = 0;
    st.disabled = 0;
  }
  __syncthreads();
  // the node's location is read only while some slot of the warp is resident
  const auto lookup = slot_lookup([&](uint32_t unit, uint32_t units, const uint2* meta) -> uint32_t {
    bool any = false;
    for (uint32_t s = 0; s < slots; ++s) any |= st.resident[s] != kNone;
    if (!any) return 0u;
    const uint32_t loc = __ldg(reinterpret_cast<const uint32_t*>(meta) + 2ull * unit + 1);
    if (loc == kNone) return 0u;
    const uint32_t d = loc >> kSlotBitsDev, u = loc & ((1u << kSlotBitsDev) - 1u);
    for (uint32_t s = 0; s < slots; ++s)
      if (st.resident[s] == d && u + units <= st.units[s]) return slot_base + s * a.slot_bytes + u * 64u;
    return 0u;
  });
  using W = Walker<CAP, true, false, false, TRACED>;  // staged launches trace one scene
  unsigned long long stack[W::kWords];
  W w;
  w.stk = stack;
  w.extra = 0;
  w.smem_reads = w.gmem_reads = 0;
  w.pin_base = pin_ok ? smem_u32(smem0) : 0u;
  w.pin_root = pin_ok ? a.pin_root : 0u;
  bool have = false, ended = false;
  int spare = (int)a.refill;  // idle lanes that end a turn; 33 once no rays are left
  uint32_t r = 0, left = 0;  // left: visits of the warp until it votes
  unsigned long long bytes = 0, staged = 0, stagings = 0;
  for (;;) {
    // --- records of finished rays, then new rays for idle lanes (as run_persistent)
    const uint32_t need = __ballot_sync(0xffffffffu, !have);
    if (need == 0xffffffffu || __popc(need) >= spare) {
      if (ended) {
        w.finish(a, r);
        bytes += 64ull * w.n_tx;
        ended = false;
      }
      if (spare > 32) break;  // every lane is idle
      const int leader = __ffs(need) - 1;
      uint32_t base = 0;
      if ((int)lane == leader) base = atomicAdd(a.queue, (uint32_t)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (base + (uint32_t)__popc(need) >= a.n) spare = 33;
      if (!have) {
        const uint32_t rr = base + (uint32_t)__popc(need & ((1u << lane) - 1u));
        if (rr < a.n) {
          r = rr;
          w.init(a, r);
          have = true;
        }
      }
      if (need == 0xffffffffu && spare <= 32 && a.n >= kTogetherRays)
        spare = rays_together(w.cx.o, w.dir()) ? 32 : (int)a.refill;
    }
    // --- staging: land a finished copy, then vote for the next one
    if (SLOTS && left == 0) {
      left = a.epoch;
      if (lane == 0 && st.pending_slot != kNone && mbar_test(&st.bar, st.phase)) {
        st.resident[st.pending_slot] = st.pending_id;
        st.units[st.pending_slot] = st.pending_units;
        st.phase ^= 1u;
        st.pending_slot = kNone;
      }
      __syncwarp();
      if (st.pending_slot == kNone && !st.disabled) {
        const uint32_t nl = have ? w.next_loc() : kNone;
        uint32_t key = nl == kNone ? kNone : (nl >> kSlotBitsDev);
        if (a.hint && key != kNone) {
          // vote for the treelet predicted to follow the one the ray enters next
          const rtm::V3 wd = w.dir();
          const uint32_t oct = (wd.x > 0.0f ? 1u : 0u) | (wd.y > 0.0f ? 2u : 0u) | (wd.z > 0.0f ? 4u : 0u);
          key = __ldg(a.hint + (size_t)key * 8 + oct);
          if (key >= a.n_treelets) key = kNone;
        }
        if (key != kNone)
          for (uint32_t s = 0; s < slots; ++s)
            if (st.resident[s] == key) key = kNone;  // already resident
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        unsigned long long v =
            key == kNone ? 0ull : (((unsigned long long)__popc(peers) << 32) | (unsigned long long)(~key));
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, s);
          v = o > v ? o : v;
        }
        const uint32_t votes = (uint32_t)(v >> 32);
        if (votes > 0 && votes >= a.min_votes && lane == 0) {
          const uint32_t d = ~(uint32_t)(v & 0xffffffffu);
          const unsigned long long off = a.image_off[d];
          uint32_t nb = (uint32_t)(a.image_off[d + 1] - off);
          if (nb > a.slot_bytes) nb = a.slot_bytes;
          if (nb > 0) {
            const uint32_t s = st.victim;
            st.victim = (s + 1 == slots) ? 0 : s + 1;
            st.resident[s] = kNone;
            st.units[s] = 0;
            mbar_expect_tx(&st.bar, nb);
            bulk_copy_g2s(my_slots + (size_t)s * a.slot_bytes, reinterpret_cast<const uint8_t*>(a.images) + off, nb,
                          &st.bar);
            st.pending_slot = s;
            st.pending_id = d;
            st.pending_units = nb / 64u;
            staged += nb;
            stagings += 1;
          }
        }
      }
      __syncwarp();
    }
    // --- node visits
    if (SLOTS) warp_turn(a, w, r, have, ended, spare, lookup, left);
    else warp_turn(a, w, r, have, ended, spare, NoLookup(), left);
  }
  rtd::touch_l1_done();
  // copies still in flight must land before the CTA's shared memory goes away
  if (lane == 0 && st.pending_slot != kNone) {
    if (!mbar_wait(&st.bar, st.phase, kWaitTries)) atomicOr(a.status, kStatusTimeout);
  }
  if (threadIdx.x == 0 && a.pin_bytes && !pin_ok) {
    if (!mbar_wait(&pin_bar, 0, kWaitTries)) atomicOr(a.status, kStatusTimeout);
  }
  __syncwarp();
  if (a.stats) {
    add_warp_total64(a.stats + ST_NODE_BYTES, bytes + (unsigned long long)(8ll * w.extra));
    add_warp_total64(a.stats + ST_SMEM_READS, w.smem_reads);
    add_warp_total64(a.stats + ST_GMEM_READS, w.gmem_reads);
    add_warp_total64(a.stats + ST_STAGED_BYTES, staged);
    add_warp_total64(a.stats + ST_STAGINGS, stagings);
  }
  if (a.stats && threadIdx.x == 0 && pin_ok && blockIdx.x == 0) {
    // the pinned image counts once as staged bytes (copied by every CTA)
    atomicAdd(a.stats + ST_STAGED_BYTES, (unsigned long long)a.pin_bytes * gridDim.x);
    atomicAdd(a.stats + ST_STAGINGS, (unsigned long long)gridDim.x);
  }
}

}  // namespace rtk
