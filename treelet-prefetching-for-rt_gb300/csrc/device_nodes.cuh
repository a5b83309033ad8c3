// Device-side node access: 32-byte vector loads of the 64 / 128-byte nodes
// from global memory (read-only path) or from a staged shared-memory image,
// and the decoders for the fields the walk uses (format.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "format.h"
#include "rtmath.h"
#include "walk_node.h"

namespace rtd {

// Raw node words.  Internal nodes and quad leaves use 16 words (64 B).
struct Node64 {
  uint32_t w[16];
};

__device__ __forceinline__ uint4 ld_global_nc(const uint4* p) { return __ldg(p); }

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr));
  return v;
}

__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t saddr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
  return v;
}

__device__ __forceinline__ uint32_t ld_shared_u16(uint32_t saddr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(saddr));
  return v;
}

// Brings the 32-byte sector of p into L1: a 4-byte asynchronous copy to a
// scratch word of shared memory that nobody reads.  The thread must wait for
// its copies (touch_l1_done) before it exits.
__device__ __forceinline__ void touch_l1(uint32_t scratch, const void* p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(scratch), "l"(p) : "memory");
}
__device__ __forceinline__ void touch_l1_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One 32-byte read-only load from global memory (256-bit loads exist on
// sm_100 and later, for the global state space only): a 64-byte node takes
// two load instructions instead of four.  p must be 32-byte aligned; nodes are
// 64-byte aligned in the blob.
__device__ __forceinline__ void ld_global_v8(const uint4* p, uint32_t* w) {
  asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
      : "l"(p));
}

// Loads a node's 64 bytes from global memory.
__device__ __forceinline__ void load64(const uint4* g, Node64& n) {
  ld_global_v8(g, n.w);
  ld_global_v8(g + 2, n.w + 8);
}

// 16 bytes: from shared memory when saddr != 0, else from global.
__device__ __forceinline__ uint4 load16(const uint4* g, uint32_t saddr, int q) {
  return saddr ? ld_shared_v4(saddr + 16u * q) : ld_global_nc(g + q);
}

__device__ __forceinline__ float f32_at(const Node64& n, int b) { return __uint_as_float(n.w[b >> 2]); }

// A bound's byte q becomes a float by one byte permute, which places it in the
// mantissa of 2^23, and a subtraction of 2^23 (both exact).  The child bound
// Origin + ldexpf(q, exp - 8) (asu.h:499-508) is one fused multiply-add:
// q * 2^(exp-8) is exact for an 8-bit q and exp in [-128, 127] (at most 8
// significant bits, all at or above 2^-149, below 2^127), so the reference's
// ldexpf is exact and its add is the only rounding; fmaf rounds the same exact
// sum once, giving the same bits (signed zeros included: q = 0 gives
// +0 * s + Origin either way).  --fmad=false stops only the compiler's own
// contraction, not this explicit fused operation.

// Three-input minimum / maximum (sm_100 and later): one instruction for two.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// The quantized bounds of one axis of a walk node, sorted into the plane a
// ray meets first and the other by the sign of its direction: children 0..3
// in the bytes of `near4` and `far4`, children 4 and 5 in `rest` (near 4,
// near 5, far 4, far 5).
struct AxisBytes {
  uint32_t near4, far4, rest;
  __device__ __forceinline__ uint32_t near_bits(int i) const {
    return __byte_perm(i < 4 ? near4 : rest, 0x4B000000u, (uint32_t)(i < 4 ? i : i - 4) | 0x7540u);
  }
  __device__ __forceinline__ uint32_t far_bits(int i) const {
    return __byte_perm(i < 4 ? far4 : rest, 0x4B000000u, (uint32_t)(i < 4 ? i : i - 2) | 0x7540u);
  }
};
__device__ __forceinline__ AxisBytes axis_bytes(const Node64& n, int k, float idir) {
  const uint32_t lo4 = n.w[7 + 3 * k], rest = n.w[8 + 3 * k], hi4 = n.w[9 + 3 * k];
  const bool up = idir > 0.0f;
  return AxisBytes{up ? lo4 : hi4, up ? hi4 : lo4, __byte_perm(rest, 0, up ? 0x3210u : 0x1032u)};
}

// The box tests of an internal node (vulkan_ray_tracing.cc:2518-2553 and the
// bottom-level twin :2714-2741): children with ChildSize > 0 are slab-tested
// with the ray's [tmin, tmax]; a hit at thit >= cull is dropped.  Bounds are
// Origin + ldexpf(q, exp - 8) (asu.h:499-508), slab values (b - o) * idir
// (vulkan_ray_tracing.cc:199-218), reduced as magic_max7 / magic_min7.
// Returns bit i for a hit child i.
//
// hit_children_exact reads the blob's node and uses the reference's ternary
// MIN/MAX macros in its order, for children [first, end).
__device__ __forceinline__ uint32_t hit_children_exact(const uint4* raw, rtm::V3 o, rtm::V3 idir, float tmin,
                                                       float tmax, float cull, uint32_t first = 0, uint32_t end = 6) {
  const uint8_t* b = reinterpret_cast<const uint8_t*>(raw);
  const float* org = reinterpret_cast<const float*>(raw);
  const float s[3] = {rtm::exp2_int((int)(int8_t)b[rtf::IN_EXP] - 8), rtm::exp2_int((int)(int8_t)b[rtf::IN_EXP + 1] - 8),
                      rtm::exp2_int((int)(int8_t)b[rtf::IN_EXP + 2] - 8)};
  uint32_t mask = 0;
#pragma unroll 1
  for (uint32_t i = first; i < end; ++i) {
    if (!(b[rtf::IN_CHILD_INFO + i] & 3u)) continue;
    const uint8_t* q = b + rtf::IN_LO_X + i;
    const rtm::V3 lo = rtm::v3(__fmaf_rn((float)q[0], s[0], org[0]), __fmaf_rn((float)q[12], s[1], org[1]),
                               __fmaf_rn((float)q[24], s[2], org[2]));
    const rtm::V3 hi = rtm::v3(__fmaf_rn((float)q[6], s[0], org[0]), __fmaf_rn((float)q[18], s[1], org[1]),
                               __fmaf_rn((float)q[30], s[2], org[2]));
    float tn;
    if (rtm::ray_box_test(lo, hi, idir, o, tmin, tmax, tn) && !(tn >= cull)) mask |= 1u << i;
  }
  return mask;
}

// hit_children is for a finite ray (finite_ray) and a walk node without
// kExact.  Every slab value then is one monotone function of its
// bound (two roundings, a finite nonzero idir), so the lower plane's value is
// the smaller one when idir > 0 and the larger one when idir < 0: the two
// planes are told apart once per node and axis by the sign of idir instead of
// by a minimum and a maximum per child and axis, and what is left of the
// reduction is a maximum and a minimum of four values.  Those agree with the
// ternary macros except on NaN operands (none here) and on the sign of a
// zero, which no comparison sees: the same hit / cull decisions.  The
// children's tests have no branch, so their chains overlap.  The test is
// bound by the integer / minmax pipe (63% busy in the staged walk): against
// six minima and maxima and one branch a child, 2M primary rays staged went
// from 3.29 to 3.12 ms on a GB300 and small frames gained 2-6%.
__device__ __forceinline__ uint32_t hit_children(const Node64& n, rtm::V3 o, rtm::V3 idir, float tmin, float tmax,
                                                 float cull) {
  const float ox = f32_at(n, 0), oy = f32_at(n, 4), oz = f32_at(n, 8);
  const float sx = __uint_as_float((n.w[4] << 23) & 0x7f800000u), sy = __uint_as_float((n.w[4] << 15) & 0x7f800000u),
              sz = __uint_as_float((n.w[4] << 7) & 0x7f800000u);
  const AxisBytes bx = axis_bytes(n, 0, idir.x), by = axis_bytes(n, 1, idir.y), bz = axis_bytes(n, 2, idir.z);
  // x and y in two-wide FP32, and the two z planes: the same roundings, half the instructions
  const unsigned long long s_xy = f2_pack(sx, sy), o_xy = f2_pack(ox, oy), s_z = f2_pack(sz, sz), o_z = f2_pack(oz, oz);
  const unsigned long long org_xy = f2_pack(o.x, o.y), id_xy = f2_pack(idir.x, idir.y);
  const unsigned long long org_z = f2_pack(o.z, o.z), id_z = f2_pack(idir.z, idir.z);
  const unsigned long long two23 = f2_pack(8388608.0f, 8388608.0f);
  uint32_t mask = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    // q as an exact float (bits - 2^23), Origin + q * 2^(e-8) fused, then (b - o) * idir
    auto slab = [&](uint32_t b0, uint32_t b1, unsigned long long s, unsigned long long org, unsigned long long ray_o,
                    unsigned long long ray_id, float& t0, float& t1) {
      const unsigned long long q = f2_sub(f2_pack_bits(b0, b1), two23);
      f2_unpack(f2_mul(f2_sub(f2_fma(q, s, org), ray_o), ray_id), t0, t1);
    };
    float nx, ny, nz, fx, fy, fz;
    slab(bx.near_bits(i), by.near_bits(i), s_xy, o_xy, org_xy, id_xy, nx, ny);
    slab(bx.far_bits(i), by.far_bits(i), s_xy, o_xy, org_xy, id_xy, fx, fy);
    slab(bz.near_bits(i), bz.far_bits(i), s_z, o_z, org_z, id_z, nz, fz);
    const float tn = fmaxf(max3(nx, ny, nz), tmin), tf = fminf(min3(fx, fy, fz), tmax);
    if (tn <= tf && !(tn >= cull)) mask |= 1u << i;
  }
  return mask & (n.w[5] | (n.w[5] >> rtw::kLeafShift)) & rtw::kChildMask;
}

// True when the slab test may tell planes apart by the direction's sign (hit_children).
__device__ __forceinline__ bool finite_ray(rtm::V3 o, rtm::V3 d, float tmin, float tmax) {
  return isfinite(o.x) && isfinite(o.y) && isfinite(o.z) && isfinite(d.x) && isfinite(d.y) && isfinite(d.z) &&
         !isnan(tmin) && !isnan(tmax);
}

// Instance leaf fields used by the walk.
struct Instance {
  rtm::Mat43 w2o;
  uint64_t bvh_address;
  uint32_t instance_id;
};

// The same fields when the leaf's first 64 bytes are already loaded in q:
// two more 16-byte loads (bytes 64..79 and 112..127).
__device__ __forceinline__ void instance_from(const Node64& q, const uint4* g, uint32_t saddr, Instance& in) {
  const uint4 d = load16(g, saddr, 4), e = load16(g, saddr, 7);
#pragma unroll
  for (int k = 0; k < 9; ++k) in.w2o.m[k / 3][k % 3] = __uint_as_float(q.w[4 + k]);
  in.w2o.m[3][0] = __uint_as_float(e.y);
  in.w2o.m[3][1] = __uint_as_float(e.z);
  in.w2o.m[3][2] = __uint_as_float(e.w);
  in.bvh_address = (uint64_t)d.x | ((uint64_t)d.y << 32);
  in.instance_id = d.z;
}

__device__ __forceinline__ void load_instance(const uint4* g, Instance& in) {
  const uint4 a = ld_global_nc(g + 1), b = ld_global_nc(g + 2), c = ld_global_nc(g + 3);
  const uint4 d = ld_global_nc(g + 4), e = ld_global_nc(g + 7);
  // bytes 16..51: world-to-object rows 0-2
  const uint32_t lin[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x};
#pragma unroll
  for (int k = 0; k < 9; ++k) in.w2o.m[k / 3][k % 3] = __uint_as_float(lin[k]);
  // bytes 116..127: translation row as the reference's struct-order read takes it
  in.w2o.m[3][0] = __uint_as_float(e.y);
  in.w2o.m[3][1] = __uint_as_float(e.z);
  in.w2o.m[3][2] = __uint_as_float(e.w);
  in.bvh_address = (uint64_t)d.x | ((uint64_t)d.y << 32);
  in.instance_id = d.z;
}

}  // namespace rtd
