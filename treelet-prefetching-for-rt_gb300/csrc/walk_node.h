// The walks' own form of an internal node (64 bytes, next to the blob's).
//
// The blob keeps a node as the reference lays it out: exponents, child sizes
// and types as bytes, bounds as six-byte rows, and the treelet walk's route
// bits in another table.  Every visit took them apart again, about a third of
// its instructions.  A walk node holds the same quantized box with that work
// done once, when the scene is created (and again when its treelets are formed,
// for the route bits).  GB300: 2M primary rays staged 2.81 -> 2.59 ms, 1M traced
// bounce rays in treelet order 2.63 -> 2.44 ms, 2M any-hit rays 1.73 -> 1.64 ms.
//   w0..2   origin
//   w3      unit of the first child, at most the blob's units (kPadUnits)
//   w4      bytes 0..2: the exponents of the x, y, z scales 2^(e-8) as biased
//           float exponents (e + 119)
//   w5      bits 0..5 children that are internal nodes, 6..11 children that
//           are leaves (a child of size 0 is neither), 12..17 and 18..23 the
//           route bits (treelets.h: same treelet root / the node's own),
//           bit 24: kExact
//   w6      nibble i: units from the first child to child i
//   w7..15  per axis: lower bounds of children 0..3; lower bounds of children
//           4 and 5 and upper bounds of 4 and 5; upper bounds of children 0..3
// kExact marks a node the walks must test from the blob's own bytes: a lower
// bound above its upper one, or a scale below the normal floats.
#pragma once
#include <stdint.h>

#include "format.h"

namespace rtw {

constexpr uint32_t kLeafShift = 6, kSameShift = 12, kOtherShift = 18, kExact = 1u << 24;
constexpr uint32_t kChildMask = 63u;

// The walks start a hit child's node on its way to L1 before its visit compares
// its unit with the blob's.  So that they need no comparison of their own, a
// child block that starts outside the blob is named by the unit past its end (its
// children are bad nodes either way), and the walk nodes' array is longer than the
// blob by the units that a node's children may lie past that.  (With a comparison
// a touch instead, 47K bounce rays plain took 318 us on a GB300 against 307, 2M
// any-hit rays in treelet order 1709 against 1667, 48 scenes in one launch 652
// against 640.)
constexpr uint32_t kPadUnits = 16;

// raw: the blob node's 16 words; units: the blob's; route: its route bits (0
// without treelets).
RT_HD void walk_node(const uint32_t* raw, uint32_t unit, uint32_t units, uint32_t route, uint32_t* out) {
  const uint32_t w4 = raw[4], w5 = raw[5], w6 = raw[6];
  bool exact = false;
  uint32_t scale = 0;
  for (int k = 0; k < 3; ++k) {
    const uint32_t b = k < 2 ? (w4 >> (16 + 8 * k)) : w5;
    const int e = (int)(int8_t)(b & 0xffu) + 119;
    if (e <= 0) exact = true;
    scale |= ((uint32_t)e & 0xffu) << (8 * k);
  }
  uint32_t internal = 0, leaf = 0, offset = 0, at = 0;
  for (int i = 0; i < 6; ++i) {
    const uint32_t info = (i < 2 ? w5 >> (16 + 8 * i) : w6 >> (8 * (i - 2))) & 0x3fu;
    offset |= (at & 15u) << (4 * i);
    at += info & 3u;
    if (!(info & 3u)) continue;
    if ((info >> 2) == rtf::CT_INTERNAL) internal |= 1u << i;
    else leaf |= 1u << i;
  }
  for (int k = 0; k < 3; ++k) {
    const uint32_t a = raw[7 + 3 * k], b = raw[8 + 3 * k], c = raw[9 + 3 * k];
    const uint32_t hi4 = (b >> 16) | (c << 16), rest = (b & 0xffffu) | (c & 0xffff0000u);
    out[7 + 3 * k] = a;
    out[8 + 3 * k] = rest;
    out[9 + 3 * k] = hi4;
    for (int i = 0; i < 6; ++i) {
      const uint32_t lo = (i < 4 ? a >> (8 * i) : rest >> (8 * (i - 4))) & 0xffu;
      const uint32_t hi = (i < 4 ? hi4 >> (8 * i) : rest >> (8 * (i - 2))) & 0xffu;
      if (((internal | leaf) >> i & 1u) && lo > hi) exact = true;
    }
  }
  out[0] = raw[0];
  out[1] = raw[1];
  out[2] = raw[2];
  const uint32_t first = unit + raw[3];
  out[3] = first < units ? first : units;
  out[4] = scale;
  out[5] = internal | leaf << kLeafShift | (route & 0xfffu) << kSameShift | (exact ? kExact : 0u);
  out[6] = offset;
}

}  // namespace rtw
