// Checks walk_node (walk_node.h) over random nodes: every child unit a walk can
// form from a walk node, its first child's unit plus a child's nibble, lies in
// the blob or less than kPadUnits past its end; it is the blob's own child when
// the child block starts inside the blob, and outside the blob otherwise.
// Prints the number of mismatches.
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "walk_node.h"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint32_t next_u32() {  // xorshift64*
  state ^= state >> 12;
  state ^= state << 25;
  state ^= state >> 27;
  return (uint32_t)((state * 0x2545F4914F6CDD1Dull) >> 32);
}

int main() {
  unsigned long long bad = 0;
  for (int k = 0; k < 2000000; ++k) {
    const uint32_t units = 2 + next_u32() % (k % 3 ? 64u : (1u << 29) - 2u), unit = next_u32() % units;
    uint32_t raw[16], node[16];
    for (uint32_t& w : raw) w = next_u32();
    if (k % 2) raw[3] = (uint32_t)((int32_t)(next_u32() % 128u) - 64);  // near the node
    rtw::walk_node(raw, unit, units, next_u32(), node);
    uint8_t b[64];
    std::memcpy(b, raw, 64);
    const uint32_t first = unit + raw[3];
    uint32_t at = 0;
    for (int i = 0; i < 6; ++i) {
      const uint32_t size = b[rtf::IN_CHILD_INFO + i] & 3u, child = node[3] + ((node[6] >> (4 * i)) & 15u);
      const bool listed = ((node[5] | node[5] >> rtw::kLeafShift) >> i) & 1u;
      bad += listed != (size != 0);
      if (size) {
        bad += child >= units + rtw::kPadUnits;
        if (first < units) bad += child != first + at;
        else bad += child < units;
      }
      at += size;
    }
  }
  std::printf("mismatches %llu\n", bad);
  return bad != 0;
}
