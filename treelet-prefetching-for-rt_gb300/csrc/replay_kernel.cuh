// RT-unit trace replay (rt_unit_replay): one warp runs one RT unit's model
// over the visit traces of its warps.  The model is the one described at
// rt_unit_replay in treelet_rt.h; this file is its GPU form.
//
// The model advances one cycle at a time and sends at most one 32-byte
// request per cycle, so a unit is a sequential loop.  The warp works the
// parts of a cycle that have lanes in them: the L1 set (one lane per way),
// the resident warps (one lane per warp), a round's 32 lanes (one lane per
// RT lane, identical requests merged with __match_any_sync), and the members
// of a treelet that is pushed onto the prefetch queue.  Lane 0 keeps the
// unit's counters and makes the single-request updates.
//
// Per unit, in shared memory: the unit's scalar state, the resident warps
// (per RT lane a trace cursor), the current round's requests, the histogram
// of next treelets (a table of counts kept as lanes move on), the stride tables
// and, when they fit, the L1 lines.  In a slice of one device scratch buffer:
//   lines     sectored L1 (128 B lines, 4 x 32 B sectors, LRU stamps), when
//             they do not fit in shared memory
//   sectors   open-addressing map keyed by 32 B sector: prefetch records of
//             the sector still unclassified, whether one has been
//             classified, and the state of the sector's most recently evicted
//             prefetch record.  A prefetch record is only ever classified
//             through the sector it filled or, once evicted, as the sector's
//             most recently evicted one, so the classification needs these
//             counts and no record list
//   queued    open-addressing map: the oldest and newest live queued prefetch
//             request of each address (a demand request finds its queued
//             copies there instead of scanning the queue)
//   pq        the prefetch queue: a ring of (address, base) with tombstones;
//             pq_next links the live requests of one address, oldest first
//   metaret   metadata fills in flight
//
// What a unit does in a cycle in which nothing is sent, retired or decided is
// known in advance, so the model steps from event to event: idle cycles are
// skipped (more than half of all cycles), rounds are retired when the earliest
// one is due, and a decision that can change nothing is only counted.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/treelet_rt.h"
#include "device_nodes.cuh"
#include "format.h"

namespace rtr {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kChunkCap = 32 * 4;     // a round: 32 lanes x 128 B
constexpr uint32_t kMaxResident = 16;
constexpr uint32_t kHistLog2 = 10, kHistSize = 1u << kHistLog2;  // at most 512 roots at a time
constexpr uint32_t kMetaRing = 4096;       // > miss latency: metadata fills in flight
constexpr uint32_t kStrideEntries = 33;    // a stride table grows while it has <= 32 entries
constexpr uint32_t kTimeCap = 0xF0000000u; // cycles are 32-bit
constexpr uint32_t kLineValid = 0x80000000u;
constexpr uint32_t kSmemLinesMax = 1536;   // lines kept in shared memory (48 KiB)

struct Line {
  unsigned long long block;
  uint32_t lru;
  uint32_t flags;  // bit k: sector k valid; bit 4+k: filled by a prefetch; bit 8+k: that record unclassified
  uint32_t ready[4];
};

struct SectorEntry {
  unsigned long long key;  // sector + 1, 0 = empty
  uint32_t n_unclassified;
  uint16_t classified;     // 1 once a record of the sector has been classified
  uint16_t evicted;        // 0 none, 1 most recent evicted record unclassified, 2 classified
};

struct QueuedEntry {
  unsigned long long key;  // address + 1, 0 = empty
  uint32_t first, last;    // queue position + 1 of its oldest / newest live request, first 0 = none
};

struct Request {
  unsigned long long addr, base;
  uint32_t first, pad;
};

struct WarpSlot {
  uint32_t gid, wid, issued;
  uint32_t ptr[32], end[32];
  uint32_t next[32], root[32];  // each lane's next transaction (visit entry) and its treelet root
};

struct StrideTable {
  uint32_t has, n;
  unsigned long long last;
  int stride[kStrideEntries];
  uint32_t count[kStrideEntries];
};

struct MetaReturn {
  uint32_t t, pad;
  unsigned long long base;
};

// The unit's scalar state (shared memory; lane 0 writes, __syncwarp, all read).
struct UnitState {
  unsigned long long most_recent_metadata;
  rt_prefetch_state ds;
  uint32_t mr_head, mr_tail;
  // histogram summary of the lanes' next treelets
  uint32_t hist_used, best, best_cnt, total, distinct, best_of, best_dense, best_nodes, second;
  uint32_t full;
  uint32_t moved[kMaxResident];  // where resident warps move from when some leave
};

struct ReplayArgs {
  const rt_hit* hits;
  const uint32_t* visits;
  uint32_t n, capacity;
  rt_unit_config cfg;
  rt_unit_stats* stats;
  // scene
  const uint2* meta;
  uint32_t n_units;
  const uint32_t* roots;
  const unsigned long long* member_first;
  const uint32_t* members;
  const uint16_t* member_bytes;
  uint32_t n_treelets;
  unsigned long long meta_base, meta_size;
  // scratch
  uint8_t* scratch;
  unsigned long long unit_bytes;
  uint32_t sec_log2, queued_log2, pq_cap;  // pq_cap: a power of two
  uint32_t cycle_cap;     // per unit: the model's own bound on its cycles (or max_cycles)
  uint32_t lines_shared;  // 1: the L1 lines live in shared memory
  uint32_t members_apart; // no two members of a treelet share an address
  unsigned long long off_lines, off_sec, off_queued, off_pq, off_pq_next, off_dead, off_meta;
};

// Dynamic shared memory of one unit (one warp per CTA).
struct UnitShared {
  UnitState s;
  WarpSlot warps[kMaxResident];
  Request chunk[kChunkCap];
  uint32_t hist_key[kHistSize], hist_cnt[kHistSize];
  uint32_t scratch;  // touch_l1's word
  StrideTable stride[kMaxResident];
};

// Table slot of a 32-byte sector: the 16 sectors of 512 bytes get neighbouring
// slots, so that the requests of one node, or of nodes next to each other,
// find their entries in a few cache lines (the tables of all units together are
// larger than L2, and a probe of its own per sector was a DRAM access).
__device__ __forceinline__ uint32_t hash_slot(unsigned long long sector, uint32_t log2) {
  return ((uint32_t)(((sector >> 4) * 0x9E3779B97F4A7C15ull) >> (68 - log2)) << 4) | (uint32_t)(sector & 15u);
}

__device__ __forceinline__ uint32_t tx_size(uint32_t type) { return type == 2 ? 128u : (type == 3 ? 8u : 64u); }
__device__ __forceinline__ uint32_t intersection_latency(uint32_t type) {
  return (type == 0 || type == 3) ? 2u : 4u;  // 2,4,4,2,4,4,4
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  return (1u << (threadIdx.x & 31u)) - 1u;
}

__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const unsigned long long o = __shfl_xor_sync(kFull, v, s);
    v = o > v ? o : v;
  }
  return v;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) { return __reduce_add_sync(kFull, v); }

struct WUnit {
  const ReplayArgs& a;
  const rt_unit_config& cfg;
  const uint32_t lane;
  UnitShared& sh;
  UnitState& S;
  Line* lines;
  SectorEntry* sec;
  QueuedEntry* queued;
  unsigned long long* pq;  // pairs (addr, base)
  uint32_t* pq_next;       // queue position + 1 of the address's next live request, 0 = none
  uint8_t* dead;
  MetaReturn* metaret;
  // lane 0's: the counters, and the records not yet classified, in all and in
  // sectors that have a classified one
  rt_unit_stats st;
  unsigned long long uncl, uncl_accessed;
  // Resident warps in order, warp o in lane o's registers: its slot, whether
  // its round is in flight and all sent, when the round's data is back, its
  // lanes with transactions left.
  uint32_t r_slot, r_ready, r_live;
  bool r_fly, r_sent;
  // The same in every lane: warps resident, free slots, the prefetch queue's
  // ends and live requests, the round being sent (its requests, the order of
  // its warp, when its data is back so far, its intersection latency), whether
  // the histogram changed, whether deciding again changes nothing until it
  // does, and the earliest cycle at which a round retires or a warp leaves.
  // (Kept in shared memory, every one of them was a 30-cycle read on the path
  // of each modeled cycle.)
  uint32_t n_res, free_mask, pq_head, pq_tail, pq_live, ch_head, ch_tail, serving, ch_ready, ch_ilat;
  uint32_t next_retire, next_gid, local;
  bool hist_dirty, quiet;

  __device__ WUnit(const ReplayArgs& args, uint32_t u, UnitShared& shm, Line* smem_lines)
      : a(args), cfg(args.cfg), lane(threadIdx.x & 31u), sh(shm), S(shm.s) {
    uint8_t* base = a.scratch + (unsigned long long)u * a.unit_bytes;
    lines = a.lines_shared ? smem_lines : reinterpret_cast<Line*>(base + a.off_lines);
    sec = reinterpret_cast<SectorEntry*>(base + a.off_sec);
    queued = reinterpret_cast<QueuedEntry*>(base + a.off_queued);
    pq = reinterpret_cast<unsigned long long*>(base + a.off_pq);
    pq_next = reinterpret_cast<uint32_t*>(base + a.off_pq_next);
    dead = base + a.off_dead;
    metaret = reinterpret_cast<MetaReturn*>(base + a.off_meta);
    st = rt_unit_stats{};
    uncl = uncl_accessed = 0;
    r_slot = r_ready = r_live = 0;
    r_fly = r_sent = false;
    n_res = 0;
    free_mask = (1u << cfg.max_warps) - 1u;
    pq_head = pq_tail = pq_live = 0;
    ch_head = ch_tail = ch_ready = ch_ilat = 0;
    serving = kNone;
    next_retire = 0;
    next_gid = u;
    local = 0;
    hist_dirty = true;
    quiet = false;
  }
  // After lane 0 has changed the queue on its own.
  __device__ void share_queue() {
    pq_head = __shfl_sync(kFull, pq_head, 0);
    pq_tail = __shfl_sync(kFull, pq_tail, 0);
    pq_live = __shfl_sync(kFull, pq_live, 0);
  }

  // ------------------------------------------------------------ tables (lane 0)
  __device__ SectorEntry* sector_entry(unsigned long long sector, bool create) {
    const unsigned long long key = sector + 1;
    const uint32_t mask = (1u << a.sec_log2) - 1u;
    uint32_t i = hash_slot(sector, a.sec_log2);
    for (uint32_t probe = 0; probe <= mask; ++probe, i = (i + 1) & mask) {
      SectorEntry& e = sec[i];
      if (e.key == key) return &e;
      if (e.key == 0) {
        if (!create) return nullptr;
        e.key = key;
        return &e;
      }
    }
    S.full = 1;
    return nullptr;
  }

  __device__ QueuedEntry* queued_entry(unsigned long long addr, bool create) {
    const unsigned long long key = addr + 1;
    const uint32_t mask = (1u << a.queued_log2) - 1u;
    uint32_t i = hash_slot(addr >> 5, a.queued_log2);
    for (uint32_t probe = 0; probe <= mask; ++probe, i = (i + 1) & mask) {
      QueuedEntry& e = queued[i];
      if (e.key == key) return &e;
      if (e.key == 0) {
        if (!create) return nullptr;
        e.key = key;
        return &e;
      }
    }
    S.full = 1;
    return nullptr;
  }

  // Starts the table entries of a request on their way to L1.
  __device__ void touch_tables(unsigned long long addr) {
    const uint32_t word = (uint32_t)__cvta_generic_to_shared(&sh.scratch);
    rtd::touch_l1(word, queued + hash_slot(addr >> 5, a.queued_log2));
    rtd::touch_l1(word, sec + hash_slot(addr >> 5, a.sec_log2));
  }

  // One of the sector's records is classified.  The final tally
  // (gpu-sim.cc:1749-1790) needs, besides the classes' counts, the
  // unclassified records of the sectors with a classified one and of the
  // others; both are kept here (scanning the table at the end took a fifth of
  // a replay).
  __device__ __forceinline__ void classify(SectorEntry* e, uint32_t cls) {  // lane 0
    e->n_unclassified--;
    --uncl;
    st.effectiveness[cls]++;
    if (e->classified) {
      --uncl_accessed;
    } else {
      e->classified = 1;
      uncl_accessed += e->n_unclassified;
    }
  }
  __device__ __forceinline__ void classify(unsigned long long sector, uint32_t cls) {
    SectorEntry* e = sector_entry(sector, false);
    if (e) classify(e, cls);
  }

  // ------------------------------------------------------------ cache (warp)
  __device__ Line* set_of(unsigned long long block) const {
    return lines + (size_t)(block & (cfg.l1_sets - 1)) * cfg.l1_ways;
  }

  // Way holding `block`, or -1 (one lane per way).
  __device__ int find_way(unsigned long long block) const {
    const Line* set = set_of(block);
    const bool m = lane < cfg.l1_ways && (set[lane].flags & kLineValid) && set[lane].block == block;
    const uint32_t b = __ballot_sync(kFull, m);
    return b ? __ffs(b) - 1 : -1;
  }

  // An unused way first, else the least recently used, lowest way on ties.
  __device__ int victim_way(unsigned long long block) const {
    const Line* set = set_of(block);
    const uint32_t inv = __ballot_sync(kFull, lane < cfg.l1_ways && !(set[lane].flags & kLineValid));
    if (inv) return __ffs(inv) - 1;
    const uint32_t lru = lane < cfg.l1_ways ? set[lane].lru : 0xFFFFFFFFu;
    const uint32_t oldest = __reduce_min_sync(kFull, lru);
    return __ffs(__ballot_sync(kFull, lane < cfg.l1_ways && lru == oldest)) - 1;
  }

  // Lane 0: installs `block` in way `w`, recording evicted prefetched sectors.
  __device__ Line* install(unsigned long long block, int w, uint32_t t) {
    Line* v = set_of(block) + w;
    if (v->flags & kLineValid) {
      for (uint32_t k = 0; k < 4; ++k)
        if ((v->flags >> k) & (v->flags >> (4 + k)) & 1u) {
          SectorEntry* e = sector_entry(v->block * 4 + k, false);
          if (e) e->evicted = ((v->flags >> (8 + k)) & 1u) ? 1u : 2u;
        }
    }
    v->block = block;
    v->flags = kLineValid;
    v->lru = t;
    return v;
  }

  // A demand request; returns the cycle its data is there (uniform).
  __device__ uint32_t demand(unsigned long long addr, uint32_t t) {
    const unsigned long long block = addr >> 7;
    const int way = find_way(block);
    Line* set = set_of(block);
    const uint32_t k = (uint32_t)((addr >> 5) & 3);
    const bool sector_valid = way >= 0 && ((set[way].flags >> k) & 1u);
    const int vic = (way < 0) ? victim_way(block) : -1;
    // every lane finds the cycle the data is there; lane 0 updates the model
    const uint32_t back = sector_valid ? set[way].ready[k] : 0u;
    const uint32_t ret = !sector_valid ? t + cfg.miss_latency : (back <= t ? t + cfg.hit_latency : back);
    __syncwarp();
    if (lane == 0) {
      const unsigned long long sector = addr >> 5;
      st.demand_requests++;
      if (sector_valid) {
        Line* l = set + way;
        l->lru = t;
        const bool pf_uncl = (l->flags >> (4 + k)) & (l->flags >> (8 + k)) & 1u;
        if (back <= t) {
          st.demand_hits++;
          if (pf_uncl) {
            classify(sector, RT_PF_TIMELY);
            l->flags &= ~(1u << (8 + k));
          }
        } else {
          st.demand_hit_reserved++;
          if (pf_uncl) {
            classify(sector, RT_PF_LATE);
            l->flags &= ~(1u << (8 + k));
          }
        }
      } else {
        st.demand_misses++;
        SectorEntry* e = sector_entry(sector, false);
        if (e && e->evicted == 1u) {
          classify(e, RT_PF_TOO_EARLY);
          e->evicted = 2u;
        }
        Line* l = way >= 0 ? set + way : install(block, vic, t);
        l->lru = t;
        l->flags = (l->flags | (1u << k)) & ~((1u << (4 + k)) | (1u << (8 + k)));
        l->ready[k] = t + cfg.miss_latency;
      }
    }
    __syncwarp();
    return ret;
  }

  __device__ bool is_metadata(unsigned long long base) const {
    return cfg.load_metadata && base >= a.meta_base && base <= a.meta_base + (unsigned long long)a.n_treelets * a.meta_size;
  }

  __device__ void prefetch(unsigned long long addr, unsigned long long base, uint32_t t) {
    const unsigned long long block = addr >> 7;
    const int way = find_way(block);
    Line* set = set_of(block);
    const uint32_t k = (uint32_t)((addr >> 5) & 3);
    const bool sector_valid = way >= 0 && ((set[way].flags >> k) & 1u);
    const int vic = (way < 0) ? victim_way(block) : -1;
    __syncwarp();
    if (lane == 0) {
      st.prefetch_issued++;
      SectorEntry* e = sector_entry(addr >> 5, true);
      if (e) {
        e->n_unclassified++;
        ++uncl;
        uncl_accessed += e->classified;
      }
      if (sector_valid) {
        Line* l = set + way;
        l->lru = t;
        // a fresh record is unclassified, so the TOO_LATE rule of
        // gpu-cache.cc:2101-2116 never applies to it
        if (l->ready[k] <= t) st.prefetch_present++;
        else st.prefetch_merged++;
      } else {
        st.prefetch_filled++;
        Line* l = way >= 0 ? set + way : install(block, vic, t);
        l->lru = t;
        l->flags |= (1u << k) | (1u << (4 + k)) | (1u << (8 + k));
        l->ready[k] = t + cfg.miss_latency;
        if (is_metadata(base)) {
          if (S.mr_tail - S.mr_head < kMetaRing) {
            metaret[S.mr_tail % kMetaRing] = MetaReturn{t + cfg.miss_latency, 0u, base};
            ++S.mr_tail;
          } else {
            S.full = 1;
          }
        }
      }
    }
    __syncwarp();
  }

  // ------------------------------------------------------------ prefetch queue
  __device__ void pq_push(unsigned long long addr, unsigned long long base) {  // lane 0
    st.prefetch_queued++;
    if (pq_tail - pq_head >= a.pq_cap) {  // ring full (live + erased entries)
      S.full = 1;
      return;
    }
    const uint32_t i = pq_tail & (a.pq_cap - 1u);
    pq[2 * i] = addr;
    pq[2 * i + 1] = base;
    dead[i] = 0;
    pq_next[i] = 0;
    const uint32_t at = ++pq_tail;  // position + 1
    ++pq_live;
    QueuedEntry* q = queued_entry(addr, true);
    if (!q) return;
    if (q->first) pq_next[(q->last - 1u) & (a.pq_cap - 1u)] = at;
    else q->first = at;
    q->last = at;
  }

  __device__ void pq_drop_dead() {  // lane 0
    while (pq_head != pq_tail && dead[pq_head & (a.pq_cap - 1u)]) ++pq_head;
  }

  // Erases queued prefetches of `addr`, stepping past the entry that follows
  // each erased one (shader.cc:4657-4668 as written): of two matches with no
  // live entry between them the second stays.  Follows the address's own
  // requests (almost always one).
  __device__ void remove_queued(unsigned long long addr) {
    QueuedEntry* q = nullptr;
    uint32_t at = 0;
    if (lane == 0) {
      q = queued_entry(addr, false);
      at = q ? q->first : 0u;
    }
    if (!__shfl_sync(kFull, at, 0)) return;
    if (lane == 0) {
        uint32_t kept = 0;  // last live request kept, position + 1
        q->first = 0;
        while (at) {
          const uint32_t i = (at - 1u) & (a.pq_cap - 1u), next = pq_next[i];
          dead[i] = 1;
          --pq_live;
          st.prefetch_removed++;
          uint32_t p = at;  // the entry stepped past: the next live one (positions at .. tail - 1)
          while (p != pq_tail && dead[p & (a.pq_cap - 1u)]) ++p;
          at = next;
          if (next && p + 1u == next) {  // it is the address's next request: it stays
            const uint32_t k = p & (a.pq_cap - 1u);
            if (kept) pq_next[(kept - 1u) & (a.pq_cap - 1u)] = next;
            else q->first = next;
            kept = next;
            at = pq_next[k];
          }
        }
        if (kept) pq_next[(kept - 1u) & (a.pq_cap - 1u)] = 0;
        q->last = kept;
        pq_drop_dead();
    }
    __syncwarp();
    share_queue();
  }

  __device__ uint32_t dense_of(uint32_t root) const {
    uint32_t lo = 0, hi = a.n_treelets;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(a.roots + mid) < root) lo = mid + 1;
      else hi = mid;
    }
    return (lo < a.n_treelets && __ldg(a.roots + lo) == root) ? lo : kNone;
  }

  __device__ void push_member(unsigned long long j, bool with_metadata) {  // lane 0
    const uint32_t m = __ldg(a.members + j);
    if (with_metadata && cfg.load_metadata) {
      const uint32_t d = dense_of(m);  // treelet_addr_to_metadata_idx: 0 for a member that is no root
      const unsigned long long ma = a.meta_base + (unsigned long long)(d == kNone ? 0u : d) * a.meta_size;
      for (unsigned long long i = 0; i < a.meta_size / 32; ++i) {
        pq_push(ma + i * 32, ma);
        st.metadata_queued++;
      }
    }
    const unsigned long long addr = (unsigned long long)m * 64;
    const uint32_t b = __ldg(a.member_bytes + j);
    for (uint32_t i = 0; i < (b + 31) / 32; ++i) pq_push(addr + 32ull * i, addr);
  }

  // Queues members [j0, j1) of the member lists, each as its 32-byte requests,
  // one member per lane.  Their addresses are distinct (a.members_apart), so
  // the lanes' table entries are too and only their keys need a
  // compare-and-swap.  False when the ring has no room for all of them.
  __device__ bool push_members(unsigned long long j0, unsigned long long j1) {
    for (unsigned long long jb = j0; jb < j1; jb += 32) {
      const unsigned long long j = jb + lane;
      const bool in = j < j1;
      const unsigned long long addr = in ? (unsigned long long)__ldg(a.members + j) * 64 : 0ull;
      const uint32_t n = in ? (__ldg(a.member_bytes + j) + 31u) / 32u : 0u;
      uint32_t incl = n;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t o = __shfl_up_sync(kFull, incl, s);
        if ((int)lane >= s) incl += o;
      }
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      const uint32_t tail = pq_tail;
      if (tail - pq_head + total > a.pq_cap) return jb == j0 ? false : push_rest(jb, j1);
      for (uint32_t i = 0; i < n; ++i) {
        const unsigned long long at_addr = addr + 32ull * i;
        const uint32_t p = tail + incl - n + i, k = p & (a.pq_cap - 1u);
        pq[2 * k] = at_addr;
        pq[2 * k + 1] = addr;
        dead[k] = 0;
        pq_next[k] = 0;
        touch_tables(at_addr);
        QueuedEntry* q = queued_claim(at_addr);
        if (!q) continue;
        if (q->first) pq_next[(q->last - 1u) & (a.pq_cap - 1u)] = p + 1u;
        else q->first = p + 1u;
        q->last = p + 1u;
      }
      __syncwarp();
      pq_tail = tail + total;
      pq_live += total;
      if (lane == 0) st.prefetch_queued += total;
    }
    return true;
  }
  // The rest of a list that no longer fits the ring: one request at a time.
  __device__ bool push_rest(unsigned long long j0, unsigned long long j1) {
    if (lane == 0)
      for (unsigned long long j = j0; j < j1; ++j) push_member(j, false);
    __syncwarp();
    share_queue();
    return true;
  }

  // queued_entry(addr, true) for lanes that claim entries at the same time.
  __device__ QueuedEntry* queued_claim(unsigned long long addr) {
    const unsigned long long key = addr + 1;
    const uint32_t mask = (1u << a.queued_log2) - 1u;
    uint32_t i = hash_slot(addr >> 5, a.queued_log2);
    for (uint32_t probe = 0; probe <= mask; ++probe, i = (i + 1) & mask) {
      unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(&queued[i].key);
      if (k == 0) k = atomicCAS(&queued[i].key, 0ull, key);
      if (k == 0 || k == key) return &queued[i];
    }
    S.full = 1;
    return nullptr;
  }

  // ------------------------------------------------------------ decision
  // Reads the calling lane's next transaction of a warp (when it has one).
  __device__ void fetch_next(WarpSlot& w) const {
    if (w.ptr[lane] >= w.end[lane]) return;
    const uint32_t v = __ldg(a.visits + (unsigned long long)(w.gid * 32 + lane) * a.capacity + w.ptr[lane]);
    w.next[lane] = v;
    w.root[lane] = (v >> 3) < a.n_units ? __ldg(&a.meta[v >> 3].x) : kNone;
  }

  // ------------------------------------------------------------ histogram
  // Lanes per treelet root over the resident warps' next transactions, kept
  // up to date as rounds retire and warps come in: an open-addressing table
  // of roots and counts (a root whose count is 0 keeps its slot until the
  // table is built anew).  Sorting up to 512 roots after every round was a
  // third of the replay's instructions.
  __device__ uint32_t hist_slot(uint32_t root) const {
    uint32_t i = (root * 0x9E3779B1u) >> (32 - kHistLog2);
    for (;; i = (i + 1) & (kHistSize - 1)) {
      const uint32_t k = sh.hist_key[i];
      if (k == root) return i;
      if (k == kNone && atomicCAS(&sh.hist_key[i], kNone, root) == kNone) {
        atomicAdd(&S.hist_used, 1u);
        return i;
      }
      if (sh.hist_key[i] == root) return i;
    }
  }
  // Adds 1 (or -1) per calling lane with `on`; all 32 lanes call.
  __device__ void hist_add(uint32_t root, bool on, uint32_t one) {
    const uint32_t key = on ? root : kNone;
    const uint32_t peers = __match_any_sync(kFull, key);
    if (key != kNone && (uint32_t)(__ffs(peers) - 1) == lane)
      atomicAdd(&sh.hist_cnt[hist_slot(key)], one * (uint32_t)__popc(peers));
    __syncwarp();
  }
  __device__ bool has_next(const WarpSlot& w) const { return w.ptr[lane] < w.end[lane]; }
  // Room for 32 new roots, or the table built anew from the resident warps'
  // lanes (true then: they are all counted).
  __device__ bool hist_renew() {
    if (S.hist_used + 32u <= kHistSize * 3 / 4) return false;
    __syncwarp();
    hist_clear();
    for (uint32_t o = 0; o < n_res; ++o) {
      const WarpSlot& w = sh.warps[__shfl_sync(kFull, r_slot, o)];
      hist_add(w.root[lane], has_next(w), 1u);
    }
    return true;
  }
  __device__ void hist_clear() {
    for (uint32_t i = lane; i < kHistSize; i += 32) {
      sh.hist_key[i] = kNone;
      sh.hist_cnt[i] = 0;
    }
    if (lane == 0) S.hist_used = 0;
    __syncwarp();
  }

  // The most popular root (ties to the lowest) and the next one, the number
  // of roots and of lanes.
  __device__ void summarize_histogram() {
    unsigned long long best = 0, second = 0;
    uint32_t runs = 0, total = 0;
    for (uint32_t i = lane; i < kHistSize; i += 32) {
      const uint32_t c = sh.hist_cnt[i];
      if (!c) continue;
      ++runs;
      total += c;
      const unsigned long long v = ((unsigned long long)c << 32) | (unsigned long long)(~sh.hist_key[i]);
      second = v > best ? best : (v > second ? v : second);
      best = v > best ? v : best;
    }
    const unsigned long long b = warp_max64(best);
    const unsigned long long b2 = warp_max64(best == b ? second : best);
    runs = warp_sum(runs);
    total = warp_sum(total);
    if (lane == 0) {
      S.second = (cfg.decision.second_prefetch && b2) ? ~(uint32_t)(b2 & 0xffffffffu) : kNone;
      S.total = total;
      S.distinct = runs;
      S.best = total ? ~(uint32_t)(b & 0xffffffffu) : kNone;
      S.best_cnt = (uint32_t)(b >> 32);
      if (S.best != S.best_of) {
        S.best_of = S.best;
        S.best_dense = S.best == kNone ? kNone : dense_of(S.best);
        S.best_nodes = S.best_dense == kNone
                           ? 0u
                           : (uint32_t)(__ldg(a.member_first + S.best_dense + 1) - __ldg(a.member_first + S.best_dense));
      }
    }
    hist_dirty = false;
    __syncwarp();
  }

  // The RT unit's decision (shader.cc:3419-3683; as prefetch_decide_kernel).
  __device__ void decide() {
    if (hist_dirty) summarize_histogram();
    else if (quiet) return;
    const rt_prefetch_params& p = cfg.decision;
    __syncwarp();
    // lane 0 decides which members are queued: [from, to) of the lists
    unsigned long long from = 0, to = 0;
    bool still = true;  // lane 0: deciding again would change nothing
    if (lane == 0) {
      const uint32_t best = S.best;
      bool submit = false;
      int num_nodes = 0;
      const int n_nodes = (int)S.best_nodes;
      const uint32_t bd = S.best_dense;
      if (p.heuristic == RT_PREFETCH_ALWAYS) {
        submit = true;
      } else if (best != kNone) {
        const double pct = (double)S.best_cnt / (double)S.total;
        if (p.heuristic == RT_PREFETCH_POPULARITY) {
          if (pct >= p.threshold) {
            S.ds.last_rejected = kNone;
            submit = true;
          } else if (S.ds.last_rejected != best) {
            S.ds.last_rejected = best;
          }
        } else {
          num_nodes = (int)(((double)n_nodes * pct) + 0.5);
          submit = true;
        }
      }
      if (submit && best != kNone && bd != kNone && S.ds.last_prefetched != best && S.ds.last_prefetched_second != best) {
        const bool partial = p.heuristic == RT_PREFETCH_PARTIAL || p.heuristic == RT_PREFETCH_LATTER;
        const int num = partial ? num_nodes : n_nodes;
        still = false;  // submitted, or waiting for room in the queue
        if ((unsigned long long)num + pq_live <= p.max_queue) {
          const int j0 = p.heuristic == RT_PREFETCH_LATTER ? n_nodes - num : 0;
          const int j1 = p.heuristic == RT_PREFETCH_LATTER ? n_nodes : num;
          const unsigned long long mf = __ldg(a.member_first + bd);
          from = mf + j0;
          to = mf + j1;
          S.ds.last_prefetched = best;
          st.treelets_prefetched++;
        }
      }
    }
    from = __shfl_sync(kFull, from, 0);
    to = __shfl_sync(kFull, to, 0);
    const unsigned long long live = pq_live;
    push_list(from, to, true);
    unsigned long long from2 = 0, to2 = 0;
    if (lane == 0) {
      const uint32_t best = S.best;
      // the queue length the decision sees: requests of the members submitted
      // count whether or not the ring had room, metadata requests do not
      unsigned long long queue = live;
      if (p.second_prefetch && live == 0)
        for (unsigned long long j = from; j < to; ++j) queue += (__ldg(a.member_bytes + j) + 31u) / 32u;
      // the second treelet may follow as soon as the queue is empty
      if (p.second_prefetch && S.total > 0 && S.distinct > 1 && S.second != kNone &&
          S.ds.last_prefetched_second != S.second)
        still = false;
      if (p.second_prefetch && queue == 0 && S.total > 0 && S.distinct > 1 && S.ds.last_prefetched == best &&
          best != kNone) {
        // the first maximum among treelets other than the last prefetched one,
        // which is `best` here (kept with the histogram)
        const uint32_t second = S.second;
        if (second != kNone && S.ds.last_prefetched_second != second) {
          const uint32_t sd = dense_of(second);
          if (sd != kNone) {
            from2 = __ldg(a.member_first + sd);
            to2 = __ldg(a.member_first + sd + 1);
          }
          S.ds.last_prefetched_second = second;
          st.treelets_prefetched++;
        }
      }
    }
    from2 = __shfl_sync(kFull, from2, 0);
    to2 = __shfl_sync(kFull, to2, 0);
    push_list(from2, to2, false);
    quiet = __shfl_sync(kFull, still ? 1u : 0u, 0) != 0;
  }

  // Queues members [j0, j1), with their treelets' metadata first when the
  // model loads it.
  __device__ void push_list(unsigned long long j0, unsigned long long j1, bool with_metadata) {
    if (j0 >= j1) return;
    if (!(with_metadata && cfg.load_metadata) && a.members_apart && push_members(j0, j1)) return;
    if (lane == 0)
      for (unsigned long long j = j0; j < j1; ++j) push_member(j, with_metadata);
    __syncwarp();
    share_queue();
  }

  // ------------------------------------------------------------ stride (Lee MICRO'10), lane 0
  __device__ void stride_prefetch(uint32_t wid, unsigned long long next_addr) {
    StrideTable& s = sh.stride[wid];
    if (!s.has) {
      s.last = next_addr;
    } else if (s.n <= 32) {
      const int d = (int)(uint32_t)(next_addr - s.last);
      uint32_t i = 0;
      while (i < s.n && s.stride[i] < d) ++i;
      if (i < s.n && s.stride[i] == d) {
        s.count[i]++;
      } else {
        for (uint32_t k = s.n; k > i; --k) {
          s.stride[k] = s.stride[k - 1];
          s.count[k] = s.count[k - 1];
        }
        s.stride[i] = d;
        s.count[i] = 1;
        s.n++;
      }
    }
    s.has = 1;  // the table lookup below creates the warp's (empty) table
    int largest = 0;
    uint32_t largest_count = 0;
    for (uint32_t i = 0; i < s.n; ++i)
      if (s.count[i] > largest_count) {
        largest = s.stride[i];
        largest_count = s.count[i];
      }
    const unsigned long long pa = next_addr + (unsigned long long)(long long)largest;
    if (cfg.decision.max_queue <= pq_live) {
      pq_push(pa, pa);
      pq_push(pa + 32, pa);
    }
  }

  // ------------------------------------------------------------ warps
  __device__ uint32_t matching_lanes(uint32_t slot) const {
    const WarpSlot& w = sh.warps[slot];
    const uint32_t lp = S.ds.last_prefetched;
    const bool m = lp != kNone && w.ptr[lane] < w.end[lane] && w.root[lane] == lp;
    return __popc(__ballot_sync(kFull, m));
  }

  // rt_unit::schedule_next_warp (shader.cc:4307-4392): the order of the warp
  // to serve, kNone if no warp is ready
  __device__ uint32_t schedule() const {
    const uint32_t ready = __ballot_sync(kFull, lane < n_res && !r_fly && r_live);
    if (!ready) return kNone;
    const bool treelet = cfg.prefetcher == RT_UNIT_PF_TREELET;
    if (treelet && cfg.scheduler == RT_UNIT_SCHED_OMR) {
      for (uint32_t m = ready; m; m &= m - 1) {
        const uint32_t o = __ffs(m) - 1;
        if (matching_lanes(__shfl_sync(kFull, r_slot, o)) > 0) return o;
      }
    } else if (treelet && cfg.scheduler == RT_UNIT_SCHED_PMR) {
      uint32_t b = kNone, bc = 0;
      for (uint32_t m = ready; m; m &= m - 1) {
        const uint32_t o = __ffs(m) - 1;
        const uint32_t c = matching_lanes(__shfl_sync(kFull, r_slot, o));
        if (c > bc) {
          b = o;
          bc = c;
        }
      }
      if (b != kNone) return b;
    }
    return __ffs(ready) - 1;
  }

  // A round: each lane's next transaction, identical (address, size) pairs
  // once in lane order, split into 32-byte requests.
  __device__ void start_round(uint32_t o) {
    WarpSlot& w = sh.warps[__shfl_sync(kFull, r_slot, o)];
    const bool has = w.ptr[lane] < w.end[lane];
    const uint32_t v = has ? w.next[lane] : 0u;
    const uint32_t size = tx_size(v & 7);
    const unsigned long long key = has ? (((unsigned long long)(v >> 3) << 8) | size) : ~0ull;
    const uint32_t peers = __match_any_sync(kFull, key);
    const bool leader = has && (uint32_t)(__ffs(peers) - 1) == lane;
    const uint32_t nch = leader ? (size + 31) / 32 : 0u;
    uint32_t incl = nch;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t o = __shfl_up_sync(kFull, incl, s);
      if ((int)lane >= s) incl += o;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    const unsigned long long addr = (unsigned long long)(v >> 3) * 64;
    for (uint32_t i = 0; i < nch; ++i) {
      sh.chunk[incl - nch + i] = Request{addr + 32ull * i, addr, i == 0 ? 1u : 0u, 0u};
      if (cfg.prefetcher != RT_UNIT_PF_NONE) touch_tables(addr + 32ull * i);
    }
    ch_ilat = __reduce_max_sync(kFull, has ? intersection_latency(v & 7) : 0u);
    const uint32_t issued = __ballot_sync(kFull, has);
    if (lane == 0) w.issued = issued;
    if (lane == o) {
      r_fly = true;
      r_sent = false;
    }
    ch_head = 0;
    ch_tail = total;
    ch_ready = 0;
    serving = o;
    __syncwarp();
  }

  __device__ void send_demand(uint32_t t) {
    const Request r = sh.chunk[ch_head];
    if (cfg.prefetcher == RT_UNIT_PF_TREELET || cfg.prefetcher == RT_UNIT_PF_STRIDE) remove_queued(r.addr);
    if (cfg.prefetcher == RT_UNIT_PF_STRIDE && r.first) {
      const uint32_t wid = sh.warps[__shfl_sync(kFull, r_slot, serving)].wid;
      if (lane == 0) stride_prefetch(wid, r.addr);
      __syncwarp();
      share_queue();
    }
    ch_ready = max(ch_ready, demand(r.addr, t));
    if (++ch_head == ch_tail) {
      const uint32_t ready = ch_ready + ch_ilat;
      if (lane == serving) {
        r_sent = true;
        r_ready = ready;
      }
      next_retire = min(next_retire, ready);
      serving = kNone;
    }
  }

  __device__ bool prefetch_issuable(unsigned long long base) const {
    if (!cfg.wait_metadata || is_metadata(base)) return true;
    // shader.cc:4469-4476: the metadata of the treelet the request's base node belongs to
    const unsigned long long unit = base >> 6;
    const uint32_t root = (base % 64 == 0 && unit < a.n_units) ? __ldg(&a.meta[unit].x) : kNone;
    const uint32_t d = root == kNone ? kNone : dense_of(root);
    return S.most_recent_metadata == a.meta_base + (unsigned long long)(d == kNone ? 0u : d) * a.meta_size;
  }

  // Rounds whose data is back advance their lanes; warps with no lanes left
  // leave; new warps come in, in order.
  __device__ void retire_and_admit(uint32_t t, uint32_t n_warps) {
    const bool treelets = cfg.prefetcher == RT_UNIT_PF_TREELET;
    const uint32_t rounds = __ballot_sync(kFull, lane < n_res && r_fly && r_sent && r_ready <= t);
    for (uint32_t m = rounds; m; m &= m - 1) {
      const uint32_t o = __ffs(m) - 1;
      WarpSlot& w = sh.warps[__shfl_sync(kFull, r_slot, o)];
      const uint32_t issued = w.issued;
      const bool mine = (issued >> lane) & 1u;
      const uint32_t old_root = w.root[lane];
      if (mine) {
        w.ptr[lane]++;
        fetch_next(w);
      }
      if (treelets) {
        __syncwarp();
        if (!hist_renew()) {
          hist_add(old_root, mine, ~0u);
          hist_add(w.root[lane], mine && has_next(w), 1u);
        }
      }
      const uint32_t live = __ballot_sync(kFull, has_next(w));
      if (lane == 0) st.transactions += __popc(issued);
      if (lane == o) {
        r_fly = false;
        r_live = live;
      }
      hist_dirty = true;
    }
    const bool gone = lane < n_res && !r_fly && r_live == 0;
    const uint32_t leave = __ballot_sync(kFull, gone);
    if (leave) {
      const uint32_t keep = __ballot_sync(kFull, lane < n_res && !gone);
      free_mask |= __reduce_or_sync(kFull, gone ? 1u << r_slot : 0u);
      if (lane < n_res && !gone) S.moved[__popc(keep & lanemask_lt())] = lane;
      __syncwarp();
      if (lane == 0) st.warps += __popc(leave);
      n_res = __popc(keep);
      const uint32_t from = lane < n_res ? S.moved[lane] : lane;
      r_slot = __shfl_sync(kFull, r_slot, from);
      r_ready = __shfl_sync(kFull, r_ready, from);
      r_live = __shfl_sync(kFull, r_live, from);
      r_fly = __shfl_sync(kFull, r_fly ? 1u : 0u, from) != 0;
      r_sent = __shfl_sync(kFull, r_sent ? 1u : 0u, from) != 0;
      if (serving != kNone) serving = __popc(keep & ((1u << serving) - 1u));
      hist_dirty = true;
      __syncwarp();
    }
    while (n_res < cfg.max_warps && next_gid < n_warps) {
      const uint32_t slot = __ffs(free_mask) - 1;
      WarpSlot& w = sh.warps[slot];
      const uint32_t gid = next_gid;
      const uint32_t r = gid * 32 + lane;
      if (lane == 0) {
        w.gid = gid;
        w.wid = local % cfg.max_warps;
        w.issued = 0;
      }
      w.ptr[lane] = 0;
      w.end[lane] = r < a.n ? min(a.hits[r].n_visits, a.capacity) : 0u;
      __syncwarp();
      fetch_next(w);
      const uint32_t live = __ballot_sync(kFull, has_next(w));
      if (lane == n_res) {
        r_slot = slot;
        r_live = live;
        r_fly = r_sent = false;
        r_ready = 0;
      }
      ++local;
      ++n_res;
      free_mask &= ~(1u << slot);
      next_gid = gid + cfg.n_rt_units;
      hist_dirty = true;
      __syncwarp();
      if (treelets && !hist_renew()) hist_add(w.root[lane], has_next(w), 1u);
    }
    // when to look again: the earliest round due, or the next cycle for a
    // warp that came in without a transaction
    uint32_t due = 0xFFFFFFFFu;
    if (lane < n_res) {
      if (r_fly && r_sent) due = r_ready;
      else if (!r_fly && r_live == 0) due = t + 1;
    }
    next_retire = __reduce_min_sync(kFull, due);
  }

  __device__ void run(uint32_t u) {
    const uint32_t n_warps = (a.n + 31) / 32;
    if (lane == 0) {
      S.most_recent_metadata = 0;
      S.ds = rt_prefetch_state{kNone, kNone, kNone, 0};
      S.mr_head = S.mr_tail = 0;
      S.best = S.best_of = kNone;
      S.best_cnt = S.total = S.distinct = S.best_nodes = 0;
      S.best_dense = S.second = kNone;
      S.full = 0;
    }
    hist_clear();
    if (lane < kMaxResident) sh.stride[lane].has = sh.stride[lane].n = 0;
    if (a.lines_shared)
      for (uint32_t i = lane; i < cfg.l1_sets * cfg.l1_ways; i += 32) lines[i].flags = 0;
    __syncwarp();
    const uint32_t tcap = a.cycle_cap;
    const bool treelets = cfg.prefetcher == RT_UNIT_PF_TREELET;
    unsigned long long decisions = 0;
    uint32_t next_decide = 0;  // the next multiple of prefetch_delay
    for (uint32_t t = 0;; ++t) {
      if (t >= next_retire) retire_and_admit(t, n_warps);
      if (n_res == 0) {
        if (lane == 0) st.cycles = t;
        break;
      }
      if (t >= tcap) {
        if (lane == 0) {
          st.cycles = t;
          st.status |= 2;
        }
        break;
      }
      if (cfg.load_metadata) {
        if (lane == 0)
          while (S.mr_head != S.mr_tail && metaret[S.mr_head % kMetaRing].t <= t) {
            S.most_recent_metadata = metaret[S.mr_head % kMetaRing].base;
            ++S.mr_head;
          }
        __syncwarp();
      }
      if (treelets && t == next_decide) {
        decide();
        ++decisions;
        next_decide += cfg.prefetch_delay;
      }
      if (ch_head != ch_tail) {
        send_demand(t);
        continue;
      }
      const uint32_t s = schedule();
      if (s != kNone) {
        start_round(s);
        send_demand(t);
        continue;
      }
      if (cfg.prefetcher != RT_UNIT_PF_NONE && pq_live > 0) {
        const uint32_t i = pq_head & (a.pq_cap - 1u);
        const unsigned long long addr = pq[2 * i], base = pq[2 * i + 1];
        if (prefetch_issuable(base)) {
          __syncwarp();
          if (lane == 0) {
            dead[i] = 1;
            QueuedEntry* q = queued_entry(addr, false);
            if (q) q->first = pq_next[i];  // the queue's head is its address's oldest request
            pq_drop_dead();
          }
          --pq_live;
          pq_head = __shfl_sync(kFull, pq_head, 0);
          prefetch(addr, base, t);
          continue;
        }
      }
      // An idle cycle: every resident warp waits for its round (schedule()
      // found none ready and no request is left to send).  Until the earliest
      // round is due nothing happens but decisions that change nothing and
      // metadata returns, which matter to a queued request that waits for one.
      uint32_t until = min(next_retire, tcap);
      if (treelets && (hist_dirty || !quiet)) until = min(until, next_decide);
      if (pq_live > 0 && S.mr_head != S.mr_tail) until = min(until, metaret[S.mr_head % kMetaRing].t);
      if (until > t + 1) {
        if (treelets && next_decide < until) {
          const uint32_t k = (until - next_decide + cfg.prefetch_delay - 1u) / cfg.prefetch_delay;
          decisions += k;
          next_decide += k * cfg.prefetch_delay;
        }
        t = until - 1u;
      }
    }
    if (lane == 0) st.decisions = decisions;
    __syncwarp();
    if (lane == 0) {
      st.effectiveness[RT_PF_NEVER_USED] = uncl - uncl_accessed;
      st.unclassified_but_accessed = uncl_accessed;
      if (S.full) st.status |= 1;
    }
    __syncwarp();
  }
};

__global__ void __launch_bounds__(32, 1) unit_replay_kernel(ReplayArgs a) {
  extern __shared__ __align__(16) uint8_t replay_smem[];
  UnitShared& sh = *reinterpret_cast<UnitShared*>(replay_smem);
  Line* smem_lines = reinterpret_cast<Line*>(replay_smem + ((sizeof(UnitShared) + 15) & ~(size_t)15));
  const uint32_t u = blockIdx.x;
  WUnit unit(a, u, sh, smem_lines);
  unit.run(u);
  rtd::touch_l1_done();
  if ((threadIdx.x & 31u) == 0) a.stats[u] = unit.st;
}

}  // namespace rtr
