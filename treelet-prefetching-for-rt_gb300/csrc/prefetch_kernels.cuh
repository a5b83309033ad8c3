// Treelet-prefetch decision of an RT unit (src/gpgpu-sim/shader.cc:3419-3683,
// or the copies the pipelined treelet queue, :3780-3932, and the treelet
// queue, :4020-4060, run) as a batched kernel: one CTA per RT unit.
//
// The reference builds std::map<treelet root, count> over the first pending
// access of every resident lane, takes the first maximum in ascending root
// order, applies the heuristic, and queues the treelet's members as 32-byte
// requests unless it was the last (or last second) treelet prefetched.  Here
// the lanes count their roots in a shared-memory table, the two most popular
// roots come out of one reduction, and the first warp applies the same
// heuristic arithmetic (IEEE double for the popularity share, as in the
// reference), searching the roots and adding up the members' requests 32 at a
// time.  A decision is a chain of small steps, bound by their latency: 152 units
// of 512 lanes take 7.7 us on a GB300 when the most popular treelet was the last
// one queued (with events around the call 10.9, and 10.9 when every unit queues
// its treelet's 256 requests); sorting the roots and walking the runs in one
// thread took 43.7 (47.8, and 49.8).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/treelet_rt.h"

namespace rtk {

constexpr int kMaxLanes = 1024;

struct PrefetchArgs {
  const uint32_t* next_unit;
  uint32_t n_groups, lanes;
  rt_prefetch_params p;
  rt_prefetch_state* state;
  rt_prefetch_decision* out;
  const uint2* meta;                 // unit -> root
  uint32_t n_units;
  const uint32_t* roots;             // dense -> root unit (ascending)
  const unsigned long long* member_first;  // dense -> first member, n + 1
  const uint16_t* member_bytes;
  uint32_t n_treelets;
};

// Dense id of a treelet root, kNone if it is none: 32 probes at a time (a full
// warp calls with the same root).
__device__ __forceinline__ uint32_t dense_of_root(const PrefetchArgs& a, uint32_t root) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lo = 0, hi = a.n_treelets;  // the first root >= `root` is in [lo, hi]
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31u) / 32u, at = lo + lane * step;
    // probes below `root` are a prefix of the lanes
    const uint32_t less = __popc(__ballot_sync(0xffffffffu, at < hi && a.roots[at] < root));
    if (less == 0) {
      hi = lo;
    } else {
      hi = min(hi, lo + less * step);
      lo += (less - 1u) * step + 1u;
    }
  }
  return (lo < a.n_treelets && a.roots[lo] == root) ? lo : kNone;
}

// Requests of members [j0, j1) (a full warp calls).
__device__ __forceinline__ uint32_t member_chunks(const PrefetchArgs& a, unsigned long long j0, unsigned long long j1) {
  uint32_t c = 0;
  for (unsigned long long j = j0 + (threadIdx.x & 31u); j < j1; j += 32) c += (a.member_bytes[j] + 31u) / 32u;
  return __reduce_add_sync(0xffffffffu, c);
}

constexpr uint32_t kCountLog2 = 11, kCountSize = 1u << kCountLog2;  // at most 1,024 roots

__global__ void __launch_bounds__(512) prefetch_decide_kernel(PrefetchArgs a) {
  __shared__ uint32_t key[kCountSize], cnt[kCountSize];
  __shared__ unsigned long long top[2][16];
  __shared__ uint32_t sums[2][16];
  const uint32_t g = blockIdx.x;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  for (uint32_t i = tid; i < kCountSize; i += blockDim.x) {
    key[i] = kNone;
    cnt[i] = 0;
  }
  __syncthreads();
  for (uint32_t l0 = 0; l0 < a.lanes; l0 += blockDim.x) {
    const uint32_t l = l0 + tid;
    uint32_t k = kNone;
    if (l < a.lanes) {
      const uint32_t u = a.next_unit[(uint64_t)g * a.lanes + l];
      if (u != kNone && u < a.n_units) k = a.meta[u].x;
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, k);
    if (k != kNone && (uint32_t)(__ffs(peers) - 1) == lane) {
      uint32_t i = (k * 0x9E3779B1u) >> (32 - kCountLog2);
      for (;; i = (i + 1) & (kCountSize - 1)) {
        const uint32_t old = atomicCAS(&key[i], kNone, k);
        if (old == kNone || old == k) break;
      }
      atomicAdd(&cnt[i], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  // the most popular root and the next one, (count << 32 | ~root): ties go to the lowest root
  unsigned long long b0 = 0, b1 = 0;
  uint32_t total = 0, distinct = 0;
  for (uint32_t i = tid; i < kCountSize; i += blockDim.x) {
    const uint32_t c = cnt[i];
    if (!c) continue;
    total += c;
    ++distinct;
    const unsigned long long v = ((unsigned long long)c << 32) | (unsigned long long)(~key[i]);
    b1 = v > b0 ? b0 : (v > b1 ? v : b1);
    b0 = v > b0 ? v : b0;
  }
  auto top_two = [](unsigned long long& x0, unsigned long long& x1) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const unsigned long long y0 = __shfl_xor_sync(0xffffffffu, x0, s), y1 = __shfl_xor_sync(0xffffffffu, x1, s);
      const unsigned long long lo = x0 > y0 ? y0 : x0, hi1 = x1 > y1 ? x1 : y1;
      x0 = x0 > y0 ? x0 : y0;
      x1 = lo > hi1 ? lo : hi1;
    }
  };
  top_two(b0, b1);
  total = __reduce_add_sync(0xffffffffu, total);
  distinct = __reduce_add_sync(0xffffffffu, distinct);
  if (lane == 0) {
    top[0][warp] = b0;
    top[1][warp] = b1;
    sums[0][warp] = total;
    sums[1][warp] = distinct;
  }
  __syncthreads();
  if (warp != 0) return;
  const uint32_t warps = blockDim.x / 32u;
  b0 = lane < warps ? top[0][lane] : 0ull;
  b1 = lane < warps ? top[1][lane] : 0ull;
  top_two(b0, b1);
  total = __reduce_add_sync(0xffffffffu, lane < warps ? sums[0][lane] : 0u);
  distinct = __reduce_add_sync(0xffffffffu, lane < warps ? sums[1][lane] : 0u);
  const uint32_t best = b0 ? ~(uint32_t)b0 : kNone, best_cnt = (uint32_t)(b0 >> 32);
  const uint32_t next = b1 ? ~(uint32_t)b1 : kNone;
  // every lane of the warp decides alike; lane 0 writes
  rt_prefetch_state st = a.state[g];
  const uint32_t copy = a.p.variant & 3u;
  const bool pipelined = copy == RT_PREFETCH_PIPELINED_QUEUE;
  const bool flush = (a.p.variant & RT_PREFETCH_FLUSH_ON_NEW_TREELET) != 0;
  rt_prefetch_decision d;
  d.treelet = best;
  d.count = best == kNone ? 0u : best_cnt;
  d.total = total;
  d.submitted = 0;
  d.first_member = 0;
  d.n_members = 0;
  d.chunks = 0;
  d.second_treelet = kNone;
  bool submit = false;
  int num_nodes = 0;
  uint32_t bd = kNone;
  int n_nodes = 0;
  if (best != kNone) {
    bd = dense_of_root(a, best);
    if (bd != kNone) n_nodes = (int)(a.member_first[bd + 1] - a.member_first[bd]);
  }
  uint64_t queue = st.queue_len;
  if (copy == RT_PREFETCH_TREELET_QUEUE) {
    // the treelet queue's copy: the whole treelet whatever the heuristic,
    // unless it was the last one prefetched; an empty histogram names no
    // treelet (an empty member list) and is recorded as the last one
    if (st.last_prefetched != best && (uint64_t)n_nodes + queue <= a.p.max_queue) {
      const uint32_t chunks =
          bd != kNone ? member_chunks(a, a.member_first[bd], a.member_first[bd] + (unsigned long long)n_nodes) : 0u;
      queue += chunks;
      d.submitted = best != kNone ? 1u : 0u;
      d.n_members = (uint32_t)n_nodes;
      d.chunks = chunks;
      st.last_prefetched = best;
    }
    st.queue_len = (uint32_t)queue;
    __syncwarp();  // every lane has read the state
    if (lane == 0) {
      a.state[g] = st;
      a.out[g] = d;
    }
    return;
  }
  if (a.p.heuristic == RT_PREFETCH_ALWAYS) {
    submit = true;
  } else if (best != kNone) {
    const double pct = (double)best_cnt / (double)total;
    if (a.p.heuristic == RT_PREFETCH_POPULARITY) {
      if (pct >= a.p.threshold) {
        st.last_rejected = kNone;
        submit = true;
      } else {
        if (st.last_rejected != best) st.last_rejected = best;
      }
    } else {
      // the pipelined queue's copy sizes LATTER at half the treelet
      const double share = (pipelined && a.p.heuristic == RT_PREFETCH_LATTER) ? 0.5 : pct;
      num_nodes = (int)(((double)n_nodes * share) + 0.5);
      submit = true;
    }
  }
  if (submit && best != kNone && bd != kNone) {
    if (st.last_prefetched != best && (pipelined || st.last_prefetched_second != best)) {
      const bool partial = a.p.heuristic == RT_PREFETCH_PARTIAL || a.p.heuristic == RT_PREFETCH_LATTER;
      const int num = partial ? num_nodes : n_nodes;
      if ((uint64_t)num + queue <= a.p.max_queue) {
        if (flush) queue = 0;
        const int j0 = a.p.heuristic == RT_PREFETCH_LATTER ? n_nodes - num : 0;
        const int j1 = a.p.heuristic == RT_PREFETCH_LATTER ? n_nodes : num;
        const unsigned long long mf = a.member_first[bd];
        const uint32_t chunks = member_chunks(a, mf + j0, mf + j1);
        queue += chunks;
        d.submitted = 1;
        d.first_member = (uint32_t)j0;
        d.n_members = (uint32_t)(j1 - j0);
        d.chunks = chunks;
        st.last_prefetched = best;
      }
    }
  }
  if (a.p.second_prefetch && !pipelined && queue == 0 && total > 0 && distinct > 1 && st.last_prefetched == best &&
      best != kNone) {
    // next most popular treelet other than the last prefetched one, `best`
    if (next != kNone && st.last_prefetched_second != next) {
      const uint32_t sd = dense_of_root(a, next);
      const uint32_t chunks = sd != kNone ? member_chunks(a, a.member_first[sd], a.member_first[sd + 1]) : 0u;
      queue += chunks;
      d.chunks += chunks;
      d.second_treelet = next;
      st.last_prefetched_second = next;
    }
  }
  st.queue_len = (uint32_t)queue;
  __syncwarp();  // every lane has read the state
  if (lane == 0) {
    a.state[g] = st;
    a.out[g] = d;
  }
}

}  // namespace rtk
