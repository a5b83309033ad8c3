// The predictor's output layer on the fifth-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory), fused with its softmax
// cross-entropy so that the batch x treelets logits never reach global memory.
//
//   z[b, c] = h2[b, :] . W3[:, c] + b3[c]            (K = 64, c over all treelets)
//   loss    = mean_b (logsumexp_c z[b, c] - z[b, target_b])
//   dz      = (softmax(z) - onehot(target)) / n
//   dW3 = h2^T dz,  db3 = column sums of dz,  dh2 = dz W3^T
//
// Two passes compute the logits tile by tile instead of storing them:
//   out_stats_kernel  per (128-row tile, column split): the online max and
//                     exp-sum of every row, and the target's logit (or, for
//                     prediction, the four largest logits);
//   out_grad_kernel   per (up to four row tiles, column split): dz of a tile,
//                     then both products of it, dh2 += dz . W3 and
//                     [dW3 | db3]^T += dz^T . [h2 | 1], on the tensor cores.
//
// Operands live in shared memory in the canonical K-major layout without
// swizzle: 8-row x 16-byte core matrices, core matrices of one row group
// 128 bytes apart along K (the leading-dimension offset), row groups 16 * (K
// extent) bytes apart (the stride-dimension offset).  A product whose K runs
// along a tile's rows reads the same tile as an MN-major operand.  One thread
// issues the MMAs and commits them to an mbarrier; every wait is bounded and a
// wait that gives up sets the status word instead of hanging.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "f32x2.cuh"

namespace tcm {

using bf16 = __nv_bfloat16;

constexpr int TM = 128;          // rows of a tile (TMEM lanes)
constexpr int TN = 128;          // columns (treelets) of a chunk
constexpr int HK = 64;           // hidden width (K of the logits product)
constexpr int HX = 80;           // [h2 | 1 | 0 ...] rows of the dW3 operand
// Eight warps a CTA: warp w reads TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31
// (the lanes a warp may access) and column half w / 4 of every chunk.
constexpr int kThreads = 256;
// TMEM columns a CTA of pass 1 allocates: four CTAs share an SM's 512, and one's
// epilogue runs while the others' MMAs and copies do.
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kTries = 1u << 22;
constexpr float kLog2e = 1.4426950408889634f;

// 2^x (MUFU ex2, flush-to-zero): the softmax exponentials in base 2.
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: K-major, no swizzle, leading-dimension
// offset 128 bytes, the given stride-dimension offset, descriptor version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) |
         ((uint64_t)1 << 46);
}

// The same tile read the other way round, its row index as K (MN-major, no
// swizzle): core matrices 128 bytes apart along M or N (the stride-dimension
// offset), the given distance apart along K (the leading-dimension offset).
__device__ __forceinline__ uint64_t sdesc_mn(uint32_t addr, uint32_t lbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)(128u >> 4) << 32) |
         ((uint64_t)1 << 46);
}
constexpr uint32_t kAMn = 1u << 15, kBMn = 1u << 16;  // instruction descriptor: A, B MN-major

// Instruction descriptor of kind::f16: BF16 A and B (both K-major), FP32 accumulator.
__host__ __device__ constexpr uint32_t idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(id), "r"(accumulate));
}

__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(bar)));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Bounded wait for the phase of the given parity; false if it gave up.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kTries; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(su32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// COLS TMEM columns for the CTA (one warp allocates); returns the base address.
// The .sync.aligned tcgen05 instructions need their whole warp converged,
// hence the __syncwarp before each.
template <uint32_t COLS = kTmemCols>
__device__ __forceinline__ uint32_t tmem_alloc(uint32_t* slot, int warp) {
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(slot)),
                 "n"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  return *slot;
}

template <uint32_t COLS = kTmemCols>
__device__ __forceinline__ void tmem_free(uint32_t base, int warp) {
  tc_before_sync();
  __syncthreads();
  __syncwarp();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLS));
}

// 32 consecutive FP32 columns of this thread's TMEM lane; every lane of the
// warp must call it (the load is warp-collective).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// 16 of them.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// Byte offset of element (row r, k) of a K-major tile whose K extent is kx.
__device__ __forceinline__ uint32_t koff(uint32_t r, uint32_t k, uint32_t kx) {
  return (r >> 3) * (kx * 16u) + (k >> 3) * 128u + (r & 7u) * 16u + (k & 7u) * 2u;
}

// Asynchronous 16-byte copy global -> shared (cp.async, L2 only).
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(su32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(su32(dst)), "l"(src) : "memory");
}
// Named barrier of `threads` threads: arrive without waiting, or wait.
__device__ __forceinline__ void nb_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void nb_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Copies rows [r0, r0 + rows) x K columns [k0, k0 + kx) of a row-major BF16
// matrix (row stride ld elements, 16-byte aligned rows) into a K-major tile;
// rows past `valid` read as zero (written directly, not copied).
__device__ __forceinline__ void load_tile(uint8_t* tile, const bf16* g, uint64_t ld, uint32_t r0, uint32_t rows,
                                          uint32_t valid, uint32_t k0, uint32_t kx) {
  const uint32_t chunks = rows * (kx / 8u);
  for (uint32_t i = threadIdx.x; i < chunks; i += blockDim.x) {
    const uint32_t r = i / (kx / 8u), c = i % (kx / 8u);
    uint8_t* dst = tile + koff(r, c * 8u, kx);
    if (r0 + r < valid) cp16(dst, g + (uint64_t)(r0 + r) * ld + k0 + c * 8u);
    else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
  }
}

struct OutArgs {
  const bf16* h2;       // [n][64] hidden activations of the last layer
  const bf16* w3t;      // [cp][64]: W3^T, rows past C zero
  const float* b3;      // [C]
  const rt_mlp_sample* s;
  uint32_t n, C, cp;    // rows, treelets, padded treelets (multiple of TN)
  uint32_t splits;      // column splits of the row-tile passes
  float* part;          // [3][splits][n]: max, exp-sum, target logit (stats); or [splits][n][8] top-4 (pairs)
  const float* lse;     // [n]
  float* dh2;           // [splits][n][64]: a partial sum per split that has chunks
  float* dw3;           // [64][C]
  float* db3;           // [C]
  uint32_t* status;     // bit 0: a bounded wait gave up
};

// Splits that have chunks: the first so many.
__host__ __device__ constexpr uint32_t live_splits(uint32_t cp, uint32_t splits) {
  const uint32_t chunks = cp / TN, per = (chunks + splits - 1) / splits;
  return (chunks + per - 1) / per;
}

// Columns [c_beg, c_end) of split `sp`, in whole chunks.
__device__ __forceinline__ void split_range(const OutArgs& a, uint32_t sp, uint32_t& c_beg, uint32_t& c_end) {
  const uint32_t chunks = a.cp / TN, per = (chunks + a.splits - 1) / a.splits;
  c_beg = min(chunks, sp * per);
  c_end = min(chunks, c_beg + per);
}

// Logits of one chunk: D[128 x 128] = A[128 x 64] . B[128 x 64]^T, issued by one thread.
__device__ __forceinline__ void mma_logits(uint32_t d, const uint8_t* a_tile, const uint8_t* b_tile) {
#pragma unroll
  for (int kk = 0; kk < HK / 16; ++kk)
    mma(d, sdesc(su32(a_tile) + kk * 256u, HK * 16u), sdesc(su32(b_tile) + kk * 256u, HK * 16u), idesc(TM, TN),
        kk > 0 ? 1u : 0u);
}

// The chunk's biases into shared memory (asynchronously; zero past C).
__device__ __forceinline__ void load_bias(float* dst, const float* b3, uint32_t c, uint32_t C) {
  for (uint32_t j = threadIdx.x; j < (uint32_t)TN; j += blockDim.x) {
    const uint32_t col = c * TN + j;
    if (col < C) cp4(dst + j, b3 + col);
    else dst[j] = 0.0f;
  }
}

// 32 logits of this thread's row, bias added; columns past C and invalid
// rows read -inf.
__device__ __forceinline__ void logits32(uint32_t taddr, const float* bias, uint32_t col0, uint32_t C, bool valid_row,
                                         float* v) {
  tmem_ld32(taddr, v);
  if (valid_row && col0 + 32 <= C) {
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 b = *reinterpret_cast<const float4*>(bias + j);
      rtd::f2_unpack(rtd::f2_add(rtd::f2_pack(v[j], v[j + 1]), rtd::f2_pack(b.x, b.y)), v[j], v[j + 1]);
      rtd::f2_unpack(rtd::f2_add(rtd::f2_pack(v[j + 2], v[j + 3]), rtd::f2_pack(b.z, b.w)), v[j + 2], v[j + 3]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = (valid_row && col0 + j < C) ? v[j] + bias[j] : -INFINITY;
  }
}

__device__ __forceinline__ float max32(const float* v) {
  float t[11];
#pragma unroll
  for (int j = 0; j < 10; ++j) t[j] = fmaxf(fmaxf(v[3 * j], v[3 * j + 1]), v[3 * j + 2]);
  t[10] = fmaxf(v[30], v[31]);
  const float a = fmaxf(fmaxf(t[0], t[1]), t[2]), b = fmaxf(fmaxf(t[3], t[4]), t[5]);
  const float c = fmaxf(fmaxf(t[6], t[7]), t[8]), d = fmaxf(t[9], t[10]);
  return fmaxf(fmaxf(fmaxf(a, b), c), d);
}

// Pass 1: per row, the running maximum and exp-sum over the split's columns
// and the target's logit (TOPK = false); or the four largest logits (TOPK).
// Each thread covers one row and one column half of every chunk, so a row's
// results are written as two partial results (index 2 * split + half).
// Four CTAs per SM hide one another's waits: 48 us for 4,096 samples and about
// 22,150 treelets on a GB300, two CTAs with two logits buffers each 57.
template <bool TOPK>
__global__ void __launch_bounds__(kThreads, 4) out_stats_kernel(OutArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* a_tile = smem;                                        // 128 x 64 bf16: 16 KiB
  uint8_t* b_tile0 = smem + 16384;                               // 128 x 64 bf16: 16 KiB, two buffers
  float* bias = reinterpret_cast<float*>(smem + 16384 + 32768);  // 2 x 128
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, quad = warp & 3, half = warp >> 2;
  const uint32_t row0 = blockIdx.x * TM;
  uint32_t c_beg, c_end;
  split_range(a, blockIdx.y, c_beg, c_end);
  if (tid == 0) bar_init(&bar);
  const uint32_t tmem = tmem_alloc(&tmem_slot, warp);
  const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
  const uint32_t row = row0 + (uint32_t)(quad * 32) + (uint32_t)(tid & 31);
  const bool valid_row = row < a.n;
  const uint32_t tgt = valid_row ? a.s[row].target : 0xFFFFFFFFu;
  float m = -INFINITY, ssum = 0.0f, zt = -INFINITY;
  float tv[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  uint32_t ti[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
  uint32_t phase = 0;
  bool ok = true;
  auto load_chunk = [&](uint32_t c, uint32_t buf) {
    load_tile(b_tile0 + buf * 16384, a.w3t, HK, c * TN, TN, a.cp, 0, HK);
    load_bias(bias + buf * TN, a.b3, c, a.C);
    cp_commit();
  };
  auto issue = [&](uint32_t buf) {  // once the chunk's operands are in place
    cp_wait_all();
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    if (tid == 0) {
      tc_after_sync();
      mma_logits(tmem, a_tile, b_tile0 + buf * 16384);
      commit(&bar);
    }
  };
  if (c_beg < c_end) {
    load_tile(a_tile, a.h2, HK, row0, TM, a.n, 0, HK);
    load_chunk(c_beg, 0);
    issue(0);
  }
  for (uint32_t c = c_beg; c < c_end; ++c) {
    const uint32_t buf = (c - c_beg) & 1u;
    // into the other buffer: its last reader, the MMA of chunk c - 1, is done
    if (c + 1 < c_end) load_chunk(c + 1, buf ^ 1u);
    if (!bar_wait(&bar, phase)) ok = false;
    phase ^= 1u;
    tc_after_sync();
#pragma unroll 1
    for (int sl = 0; sl < 2; ++sl) {
      const uint32_t cl0 = (uint32_t)(half * 64 + sl * 32);  // column within the chunk
      const uint32_t col0 = c * TN + cl0;
      float v[32];
      logits32(lanes + cl0, bias + buf * TN + cl0, col0, a.C, valid_row, v);
      if (TOPK) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float x = v[j];
          const uint32_t ix = col0 + j;
          if (x > tv[3]) {  // columns arrive in ascending order: ties keep the lower index
            if (x > tv[2]) {
              tv[3] = tv[2], ti[3] = ti[2];
              if (x > tv[1]) {
                tv[2] = tv[1], ti[2] = ti[1];
                if (x > tv[0]) {
                  tv[1] = tv[0], ti[1] = ti[0];
                  tv[0] = x, ti[0] = ix;
                } else {
                  tv[1] = x, ti[1] = ix;
                }
              } else {
                tv[2] = x, ti[2] = ix;
              }
            } else {
              tv[3] = x, ti[3] = ix;
            }
          }
        }
      } else {
        if (tgt - col0 < 32u) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (col0 + j == tgt) zt = v[j];
        }
        const float mx = max32(v);
        if (mx > -INFINITY) {
          const float mn = fmaxf(m, mx), sh = mn * kLog2e;
          unsigned long long acc = rtd::f2_pack(ssum * ex2(fmaf(m, kLog2e, -sh)), 0.0f);
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float x, y;
            rtd::f2_unpack(rtd::f2_fma(rtd::f2_pack(v[j], v[j + 1]), rtd::f2_pack(kLog2e, kLog2e), rtd::f2_pack(-sh, -sh)), x, y);
            acc = rtd::f2_add(acc, rtd::f2_pack(ex2(x), ex2(y)));
          }
          float acc0, acc1;
          rtd::f2_unpack(acc, acc0, acc1);
          ssum = acc0 + acc1;
          m = mn;
        }
      }
    }
    if (c + 1 < c_end) issue(buf ^ 1u);  // every thread has read chunk c's logits
  }
  if (!ok) atomicOr(a.status, 1u);
  cp_wait_all();  // no copy may still be landing when the CTA exits
  const uint32_t splits2 = a.splits * 2, sp = blockIdx.y * 2 + (uint32_t)half;
  if (valid_row) {
    if (TOPK) {
      float* p = a.part + ((uint64_t)sp * a.n + row) * 8;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        p[2 * k] = tv[k];
        p[2 * k + 1] = __uint_as_float(ti[k]);
      }
    } else {
      a.part[((uint64_t)0 * splits2 + sp) * a.n + row] = m;
      a.part[((uint64_t)1 * splits2 + sp) * a.n + row] = ssum;
      a.part[((uint64_t)2 * splits2 + sp) * a.n + row] = zt;
    }
  }
  tmem_free(tmem, warp);
}

// Pass 1 combined over the partial results: lse per row and the mean loss.
// A block takes 32 rows, each of its warps every eighth partial result of
// them; the terms' sum is taken in the splits' order (one thread per row walking
// up to 304 partial results took 19 us for 4,096 rows on a GB300, now 9).
// The rows' losses are added up in double, so that the sum does not depend on
// the order of the CTAs.
constexpr int kLseRows = 32, kLseWarps = 8, kMaxPartials = 2 * 152;
__global__ void __launch_bounds__(kLseWarps * 32) out_lse_kernel(const float* __restrict__ part, uint32_t splits,
                                                                 uint32_t n, const rt_mlp_sample* s, uint32_t C,
                                                                 float* __restrict__ lse, double* __restrict__ loss) {
  __shared__ float term[kMaxPartials][kLseRows], top[kLseWarps][kLseRows], tz[kLseWarps][kLseRows];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, b = blockIdx.x * kLseRows + lane;
  float m = -INFINITY, zt = -INFINITY;
  if (b < n)
    for (uint32_t k = warp; k < splits; k += kLseWarps) {
      m = fmaxf(m, part[(uint64_t)k * n + b]);
      zt = fmaxf(zt, part[((uint64_t)2 * splits + k) * n + b]);
    }
  top[warp][lane] = m;
  tz[warp][lane] = zt;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kLseWarps; ++w) {
    m = fmaxf(m, top[w][lane]);
    zt = fmaxf(zt, tz[w][lane]);
  }
  for (uint32_t k = warp; k < splits; k += kLseWarps) {
    const float mk = b < n ? part[(uint64_t)k * n + b] : -INFINITY;
    term[k][lane] = mk > -INFINITY ? part[((uint64_t)splits + k) * n + b] * __expf(mk - m) : 0.0f;
  }
  __syncthreads();
  if (warp != 0) return;
  float sum = 0.0f;
  for (uint32_t k = 0; k < splits; ++k) sum += term[k][lane];
  double mine = 0.0;
  if (b < n) {
    const float l = m + logf(sum);
    lse[b] = l;
    if (s[b].target < C) mine = (double)(l - zt) / (double)n;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, d);
  if (lane == 0) atomicAdd(loss, mine);
}

// Pass 1 (TOPK) combined: the four largest over the partial results' candidates.
__global__ void out_top4_kernel(const float* __restrict__ part, uint32_t splits, uint32_t n, uint32_t* __restrict__ out) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  float tv[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  uint32_t ti[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
  for (uint32_t k = 0; k < splits; ++k)
    for (int q = 0; q < 4; ++q) {
      const float* p = part + ((uint64_t)k * n + b) * 8 + 2 * q;
      const float x = p[0];
      const uint32_t ix = __float_as_uint(p[1]);
      if (ix == 0xFFFFFFFFu) continue;
      // insert, ties to the lower index
      int pos = 4;
      while (pos > 0 && (x > tv[pos - 1] || (x == tv[pos - 1] && ix < ti[pos - 1]))) --pos;
      if (pos < 4) {
        for (int t = 3; t > pos; --t) tv[t] = tv[t - 1], ti[t] = ti[t - 1];
        tv[pos] = x, ti[pos] = ix;
      }
    }
  for (int q = 0; q < 4; ++q) out[(uint64_t)b * 4 + q] = ti[q];
}

// Pass 2, both gradients from one recomputation.  A CTA takes up to kTiles
// 128-row tiles through the chunks of a column split; per chunk and tile the
// logits (A = h2 tile, B = W3^T chunk), dz from them into shared memory, and
// from that one tile
//   dh2[tile]            += dz . W3             (A = dz,   B = W3^T chunk, read along its rows)
//   [dW3 | db3]^T[chunk] += dz^T . [h2 | 1]     (A = dz read along its rows, B = [h2 | 1] tile, too)
// so that neither operand is kept or stored a second time in transposed form.
// Tensor memory holds the logits, the chunk's dW3 and every tile's dh2; dh2
// leaves it once per split, as a partial sum, dW3 once per chunk, added into the
// zeroed gradient.
//
// What bounds it: each tile's chain from logits through tensor memory, the
// exponentials and dz to the products (tensor pipe 46% of the time, issue 35%).
// The next logits and the last products run under the epilogue of sixteen
// warps; a seventeenth issues them, so that no warp waits for another but at a
// chunk's start; W3 chunks arrive two ahead.  GB300, 4,096 samples, about
// 22,150 treelets: 68 us; with CTA-wide barriers and one thread of the epilogue
// issuing 90; with dz in two buffers 76 (spills); as two kernels that
// recompute the logits each and wait for every product, 111 and 148.
constexpr uint32_t kTiles = 4;
constexpr uint32_t kColDw3 = TN, kColDh2 = kColDw3 + 96;  // TMEM columns (dW3 uses 80)
static_assert(kColDh2 + kTiles * HK <= 512, "tensor memory");
// Epilogue threads: warp w has TMEM lanes 32 (w % 4) .. + 31 and column quarter
// w / 4 of a chunk.  One more warp issues the products.
constexpr int kGradThreads = 512;
constexpr uint32_t kH2Bytes = TM * HX * 2, kW3Bytes = TN * HK * 2, kDzBytes = TM * TN * 2;
constexpr uint32_t kW3Bufs = 3;    // read until a chunk's last product, loaded two chunks ahead
constexpr uint32_t kGradSmem = kTiles * kH2Bytes + kW3Bufs * (kW3Bytes + TN * 4) + kDzBytes;

constexpr int kBarRead = 1, kBarDz = 2, kBarChunk = 3;  // named barriers

__global__ void __launch_bounds__(kGradThreads + 32, 1) out_grad_kernel(OutArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* const h2 = smem;                          // the tiles' [h2 | 1 | 0], 128 x 80 each
  uint8_t* const w3 = h2 + kTiles * kH2Bytes;        // W3^T chunks, 128 x 64 each
  uint8_t* const dz = w3 + kW3Bufs * kW3Bytes;       // 128 x 128
  float* const bias = reinterpret_cast<float*>(dz + kDzBytes);
  __shared__ __align__(8) uint64_t bar_l, bar_g;     // logits ready; gradient products done
  __shared__ uint32_t tmem_slot, s_tgt[kTiles][TM];
  __shared__ float s_sh[kTiles][TM];                 // lse * log2(e)
  const uint32_t tid = threadIdx.x, warp = tid >> 5, quad = warp & 3u, quarter = warp >> 2;
  if (tid == 0) {
    bar_init(&bar_l);
    bar_init(&bar_g);
  }
  const uint32_t tmem = tmem_alloc<512>(&tmem_slot, (int)warp);
  const uint32_t lanes = tmem + ((quad * 32u) << 16);
  const uint32_t r = quad * 32u + (tid & 31u);
  const float inv_n = 1.0f / (float)a.n;
  if (tid < kGradThreads) {  // the one and the zeros behind every h2 row
    *reinterpret_cast<uint4*>(h2 + (tid / TM) * kH2Bytes + koff(tid % TM, HK, HX)) = make_uint4(0x3f80u, 0, 0, 0);
    *reinterpret_cast<uint4*>(h2 + (tid / TM) * kH2Bytes + koff(tid % TM, HK + 8, HX)) = make_uint4(0, 0, 0, 0);
  }
  const uint32_t tiles = (a.n + TM - 1) / TM, units = a.splits * tiles;  // unit: a split of a tile
  const uint32_t u_end = (uint32_t)((uint64_t)units * (blockIdx.x + 1u) / gridDim.x);
  uint32_t u = (uint32_t)((uint64_t)units * blockIdx.x / gridDim.x), par_l = 0, par_g = 0;
  bool ok = true;
  auto load_chunk = [&](uint32_t c, uint32_t buf) {  // by the epilogue threads
    for (uint32_t x = tid; x < TN * (HK / 8u); x += kGradThreads) {
      const uint32_t row = x / (HK / 8u), k = x % (HK / 8u) * 8u;
      cp16(w3 + buf * kW3Bytes + koff(row, k, HK), a.w3t + (uint64_t)(c * TN + row) * HK + k);
    }
    load_bias(bias + buf * TN, a.b3, c, a.C);
    cp_commit();
  };
  auto issue_logits = [&](uint32_t i, uint32_t buf) {
    tc_after_sync();
#pragma unroll
    for (uint32_t kk = 0; kk < HK / 16; ++kk)
      mma(tmem, sdesc(su32(h2 + i * kH2Bytes) + kk * 256u, HX * 16u), sdesc(su32(w3 + buf * kW3Bytes) + kk * 256u, HK * 16u),
          idesc(TM, TN), kk > 0 ? 1u : 0u);
    commit(&bar_l);
  };
  auto issue_products = [&](uint32_t i, uint32_t buf, bool more) {
    tc_after_sync();
#pragma unroll
    for (uint32_t kk = 0; kk < TN / 16; ++kk)
      mma(tmem + kColDh2 + i * HK, sdesc(su32(dz) + kk * 256u, TN * 16u),
          sdesc_mn(su32(w3 + buf * kW3Bytes) + kk * (2u * HK * 16u), HK * 16u), idesc(TM, HK) | kBMn,
          (more || kk > 0) ? 1u : 0u);
#pragma unroll
    for (uint32_t kk = 0; kk < TM / 16; ++kk)
      mma(tmem + kColDw3, sdesc_mn(su32(dz) + kk * (2u * TN * 16u), TN * 16u),
          sdesc_mn(su32(h2 + i * kH2Bytes) + kk * (2u * HX * 16u), HX * 16u), idesc(TM, HX) | kAMn | kBMn,
          (i > 0 || kk > 0) ? 1u : 0u);
    commit(&bar_g);
  };
  auto next = [](uint32_t buf) { return buf + 1 == kW3Bufs ? 0u : buf + 1; };
  // lane r of the accumulator is the chunk's column r: 64 weight gradients, then the bias gradient
  auto add_dw3 = [&](uint32_t c) {
    const uint32_t col = c * TN + r, k0 = quarter * 16u;
    float v[16];
    tmem_ld16(lanes + kColDw3 + k0, v);
    if (col < a.C) {
#pragma unroll
      for (int k = 0; k < 16; ++k) atomicAdd(a.dw3 + (uint64_t)(k0 + k) * a.C + col, v[k]);
    }
    if (quarter == 0) {
      tmem_ld16(lanes + kColDw3 + HK, v);
      if (col < a.C) atomicAdd(a.db3 + col, v[0]);
    }
  };
  while (u < u_end) {
    // this CTA's tiles t0 .. t0 + nt - 1 of one split
    const uint32_t split = u / tiles, t0 = u % tiles, nt = min(min(tiles - t0, u_end - u), kTiles);
    uint32_t c_beg, c_end;
    split_range(a, split, c_beg, c_end);
    u += nt;
    if (c_beg >= c_end) continue;
    for (uint32_t x = tid; x < nt * TM * (HK / 8u); x += blockDim.x) {
      const uint32_t row = x / (HK / 8u), k = x % (HK / 8u) * 8u;
      uint8_t* dst = h2 + row / TM * kH2Bytes + koff(row % TM, k, HX);
      if (t0 * TM + row < a.n) cp16(dst, a.h2 + (uint64_t)(t0 * TM + row) * HK + k);
      else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    }
    if (tid < nt * TM) {
      const uint32_t row = t0 * TM + tid;
      s_tgt[tid / TM][tid % TM] = row < a.n ? a.s[row].target : 0xFFFFFFFFu;
      s_sh[tid / TM][tid % TM] = row < a.n ? a.lse[row] * kLog2e : 0.0f;
    }
    if (tid < kGradThreads) {
      load_chunk(c_beg, 0);
      if (c_beg + 1 < c_end) load_chunk(c_beg + 1, 1);
    }
    cp_wait_all();
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    if (warp == kGradThreads / 32) {
      if (tid == kGradThreads) issue_logits(0, 0);
      uint32_t buf = 0;
      for (uint32_t c = c_beg; c < c_end; ++c, buf = next(buf))
        for (uint32_t i = 0; i < nt; ++i) {
          const bool last = i + 1 == nt && c + 1 == c_end;
          nb_sync(kBarRead, kGradThreads + 32);
          if (tid == kGradThreads && !last) issue_logits(i + 1 == nt ? 0u : i + 1, i + 1 == nt ? next(buf) : buf);
          __syncwarp();
          nb_sync(kBarDz, kGradThreads + 32);
          if (tid == kGradThreads) issue_products(i, buf, c > c_beg);
          __syncwarp();
        }
    } else {
      uint32_t buf = 0;
      for (uint32_t c = c_beg; c < c_end; ++c, buf = next(buf)) {
        if (c > c_beg) nb_sync(kBarChunk, kGradThreads);  // every thread's part of the chunk's biases is in place
        for (uint32_t i = 0; i < nt; ++i) {
          const uint32_t tgt = s_tgt[i][r];
          const float sh = s_sh[i][r];
          if (!bar_wait(&bar_l, par_l)) ok = false;
          par_l ^= 1u;
          tc_after_sync();
          const uint32_t cl0 = quarter * 32u, col0 = c * TN + cl0;
          float v[32];
          logits32(lanes + cl0, bias + buf * TN + cl0, col0, a.C, (t0 + i) * TM + r < a.n, v);
          cp_wait_all();  // the chunk asked for one chunk ago
          fence_async_smem();
          tc_before_sync();
          nb_arrive(kBarRead, kGradThreads + 32);
#pragma unroll
          for (int k = 0; k < 32; k += 2) {  // ex2(-inf) = 0: dead columns give 0
            rtd::f2_unpack(rtd::f2_fma(rtd::f2_pack(v[k], v[k + 1]), rtd::f2_pack(kLog2e, kLog2e), rtd::f2_pack(-sh, -sh)), v[k], v[k + 1]);
            v[k] = ex2(v[k]);
            v[k + 1] = ex2(v[k + 1]);
          }
          if (tgt - col0 < 32u) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (col0 + k == tgt) v[k] -= 1.0f;
          }
          uint32_t w[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float x, y;
            rtd::f2_unpack(rtd::f2_mul(rtd::f2_pack(v[2 * k], v[2 * k + 1]), rtd::f2_pack(inv_n, inv_n)), x, y);
            const __nv_bfloat162 pr = __floats2bfloat162_rn(x, y);
            w[k] = *reinterpret_cast<const uint32_t*>(&pr);
          }
          if (i > 0 || c > c_beg) {
            if (!bar_wait(&bar_g, par_g)) ok = false;  // the last products have read dz
            par_g ^= 1u;
            tc_after_sync();
          }
          if (i == 0) {
            if (c > c_beg) add_dw3(c - 1);
            if (c + 2 < c_end) load_chunk(c + 2, next(next(buf)));  // over chunk c - 1
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<uint4*>(dz + koff(r, cl0 + (uint32_t)(q * 8), TN)) =
                make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
          fence_async_smem();
          tc_before_sync();
          nb_arrive(kBarDz, kGradThreads + 32);
        }
      }
      if (!bar_wait(&bar_g, par_g)) ok = false;
      par_g ^= 1u;
      tc_after_sync();
      add_dw3(c_end - 1);
      for (uint32_t i = 0; i < nt; ++i) {  // a quarter of the tile's columns each
        float v[16];
        tmem_ld16(lanes + kColDh2 + i * HK + quarter * 16u, v);
        const uint32_t row = (t0 + i) * TM + r;
        if (row < a.n) {
          float4* p = reinterpret_cast<float4*>(a.dh2 + ((uint64_t)split * a.n + row) * HK + quarter * 16u);
#pragma unroll
          for (int q = 0; q < 4; ++q) p[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
      }
    }
    tc_before_sync();
    __syncthreads();  // the next tiles' operands and accumulators may replace these
    tc_after_sync();
  }
  if (!ok) atomicOr(a.status, 1u);
  tmem_free<512>(tmem, (int)warp);
}

// W3 (FP32 master, [64][C]) as the padded BF16 operand W3^T ([cp][64]).  One
// block per 32 columns: W3's rows are read along the columns, W3^T's written
// through a shared-memory transpose (one thread per column wrote 2-byte entries
// 128 bytes apart).
__global__ void __launch_bounds__(256) w3_operand_kernel(const float* __restrict__ w3, uint32_t C,
                                                         bf16* __restrict__ w3t) {
  __shared__ __align__(4) bf16 t[32][HK + 2];  // [column][k]: rows 132 bytes apart, no bank conflicts
  const uint32_t c0 = blockIdx.x * 32, tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;
  const uint32_t c = c0 + tx;
  for (uint32_t k = ty; k < (uint32_t)HK; k += 8)
    t[tx][k] = __float2bfloat16_rn(c < C ? w3[(uint64_t)k * C + c] : 0.0f);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 32u * (HK / 2); i += blockDim.x) {
    const uint32_t cl = i / (HK / 2), kp = i % (HK / 2);
    reinterpret_cast<uint32_t*>(w3t + (uint64_t)(c0 + cl) * HK)[kp] = *reinterpret_cast<const uint32_t*>(&t[cl][2 * kp]);
  }
}

}  // namespace tcm
