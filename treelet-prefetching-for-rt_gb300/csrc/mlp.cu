// The learned treelet predictor: forward, softmax cross-entropy, backward,
// Adam and top-4, all on the GPU.
//
//   x  = [origin(3), dir(3), E[current](16)]           22 inputs (padded to 32)
//   h1 = GELU(x W1 + b1)                                64
//   h2 = GELU(h1 W2 + b2)                               64
//   z  = h2 W3 + b3                                     one logit per treelet
//
// Weights are used in BF16 with FP32 accumulation; FP32 master copies are
// what Adam updates.  The output layer, whose products span every treelet,
// runs on the fifth-generation tensor cores (tcgen05.mma with accumulators in
// tensor memory) fused with the softmax cross-entropy, so the batch x
// treelets logits are never stored (mlp_tc.cuh).  The two hidden layers
// (4096 x 64 x 64 at most) run on mma.sync m16n8k16 tiles, one fused kernel each way.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <vector>

#include "capi_internal.h"
#include "mlp_tc.cuh"

namespace {

constexpr int H = RT_MLP_HIDDEN;  // 64
constexpr int EMB = RT_MLP_EMBED; // 16
constexpr int XIN = 22;           // real inputs
constexpr int XP = 32;            // padded input width
using bf16 = __nv_bfloat16;

// ------------------------------------------------------------ hidden layers
// One CTA of eight warps per 64 samples runs both hidden layers, forward or
// backward, with its operands in shared memory; warp w owns rows 16 (w % 4) ..
// + 15 and column half w / 4 of a product's output (mma.sync m16n8k16, K
// ascending).  As separate products and elementwise kernels of 10-64 CTAs each,
// the two directions took 15 launches and 150 us of a 4,096-sample step on a
// GB300, nearly all of it latency; fused they take 24 us.
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.3989422804014327f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

constexpr int HB = 64;        // samples per CTA
constexpr int HT = 256;       // threads per CTA
constexpr int HP = H + 8;     // padded rows of the 64-wide tiles (16-byte rows, fragments on distinct banks)
constexpr int XPP = XP + 8;   // padded rows of the 32-wide tiles

__device__ __forceinline__ uint32_t pair_at(const bf16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// acc[j] (16 rows from `row0`, columns col0 + 8j .. + 7) = A[row][k] . B[n][k]^T,
// both K-contiguous in shared memory, over K = 16 KS.
template <int NT, int KS, int LDA, int LDB>
__device__ __forceinline__ void tile_mma(float (&acc)[NT][4], const bf16 (*A)[LDA], int row0, const bf16 (*B)[LDB],
                                         int col0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    const int k = ks * 16 + 2 * t;
    const uint32_t a0 = pair_at(&A[row0 + g][k]), a1 = pair_at(&A[row0 + g + 8][k]);
    const uint32_t a2 = pair_at(&A[row0 + g][k + 8]), a3 = pair_at(&A[row0 + g + 8][k + 8]);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const uint32_t b0 = pair_at(&B[col0 + j * 8 + g][k]), b1 = pair_at(&B[col0 + j * 8 + g][k + 8]);
      asm volatile(
          "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
          "{%0,%1,%2,%3};\n"
          : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
          : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
  }
}

// Row and column of accumulator element (j, r) of the calling lane.
__device__ __forceinline__ int acc_row(int row0, int r) { return row0 + ((threadIdx.x & 31) >> 2) + (r >= 2 ? 8 : 0); }
__device__ __forceinline__ int acc_col(int col0, int j, int r) { return col0 + j * 8 + 2 * (threadIdx.x & 3) + (r & 1); }

// Eight consecutive elements at once.
struct Eight {
  bf16 v[8];
};
__device__ __forceinline__ Eight load8(const bf16* p) {
  Eight e;
  *reinterpret_cast<uint4*>(e.v) = *reinterpret_cast<const uint4*>(p);
  return e;
}
__device__ __forceinline__ void store8(bf16* p, const Eight& e) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(e.v);
}
__device__ __forceinline__ void load8f(const float* p, float* v) {
  *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
  *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + 4);
}

// x = [origin, dir, E[current]] (a sample whose current treelet is out of range
// gets a zero embedding); h1 = GELU(x W1 + b1), h2 = GELU(h1 W2 + b2).  Stores
// x, z1, h1, z2 and h2.
__global__ void __launch_bounds__(HT) hidden_forward_kernel(
    const rt_mlp_sample* __restrict__ s, int n, const bf16* __restrict__ E, uint32_t C, const bf16* __restrict__ W1,
    const float* __restrict__ b1, const bf16* __restrict__ W2, const float* __restrict__ b2, bf16* __restrict__ X,
    float* __restrict__ Z1, bf16* __restrict__ H1, float* __restrict__ Z2, bf16* __restrict__ H2) {
  __shared__ __align__(16) bf16 xs[HB][XPP], w1[H][XPP], w2[H][HP], h1[HB][HP];
  const int tid = threadIdx.x, row0 = ((tid >> 5) & 3) * 16, col0 = (tid >> 7) * 32, base = blockIdx.x * HB;
  {  // four threads a sample: origin and direction, the embedding's halves, zeros
    const int b = tid >> 2, part = tid & 3;
    Eight e;
#pragma unroll
    for (int q = 0; q < 8; ++q) e.v[q] = __float2bfloat16(0.0f);
    if (base + b < n) {
      const rt_mlp_sample q = s[base + b];
      const bool has = q.current < C;
      if (part == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          e.v[k] = __float2bfloat16(q.origin[k]);
          e.v[3 + k] = __float2bfloat16(q.dir[k]);
        }
        if (has) e.v[6] = E[(size_t)q.current * EMB], e.v[7] = E[(size_t)q.current * EMB + 1];
      } else if (has) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (part * 8 + k < XIN) e.v[k] = E[(size_t)q.current * EMB + part * 8 + k - 6];
      }
      store8(X + (size_t)(base + b) * XP + part * 8, e);
    }
    store8(&xs[b][part * 8], e);
  }
  {  // W1 (32 x 64) and W2 (64 x 64) transposed
    const Eight e = load8(W1 + tid * 8), f = load8(W2 + tid * 8), g = load8(W2 + (HT + tid) * 8);
    const int r = tid / 8, c = tid % 8 * 8;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      w1[c + q][r] = e.v[q];
      w2[c + q][r] = f.v[q];
      w2[c + q][r + 32] = g.v[q];
    }
  }
  __syncthreads();
  float acc[4][4];
  tile_mma<4, XP / 16, XPP, XPP>(acc, xs, row0, w1, col0);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = acc_row(row0, r), c = acc_col(col0, j, r);
      const float z = acc[j][r] + b1[c];
      const bf16 h = __float2bfloat16(gelu(z));
      h1[m][c] = h;
      if (base + m < n) {
        Z1[(size_t)(base + m) * H + c] = z;
        H1[(size_t)(base + m) * H + c] = h;
      }
    }
  __syncthreads();
  tile_mma<4, H / 16, HP, HP>(acc, h1, row0, w2, col0);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = acc_row(row0, r), c = acc_col(col0, j, r);
      const float z = acc[j][r] + b2[c];
      if (base + m < n) {
        Z2[(size_t)(base + m) * H + c] = z;
        H2[(size_t)(base + m) * H + c] = __float2bfloat16(gelu(z));
      }
    }
}

// dz2 = dh2 * GELU'(z2), [dW2, db2] += h1^T [dz2], dh1 = dz2 W2^T, dz1 = dh1 *
// GELU'(z1), [dW1, db1] += x^T [dz1], dx = dz1 W1^T into the embedding's rows.
// The dz are BF16, products FP32; weight gradients are added into G.  dh2
// arrives as one partial sum per column split of the output layer.
__global__ void __launch_bounds__(HT) hidden_backward_kernel(
    const rt_mlp_sample* __restrict__ s, int n, uint32_t C, const bf16* __restrict__ W1, const bf16* __restrict__ W2,
    const bf16* __restrict__ X, const float* __restrict__ Z1, const bf16* __restrict__ H1,
    const float* __restrict__ Z2, const float* __restrict__ dH2, uint32_t splits, float* __restrict__ gE,
    float* __restrict__ gW1, float* __restrict__ gb1, float* __restrict__ gW2, float* __restrict__ gb2) {
  __shared__ __align__(16) bf16 dz[HB][HP], dzt[H][HP], ht[H][HP], w[H][HP], xt[XP][HP];
  const int tid = threadIdx.x, warp = tid >> 5, row0 = (warp & 3) * 16, col0 = (warp >> 2) * 32, base = blockIdx.x * HB;
  const bf16 zero = __float2bfloat16(0.0f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // eight columns of a sample at a time
    const int i = h * HT + tid, b = i / 8, c = i % 8 * 8;
    Eight d, e;
#pragma unroll
    for (int q = 0; q < 8; ++q) d.v[q] = e.v[q] = zero;
    if (base + b < n) {
      float g[8], z[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) g[q] = 0.0f;
#pragma unroll 8
      for (uint32_t k = 0; k < splits; ++k) {  // in the splits' order: the sum is the same on every run
        float p[8];
        load8f(dH2 + ((size_t)k * n + base + b) * H + c, p);
#pragma unroll
        for (int q = 0; q < 8; ++q) g[q] += p[q];
      }
      load8f(Z2 + (size_t)(base + b) * H + c, z);
      e = load8(H1 + (size_t)(base + b) * H + c);
#pragma unroll
      for (int q = 0; q < 8; ++q) d.v[q] = __float2bfloat16(g[q] * gelu_grad(z[q]));
    }
    store8(&dz[b][c], d);
    store8(&w[b][c], load8(W2 + i * 8));  // 64 x 64 as well: W2[k][c] row-major
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      dzt[c + q][b] = d.v[q];
      ht[c + q][b] = e.v[q];
    }
  }
  {
    const int b = tid >> 2, c = (tid & 3) * 8;
    Eight e;
#pragma unroll
    for (int q = 0; q < 8; ++q) e.v[q] = zero;
    if (base + b < n) e = load8(X + (size_t)(base + b) * XP + c);
#pragma unroll
    for (int q = 0; q < 8; ++q) xt[c + q][b] = e.v[q];
  }
  // z1 of this thread's accumulator elements, on its way while the products run
  float z1[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int b = base + acc_row(row0, r);
      z1[j][r] = b < n ? Z1[(size_t)b * H + acc_col(col0, j, r)] : 0.0f;
    }
  __syncthreads();
  float acc[4][4];
  // dW2[i][c] = sum_b h1[b][i] dz2[b][c]
  tile_mma<4, HB / 16, HP, HP>(acc, ht, row0, dzt, col0);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) atomicAdd(gW2 + acc_row(row0, r) * H + acc_col(col0, j, r), acc[j][r]);
  auto column_sum = [&](int c, float* out) {  // four threads a column
    float sum = 0.0f;
#pragma unroll
    for (int b = 0; b < HB / 4; ++b) sum += __bfloat162float(dzt[c >> 2][(c & 3) * (HB / 4) + b]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if ((c & 3) == 0) atomicAdd(out + (c >> 2), sum);
  };
  column_sum(tid, gb2);
  // dh1[b][k] = sum_c dz2[b][c] W2[k][c]
  tile_mma<4, H / 16, HP, HP>(acc, dz, row0, w, col0);
  __syncthreads();  // every reader of dz, dzt and w is done
  store8(&w[tid / 8][tid % 8 * 8], load8(W1 + tid * 8));
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int b = acc_row(row0, r), c = acc_col(col0, j, r);
      const bf16 d = base + b < n ? __float2bfloat16(acc[j][r] * gelu_grad(z1[j][r])) : zero;
      dz[b][c] = d;
      dzt[c][b] = d;
    }
  __syncthreads();
  column_sum(tid, gb1);
  if (row0 < XP) {  // dW1[i][c] = sum_b x[b][i] dz1[b][c], 22 of the 32 padded rows
    tile_mma<4, HB / 16, HP, HP>(acc, xt, row0, dzt, col0);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (acc_row(row0, r) < XIN) atomicAdd(gW1 + acc_row(row0, r) * H + acc_col(col0, j, r), acc[j][r]);
  }
  // dx[b][i] = sum_c dz1[b][c] W1[i][c]; columns 6 .. 21 are the embedding's
  float dx[2][4];
  tile_mma<2, H / 16, HP, HP>(dx, dz, row0, w, col0 / 2);
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int b = acc_row(row0, r), c = acc_col(col0 / 2, j, r);
      if (c < 6 || c >= XIN || base + b >= n) continue;
      const uint32_t cur = s[base + b].current;
      if (cur < C) atomicAdd(gE + (size_t)cur * EMB + (c - 6), dx[j][r]);
    }
}

__global__ void adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, const float* __restrict__ g,
                     uint64_t n, float lr, float c1, float c2) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = 0.9f * m[i] + 0.1f * gi;
  const float vi = 0.999f * v[i] + 0.001f * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

__global__ void to_bf16(const float* __restrict__ src, bf16* __restrict__ dst, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __float2bfloat16(src[i]);
}

// W1 (22 x 64) -> padded BF16 (32 x 64, rows 22..31 zero)
__global__ void w1_to_bf16(const float* __restrict__ w1, bf16* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < XP * H) dst[i] = __float2bfloat16(i < XIN * H ? w1[i] : 0.0f);
}

// Deterministic initial values from a hash of (seed, index).
__global__ void init_params(float* __restrict__ p, uint64_t n, uint64_t seed, uint64_t offW1, uint64_t offb1,
                            uint64_t offW2, uint64_t offb2, uint64_t offW3, uint64_t offb3) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t h = rti::pcg_hash((uint32_t)i ^ rti::pcg_hash((uint32_t)seed));
  h = rti::pcg_hash(h ^ (uint32_t)(i >> 32));
  const float u = ((float)(h >> 8) * (1.0f / 16777216.0f)) * 2.0f - 1.0f;  // [-1, 1)
  float v;
  if (i < offW1) v = 0.1f * u;                       // embedding
  else if (i < offb1) v = u * 0.2132f;               // W1: 1/sqrt(22)
  else if (i < offW2) v = 0.0f;
  else if (i < offb2) v = u * 0.125f;                // W2: 1/sqrt(64)
  else if (i < offW3) v = 0.0f;
  else if (i < offb3) v = u * 0.125f;                // W3
  else v = 0.0f;
  p[i] = v;
}

}  // namespace

struct rt_mlp {
  int device = 0;
  uint32_t C = 0;
  uint64_t n_params = 0, offW1 = 0, offb1 = 0, offW2 = 0, offb2 = 0, offW3 = 0, offb3 = 0;
  float *P = nullptr, *M = nullptr, *V = nullptr, *G = nullptr;
  bf16 *E16 = nullptr, *W1_16 = nullptr, *W2_16 = nullptr;
  bf16 *W3T = nullptr;                                 // output-layer operand (mlp_tc.cuh)
  uint32_t Cp = 0;                                     // treelets padded to the output chunk
  bf16 *X = nullptr, *H1 = nullptr, *H2 = nullptr;
  float *Z1 = nullptr, *Z2 = nullptr;
  float *lse = nullptr, *part = nullptr;
  uint32_t* tstatus = nullptr;                         // bit 0: a bounded wait of the output layer gave up
  double* loss = nullptr;                              // sum over the samples of their loss / n
  uint64_t step = 0;
  cudaStream_t st = nullptr;
};

namespace {

rt_status cfail(cudaError_t e, const char* what) {
  return rti::fail(RT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
#define MLP_CUDA(call)                                  \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return cfail(e_, #call);     \
  } while (0)

template <class T>
cudaError_t mk(T** p, size_t count) {
  return cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
}

unsigned blocks(uint64_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

void refresh_bf16(rt_mlp* m) {
  to_bf16<<<blocks((uint64_t)m->C * EMB), 256, 0, m->st>>>(m->P, m->E16, (uint64_t)m->C * EMB);
  w1_to_bf16<<<blocks(XP * H), 256, 0, m->st>>>(m->P + m->offW1, m->W1_16);
  to_bf16<<<blocks(H * H), 256, 0, m->st>>>(m->P + m->offW2, m->W2_16, H * H);
  tcm::w3_operand_kernel<<<m->Cp / 32, 256, 0, m->st>>>(m->P + m->offW3, m->C, m->W3T);
}

// Column splits of the row-tile passes of the output layer: one wave of
// four CTAs per SM over the row tiles of the batch (at most 152 splits: the
// partial-result buffer holds 2 x 152 per row).
uint32_t out_splits(const rt_mlp* m, uint32_t n) {
  const uint32_t tiles = (n + tcm::TM - 1) / tcm::TM, chunks = m->Cp / tcm::TN;
  const uint32_t want = (4 * 152 + tiles - 1) / tiles;
  return std::max<uint32_t>(1, std::min(std::min(chunks, want), 152u));
}

// Shared memory per CTA of pass 1: an h2 tile, two W3 chunks and their biases.
constexpr size_t kSmemStats = 16384 + 2 * 16384 + 1024;

tcm::OutArgs out_args(rt_mlp* m, const rt_mlp_sample* s, uint32_t n) {
  tcm::OutArgs a{};
  a.h2 = m->H2;
  a.w3t = m->W3T;
  a.b3 = m->P + m->offb3;
  a.s = s;
  a.n = n;
  a.C = m->C;
  a.cp = m->Cp;
  a.splits = out_splits(m, n);
  a.part = m->part;
  a.lse = m->lse;
  a.dh2 = m->part;  // pass 1's partial results are used up by then
  a.dw3 = m->G + m->offW3;
  a.db3 = m->G + m->offb3;
  a.status = m->tstatus;
  return a;
}

// Loss (and lse per row) of the output layer for n samples, or with top4 set
// the four largest logits of each sample instead.
void output_forward(rt_mlp* m, const rt_mlp_sample* s, uint32_t n, uint32_t* top4) {
  const tcm::OutArgs a = out_args(m, s, n);
  const dim3 grid((n + tcm::TM - 1) / tcm::TM, a.splits);
  if (top4) {
    tcm::out_stats_kernel<true><<<grid, tcm::kThreads, kSmemStats, m->st>>>(a);
    tcm::out_top4_kernel<<<blocks(n), 256, 0, m->st>>>(m->part, 2 * a.splits, n, top4);
    return;
  }
  tcm::out_stats_kernel<false><<<grid, tcm::kThreads, kSmemStats, m->st>>>(a);
  tcm::out_lse_kernel<<<blocks(n, tcm::kLseRows), tcm::kLseWarps * 32, 0, m->st>>>(m->part, 2 * a.splits, n, s, m->C,
                                                                                  m->lse, m->loss);
}

// Gradients of the output layer: dW3 and db3 into the zeroed G, dH2 as partial sums into part.
void output_backward(rt_mlp* m, const rt_mlp_sample* s, uint32_t n) {
  const tcm::OutArgs a = out_args(m, s, n);
  // one CTA per SM, each with an even share of the splits' tiles
  const uint32_t units = (n + tcm::TM - 1) / tcm::TM * a.splits;
  tcm::out_grad_kernel<<<std::min(units, 152u), tcm::kGradThreads + 32, tcm::kGradSmem, m->st>>>(a);
}

// Forward (and, when grads is true, backward into G) for n samples.
rt_status run(rt_mlp* m, const rt_mlp_sample* s, uint32_t n, bool grads, uint32_t* top4) {
  const int B = (int)n;
  cudaStream_t st = m->st;
  hidden_forward_kernel<<<(B + HB - 1) / HB, HT, 0, st>>>(s, B, m->E16, m->C, m->W1_16, m->P + m->offb1, m->W2_16,
                                                          m->P + m->offb2, m->X, m->Z1, m->H1, m->Z2, m->H2);
  if (top4) {
    output_forward(m, s, n, top4);
    return RT_OK;
  }
  MLP_CUDA(cudaMemsetAsync(m->loss, 0, sizeof(double), st));
  output_forward(m, s, n, nullptr);
  if (!grads) return RT_OK;
  MLP_CUDA(cudaMemsetAsync(m->G, 0, sizeof(float) * m->n_params, st));
  output_backward(m, s, n);
  hidden_backward_kernel<<<(B + HB - 1) / HB, HT, 0, st>>>(s, B, m->C, m->W1_16, m->W2_16, m->X, m->Z1, m->H1, m->Z2,
                                                           m->part, tcm::live_splits(m->Cp, out_splits(m, n)), m->G,
                                                           m->G + m->offW1, m->G + m->offb1, m->G + m->offW2,
                                                           m->G + m->offb2);
  return RT_OK;
}

// After the stream has been synchronised: RT_ERR_TIMEOUT (and the flag
// cleared) if a bounded wait of the output layer gave up.
rt_status check_status(rt_mlp* m, const char* who) {
  uint32_t st = 0;
  MLP_CUDA(cudaMemcpy(&st, m->tstatus, sizeof(st), cudaMemcpyDeviceToHost));
  if (st == 0) return RT_OK;
  MLP_CUDA(cudaMemset(m->tstatus, 0, sizeof(uint32_t)));
  return rti::fail(RT_ERR_TIMEOUT, std::string(who) + ": a bounded tensor-core wait gave up; results are invalid");
}

}  // namespace

extern "C" {

rt_status rt_mlp_create(rt_ctx* ctx, uint32_t n_treelets, uint64_t seed, rt_mlp** out) {
  if (!ctx || !out || n_treelets == 0) return rti::fail(RT_ERR_INVALID, "rt_mlp_create: bad argument");
  if (n_treelets > (1u << 24)) return rti::fail(RT_ERR_TOO_LARGE, "rt_mlp_create: at most 16M treelets");
  *out = nullptr;
  MLP_CUDA(cudaSetDevice(ctx->device));
  auto* m = new rt_mlp();
  m->device = ctx->device;
  const uint64_t C = n_treelets;
  m->C = n_treelets;
  m->offW1 = C * EMB;
  m->offb1 = m->offW1 + XIN * H;
  m->offW2 = m->offb1 + H;
  m->offb2 = m->offW2 + H * H;
  m->offW3 = m->offb2 + H;
  m->offb3 = m->offW3 + H * C;
  m->n_params = m->offb3 + C;
  const size_t MB = RT_MLP_MAX_BATCH;
  cudaError_t e = cudaSuccess;
  auto chk = [&](cudaError_t x) {
    if (e == cudaSuccess) e = x;
  };
  chk(mk(&m->P, m->n_params));
  chk(mk(&m->M, m->n_params));
  chk(mk(&m->V, m->n_params));
  chk(mk(&m->G, m->n_params));
  chk(mk(&m->E16, C * EMB));
  chk(mk(&m->W1_16, XP * H));
  chk(mk(&m->W2_16, H * H));
  m->Cp = (uint32_t)((C + tcm::TN - 1) / tcm::TN * tcm::TN);
  chk(mk(&m->W3T, (size_t)m->Cp * H));
  chk(mk(&m->X, MB * XP));
  chk(mk(&m->H1, MB * H));
  chk(mk(&m->H2, MB * H));
  chk(mk(&m->Z1, MB * H));
  chk(mk(&m->Z2, MB * H));
  chk(mk(&m->lse, MB));
  // 2 x 152 partial results of 8 floats per row; or dH2's partial sums: at most
  // 4 x 152 + 31 row tiles' splits (out_splits) of 128 x 64 floats
  static_assert(8 * 152 * 2 * (uint64_t)RT_MLP_MAX_BATCH >= (4 * 152 + RT_MLP_MAX_BATCH / tcm::TM) * (uint64_t)tcm::TM * H);
  chk(mk(&m->part, 8 * 152 * 2 * MB));
  chk(mk(&m->tstatus, 1));
  chk(mk(&m->loss, 1));
  chk(cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking));
  chk(cudaFuncSetAttribute(tcm::out_stats_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemStats));
  chk(cudaFuncSetAttribute(tcm::out_stats_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemStats));
  chk(cudaFuncSetAttribute(tcm::out_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tcm::kGradSmem));
  if (e == cudaSuccess) e = cudaMemset(m->tstatus, 0, sizeof(uint32_t));
  if (e != cudaSuccess) {
    rt_mlp_destroy(m);
    return rti::fail(RT_ERR_OOM, std::string("rt_mlp_create: ") + cudaGetErrorString(e));
  }
  init_params<<<blocks(m->n_params), 256, 0, m->st>>>(m->P, m->n_params, seed, m->offW1, m->offb1, m->offW2,
                                                         m->offb2, m->offW3, m->offb3);
  cudaMemsetAsync(m->M, 0, sizeof(float) * m->n_params, m->st);
  cudaMemsetAsync(m->V, 0, sizeof(float) * m->n_params, m->st);
  refresh_bf16(m);
  e = cudaStreamSynchronize(m->st);
  if (e != cudaSuccess) {
    rt_mlp_destroy(m);
    return cfail(e, "rt_mlp_create");
  }
  *out = m;
  return RT_OK;
}

rt_status rt_mlp_destroy(rt_mlp* m) {
  if (!m) return RT_OK;
  cudaSetDevice(m->device);
  void* ptrs[] = {m->P, m->M, m->V, m->G, m->E16, m->W1_16, m->W2_16, m->W3T, m->X, m->H1,
                  m->H2, m->Z1, m->Z2, m->lse, m->part, m->tstatus, m->loss};
  for (void* p : ptrs) cudaFree(p);
  if (m->st) cudaStreamDestroy(m->st);
  delete m;
  return RT_OK;
}

rt_status rt_mlp_num_params(const rt_mlp* m, uint64_t* n) {
  if (!m || !n) return rti::fail(RT_ERR_INVALID, "rt_mlp_num_params: NULL");
  *n = m->n_params;
  return RT_OK;
}

rt_status rt_mlp_get_params(const rt_mlp* m, float* host) {
  if (!m || !host) return rti::fail(RT_ERR_INVALID, "rt_mlp_get_params: NULL");
  MLP_CUDA(cudaSetDevice(m->device));
  MLP_CUDA(cudaStreamSynchronize(m->st));
  MLP_CUDA(cudaMemcpy(host, m->P, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost));
  return RT_OK;
}

rt_status rt_mlp_set_params(rt_mlp* m, const float* host) {
  if (!m || !host) return rti::fail(RT_ERR_INVALID, "rt_mlp_set_params: NULL");
  MLP_CUDA(cudaSetDevice(m->device));
  MLP_CUDA(cudaStreamSynchronize(m->st));
  MLP_CUDA(cudaMemcpy(m->P, host, sizeof(float) * m->n_params, cudaMemcpyHostToDevice));
  refresh_bf16(m);
  MLP_CUDA(cudaStreamSynchronize(m->st));
  return RT_OK;
}

rt_status rt_mlp_loss_grad(rt_mlp* m, const rt_mlp_sample* s, uint32_t n, float* loss, float* grads_host) {
  if (!m || !s || n == 0) return rti::fail(RT_ERR_INVALID, "rt_mlp_loss_grad: bad argument");
  if (n > RT_MLP_MAX_BATCH) return rti::fail(RT_ERR_TOO_LARGE, "rt_mlp_loss_grad: batch above RT_MLP_MAX_BATCH");
  MLP_CUDA(cudaSetDevice(m->device));
  rt_status st = run(m, s, n, grads_host != nullptr, nullptr);
  if (st != RT_OK) return st;
  MLP_CUDA(cudaGetLastError());
  MLP_CUDA(cudaStreamSynchronize(m->st));
  st = check_status(m, "rt_mlp_loss_grad");
  if (st != RT_OK) return st;
  if (loss) {
    double sum = 0.0;
    MLP_CUDA(cudaMemcpy(&sum, m->loss, sizeof(sum), cudaMemcpyDeviceToHost));
    *loss = (float)sum;
  }
  if (grads_host) MLP_CUDA(cudaMemcpy(grads_host, m->G, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost));
  return RT_OK;
}

rt_status rt_mlp_train_step(rt_mlp* m, const rt_mlp_sample* s, uint32_t n, float lr, float* loss) {
  if (!m || !s || n == 0) return rti::fail(RT_ERR_INVALID, "rt_mlp_train_step: bad argument");
  if (n > RT_MLP_MAX_BATCH) return rti::fail(RT_ERR_TOO_LARGE, "rt_mlp_train_step: batch above RT_MLP_MAX_BATCH");
  MLP_CUDA(cudaSetDevice(m->device));
  rt_status st = run(m, s, n, true, nullptr);
  if (st != RT_OK) return st;
  m->step += 1;
  const float c1 = 1.0f - powf(0.9f, (float)m->step), c2 = 1.0f - powf(0.999f, (float)m->step);
  adam<<<blocks(m->n_params), 256, 0, m->st>>>(m->P, m->M, m->V, m->G, m->n_params, lr, c1, c2);
  refresh_bf16(m);
  MLP_CUDA(cudaGetLastError());
  if (loss) {
    double sum = 0.0;
    MLP_CUDA(cudaMemcpyAsync(&sum, m->loss, sizeof(sum), cudaMemcpyDeviceToHost, m->st));
    MLP_CUDA(cudaStreamSynchronize(m->st));
    *loss = (float)sum;
    return check_status(m, "rt_mlp_train_step");
  }
  return RT_OK;
}

rt_status rt_mlp_topk(rt_mlp* m, const rt_mlp_sample* s, uint32_t n, uint32_t* top4) {
  if (!m || !s || !top4) return rti::fail(RT_ERR_INVALID, "rt_mlp_topk: NULL");
  MLP_CUDA(cudaSetDevice(m->device));
  for (uint32_t b0 = 0; b0 < n; b0 += RT_MLP_MAX_BATCH) {
    const uint32_t nb = std::min<uint32_t>(RT_MLP_MAX_BATCH, n - b0);
    rt_status st = run(m, s + b0, nb, false, top4 + (size_t)b0 * 4);
    if (st != RT_OK) return st;
  }
  MLP_CUDA(cudaGetLastError());
  MLP_CUDA(cudaStreamSynchronize(m->st));
  return check_status(m, "rt_mlp_topk");
}

}  // extern "C"
