// k_mlp.cu -- the Monte Carlo surrogate network, trained and evaluated with
// hand-written BF16-in / FP32-accumulate kernels; every matrix product runs
// on the 5th-generation tensor cores (tcgen05.mma, accumulator in tensor
// memory).
//
// Network: g(x) = w3 . silu(W2 silu(W1 x' + b1) + b2) + b3 with 64 inputs,
// two hidden layers of 128 and one output; x' = (x - mean) / std per input.
// A trial move is scored by the difference g(x_new) - g(x_old) of its
// descriptors after and before the move, which makes the predicted energy
// change antisymmetric under reversing the move (what the delayed-acceptance
// second stage relies on).  Training minimises the mean squared error of
// that difference against the exact reciprocal-space energy change with
// Adam (Kingma & Ba 2015).
//
// Training runs as one kernel (k_mlp_train).  Pass 1: a CTA takes tiles of 64
// samples -- 128 rows, before and after -- forward and back, activations in
// shared memory, products accumulated in tensor memory, and leaves what the
// gradients need in L2.  Pass 2: eight parts each take 16 columns of dW2, four
// of them 16 of dW1 and the other four the column sums, and apply Adam to what
// they summed.  Eight CTAs form a cluster that runs a whole epoch with a
// barrier after each pass.  Every sum runs in one order whatever the number of
// CTAs (products along K in one accumulator, column sums row by row).  A batch
// of 512 took 13 launches, dW on one CTA, serial column sums from global memory
// and a synchronisation: 600 us.
//
// GEMM kernel (test entry): one CTA of 4 warps computes a 128 x N tile of
// D = A B^T (A: M x K, B: N x K, both bf16 with K contiguous; D fp32).  K is streamed
// through shared memory in chunks of 64; thread 0 issues the MMAs (K = 16
// each) and commits them to an mbarrier that all threads wait on (bounded),
// then each warp reads its 32 accumulator rows from tensor memory.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "fe_internal.h"
#include "fe_rng.cuh"
#include "fe_tc.cuh"

namespace fe {

constexpr int kMlpIn = 64, kMlpH = 128;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kMlpH * kMlpIn, kOffW2 = kOffB1 + kMlpH,
              kOffB2 = kOffW2 + kMlpH * kMlpH, kOffW3 = kOffB2 + kMlpH, kOffB3 = kOffW3 + kMlpH,
              kMlpParams = kOffB3 + 1;
constexpr int kTcKc = 64;  // K per shared-memory chunk
constexpr long kTcWaitPolls = 1L << 20;

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------------------
// D[M x N] (row stride ldd) = A[M x K] B[N x K]^T + bias; M % 128 == 0,
// N in {32, 64, 96, 128, ..., 256}, K % 64 == 0; rows 16-byte aligned.
__global__ void __launch_bounds__(128) k_gemm_tc(const bf16 *__restrict__ A, int lda,
                                                 const bf16 *__restrict__ B, int ldb,
                                                 const float *__restrict__ bias,
                                                 float *__restrict__ D, int ldd, int N, int K,
                                                 int *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * 128;
  const uint32_t ncols = N <= 32 ? 32u : N <= 64 ? 64u : N <= 128 ? 128u : 256u;
  unsigned char *sA = tc_smem;
  unsigned char *sB = tc_smem + 128 * kTcKc * 2;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&tmem_base), ncols);
    tc::tmem_relinquish();
  }
  if (tid == 0) tc::mbar_init(tc::smem_u32(&mbar), 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = tc::idesc_bf16_f32(128, N);
  uint32_t phase = 0;
  bool ok = true;
  for (int k0 = 0; k0 < K && ok; k0 += kTcKc) {
    for (int u = tid; u < 128 * (kTcKc / 8); u += blockDim.x) {
      int r = u / (kTcKc / 8), c = u % (kTcKc / 8);
      uint4 v = *reinterpret_cast<const uint4 *>(A + (size_t)(m0 + r) * lda + k0 + c * 8);
      *reinterpret_cast<uint4 *>(sA + tc::tile_offset(r, c * 8, kTcKc)) = v;
    }
    for (int u = tid; u < N * (kTcKc / 8); u += blockDim.x) {
      int r = u / (kTcKc / 8), c = u % (kTcKc / 8);
      uint4 v = *reinterpret_cast<const uint4 *>(B + (size_t)r * ldb + k0 + c * 8);
      *reinterpret_cast<uint4 *>(sB + tc::tile_offset(r, c * 8, kTcKc)) = v;
    }
    tc::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int ks = 0; ks < kTcKc / 16; ks++) {
        uint64_t ad = tc::smem_desc(tc::smem_u32(sA) + ks * 2 * tc::kLbo, tc::kLbo,
                                    tc::sbo_bytes(kTcKc));
        uint64_t bd = tc::smem_desc(tc::smem_u32(sB) + ks * 2 * tc::kLbo, tc::kLbo,
                                    tc::sbo_bytes(kTcKc));
        tc::mma_bf16(tmem, ad, bd, idesc, (k0 > 0 || ks > 0) ? 1u : 0u);
      }
      tc::mma_commit(tc::smem_u32(&mbar));
    }
    // the chunk buffers are rewritten next: wait for the MMAs to finish
    ok = tc::mbar_wait(tc::smem_u32(&mbar), phase, kTcWaitPolls);
    phase ^= 1u;
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
  }
  if (ok) {
    tc::fence_after_sync();
    const int row = m0 + warp * 32 + lane;
    for (int cg = 0; cg < N / 32; cg++) {
      float v[32];
      tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cg * 32), v);
      float *d = D + (size_t)row * ldd + cg * 32;
#pragma unroll
      for (int j = 0; j < 32; j++) d[j] = v[j] + (bias ? bias[cg * 32 + j] : 0.f);
    }
  } else {
    // give the tensor core a last bounded chance to finish before freeing its memory
    if (tid == 0) atomicExch(err, 1);
    tc::mbar_wait(tc::smem_u32(&mbar), phase ^ 1u, kTcWaitPolls);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

static int gemm_tc(cudaStream_t st, const bf16 *A, int lda, const bf16 *B, int ldb,
                   const float *bias, float *D, int ldd, int M, int N, int K, int *err) {
  if (M % 128 || N % 32 || N < 32 || N > 256 || K % kTcKc || lda % 8 || ldb % 8) {
    set_error("tensor-core GEMM: M % 128, N in 32..256 step 32, K % 64 and 8-element strides");
    return FE_ERR_ARG;
  }
  size_t smem = (size_t)(128 + N) * kTcKc * 2;
  static bool attr = false;
  if (!attr) {
    FE_CUDA(cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)((128 + 256) * kTcKc * 2)));
    attr = true;
  }
  k_gemm_tc<<<M / 128, 128, smem, st>>>(A, lda, B, ldb, bias, D, ldd, N, K, err);
  FE_LAUNCH_CHECK("k_gemm_tc");
  return FE_OK;
}

// ---------------------------------------------------------------------------
// training

__device__ __forceinline__ float sigm(float z) { return 1.f / (1.f + __expf(-z)); }

constexpr int kTrThreads = 512;   // four threads per row, 32 columns each
constexpr int kTrCluster = 8;     // CTAs of a cluster at most (the portable size)
constexpr int kTrRows = 128, kTrSamples = 64;
constexpr int kTrParts = 8;       // of pass 2
constexpr int kTrCols = kMlpH / kTrParts;                  // columns of dW2 per part
constexpr int kTrSums = 3 * kMlpH / (kTrParts / 2);        // column sums of parts 4 to 7
// pass 1's operand tiles (K-major core matrices); dZ2 takes H1's
constexpr int kTrX = 0, kTrW1 = kTrX + kTrRows * kMlpIn * 2, kTrH1 = kTrW1 + kMlpH * kMlpIn * 2,
              kTrW2 = kTrH1 + kTrRows * kMlpH * 2, kTrW2t = kTrW2 + kMlpH * kMlpH * 2,
              kTrSg = kTrW2t + kMlpH * kMlpH * 2;
// sigmoid(Z1) of the tile, kept for the way back: [column][row] fp32
constexpr int kTrEnd1 = kTrSg + kMlpH * kTrRows * 4;
// pass 2's ring over the rows: stages of 128 rows of dZ^T (128 units) and 16
// columns, or of 64 rows of 96 columns to sum with dout and the squared errors
constexpr int kTrStages = 4, kTrStageA = kMlpH * 128 * 2, kTrStageB = kTrCols * 128 * 2,
              kTrStage = kTrStageA + kTrStageB, kTrSumRows = 64;
static_assert(kTrSumRows * (kTrSums + 2) * 4 <= kTrStage, "the sums' stages fit the ring");
constexpr int kTrF = kTrStages * kTrStage > kTrEnd1 ? kTrStages * kTrStage : kTrEnd1;
// floats: b1, b2, w3, mean, istd, head (128), dout (128), y (64)
constexpr int kTrFloats = 3 * kMlpH + 2 * kMlpIn + 2 * kTrRows + kTrSamples;
constexpr int kTrSmem = kTrF + kTrFloats * 4;

struct TrainArgs {
  int B, nbatch;
  int passes;              // 1, 2 or both (3: one cluster, barriers between)
  int update;              // Adam; else the gradient to G
  const int *idx;          // nbatch * B sample indices
  const float *data, *y, *mean, *istd;
  float *P, *Am, *Av, *G;
  bf16 *W1b, *W2b, *W2tb;
  // pass 1's results over the batch's R = 2 B rows: bf16 transposed [unit][R],
  // fp32 [R][128], per row dout and (first B) the squared error
  bf16 *Xt, *H1t, *dZ1t, *dZ2t;
  float *dZ1f, *dZ2f, *S2f, *dout, *err2;
  const float2 *bc;        // Adam's bias corrections per batch
  float lr;
  double *loss;            // += the batch losses
  float *out;              // R outputs (optional)
  int *err;
};

// D (tensor memory) [+]= A (128 x K) B (N x K)^T from tiles of K columns
__device__ __forceinline__ void train_mma(uint32_t d, uint32_t a, uint32_t b, int N, int K,
                                          bool add) {
  const uint32_t idesc = tc::idesc_bf16_f32(128, N);
  for (int ks = 0; ks < K / 16; ks++)
    tc::mma_bf16(d, tc::smem_desc(a + ks * 2 * tc::kLbo, tc::kLbo, tc::sbo_bytes(K)),
                 tc::smem_desc(b + ks * 2 * tc::kLbo, tc::kLbo, tc::sbo_bytes(K)), idesc,
                 (add || ks > 0) ? 1u : 0u);
}

// eight consecutive values of a row as one 16-byte store (k % 8 == 0)
__device__ __forceinline__ void tile_put8(unsigned char *tile, int r, int k, int kc,
                                          const bf16 (&h)[8]) {
  uint4 v;
  memcpy(&v, h, 16);
  *reinterpret_cast<uint4 *>(tile + tc::tile_offset(r, k, kc)) = v;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// 16 bytes from L2 to shared memory, asynchronously (PTX cp.async)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// a weight tile (K columns, uint4 per 8) into core matrices: eight lanes take
// the eight rows of one, so that a warp writes four whole ones
template <int K>
__device__ __forceinline__ void tile_load(unsigned char *tile, const bf16 *src) {
  for (int u = threadIdx.x; u < kMlpH * K / 8; u += kTrThreads) {
    const int r = (u & 7) + u / K * 8, c = (u >> 3) % (K / 8) * 8;
    *reinterpret_cast<uint4 *>(tile + tc::tile_offset(r, c, K)) =
        __ldcg(reinterpret_cast<const uint4 *>(src + r * K + c));
  }
}

// Adam (Kingma & Ba 2015) on N consecutive parameters from i and their bf16
// copies, or their gradients; all loads first
template <int N>
__device__ __forceinline__ void train_apply(const TrainArgs &a, int i, const float (&g)[N],
                                            float2 c) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  float m[N], v[N], p[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    if (!a.update) {
      a.G[i + k] = g[k];
      continue;
    }
    m[k] = a.Am[i + k];
    v[k] = a.Av[i + k];
    p[k] = a.P[i + k];
  }
  if (!a.update) return;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const float mi = fmaf(1.f - b1, g[k], b1 * m[k]);
    const float vi = fmaf((1.f - b2) * g[k], g[k], b2 * v[k]);
    m[k] = mi;
    v[k] = vi;
    p[k] -= a.lr * (mi / c.x) / (sqrtf(vi / c.y) + eps);
  }
#pragma unroll
  for (int k = 0; k < N; k++) {
    a.Am[i + k] = m[k];
    a.Av[i + k] = v[k];
    a.P[i + k] = p[k];
    const bf16 h = __float2bfloat16_rn(p[k]);
    if (i < kOffB1) {
      a.W1b[i + k] = h;
    } else if (i >= kOffW2 && i < kOffB2) {
      const int t = i + k - kOffW2;
      a.W2b[t] = h;
      a.W2tb[t % kMlpH * kMlpH + t / kMlpH] = h;
    }
  }
}

__global__ void __launch_bounds__(kTrThreads, 1) k_mlp_train(TrainArgs a) {
  extern __shared__ __align__(1024) unsigned char tr[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = (warp >> 2) * 32, row = (warp & 3) * 32 + lane;  // columns c0 .. c0 + 31
  float *f = reinterpret_cast<float *>(tr + kTrF);
  float *b1 = f, *b2 = b1 + kMlpH, *w3 = b2 + kMlpH, *mean = w3 + kMlpH, *istd = mean + kMlpIn,
        *so = istd + kMlpIn, *dout = so + kTrRows, *yb = dout + kTrRows;
  float *sg1 = reinterpret_cast<float *>(tr + kTrSg);
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&tmem_base), 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) tc::mbar_init(tc::smem_u32(&mbar), 1);
  if (tid < kMlpIn) {
    mean[tid] = a.mean[tid];
    istd[tid] = a.istd[tid];
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tm = tmem_base, sm = tc::smem_u32(tr), lanes = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t tZ1 = tm, tZ2 = tm + 128, tG = tm + 256;  // dH1 takes Z2's columns
  uint32_t phase = 0;
  bool ok = true;
  // operands written; products issued by thread 0 through `issue` and waited
  // for (bounded: where that runs out, the CTA skips to the next barrier)
  auto products = [&](auto issue) {
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (!ok) return;
    if (tid == 0) {
      tc::fence_after_sync();
      issue();
      tc::mma_commit(tc::smem_u32(&mbar));
    }
    const bool done = tc::mbar_wait(tc::smem_u32(&mbar), phase, kTcWaitPolls);
    phase ^= 1u;
    ok = __syncthreads_and(done ? 1 : 0) != 0;
    if (!ok && tid == 0) atomicExch(a.err, 1);
    tc::fence_after_sync();
  };
  const int R = 2 * a.B, ntile = a.B / kTrSamples, ncta = gridDim.x, cta = blockIdx.x;
  for (int bi = 0; bi < a.nbatch; bi++) {
    if (a.passes & 1) {
      // the weights as the last update left them (in L2: other CTAs wrote them)
      tile_load<kMlpIn>(tr + kTrW1, a.W1b);
      tile_load<kMlpH>(tr + kTrW2, a.W2b);
      tile_load<kMlpH>(tr + kTrW2t, a.W2tb);
      if (tid < kMlpH) {
        b1[tid] = __ldcg(a.P + kOffB1 + tid);
        b2[tid] = __ldcg(a.P + kOffB2 + tid);
        w3[tid] = __ldcg(a.P + kOffW3 + tid);
      }
      const float b3 = __ldcg(a.P + kOffB3);
      for (int tile = cta; tile < ntile && ok; tile += ncta) {
        const int s0 = tile * kTrSamples;
        const int *id = a.idx + (size_t)bi * a.B + s0;
        // row of the batch: samples before the move first, then after
        const int gr = (row < kTrSamples ? row : a.B + row - kTrSamples) + s0;
        // inputs, normalised
        for (int u = tid; u < kTrRows * kMlpIn / 8; u += kTrThreads) {
          const int r = u & 127, c = (u >> 7) * 8, s = id[r & 63];
          const int q = (r < kTrSamples ? r : a.B + r - kTrSamples) + s0;
          const float4 *src = reinterpret_cast<const float4 *>(
              a.data + (size_t)s * 2 * kMlpIn + (r >= kTrSamples ? kMlpIn : 0) + c);
          const float4 lo = src[0], hi = src[1];
          const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
          bf16 h[8];
#pragma unroll
          for (int k = 0; k < 8; k++) {
            h[k] = __float2bfloat16_rn((v[k] - mean[c + k]) * istd[c + k]);
            a.Xt[(size_t)(c + k) * R + q] = h[k];
          }
          tile_put8(tr + kTrX, r, c, kMlpIn, h);
        }
        if (tid < kTrSamples) yb[tid] = a.y[id[tid]];
        products([&] { train_mma(tZ1, sm + kTrX, sm + kTrW1, kMlpH, kMlpIn, false); });
        if (!ok) break;
        // H1 = silu(Z1 + b1)
        {
          float z[32];
          tc::tmem_ld32(tZ1 + lanes + c0, z);
#pragma unroll
          for (int k = 0; k < 32; k += 8) {
            bf16 h[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
              const float x = z[k + q] + b1[c0 + k + q], sg = sigm(x);
              h[q] = __float2bfloat16_rn(x * sg);
              sg1[(c0 + k + q) * kTrRows + row] = sg;
              a.H1t[(size_t)(c0 + k + q) * R + gr] = h[q];
            }
            tile_put8(tr + kTrH1, row, c0 + k, kMlpH, h);
          }
        }
        products([&] { train_mma(tZ2, sm + kTrH1, sm + kTrW2, kMlpH, kMlpH, false); });
        if (!ok) break;
        // the outputs (columns in order: each group hands its sum on), the loss
        // and its gradient
        float z2[32], sg2[32];
        tc::tmem_ld32(tZ2 + lanes + c0, z2);
#pragma unroll
        for (int k = 0; k < 32; k++) {
          z2[k] += b2[c0 + k];
          sg2[k] = sigm(z2[k]);
        }
        for (int g = 0; g < kMlpH; g += 32) {
          if (c0 == g) {
            float o = g == 0 ? b3 : so[row];
#pragma unroll
            for (int k = 0; k < 32; k++) o = fmaf(w3[c0 + k], z2[k] * sg2[k], o);
            so[row] = o;
          }
          __syncthreads();
        }
        if (tid < kTrSamples) {
          const float o0 = so[tid], o1 = so[tid + kTrSamples];
          const float e = (o1 - o0) - yb[tid], g = 2.f * e / (float)a.B;
          dout[tid + kTrSamples] = g;
          dout[tid] = -g;
          a.dout[a.B + s0 + tid] = g;
          a.dout[s0 + tid] = -g;
          a.err2[s0 + tid] = e * e;
          if (a.out) {
            a.out[s0 + tid] = o0;
            a.out[a.B + s0 + tid] = o1;
          }
        }
        __syncthreads();
        // dZ2 = dout w3 silu'(Z2)
        const float d = dout[row];
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
          bf16 h[8];
          float dz[8], sv[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const float z = z2[k + q], sg = sg2[k + q];
            dz[q] = d * w3[c0 + k + q] * sg * (1.f + z * (1.f - sg));
            sv[q] = z * sg;
            h[q] = __float2bfloat16_rn(dz[q]);
            a.dZ2t[(size_t)(c0 + k + q) * R + gr] = h[q];
          }
          tile_put8(tr + kTrH1, row, c0 + k, kMlpH, h);
          float4 *zf = reinterpret_cast<float4 *>(a.dZ2f + (size_t)gr * kMlpH + c0 + k);
          float4 *sf = reinterpret_cast<float4 *>(a.S2f + (size_t)gr * kMlpH + c0 + k);
          zf[0] = make_float4(dz[0], dz[1], dz[2], dz[3]);
          zf[1] = make_float4(dz[4], dz[5], dz[6], dz[7]);
          sf[0] = make_float4(sv[0], sv[1], sv[2], sv[3]);
          sf[1] = make_float4(sv[4], sv[5], sv[6], sv[7]);
        }
        products([&] { train_mma(tZ2, sm + kTrH1, sm + kTrW2t, kMlpH, kMlpH, false); });
        if (!ok) break;
        // dZ1 = dH1 silu'(Z1)
        float z[32], dz[32];
        tc::tmem_ld32(tZ1 + lanes + c0, z);
        tc::tmem_ld32(tZ2 + lanes + c0, dz);
#pragma unroll
        for (int k = 0; k < 32; k++) {
          const float x = z[k] + b1[c0 + k], sg = sg1[(c0 + k) * kTrRows + row];
          dz[k] = dz[k] * sg * (1.f + x * (1.f - sg));
          a.dZ1t[(size_t)(c0 + k) * R + gr] = __float2bfloat16_rn(dz[k]);
        }
        float4 *zf = reinterpret_cast<float4 *>(a.dZ1f + (size_t)gr * kMlpH + c0);
#pragma unroll
        for (int k = 0; k < 8; k++)
          zf[k] = make_float4(dz[4 * k], dz[4 * k + 1], dz[4 * k + 2], dz[4 * k + 3]);
      }
    }
    if (a.passes == 3) {
      cluster_barrier();
      if (__ldcg(a.err)) break;  // the same for every CTA of the cluster
    }
    if (a.passes & 2) {
      const float2 bc = a.update ? a.bc[bi] : make_float2(1.f, 1.f);
      for (int part = cta; part < kTrParts && ok; part += ncta) {
        // 16 columns of dW2 (dZ2^T H1), of parts 0 to 3 also of dW1 (dZ1^T X)
        for (int job = 0; job < (part < kTrParts / 2 ? 2 : 1) && ok; job++) {
          const bf16 *A = job ? a.dZ1t : a.dZ2t;
          const bf16 *Bm = (job ? a.Xt : a.H1t) + (size_t)part * kTrCols * R;
          const int nk = R / 128;
          auto load = [&](int kc) {
            if (kc < nk) {
              const uint32_t st = sm + (kc % kTrStages) * kTrStage;
              // eight lanes take a core matrix's eight rows
              for (int u = tid; u < kMlpH * 16; u += kTrThreads) {
                const int r = (u & 7) + (u >> 7) * 8, c = (u >> 3 & 15) * 8;
                cp_async16(st + tc::tile_offset(r, c, 128), A + (size_t)r * R + kc * 128 + c);
              }
              for (int u = tid; u < kTrCols * 16; u += kTrThreads) {
                const int r = (u & 7) + (u >> 7) * 8, c = (u >> 3 & 15) * 8;
                cp_async16(st + kTrStageA + tc::tile_offset(r, c, 128),
                           Bm + (size_t)r * R + kc * 128 + c);
              }
            }
            cp_async_commit();
          };
          __syncthreads();  // the ring's last readers are done
          for (int kc = 0; kc < kTrStages; kc++) load(kc);
          for (int kc = 0; kc < nk && ok; kc++) {
            cp_async_wait<kTrStages - 1>();
            const uint32_t st = sm + (kc % kTrStages) * kTrStage;
            products([&] { train_mma(tG, st, st + kTrStageA, kTrCols, 128, kc > 0); });
            load(kc + kTrStages);
          }
          cp_async_wait<0>();
          if (!ok) break;
          float v[32], g[4];
          tc::tmem_ld32(tG + lanes, v);  // 16 of the columns are this product's
#pragma unroll
          for (int k = 0; k < kTrCols; k++)
            if (k / 4 == c0 / 32) g[k % 4] = v[k];
          const int i0 = job ? kOffW1 + row * kMlpIn + part * kTrCols
                             : kOffW2 + row * kMlpH + part * kTrCols;
          train_apply<4>(a, i0 + c0 / 8, g, bc);
        }
        if (part < kTrParts / 2) continue;
        // db1, db2, dw3: 96 columns, row by row; db3 and the loss in part 7
        const int c00 = (part - kTrParts / 2) * kTrSums, nr = R / kTrSumRows;
        auto load = [&](int kr) {
          if (kr < nr) {
            const uint32_t st = sm + (kr % kTrStages) * kTrStage;
            for (int u = tid; u < kTrSumRows * (kTrSums / 4); u += kTrThreads) {
              const int r = u / (kTrSums / 4), q = u % (kTrSums / 4), c = c00 + q * 4;
              const float *src = c < kMlpH ? a.dZ1f : c < 2 * kMlpH ? a.dZ2f : a.S2f;
              cp_async16(st + (r * kTrSums + q * 4) * 4,
                         src + (size_t)(kr * kTrSumRows + r) * kMlpH + (c & (kMlpH - 1)));
            }
            if (tid < kTrSumRows / 4)
              cp_async16(st + (kTrSumRows * kTrSums + tid * 4) * 4,
                         a.dout + kr * kTrSumRows + tid * 4);
            else if (tid < kTrSumRows / 2 && kr * kTrSumRows < a.B)
              cp_async16(st + (kTrSumRows * kTrSums + tid * 4) * 4,
                         a.err2 + kr * kTrSumRows + (tid - kTrSumRows / 4) * 4);
          }
          cp_async_commit();
        };
        __syncthreads();
        for (int kr = 0; kr < kTrStages - 1; kr++) load(kr);
        float acc = 0.f;
        const int c = c00 + tid;
        for (int kr = 0; kr < nr; kr++) {
          cp_async_wait<kTrStages - 2>();
          __syncthreads();
          load(kr + kTrStages - 1);  // into the stage read last round
          const float *st = reinterpret_cast<const float *>(tr + (kr % kTrStages) * kTrStage);
          const float *dq = st + kTrSumRows * kTrSums;
          // one thread per sum, its values sixteen at a time
          const float *src = tid < kTrSums ? st + tid : tid == kTrSums ? dq : dq + kTrSumRows;
          const int ld = tid < kTrSums ? kTrSums : 1;
          const bool on = tid <= kTrSums || (tid == kTrSums + 32 && kr * kTrSumRows < a.B);
          const bool scaled = tid < kTrSums && c >= 2 * kMlpH;
          if (on)
            for (int r0 = 0; r0 < kTrSumRows; r0 += 16) {
              float x[16], w[16];
#pragma unroll
              for (int r = 0; r < 16; r++) {
                x[r] = src[(r0 + r) * ld];
                w[r] = dq[r0 + r];
              }
#pragma unroll
              for (int r = 0; r < 16; r++) acc = scaled ? fmaf(w[r], x[r], acc) : acc + x[r];
            }
        }
        cp_async_wait<0>();
        const float g[1] = {acc};
        if (tid < kTrSums)
          train_apply<1>(a, (c < kMlpH ? kOffB1 : c < 2 * kMlpH ? kOffB2 - kMlpH
                                                                : kOffW3 - 2 * kMlpH) + c, g, bc);
        else if (part == kTrParts - 1 && tid == kTrSums)
          train_apply<1>(a, kOffB3, g, bc);
        else if (part == kTrParts - 1 && tid == kTrSums + 32)
          *a.loss += (double)(acc / (float)a.B);
      }
    }
    if (a.passes == 3) {
      cluster_barrier();
      if (__ldcg(a.err)) break;
    }
  }
  // give the tensor core a last bounded chance to finish before freeing its memory
  if (!ok) tc::mbar_wait(tc::smem_u32(&mbar), phase ^ 1u, kTcWaitPolls);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tm, 512);
}

// per-feature sums of v and v^2 over both halves of every sample: one row of
// 128 sums per block (feature, then squares)
constexpr int kNormBlocks = 304;
__global__ void __launch_bounds__(256) k_mlp_moments(long long n, const float *__restrict__ data,
                                                     double *__restrict__ part) {
  __shared__ double sh[2][256];
  const int feat = threadIdx.x & 63, sub = threadIdx.x >> 6;
  double s = 0.0, s2 = 0.0;
  for (long long r = (long long)blockIdx.x * 4 + sub; r < 2 * n; r += (long long)gridDim.x * 4) {
    const double v = data[(size_t)r * kMlpIn + feat];
    s += v;
    s2 += v * v;
  }
  sh[0][threadIdx.x] = s;
  sh[1][threadIdx.x] = s2;
  __syncthreads();
  if (threadIdx.x < 128) {
    const double *q = sh[threadIdx.x >> 6] + feat;
    part[blockIdx.x * 128 + threadIdx.x] = (q[0] + q[64]) + (q[128] + q[192]);
  }
}

// 1024 threads: eight row groups of 128 sums
__global__ void __launch_bounds__(1024)
k_mlp_normalise(long long n, int rows, const double *__restrict__ part, float *__restrict__ mean,
                float *__restrict__ istd) {
  __shared__ double sh[8][128];
  const int c = threadIdx.x & 127, g = threadIdx.x >> 7;
  double s = 0.0;
#pragma unroll 8
  for (int r = g; r < rows; r += 8) s += part[r * 128 + c];
  sh[g][c] = s;
  __syncthreads();
  if (threadIdx.x < 128) {
    for (int k = 1; k < 8; k++) s += sh[k][c];
    sh[0][c] = s;
  }
  __syncthreads();
  if (threadIdx.x < kMlpIn) {
    const double mu = sh[0][c] / (2.0 * n), var = sh[0][64 + c] / (2.0 * n) - mu * mu;
    mean[c] = (float)mu;
    istd[c] = (float)(var > 1e-12 ? 1.0 / sqrt(var) : 1.0);
  }
}

// the Fisher-Yates partners of one epoch: j <= i uniform
__global__ void k_mlp_draws(long long n, uint64_t seed, uint64_t event0, int *__restrict__ j) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long v =
      (long long)(fe_uniform(seed, 0x50524D31u, event0 + (uint64_t)i, 0) * (double)(i + 1));
  j[i] = (int)(v > i ? i : v);
}

// bf16 weight copies for the GEMMs: W1 [128 x 64], W2 [128 x 128], W2^T
__global__ void k_mlp_refresh(const float *__restrict__ P, bf16 *__restrict__ W1b,
                              bf16 *__restrict__ W2b, bf16 *__restrict__ W2tb) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < kMlpH * kMlpIn) W1b[t] = __float2bfloat16_rn(P[kOffW1 + t]);
  if (t < kMlpH * kMlpH) {
    int j = t / kMlpH, i = t % kMlpH;
    bf16 h = __float2bfloat16_rn(P[kOffW2 + t]);
    W2b[t] = h;
    W2tb[(size_t)i * kMlpH + j] = h;
  }
}

// ---------------------------------------------------------------------------

struct Mlp {
  int dev = 0, nsm = 0;
  cudaStream_t st = nullptr, st_draw = nullptr;
  cudaEvent_t ev_draw[2] = {nullptr, nullptr}, ev_idx[2] = {nullptr, nullptr};
  float *P = nullptr, *G = nullptr, *Am = nullptr, *Av = nullptr;
  long long step = 0;
  float *mean = nullptr, *istd = nullptr;
  bf16 *W1b = nullptr, *W2b = nullptr, *W2tb = nullptr;
  int cap = 0;  // rows (2 B) the batch buffers hold, one allocation
  char *batch = nullptr;
  bf16 *Xt = nullptr, *H1t = nullptr, *dZ1t = nullptr, *dZ2t = nullptr;
  float *dZ1f = nullptr, *dZ2f = nullptr, *S2f = nullptr, *dout = nullptr, *err2 = nullptr;
  double *loss = nullptr, *moments = nullptr;
  float *out = nullptr;  // 2 B outputs of fe_mlp_grad
  int *idx1 = nullptr;   // and its samples' indices
  // Training alone, from the first on, one allocation on the device and a pinned one:
  // an epoch's permutation (Fisher-Yates partners, shuffled indices) and Adam's
  // bias corrections, for two epochs; the epochs' loss sums, and on the host err
  // behind them
  long long perm_cap = 0;
  int loss_cap = 0;
  char *train_dev = nullptr, *train_host = nullptr;
  double *ep_loss = nullptr, *h_loss = nullptr;
  int *draws[2] = {nullptr, nullptr}, *h_draws[2] = {nullptr, nullptr};
  int *h_idx[2] = {nullptr, nullptr}, *idx[2] = {nullptr, nullptr};
  float2 *h_bc[2] = {nullptr, nullptr}, *bc[2] = {nullptr, nullptr};
  int *err = nullptr;
  float *data = nullptr, *y = nullptr;  // uploaded samples
  long long ndata = 0, data_cap = 0;
};

static void mlp_free(Mlp *m) {
  cudaFreeHost(m->train_host);
  void *p[] = {m->batch, m->train_dev, m->P, m->G, m->Am, m->Av, m->mean, m->istd, m->W1b,
               m->W2b, m->W2tb, m->loss, m->moments, m->err, m->data, m->y};
  for (void *q : p)
    if (q) cudaFree(q);
  for (cudaEvent_t e : {m->ev_draw[0], m->ev_draw[1], m->ev_idx[0], m->ev_idx[1]})
    if (e) cudaEventDestroy(e);
  if (m->st_draw) cudaStreamDestroy(m->st_draw);
  if (m->st) cudaStreamDestroy(m->st);
}

// the next `bytes` of an allocation, every part on a 256-byte line; with base null
// the parts only add up
template <typename T>
static void mlp_part(char *base, size_t *at, T **p, size_t n) {
  *p = base ? reinterpret_cast<T *>(base + *at) : nullptr;
  *at = (*at + sizeof(T) * n + 255) & ~(size_t)255;
}

static size_t mlp_batch_parts(Mlp *m, size_t R) {
  size_t at = 0;
  for (bf16 **q : {&m->H1t, &m->dZ1t, &m->dZ2t}) mlp_part(m->batch, &at, q, R * kMlpH);
  mlp_part(m->batch, &at, &m->Xt, R * kMlpIn);
  for (float **q : {&m->dZ1f, &m->dZ2f, &m->S2f}) mlp_part(m->batch, &at, q, R * kMlpH);
  for (float **q : {&m->dout, &m->err2, &m->out}) mlp_part(m->batch, &at, q, R);
  mlp_part(m->batch, &at, &m->idx1, R);
  return at;
}

// buffers for batches of B samples
static int mlp_reserve_batch(Mlp *m, int B) {
  const int R = 2 * B;
  if (R <= m->cap) return FE_OK;
  cudaFree(m->batch);
  m->batch = nullptr;
  m->cap = 0;
  FE_CUDA(cudaMalloc(&m->batch, mlp_batch_parts(m, (size_t)R)));
  mlp_batch_parts(m, (size_t)R);
  m->cap = R;
  return FE_OK;
}

static size_t mlp_train_parts(Mlp *m, size_t n, size_t epochs, bool host) {
  char *base = host ? m->train_host : m->train_dev;
  const size_t nb = n / kTrSamples + 1;
  size_t at = 0;
  for (int k = 0; k < 2; k++) {
    mlp_part(base, &at, host ? &m->h_draws[k] : &m->draws[k], n);
    mlp_part(base, &at, host ? &m->h_idx[k] : &m->idx[k], n);
    mlp_part(base, &at, host ? &m->h_bc[k] : &m->bc[k], nb);
  }
  mlp_part(base, &at, host ? &m->h_loss : &m->ep_loss, epochs + (host ? 1 : 0));
  return at;
}

// buffers for trainings on n samples, the events and the stream of their draws
static int mlp_reserve_train(Mlp *m, long long n, int epochs) {
  if (!m->st_draw) {
    FE_CUDA(cudaStreamCreateWithFlags(&m->st_draw, cudaStreamNonBlocking));
    for (cudaEvent_t *e : {&m->ev_draw[0], &m->ev_draw[1], &m->ev_idx[0], &m->ev_idx[1]})
      FE_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  if (n <= m->perm_cap && epochs <= m->loss_cap) return FE_OK;
  const long long N = n > m->perm_cap ? n : m->perm_cap;
  const int E = epochs > m->loss_cap ? epochs : m->loss_cap;
  cudaFree(m->train_dev);
  cudaFreeHost(m->train_host);
  m->train_dev = m->train_host = nullptr;
  m->perm_cap = m->loss_cap = 0;
  FE_CUDA(cudaMalloc(&m->train_dev, mlp_train_parts(m, (size_t)N, (size_t)E, false)));
  FE_CUDA(cudaMallocHost(&m->train_host, mlp_train_parts(m, (size_t)N, (size_t)E, true)));
  mlp_train_parts(m, (size_t)N, (size_t)E, false);
  mlp_train_parts(m, (size_t)N, (size_t)E, true);
  m->perm_cap = N;
  m->loss_cap = E;
  return FE_OK;
}

static int mlp_refresh(Mlp *m) {
  k_mlp_refresh<<<(kMlpH * kMlpH + 255) / 256, 256, 0, m->st>>>(m->P, m->W1b, m->W2b, m->W2tb);
  FE_LAUNCH_CHECK("k_mlp_refresh");
  return FE_OK;
}

static int mlp_create(Mlp *m, int dev, uint64_t seed) {
  m->dev = dev;
  FE_CUDA(cudaSetDevice(dev));
  FE_CUDA(cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking));
  FE_CUDA(cudaMalloc(&m->P, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMalloc(&m->G, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMalloc(&m->Am, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMalloc(&m->Av, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMalloc(&m->mean, sizeof(float) * kMlpIn));
  FE_CUDA(cudaMalloc(&m->istd, sizeof(float) * kMlpIn));
  FE_CUDA(cudaMalloc(&m->W1b, 2 * kMlpH * kMlpIn));
  FE_CUDA(cudaMalloc(&m->W2b, 2 * kMlpH * kMlpH));
  FE_CUDA(cudaMalloc(&m->W2tb, 2 * kMlpH * kMlpH));
  FE_CUDA(cudaDeviceGetAttribute(&m->nsm, cudaDevAttrMultiProcessorCount, dev));
  FE_CUDA(cudaMalloc(&m->loss, sizeof(double)));
  FE_CUDA(cudaMalloc(&m->moments, sizeof(double) * 128 * kNormBlocks));
  FE_CUDA(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem));
  FE_CUDA(cudaMalloc(&m->err, sizeof(int)));
  FE_CUDA(cudaMemset(m->err, 0, sizeof(int)));
  FE_CUDA(cudaMemset(m->G, 0, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMemset(m->Am, 0, sizeof(float) * kMlpParams));
  FE_CUDA(cudaMemset(m->Av, 0, sizeof(float) * kMlpParams));
  // Glorot-uniform weights from Philox draws, zero biases, identity normalisation
  std::vector<float> P(kMlpParams, 0.f), mean(kMlpIn, 0.f), istd(kMlpIn, 1.f);
  auto fill = [&](int off, int fan_out, int fan_in, uint32_t tag) {
    float a = sqrtf(6.f / (float)(fan_in + fan_out));
    for (int i = 0; i < fan_out * fan_in; i++)
      P[off + i] = (float)((2.0 * fe_uniform(seed, tag, (uint64_t)i, 0) - 1.0) * a);
  };
  fill(kOffW1, kMlpH, kMlpIn, 0x4D4C5031u);
  fill(kOffW2, kMlpH, kMlpH, 0x4D4C5032u);
  fill(kOffW3, 1, kMlpH, 0x4D4C5033u);
  FE_CUDA(cudaMemcpy(m->P, P.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMemcpy(m->mean, mean.data(), sizeof(float) * kMlpIn, cudaMemcpyHostToDevice));
  FE_CUDA(cudaMemcpy(m->istd, istd.data(), sizeof(float) * kMlpIn, cudaMemcpyHostToDevice));
  int rc = mlp_refresh(m);
  if (rc) return rc;
  FE_CUDA(cudaStreamSynchronize(m->st));
  return FE_OK;
}

static TrainArgs train_args(Mlp *m, const float *data, const float *y, int B) {
  TrainArgs a;
  memset(&a, 0, sizeof a);
  a.B = B;
  a.nbatch = 1;
  a.data = data;
  a.y = y;
  a.mean = m->mean;
  a.istd = m->istd;
  a.P = m->P;
  a.Am = m->Am;
  a.Av = m->Av;
  a.G = m->G;
  a.W1b = m->W1b;
  a.W2b = m->W2b;
  a.W2tb = m->W2tb;
  a.Xt = m->Xt;
  a.H1t = m->H1t;
  a.dZ1t = m->dZ1t;
  a.dZ2t = m->dZ2t;
  a.dZ1f = m->dZ1f;
  a.dZ2f = m->dZ2f;
  a.S2f = m->S2f;
  a.dout = m->dout;
  a.err2 = m->err2;
  a.loss = m->loss;
  a.err = m->err;
  return a;
}

static int launch_train(Mlp *m, const TrainArgs &a, int ncta, bool cluster) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster ? ncta : 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)ncta);
  cfg.blockDim = dim3(kTrThreads);
  cfg.dynamicSmemBytes = kTrSmem;
  cfg.stream = m->st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  FE_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_train, a));
  FE_LAUNCH_CHECK("k_mlp_train");
  return FE_OK;
}

// One batch as two launches, pass 1 over as many CTAs as it has tiles
static int train_batch(Mlp *m, const TrainArgs &a0, int bi) {
  TrainArgs a = a0;
  const int ntile = a.B / kTrSamples;
  a.nbatch = 1;
  a.idx = a0.idx + (size_t)bi * a.B;
  if (a0.bc) a.bc = a0.bc + bi;
  a.passes = 1;
  int rc = launch_train(m, a, ntile < m->nsm ? ntile : m->nsm, false);
  if (rc) return rc;
  a.passes = 2;
  return launch_train(m, a, kTrParts, false);
}

// the kernels' error flag, once the stream is done; e: its copy on the host
static int mlp_check_err(Mlp *m, int e) {
  if (e) {
    set_error("tensor-core GEMM: an MMA completion wait ran out");
    FE_CUDA(cudaMemset(m->err, 0, sizeof(int)));
    return FE_ERR_DEVICE;
  }
  return FE_OK;
}

static int mlp_upload(Mlp *m, const float *data, const float *y, long long n) {
  if (n > m->data_cap) {
    if (m->data) cudaFree(m->data);
    if (m->y) cudaFree(m->y);
    m->data = nullptr;
    m->y = nullptr;
    FE_CUDA(cudaMalloc(&m->data, sizeof(float) * 2 * kMlpIn * (size_t)n));
    FE_CUDA(cudaMalloc(&m->y, sizeof(float) * (size_t)n));
    m->data_cap = n;
  }
  FE_CUDA(cudaMemcpyAsync(m->data, data, sizeof(float) * 2 * kMlpIn * (size_t)n,
                          cudaMemcpyHostToDevice, m->st));
  FE_CUDA(cudaMemcpyAsync(m->y, y, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, m->st));
  m->ndata = n;
  return FE_OK;
}

// Trains on n samples resident on the device (data: n x [64 before | 64
// after], y: n).  Epochs of shuffled batches (Philox permutation keys);
// loss_hist[e] = mean batch loss of epoch e.
int mlp_train_device(Mlp *m, const float *data, const float *y, long long n, int epochs, int B,
                     float lr, uint64_t seed, float *loss_hist) {
  if (B < 64 || B % 64 || n < B || epochs < 1) {
    set_error("fe_mlp_train: batch must be a multiple of 64 and at most the sample count");
    return FE_ERR_ARG;
  }
  int rc;
  if ((rc = mlp_reserve_batch(m, B)) || (rc = mlp_reserve_train(m, n, epochs))) return rc;
  // per-feature normalisation from the samples (both halves)
  const int nblk = (int)(n < 2 * kNormBlocks ? (n + 1) / 2 : kNormBlocks);
  k_mlp_moments<<<nblk, 256, 0, m->st>>>(n, data, m->moments);
  FE_LAUNCH_CHECK("k_mlp_moments");
  k_mlp_normalise<<<1, 1024, 0, m->st>>>(n, nblk, m->moments, m->mean, m->istd);
  FE_LAUNCH_CHECK("k_mlp_normalise");
  const long long nbatch = n / B;
  // One cluster runs an epoch while a CTA has at most two tiles a batch; above
  // that two launches a batch, pass 1 over more CTAs.  Pass 2 has eight parts
  // whatever the batch: 2,048 samples in batches of 64, 128 and 256 take 2.01, 1.19
  // and 0.79 ms on eight CTAs; on 1, 2 and 4, as many as the batch has tiles, 6.73,
  // 2.31 and 1.00.
  const bool cluster = B / kTrSamples <= 2 * kTrCluster;
  const float b1 = 0.9f, b2 = 0.999f;
  // Fisher-Yates with Philox draws: the draws on the device one epoch ahead, the
  // swaps here while the device trains
  auto draw = [&](int e) -> int {
    const int k = e & 1;
    k_mlp_draws<<<(unsigned)((n + 255) / 256), 256, 0, m->st_draw>>>(
        n, seed, (uint64_t)e * (uint64_t)n, m->draws[k]);
    FE_LAUNCH_CHECK("k_mlp_draws");
    FE_CUDA(cudaMemcpyAsync(m->h_draws[k], m->draws[k], sizeof(int) * (size_t)n,
                            cudaMemcpyDeviceToHost, m->st_draw));
    FE_CUDA(cudaEventRecord(m->ev_draw[k], m->st_draw));
    return FE_OK;
  };
  FE_CUDA(cudaMemsetAsync(m->ep_loss, 0, sizeof(double) * (size_t)epochs, m->st));
  int *h_err = reinterpret_cast<int *>(m->h_loss + epochs);
  auto run = [&]() -> int {
    int rc;
    if ((rc = draw(0))) return rc;
    for (int e = 0; e < epochs; e++) {
      const int k = e & 1;
      if (e >= 2) FE_CUDA(cudaEventSynchronize(m->ev_idx[k]));  // pinned buffers free again
      if (e + 1 < epochs && (rc = draw(e + 1))) return rc;
      int *perm = m->h_idx[k];
      for (long long i = 0; i < n; i++) perm[i] = (int)i;
      FE_CUDA(cudaEventSynchronize(m->ev_draw[k]));
      const int *j = m->h_draws[k];
      for (long long i = n - 1; i > 0; i--) std::swap(perm[i], perm[j[i]]);
      for (long long bi = 0; bi < nbatch; bi++) {
        m->step++;
        m->h_bc[k][bi] = make_float2(1.f - powf(b1, (float)m->step),
                                     1.f - powf(b2, (float)m->step));
      }
      FE_CUDA(cudaMemcpyAsync(m->idx[k], perm, sizeof(int) * (size_t)(nbatch * B),
                              cudaMemcpyHostToDevice, m->st));
      FE_CUDA(cudaMemcpyAsync(m->bc[k], m->h_bc[k], sizeof(float2) * (size_t)nbatch,
                              cudaMemcpyHostToDevice, m->st));
      FE_CUDA(cudaEventRecord(m->ev_idx[k], m->st));
      TrainArgs a = train_args(m, data, y, B);
      a.nbatch = (int)nbatch;
      a.passes = 3;
      a.update = 1;
      a.idx = m->idx[k];
      a.bc = m->bc[k];
      a.lr = lr;
      a.loss = m->ep_loss + e;
      if (cluster) {
        if ((rc = launch_train(m, a, kTrCluster, true))) return rc;
      } else {
        for (long long bi = 0; bi < nbatch; bi++)
          if ((rc = train_batch(m, a, (int)bi))) return rc;
      }
    }
    FE_CUDA(cudaMemcpyAsync(m->h_loss, m->ep_loss, sizeof(double) * (size_t)epochs,
                            cudaMemcpyDeviceToHost, m->st));
    FE_CUDA(cudaMemcpyAsync(h_err, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->st));
    return FE_OK;
  };
  rc = run();
  cudaStreamSynchronize(m->st_draw);
  if (rc) {
    cudaStreamSynchronize(m->st);
    return rc;
  }
  FE_CUDA(cudaStreamSynchronize(m->st));
  if (loss_hist)
    for (int e = 0; e < epochs; e++) loss_hist[e] = (float)(m->h_loss[e] / (double)nbatch);
  return mlp_check_err(m, *h_err);
}

}  // namespace fe

using namespace fe;

struct fe_mlp {
  Mlp m;
};

namespace fe {
Mlp *mlp_from_handle(fe_mlp *h) { return &h->m; }
}  // namespace fe

extern "C" {

int fe_mlp_create(fe_mlp **out, int device, uint64_t seed) {
  if (!out) return FE_ERR_ARG;
  fe_mlp *h = new fe_mlp();
  int rc = mlp_create(&h->m, device, seed);
  if (rc) {
    mlp_free(&h->m);
    delete h;
    return rc;
  }
  *out = h;
  return FE_OK;
}

void fe_mlp_destroy(fe_mlp *h) {
  if (!h) return;
  if (h->m.st) cudaStreamSynchronize(h->m.st);
  mlp_free(&h->m);
  delete h;
}

int fe_mlp_param_count(void) { return kMlpParams; }

int fe_mlp_set_params(fe_mlp *h, const float *params, const float *mean, const float *istd) {
  if (!h || !params) return FE_ERR_ARG;
  Mlp *m = &h->m;
  FE_CUDA(cudaMemcpyAsync(m->P, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, m->st));
  if (mean)
    FE_CUDA(cudaMemcpyAsync(m->mean, mean, sizeof(float) * kMlpIn, cudaMemcpyHostToDevice, m->st));
  if (istd)
    FE_CUDA(cudaMemcpyAsync(m->istd, istd, sizeof(float) * kMlpIn, cudaMemcpyHostToDevice, m->st));
  int rc = mlp_refresh(m);
  if (rc) return rc;
  FE_CUDA(cudaStreamSynchronize(m->st));
  return FE_OK;
}

int fe_mlp_get_params(fe_mlp *h, float *params, float *mean, float *istd) {
  if (!h) return FE_ERR_ARG;
  Mlp *m = &h->m;
  if (params)
    FE_CUDA(cudaMemcpyAsync(params, m->P, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, m->st));
  if (mean)
    FE_CUDA(cudaMemcpyAsync(mean, m->mean, sizeof(float) * kMlpIn, cudaMemcpyDeviceToHost, m->st));
  if (istd)
    FE_CUDA(cudaMemcpyAsync(istd, m->istd, sizeof(float) * kMlpIn, cudaMemcpyDeviceToHost, m->st));
  FE_CUDA(cudaStreamSynchronize(m->st));
  return FE_OK;
}

// Gradient of the batch loss at the current parameters (no update): B
// samples of 128 inputs (64 before, 64 after) and targets y; B % 64 == 0.
int fe_mlp_grad(fe_mlp *h, const float *data, const float *y, int B, float *grad, float *loss,
                float *out2B) {
  if (!h || !data || !y || B < 64 || B % 64) return FE_ERR_ARG;
  Mlp *m = &h->m;
  int rc;
  if ((rc = mlp_reserve_batch(m, B))) return rc;
  if ((rc = mlp_upload(m, data, y, B))) return rc;
  std::vector<int> order(B);
  for (int i = 0; i < B; i++) order[i] = i;
  FE_CUDA(cudaMemcpyAsync(m->idx1, order.data(), sizeof(int) * B, cudaMemcpyHostToDevice, m->st));
  FE_CUDA(cudaMemsetAsync(m->loss, 0, sizeof(double), m->st));
  TrainArgs a = train_args(m, m->data, m->y, B);
  a.idx = m->idx1;
  a.out = m->out;
  if ((rc = train_batch(m, a, 0))) return rc;
  double dl = 0.0;
  int e = 0;
  if (grad)
    FE_CUDA(cudaMemcpyAsync(grad, m->G, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, m->st));
  FE_CUDA(cudaMemcpyAsync(&dl, m->loss, sizeof(double), cudaMemcpyDeviceToHost, m->st));
  FE_CUDA(cudaMemcpyAsync(&e, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->st));
  if (out2B)
    FE_CUDA(cudaMemcpyAsync(out2B, m->out, sizeof(float) * 2 * B, cudaMemcpyDeviceToHost, m->st));
  FE_CUDA(cudaStreamSynchronize(m->st));
  if (loss) *loss = (float)dl;
  return mlp_check_err(m, e);
}

int fe_mlp_train(fe_mlp *h, const float *data, const float *y, int64_t n, int epochs, int batch,
                 float lr, uint64_t seed, float *loss_hist) {
  if (!h || !data || !y || n < 1) return FE_ERR_ARG;
  Mlp *m = &h->m;
  int rc;
  if ((rc = mlp_upload(m, data, y, n))) return rc;
  return mlp_train_device(m, m->data, m->y, n, epochs, batch, lr, seed, loss_hist);
}

// Test entry for the tensor-core GEMM alone: D = A B^T (+ bias), host arrays,
// A: M x K, B: N x K bf16 bit patterns, D: M x N fp32.
int fe_tc_gemm_bf16(const uint16_t *A, const uint16_t *B, const float *bias, float *D, int M,
                    int N, int K) {
  if (!A || !B || !D) return FE_ERR_ARG;
  bf16 *dA = nullptr, *dB = nullptr;
  float *dD = nullptr, *dbias = nullptr;
  int *derr = nullptr;
  int rc = FE_OK;
  cudaError_t e = cudaSuccess;
  do {
    if ((e = cudaMalloc(&dA, 2 * (size_t)M * K))) break;
    if ((e = cudaMalloc(&dB, 2 * (size_t)N * K))) break;
    if ((e = cudaMalloc(&dD, 4 * (size_t)M * N))) break;
    if ((e = cudaMalloc(&derr, sizeof(int)))) break;
    if ((e = cudaMemset(derr, 0, sizeof(int)))) break;
    if (bias && (e = cudaMalloc(&dbias, 4 * (size_t)N))) break;
    if ((e = cudaMemcpy(dA, A, 2 * (size_t)M * K, cudaMemcpyHostToDevice))) break;
    if ((e = cudaMemcpy(dB, B, 2 * (size_t)N * K, cudaMemcpyHostToDevice))) break;
    if (bias && (e = cudaMemcpy(dbias, bias, 4 * (size_t)N, cudaMemcpyHostToDevice))) break;
    rc = gemm_tc(0, dA, K, dB, K, dbias, dD, N, M, N, K, derr);
    if (rc) break;
    if ((e = cudaDeviceSynchronize())) break;
    int he = 0;
    if ((e = cudaMemcpy(&he, derr, sizeof(int), cudaMemcpyDeviceToHost))) break;
    if (he) {
      set_error("tensor-core GEMM: an MMA completion wait ran out");
      rc = FE_ERR_DEVICE;
      break;
    }
    e = cudaMemcpy(D, dD, 4 * (size_t)M * N, cudaMemcpyDeviceToHost);
  } while (0);
  cudaFree(dA);
  cudaFree(dB);
  cudaFree(dD);
  cudaFree(dbias);
  cudaFree(derr);
  if (e != cudaSuccess) return cuda_fail(e, "fe_tc_gemm_bf16");
  return rc;
}

}  // extern "C"
