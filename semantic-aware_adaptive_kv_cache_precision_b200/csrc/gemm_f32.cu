// The true 32-bit matrix product of the fp32 path:
//   C[m, n] (+)= sum_k A[m, k] W[n, k]  (+ bias[n])
// with W stored (out, in) row-major as in the checkpoint, plain FFMA in fp32 (no
// TF32, no tensor cores). Each output element adds its products for k = 0, 1,
// 2, ... in that order whatever the tile and whatever M is, so a row's result
// is the same to the bit whether it is computed alone or among 2,048 others.
// This is what makes "whole prompt == token by token == batched" exact in the
// fp32 path. The reference's counterpart is cuBLAS with fp32 accumulation
// (`src/core_kernels/linear.cu:85-142`).
#include "common.cuh"

namespace {

__device__ __forceinline__ void copy_async16(uint32_t dst, const float* src, bool real) {
  const int n = real ? 16 : 0;                    // (0: zeros, nothing is read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t dst, const float* src, bool real) {
  const int n = real ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// A BM x BN tile of the output a block, TM x TN outputs a thread (rows ty, ty + BM / TM, ...; columns
// likewise), K in steps of BK through a ring of STAGES copied with cp.async. The order of a sum makes
// a chain of K dependent multiply-adds, some 4 cycles each, that no split may shorten: what is left to
// win is that nothing else stands in it (four of them a pair of 16-byte reads, the copies STAGES - 1
// steps ahead) and that there are enough tiles for every SM (`sakv_gemm_f32`). `wide`: rows that begin at
// multiples of 16 bytes.
template <int BM, int BN, int TM, int TN, int BK, int STAGES>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W,
                const float* __restrict__ bias, float* __restrict__ C, long long ldc, int M,
                int N, int K, int accumulate, int wide) {
  constexpr int kThreads = (BM / TM) * (BN / TN), kLd = BK + 4;
  extern __shared__ __align__(16) float smem[];       // [STAGES][BM + BN][kLd]
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int steps = (K + BK - 1) / BK;
  auto fill = [&](int step, const float* from, long long ld, int first, int end, int rows, int row0) {
    const int k0 = step * BK;
    const uint32_t to = base + ((step % STAGES) * (BM + BN) + row0) * kLd * 4;
    if (wide) {
      for (int i = threadIdx.x; i < rows * (BK / 4); i += kThreads) {
        const int r = i / (BK / 4), c = i % (BK / 4) * 4;
        const bool real = first + r < end && k0 + c < K;
        copy_async16(to + (r * kLd + c) * 4, real ? from + (first + r) * ld + k0 + c : from, real);
      }
    } else {
      for (int i = threadIdx.x; i < rows * BK; i += kThreads) {
        const int r = i / BK, c = i % BK;
        const bool real = first + r < end && k0 + c < K;
        copy_async4(to + (r * kLd + c) * 4, real ? from + (first + r) * ld + k0 + c : from, real);
      }
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) {
      fill(s, W, K, n0, N, BN, BM);
      fill(s, A, lda, m0, M, BM, 0);
    }
    commit();
  }
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    if (step + STAGES - 1 < steps) {
      fill(step + STAGES - 1, W, K, n0, N, BN, BM);
      fill(step + STAGES - 1, A, lda, m0, M, BM, 0);
    }
    commit();
    const float* as = smem + (step % STAGES) * (BM + BN) * kLd;
    const float* ws = as + BM * kLd;
    // (a run of kRun k's is read while the one before it is summed)
    constexpr int kRun = TM * TN == 1 ? 16 : 4;
    float4 a[2][kRun / 4][TM], w[2][kRun / 4][TN];
    auto read = [&](int k, int to) {
#pragma unroll
      for (int u = 0; u < kRun / 4; ++u) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
          a[to][u][i] = *reinterpret_cast<const float4*>(as + (ty + i * (BM / TM)) * kLd + k + 4 * u);
#pragma unroll
        for (int j = 0; j < TN; ++j)
          w[to][u][j] = *reinterpret_cast<const float4*>(ws + (tx + j * (BN / TN)) * kLd + k + 4 * u);
      }
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; k += kRun) {
      const int now = k / kRun & 1;
      if (k + kRun < BK) read(k + kRun, now ^ 1);
#pragma unroll
      for (int u = 0; u < kRun / 4; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j)
              acc[i][j] = fmaf(reinterpret_cast<const float*>(&a[now][u][i])[e],
                               reinterpret_cast<const float*>(&w[now][u][j])[e], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * (BM / TM);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * (BN / TN);
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      float* c = C + (long long)m * ldc + n;
      *c = accumulate ? *c + v : v;
    }
  }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
int launch(const float* A, long long lda, const float* W, const float* bias, float* C, long long ldc,
           int M, int N, int K, int accumulate, cudaStream_t stream) {
  constexpr int kSmem = STAGES * (BM + BN) * (BK + 4) * 4;
  auto kernel = gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>;
  static PerDeviceOnce configured;
  if (configured.needs()) {
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return (int)e;
    configured.done();
  }
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return cudaErrorInvalidValue;
  const int wide = K % 4 == 0 && lda % 4 == 0 && !(((uintptr_t)A | (uintptr_t)W) & 15);
  return launch_ordered(kernel, grid, dim3((BM / TM) * (BN / TN)), kSmem, stream, A, lda, W, bias, C,
                           ldc, M, N, K, accumulate, wide);
}

}  // namespace

SAKV_EXPORT int sakv_gemm_f32(const float* A, long long lda, const float* W, const float* bias,
                              float* C, long long ldc, int M, int N, int K, int accumulate,
                              cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldc < N) return cudaErrorInvalidValue;
  if (M == 0) return 0;
  // The largest tile that still gives every SM one (larger tiles read less shared memory a product,
  // more tiles fill the GPU). Up to 4 tokens the tile is one warp's, with four columns a
  // thread where there are enough of them. Before (64 columns a block, one step of 16 k's at a time) and
  // now, us: 4 tokens 192 -> 704 17.4 / 2.7, 1536 -> 17920 247 / 43, 8960 -> 1536 1347 / 62; 24 tokens
  // 1536 -> 17920 358 / 89; 96 tokens 8960 -> 1536 1762 / 260, 200 tokens 1536 -> 17920 803 / 402
  auto tiles = [&](long long bm, long long bn) { return (M + bm - 1) / bm * ((N + bn - 1) / bn); };
#define SAKV_F32_TILE(BM, BN, TM, TN, BK, STAGES) \
  return launch<BM, BN, TM, TN, BK, STAGES>(A, lda, W, bias, C, ldc, M, N, K, accumulate, stream)
  if (M <= 4 && tiles(4, 32) >= 3LL * sm_count()) SAKV_F32_TILE(4, 32, 1, 4, 64, 4);
  if (M <= 4) SAKV_F32_TILE(4, 8, 1, 1, 128, 5);
  const int sms = sm_count();
  if (M > 32 && (tiles(64, 64) >= sms || (M + 15) / 16 > 65535)) SAKV_F32_TILE(64, 64, 4, 4, 32, 3);
  if (M > 16 && (tiles(32, 32) >= sms || (M + 15) / 16 > 65535)) SAKV_F32_TILE(32, 32, 2, 2, 64, 3);
  SAKV_F32_TILE(16, 8, 1, 1, 128, 4);
#undef SAKV_F32_TILE
}
