// The bf16 matrix product of a step of up to 16 tokens: C[m, n] = sum_k X[m, k] W[n, k], every thread its own
// numbers from memory to the tensor cores.
//
// With this few tokens a product is the streaming of its weights plus what a kernel costs before the first
// and after the last of them, and in a decode step, a chain of such products of a few megabytes, it is
// mostly the latter. csrc/gemm_tc.cu (tensor maps, mbarriers, tensor memory, clusters that add their K
// ranges through each other's shared memory) pays 4 us from one kernel's end to the next for products
// whose bytes take 1. Here a block of eight warps has 16 rows of W and all of K; a warp asks for its first
// weights while the kernel before is still running, with nothing to set up; after the wait come one trip to
// L2 for x, the products (mma.sync m16n8k16), one meeting of the block and the store.
//
// The tensor cores' K index may be any permutation of the columns as long as both operands use the same
// one: a lane takes eight neighbouring columns of a row with one 16-byte copy, and they serve as its
// numbers of two products. So a thread needs what it asked for itself and nothing else, and a warp's copy is
// 64 contiguous bytes of each of eight rows. The warps take groups of 32 columns in turn. Sums are fp32, a
// warp's own first, then the eight warps' in their order.
//
// Bound by the bytes in flight (96 KB of weights an SM), which have to be somewhere while they are: in slots of
// shared memory that belong to the thread (cp.async), not in registers by plain loads. Those are in flight in
// L1, and an SM whose neighbours in the stream use much shared memory (csrc/gemm_tc.cu, the attention of
// decoded tokens) has 28 KB of it left: the gated product of 55 MB took 17.6 us there and 10.8 alone, now 10.5
// in both; steps of 8 users behind 16,384 tokens, width 1,536, 1,599 us for 2,096; of width 2,048 and 8 users
// 994 for 1,360. Weights are the first to leave L2, or a step's states and activations leave with them
// (width 2,048, 4 users: 397 us a step for 434, and 415 with plain loads).
//
// Epilogues as in csrc/gemm_tc.cu. `parts` > 1: K is cut into that many ranges for blocks of their own
// (few rows, long K), whose sums are left apart for the reader to add.
#include "common.cuh"
#include "mma.cuh"

namespace {

constexpr int kWarps = 8, kThreads = 32 * kWarps;
constexpr int kRows = 16;

enum : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_ACCUM = 2, EPI_GATED = 3, EPI_CLAMPED = 4, EPI_RELU2 = 5 };
constexpr bool gated_epi(int epi) { return epi == EPI_GATED || epi == EPI_CLAMPED; }

// groups of columns a warp asks for at a time, at most
constexpr int ahead(int epi) { return gated_epi(epi) ? 3 : 6; }

// pieces of 16 bytes that a thread has of a group: of the weights' rows, and of x
constexpr int pieces(int epi, int nt) { return (gated_epi(epi) ? 4 : 2) + nt; }

struct Few {
  const __nv_bfloat16* x;
  long long ldx;
  const __nv_bfloat16* w;            // [rows, K]
  int M, N, K;
  int groups;                        // groups of 32 columns of one part
  int each;                          // groups a warp takes at a time
  int dual_offset;
  float limit, alpha, plus;
  const void* bias;
  int bias_dtype;
  void* out;
  long long ldo, part_stride;
};

// 16 bytes to shared memory, past L1 (zeros, and nothing read, where `in` is false).
__device__ __forceinline__ void copy16(uint32_t to, const __nv_bfloat16* from, bool in) {
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(n) : "memory");
}
// The same of what is read once a step: the first to leave L2, which keeps states and activations instead.
__device__ __forceinline__ void copy16_once(uint32_t to, const __nv_bfloat16* from, bool in, uint64_t policy) {
  const int n = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(to), "l"(from),
               "r"(n), "l"(policy)
               : "memory");
}
__device__ __forceinline__ uint64_t leaves_first() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint4 copied16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(at)
               : "memory");
  return v;
}

__device__ __forceinline__ float bias_of(const Few& p, int n) {
  if (!p.bias) return 0.f;
  return p.bias_dtype == SAKV_F32 ? static_cast<const float*>(p.bias)[n]
                                  : widen(static_cast<const __nv_bfloat16*>(p.bias)[n]);
}

// NT: groups of eight tokens. FULL: a warp takes as many groups of columns at a time as it has slots for, known
// when compiled; else `each` of them, so that all warps have the same (K 1,024: four, not six for five warps
// and two for the sixth; at K 512 the error against 64 bits is 7.4e-8, not 9.9e-8).
template <int NT, int kEpi, bool FULL>
__global__ void __launch_bounds__(kThreads, 2) gemm_few_kernel(const Few p) {
  constexpr int kSets = gated_epi(kEpi) ? 2 : 1;       // gate and up rows
  constexpr int kAhead = ahead(kEpi);
  const int each = FULL ? kAhead : p.each;
  __shared__ float sums[kSets][kWarps][NT * 8][kRows + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kRows, part = blockIdx.y;
  const int row = lane >> 2, col = (lane & 3) * 8;
  // (rows beyond the last are the last one again, and not stored)
  const __nv_bfloat16* from[kSets][2];
#pragma unroll
  for (int s = 0; s < kSets; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      from[s][h] = p.w + ((long long)s * p.dual_offset + min(n0 + row + 8 * h, p.N - 1)) * p.K + col;
  const int first = part * p.groups, last = min(first + p.groups, (p.K + 31) / 32);
  // what a thread has asked for, and nobody else reads
  extern __shared__ __align__(16) uint4 ring[];          // [kAhead][kPieces][kThreads]
  constexpr int kPieces = pieces(kEpi, NT);
  const uint32_t mine = static_cast<uint32_t>(__cvta_generic_to_shared(ring)) + threadIdx.x * 16;
  auto slot = [&](int i, int piece) { return mine + (i * kPieces + piece) * (kThreads * 16); };
  const uint64_t once = leaves_first();
  auto ask = [&](int i, int g) {
    if (g >= last || (!FULL && i >= each)) return;       // (the whole warp)
    const bool in = g * 32 + col < p.K;
#pragma unroll
    for (int s = 0; s < kSets; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) copy16_once(slot(i, 2 * s + h), in ? from[s][h] + g * 32 : p.w, in, once);
  };
  auto ask_x = [&](int i, int g) {
    if (g >= last || (!FULL && i >= each)) return;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int m = t * 8 + row;
      const bool in = g * 32 + col < p.K && m < p.M;
      copy16(slot(i, 2 * kSets + t), in ? p.x + m * p.ldx + g * 32 + col : p.x, in);
    }
  };
  // two sums an output, of every second product: the tensor cores cut where they add, and a chain of half
  // the length loses half as much (relative error at K 1,536: 1.2e-7 as csrc/gemm_tc.cu; in one chain 1.8e-7)
  float acc[kSets][NT][2][4];
#pragma unroll
  for (int s = 0; s < kSets; ++s)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[s][t][0][k] = acc[s][t][1][k] = 0.f;

#pragma unroll
  for (int i = 0; i < kAhead; ++i) ask(i, first + warp * each + i);
  copies_commit();
  float bias = 0.f;
  if (threadIdx.x < NT * 8 * kRows && n0 + (int)(threadIdx.x & 15) < p.N && part == 0)
    bias = bias_of(p, n0 + (threadIdx.x & 15));
  wait_for_previous_kernel();
  let_next_kernel_start();
#pragma unroll
  for (int i = 0; i < kAhead; ++i) {
    ask_x(i, first + warp * each + i);
    copies_commit();
  }
  for (int g0 = first + warp * each; g0 < last; g0 += each * kWarps) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      // (a set of copies, empty or not, is committed for every group: all but the newest kAhead - 1 are there)
      copies_wait<kAhead - 1>();
      if (g0 + i < last && (FULL || i < each)) {
        uint4 x[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) x[t] = copied16(slot(i, 2 * kSets + t));
#pragma unroll
        for (int s = 0; s < kSets; ++s) {
          const uint4 lo = copied16(slot(i, 2 * s)), hi = copied16(slot(i, 2 * s + 1));
          const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            mma::bf16_16816(acc[s][t][0], a0, x[t].x, x[t].y);
            mma::bf16_16816(acc[s][t][1], a1, x[t].z, x[t].w);
          }
        }
        ask(i, g0 + each * kWarps + i);
        ask_x(i, g0 + each * kWarps + i);
      }
      copies_commit();
    }
  }
#pragma unroll
  for (int s = 0; s < kSets; ++s)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        sums[s][warp][t * 8 + (lane & 3) * 2 + (k & 1)][row + 8 * (k >> 1)] =
            acc[s][t][0][k] + acc[s][t][1][k];
  __syncthreads();
  const int r = threadIdx.x & 15, m = threadIdx.x >> 4, n = n0 + r;
  if (m >= NT * 8 || m >= p.M || n >= p.N) return;
  float c[kSets];
#pragma unroll
  for (int s = 0; s < kSets; ++s) {
    c[s] = sums[s][0][m][r];
#pragma unroll
    for (int i = 1; i < kWarps; ++i) c[s] += sums[s][i][m][r];
  }
  const long long at = m * p.ldo + n + part * p.part_stride;
  float* out32 = static_cast<float*>(p.out);
  __nv_bfloat16* out16 = static_cast<__nv_bfloat16*>(p.out);
  if (kEpi == EPI_F32) {
    out32[at] = c[0] + bias;
  } else if (kEpi == EPI_ACCUM) {
    atomicAdd(out32 + at, c[0] + bias);      // (the only addition to this element)
  } else if (kEpi == EPI_BF16) {
    out16[at] = narrow<__nv_bfloat16>(c[0] + bias);
  } else if (kEpi == EPI_RELU2) {
    const float z = fmaxf(c[0] + bias, 0.f);
    out16[at] = narrow<__nv_bfloat16>(z * z);
  } else if (kEpi == EPI_CLAMPED) {
    const float g = fminf(c[0], p.limit), u = fminf(fmaxf(c[kSets - 1], -p.limit), p.limit);
    out16[at] = narrow<__nv_bfloat16>(g / (1.0f + expf(-p.alpha * g)) * (u + p.plus));
  } else {
    out16[at] = narrow<__nv_bfloat16>(c[0] / (1.0f + expf(-c[0])) * c[kSets - 1]);
  }
}

template <int NT, int kEpi, bool FULL>
int launch(dim3 grid, cudaStream_t stream, const Few& p) {
  constexpr int kRing = ahead(kEpi) * pieces(kEpi, NT) * kThreads * 16;      // (61 to 98 KB)
  static PerDeviceOnce once;
  if (once.needs()) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<NT, kEpi, FULL>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, kRing);
    if (e != cudaSuccess) return static_cast<int>(e);
    once.done();
  }
  return launch_overlapped(gemm_few_kernel<NT, kEpi, FULL>, grid, dim3(kThreads), kRing, stream, 1, p);
}

}  // namespace

// x: [M, K] bf16 rows `ldx` apart; w: [N, K] bf16 (gated: gate rows, and up rows from `dual_offset` on);
// M up to 16, K and ldx multiples of 8, x and w at multiples of 16 bytes. epi, bias, out, ldo, clamp: as
// `sakv_gemm_tc`. parts > 1 (EPI_F32): part i's sums at out + i * part_stride, the bias in part 0.
SAKV_EXPORT int sakv_gemm_few(const void* x, long long ldx, const void* w, int M, int N, int K, int parts,
                              int epi, int dual_offset, const void* bias, int bias_dtype, void* out,
                              long long ldo, long long part_stride, float limit, float alpha, float plus,
                              cudaStream_t stream) {
  if (M <= 0 || M > 16 || N <= 0 || K <= 0 || K % 8 || ldx % 8 || parts < 1 || parts > 64 || ldo < N ||
      epi < 0 || epi > EPI_RELU2 || (parts > 1 && epi != EPI_F32) ||
      (((uintptr_t)x | (uintptr_t)w) & 15))
    return cudaErrorInvalidValue;
  const int groups = (K + 31) / 32;
  Few p = {(const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, M, N, K, (groups + parts - 1) / parts, 1,
           dual_offset, limit, alpha, plus, bias, bias_dtype, out, ldo, part_stride};
  const int most = kWarps * ahead(epi), rounds = (p.groups + most - 1) / most;
  p.each = (p.groups + kWarps * rounds - 1) / (kWarps * rounds);     // (the same for all warps, nearly)
  const dim3 grid((unsigned)((N + kRows - 1) / kRows), (unsigned)parts);
  const bool full = p.each == ahead(epi);
#define SAKV_FEW(EPI)                                                                            \
  if (epi == EPI)                                                                                \
    return M <= 8 ? full ? launch<1, EPI, true>(grid, stream, p) : launch<1, EPI, false>(grid, stream, p) \
                  : full ? launch<2, EPI, true>(grid, stream, p) : launch<2, EPI, false>(grid, stream, p)
  SAKV_FEW(EPI_BF16);
  SAKV_FEW(EPI_F32);
  SAKV_FEW(EPI_ACCUM);
  SAKV_FEW(EPI_GATED);
  SAKV_FEW(EPI_CLAMPED);
  SAKV_FEW(EPI_RELU2);
#undef SAKV_FEW
  return cudaErrorInvalidValue;
}
