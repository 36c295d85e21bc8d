// The grouped products of a mixture of experts on tcgen05: rows sorted by expert, every expert's rows
// times its own weights.
//
//   DUAL   out[r, n] = act((rows W0[e]^T)[r, n], (rows W1[e]^T)[r, n])      bf16
//   else   out[r, n] = (rows W0[e]^T)[r, n]                                 fp32
//   act(g, u) = g' sigmoid(alpha g') (u' + plus), g' = min(g, limit), u' within +-limit
//
// A tile is XR rows of one expert x 2 HB weight rows (HB of each matrix, or 2 HB of the one); rows on
// the MMA's 128 lanes, weight rows on its columns, fp32 sums in tensor memory, twice, so that a
// tile's epilogue runs under the next tile's products. Persistent blocks, one an SM, take tiles in
// turn; an expert's tiles lie together, its rows fastest, so that the blocks that run at one time
// share weight tiles in L2. Nothing is read back by the host: each block works the tiles out from
// the experts' row offsets on the device.
//
//   XR 128, HB 128   prompts: one tcgen05.mma is 128 x 256 x 16 (the tensor cores' full rate), four
//                    stages of 48 KB. 3,001 tokens of 4 choices among 32 experts, 2 x 1024 x 2048: 101
//                    us (1.0 PFLOP/s), 530 before on mma.sync in tiles of 32 x 64; 3,160 tokens with 2
//                    experts, 2 x 1024 x 1024, 27 us, 156 before
//   XR 32, HB 32     few rows an expert: what counts is that the weights stream, through as many SMs
//                    as there are tiles; a box of 32 rows, the MMA's other 96 lanes hold whatever lies
//                    behind them and nobody reads their sums. One token of 4 experts, 2 x
//                    1024 x 2048: 14 us, 32 before
//
//   warp 0     TMA: boxes of 64 columns of the rows and of the weights into the ring
//   warp 1     tensor memory; lane 0 issues the products and commits stages and accumulators
//   the others epilogue: thread = row, warps of one quarter of the rows share out the columns. The
//              activation (expf and a division, as the general kernel takes it) of a tile's 128 x 128
//              outputs takes four warps longer than the tile's products: 4,136 tokens of 2 choices
//              among 16 experts, 2 x 1024 x 1024: 58 us with four warps, 40 with eight, 39 with sixteen;
//              16 tokens 27.8, 23.2 and 21.2
#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace {

constexpr int BK = 64;                     // K step: one 128-byte swizzle row of bf16
constexpr int kMaxExperts = 1024;

struct Params {
  const int32_t* offsets;                  // [experts + 1]: where each expert's rows begin
  void* out;
  int experts, N, K;                       // N: output columns = rows of a weight matrix
  float limit, alpha, plus;
  int* error;
};

template <int XR, int HB>
struct Ring {
  static constexpr int kXBytes = XR * BK * 2, kWBytes = 2 * HB * BK * 2;
  static constexpr int kStageBytes = kXBytes + kWBytes;
  static constexpr int kStages = XR == 128 ? 4 : 12;
  static constexpr int kEpilogue = HB == 128 ? 512 : 256;     // threads of the epilogue
  static constexpr int kThreads = 64 + kEpilogue;
  static constexpr int kSlack = 128 * BK * 2 - kXBytes;       // (the MMA reads 128 rows)
  static constexpr int kSmem = kStages * kStageBytes + kSlack + 1024 + 512 + (kMaxExperts + 1) * 4;
};

template <int STAGES>
struct Barriers {
  uint64_t full[STAGES], empty[STAGES];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem;
};

template <int XR, int HB, bool DUAL>
__global__ void __launch_bounds__(Ring<XR, HB>::kThreads, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w0_map,
              const __grid_constant__ CUtensorMap w1_map, const Params p) {
  using R = Ring<XR, HB>;
  constexpr int BN = 2 * HB, kStages = R::kStages;
  constexpr uint32_t kTmemCols = 2 * BN;
  static_assert(R::kXBytes % 1024 == 0 && R::kStageBytes % 1024 == 0, "swizzled tiles begin at 1024 bytes");
  static_assert(sizeof(Barriers<kStages>) <= 512 && R::kSmem <= 227 * 1024, "");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  auto* bar = reinterpret_cast<Barriers<kStages>*>(smem + kStages * R::kStageBytes + R::kSlack);
  int32_t* first_tile = reinterpret_cast<int32_t*>(reinterpret_cast<uint8_t*>(bar) + 512);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_kb = (p.K + BK - 1) / BK;
  constexpr int kCols = DUAL ? HB : BN;                 // output columns of a tile
  const int n_tiles = (p.N + kCols - 1) / kCols;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      tma::mbar_init(&bar->full[s], 1);
      tma::mbar_init(&bar->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tma::mbar_init(&bar->acc_full[i], 1);
      tma::mbar_init(&bar->acc_empty[i], R::kEpilogue);
    }
    tma::fence_barrier_init();
    tma::prefetch_map(&x_map);
    tma::prefetch_map(&w0_map);
    if (DUAL) tma::prefetch_map(&w1_map);
  }
  if (warp == 1) tc::tmem_alloc(&bar->tmem, kTmemCols);
  if (warp == 0) {                          // the experts' first row tiles
    int base = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int mine = e < p.experts ? (p.offsets[e + 1] - p.offsets[e] + XR - 1) / XR : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (e < p.experts) first_tile[e] = base + sum - mine;
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first_tile[p.experts] = base;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = bar->tmem;
  const int tiles = first_tile[p.experts] * n_tiles;

  struct Tile {
    int expert, row0, rows, n0;             // its first row, rows of it, its first output column
  };
  auto tile_at = [&](int i) {
    int lo = 0, hi = p.experts;             // the last expert whose tiles begin at or before i
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first_tile[mid] * n_tiles <= i) lo = mid;
      else hi = mid;
    }
    const int row_tiles = first_tile[lo + 1] - first_tile[lo];
    const int at = i - first_tile[lo] * n_tiles;
    Tile t;
    t.expert = lo;
    t.row0 = p.offsets[lo] + at % row_tiles * XR;
    t.rows = min(XR, p.offsets[lo + 1] - t.row0);
    t.n0 = at / row_tiles * kCols;
    return t;
  };

  if (warp == 0) {
    // ---- TMA producer -----------------------------------------------------------------
    if (lane == 0) {
      int stage = 0, phase = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < tiles && ok; i += gridDim.x) {
        const Tile t = tile_at(i);
        const int w_row = t.expert * p.N + t.n0;
        for (int kb = 0; kb < n_kb; ++kb) {
          // (waiting for the parity before the ring's own: the first pass finds every stage free)
          if (!tma::mbar_wait(&bar->empty[stage], phase ^ 1, p.error, 801)) {
            ok = false;
            break;
          }
          uint8_t* dst = smem + stage * R::kStageBytes;
          tma::mbar_expect_tx(&bar->full[stage], R::kStageBytes);
          tma::load_2d(dst, &x_map, kb * BK, t.row0, &bar->full[stage]);
          tma::load_2d(dst + R::kXBytes, &w0_map, kb * BK, w_row, &bar->full[stage]);
          tma::load_2d(dst + R::kXBytes + R::kWBytes / 2, DUAL ? &w1_map : &w0_map, kb * BK,
                       DUAL ? w_row : w_row + HB, &bar->full[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // before this block may leave: every stage it filled has been given back
      for (int s = 0; s < kStages && ok; ++s) {
        ok = tma::mbar_wait(&bar->empty[stage], phase ^ 1, p.error, 805);
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issue ----------------------------------------------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(128, BN);
      int stage = 0, phase = 0, round = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < tiles && ok; i += gridDim.x, ++round) {
        const int buf = round & 1;
        // the accumulator may be written again once the epilogue has read its last tile
        if (round >= 2 && !tma::mbar_wait(&bar->acc_empty[buf], ((round >> 1) - 1) & 1, p.error, 802)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!tma::mbar_wait(&bar->full[stage], phase, p.error, 803)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint32_t a = tma::smem_u32(smem + stage * R::kStageBytes);
          const uint32_t b = a + R::kXBytes;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            tc::mma_ss(tmem + buf * BN, tc::smem_desc_k_major_sw128(a + k * 32),
                       tc::smem_desc_k_major_sw128(b + k * 32), idesc, kb > 0 || k > 0);
          tc::commit(&bar->empty[stage]);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) tc::commit(&bar->acc_full[buf]);
      }
    }
  } else {
    // ---- epilogue: thread = row, the warps of one quarter of the rows share out the columns ----
    const int quarter = warp & 3;         // (the quarter of tensor memory that a warp may read)
    constexpr int kShare = kCols / (R::kEpilogue / 128);
    static_assert(kShare % 16 == 0, "columns in pieces of 16");
    const int c0 = (warp - 2) / 4 * kShare;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    int round = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < tiles; i += gridDim.x, ++round) {
      const Tile t = tile_at(i);
      const int buf = round & 1;
      ok = ok && tma::mbar_wait(&bar->acc_full[buf], (round >> 1) & 1, p.error, 804);
      tc::fence_after_sync();
      const uint32_t acc = lane_base + buf * BN;
      const long long to = (long long)(t.row0 + row) * p.N + t.n0;
      if (quarter * 32 < t.rows) {
#pragma unroll 1
        for (int c = c0; c < c0 + kShare && ok; c += 16) {
          if (t.n0 + c >= p.N) break;
          float g[16];
          tc::ld_32x32b_x16(acc + c, g);
          if constexpr (DUAL) {
            float u[16];
            tc::ld_32x32b_x16(acc + HB + c, u);
            if (row < t.rows) {
              uint32_t w[8];
#pragma unroll
              for (int k = 0; k < 16; ++k) {
                const float gg = fminf(g[k], p.limit);
                const float uu = fminf(fmaxf(u[k], -p.limit), p.limit);
                g[k] = gg / (1.f + expf(-p.alpha * gg)) * (uu + p.plus);
              }
#pragma unroll
              for (int k = 0; k < 8; ++k) w[k] = mma::pack_bf16(g[2 * k], g[2 * k + 1]);
              uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + to + c);
              dst[0] = make_uint4(w[0], w[1], w[2], w[3]);          // (N is a multiple of 8)
              if (t.n0 + c + 8 < p.N) dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
            }
          } else if (row < t.rows) {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.out) + to + c);
            dst[0] = make_float4(g[0], g[1], g[2], g[3]);
            dst[1] = make_float4(g[4], g[5], g[6], g[7]);
            if (t.n0 + c + 8 < p.N) {
              dst[2] = make_float4(g[8], g[9], g[10], g[11]);
              dst[3] = make_float4(g[12], g[13], g[14], g[15]);
            }
          }
        }
      }
      tc::fence_before_sync();
      tma::mbar_arrive(&bar->acc_empty[buf]);       // (whatever happened)
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kTmemCols);
  }
}

__device__ int g_error;

template <int XR, int HB, bool DUAL>
int launch(const CUtensorMap& x, const CUtensorMap& w0, const CUtensorMap& w1, const Params& p,
           long long most_tiles, cudaStream_t stream) {
  auto kernel = moe_tc_kernel<XR, HB, DUAL>;
  static PerDeviceOnce configured;
  if (configured.needs()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               Ring<XR, HB>::kSmem);
    if (e != cudaSuccess) return (int)e;
    configured.done();
  }
  const int blocks = most_tiles < sm_count() ? (int)most_tiles : sm_count();
  return launch_ordered(kernel, dim3(blocks), dim3(Ring<XR, HB>::kThreads), Ring<XR, HB>::kSmem, stream, x, w0, w1, p);
}

}  // namespace

// rows: bf16 [total, K], sorted by expert: expert e's are offsets[e] .. offsets[e + 1] - 1 (int32,
// on the device, offsets[experts] <= total). w0, w1: bf16 [experts, N, K], contiguous. w1 null: out
// fp32 [total, N] = rows w0[e]^T; else out bf16 [total, N] = act(rows w0[e]^T, rows w1[e]^T). few: the
// form for few rows an expert. K and N multiples of 8, everything at multiples of 16 bytes.
SAKV_EXPORT int sakv_moe_tc(const void* rows, long long total, const void* w0, const void* w1,
                            const int32_t* offsets, int experts, void* out, int N, int K, float limit,
                            float alpha, float plus, int few, cudaStream_t stream) {
  if (total < 0 || experts <= 0 || experts > kMaxExperts || N <= 0 || K <= 0 || (N % 8) || (K % 8) ||
      total > 0x7fffffffLL || (long long)experts * N > 0x7fffffffLL ||
      (((uintptr_t)rows | (uintptr_t)w0 | (uintptr_t)w1 | (uintptr_t)out) & 15))
    return cudaErrorInvalidValue;
  if (total == 0) return 0;
  const int xr = few ? 32 : 128, hb = few ? 32 : 128;
  const int cols = w1 != nullptr ? hb : 2 * hb;
  const long long most = ((total + xr - 1) / xr + (experts < total ? experts : total)) *
                         ((N + cols - 1) / cols);
  if (most > 0x7fffffffLL) return cudaErrorInvalidValue;
  CUtensorMap x, a, b;
  int code = tma::make_map_bf16_2d(&x, rows, (uint64_t)total, (uint64_t)K, (uint64_t)K * 2, xr, BK);
  if (code == 0)
    code = tma::make_map_bf16_2d(&a, w0, (uint64_t)experts * N, (uint64_t)K, (uint64_t)K * 2, hb, BK);
  if (code == 0)
    code = tma::make_map_bf16_2d(&b, w1 != nullptr ? w1 : w0, (uint64_t)experts * N, (uint64_t)K,
                                 (uint64_t)K * 2, hb, BK);
  if (code != 0) return code;
  Params p;
  p.offsets = offsets;
  p.out = out;
  p.experts = experts;
  p.N = N;
  p.K = K;
  p.limit = limit;
  p.alpha = alpha;
  p.plus = plus;
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p.error), g_error) != cudaSuccess)
    return cudaErrorInvalidValue;
  if (few)
    return w1 != nullptr ? launch<32, 32, true>(x, a, b, p, most, stream)
                         : launch<32, 32, false>(x, a, b, p, most, stream);
  return w1 != nullptr ? launch<128, 128, true>(x, a, b, p, most, stream)
                       : launch<128, 128, false>(x, a, b, p, most, stream);
}

SAKV_EXPORT int sakv_moe_tc_error(int* value) {
  return static_cast<int>(cudaMemcpyFromSymbol(value, g_error, sizeof(int)));
}
