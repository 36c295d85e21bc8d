// Causal attention over the cache in bfloat16 on the tensor cores, for the sizes the designs
// use: keys of 64 or 128 columns with values of 64, 128 or 256, and one shared latent row of 576
// columns whose first 512 are the values. The scores and options are those of
// `csrc/attention_distance.cu` (logarithmic or linear distance penalty, soft cap, window with kept
// first tokens, chunks, sinks, gates, two maps a head), which takes every other size and type.
//
// Precision: queries, keys and values are bfloat16 and their products exact in fp32; scores,
// softmax weights, running maxima and sums are fp32, worked out with the functions of the general
// kernel (expf, log1pf). A weight enters the second product as the sum of three bfloat16 numbers,
// which hold all 24 of its bits, so every value tile is multiplied three times.
//
// A block takes the rows of one key/value head: ROWS = 16 WR rows are tokens x query heads of the
// group (x maps in a prompt, decoded tokens: of one map), so a group's heads share each tile of keys. WR warps go along the rows and WC
// along the keys of a tile for the scores and along the values' columns for the weighted sum:
//   * prompts, 128 columns: WR 4, WC 1 (weights stay in registers); tiles of 64 keys, two blocks
//     an SM.
//   * prompts, two maps a head: the same with tiles of 32 keys; half of the warps take one map, half the
//     other, and the block combines them (as blocks of one map each through fp32 sums in device memory,
//     values of 256 columns: 2 KB a token and head, and 109 us instead of 77 for 16 prompts of 17 to
//     500 tokens with 4 heads, 313 instead of 296 for one of 3,001).
//   * prompts, latent rows: WR 4, WC 2, tiles of 32 keys: 64 rows x 512 columns of fp32 sums are
//     128 registers a thread of 256, and the queries and three tiles fill the shared memory.
//   * decoded tokens: WR 1, WC 8 and `key_splits` blocks a token; what bounds them is the trip to
//     memory, so a whole tile of 64 keys is asked for at once by 256 threads.
// Tiles lie at multiples of their size in the sequence and a row that sees nothing of a tile is
// left exactly as it was, so in a prompt a token's result does not depend on which tokens came with
// it, as long as all values are finite (a block that meets one that is not walks its rows' keys one
// by one). A decoded token's keys are split by rules that count the step's tokens.
//
// The products run on mma.sync. Over latent rows the sums of 128 rows x 512 columns would fill the whole
// of tensor memory and the weights' pieces would pass through it three times. At 128 / 128 columns a
// form on tcgen05 (as `csrc/attention_prefill_tc.cu`) is possible and not built: 3,001 tokens of 8 heads
// of 2 take 245 us, 0.075 PFLOP/s of useful work, 0.15 with three products of P V to one of Q K^T.
#include <float.h>

#include "common.cuh"
#include "mma.cuh"

struct MmaAttention {
  const __nv_bfloat16* q;      // row t: + t * q_stride, virtual head h: + h * q_head_stride
  long long q_stride;
  int q_head_stride;
  const __nv_bfloat16* q2;     // columns from q_split on (null: none)
  long long q2_stride;
  int q2_head_stride, q_split;
  const __nv_bfloat16* k_cache;
  const __nv_bfloat16* v_cache;      // null: the values are the first columns of the key rows
  int k_row, v_row;
  const int32_t* positions;
  const int32_t* token_seq;
  const int32_t* cu_seqlens;   // prompts: where each of `sequences` begins among the tokens, or null
  int sequences;
  const int32_t* block_table;
  int max_blocks, tokens, heads, kv_heads, maps;      // heads: query heads (each of `maps` maps)
  float scale;
  int window, chunk, keep;
  const float* slope;          // logarithmic penalty, with `rate`
  const float* rate;
  float softcap;
  const float* linear;
  int key_splits;
  // the outputs: directly, or (decoded: two maps or several splits) through `sums` and a second kernel
  __nv_bfloat16* out;          // [tokens, heads * DV]
  float* sums;                 // [key_splits, tokens, heads * maps, DV], not yet divided
  float* stats;                // [key_splits, tokens, heads * maps, 2]: maximum, sum
  const float* sink;
  const __nv_bfloat16* gate;   // a gate a head: + t * gate_stride + h (null: none)
  long long gate_stride;
  const float* elem_gate;      // fp32, + t * elem_stride + h * DV + c (null: none)
  long long elem_stride;
  const __nv_bfloat16* map_gate;   // two maps: + t * map_gate_stride + h * DV + c (null: none)
  long long map_gate_stride;
  float out_scale, lambda, eps;
  int ordered;                 // in plain stream order: see `launch_shape`
  // the split of the work
  int heads_per_tile, tokens_per_tile, head_tiles;
  int windows_shared;          // grid z are the runs of a window of tokens instead of splits
};

namespace {

__device__ __forceinline__ int first_visible(int pos, int window, int chunk) {
  if (chunk > 0) return pos - pos % chunk;
  return (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
}

// 16 bytes into shared memory; zeros without reading where `real` is false
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool real) {
  const int n = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= FLT_MAX; }

// A score from a product: scale, soft cap (as the general kernel takes it of 16-bit keys), penalty.
__device__ __forceinline__ float score_of(const MmaAttention& a, float s, float dist, float sl, float rt) {
  s *= a.scale;
  if (a.softcap > 0.f)       // cap * tanh(s / cap) as cap * (1 - 2 / (e^(2z) + 1))
    s = a.softcap * (1.f - __fdividef(2.f, __expf(2.f * __fdividef(s, a.softcap)) + 1.f));
  if (a.slope != nullptr) s -= sl * log1pf(rt * dist);
  else if (a.linear != nullptr) s = fmaf(-sl, dist, s);
  return s;
}

// What a row's sums become in the output: one warp a row, columns dealt to the lanes by fours.
template <int DV>
__device__ __forceinline__ void write_row(const MmaAttention& a, const float* acc, float m, float l,
                                          int t, int h, int lane) {
  float corr = 1.f;
  if (a.sink != nullptr) {       // one more logit in the denominator
    const float s = a.sink[h];
    const float top = fmaxf(m, s);
    corr = expf(m - top);
    l = fmaf(l, corr, expf(s - top));
  }
  float f = a.out_scale * corr / l;
  if (a.gate != nullptr)
    f *= 1.f / (1.f + expf(-widen(a.gate[(long long)t * a.gate_stride + h])));
  const float* eg = a.elem_gate == nullptr ? nullptr
                                           : a.elem_gate + (long long)t * a.elem_stride + (long long)h * DV;
  __nv_bfloat16* o = a.out + ((long long)t * a.heads + h) * DV;
  for (int c = lane * 4; c < DV; c += 128) {
    const float4 v = *reinterpret_cast<const float4*>(acc + c);
    float r[4] = {v.x * f, v.y * f, v.z * f, v.w * f};
    if (eg != nullptr) {
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] /= 1.f + expf(-eg[c + i]);
    }
    *reinterpret_cast<uint2*>(o + c) = make_uint2(mma::pack_bf16(r[0], r[1]), mma::pack_bf16(r[2], r[3]));
  }
}

// The same of a head's two maps: a1 - lambda a2 over its root mean square.
template <int DV>
__device__ __forceinline__ void write_pair(const MmaAttention& a, const float* acc1, const float* acc2,
                                           float2 m, float2 l, int t, int h, int lane) {
  constexpr int N = DV / 128;
  float2 corr = make_float2(1.f, 1.f);
  if (a.sink != nullptr) {
    const float s = a.sink[h];
    const float2 top = make_float2(fmaxf(m.x, s), fmaxf(m.y, s));
    corr = make_float2(expf(m.x - top.x), expf(m.y - top.y));
    l = make_float2(fmaf(l.x, corr.x, expf(s - top.x)), fmaf(l.y, corr.y, expf(s - top.y)));
  }
  const float f1 = corr.x / l.x, f2 = a.lambda * corr.y / l.y;
  float o[N][4], ss = 0.f;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const float4 x = *reinterpret_cast<const float4*>(acc1 + n * 128 + lane * 4);
    const float4 y = *reinterpret_cast<const float4*>(acc2 + n * 128 + lane * 4);
    o[n][0] = x.x * f1 - y.x * f2;
    o[n][1] = x.y * f1 - y.y * f2;
    o[n][2] = x.z * f1 - y.z * f2;
    o[n][3] = x.w * f1 - y.w * f2;
#pragma unroll
    for (int i = 0; i < 4; ++i) ss = fmaf(o[n][i], o[n][i], ss);
  }
  const float r = rsqrtf(warp_sum(ss) / (float)DV + a.eps) * a.out_scale;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int c = n * 128 + lane * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      o[n][i] *= r;
      if (a.map_gate != nullptr)
        o[n][i] *= 1.f / (1.f + expf(-widen(a.map_gate[(long long)t * a.map_gate_stride +
                                                      (long long)h * DV + c + i])));
    }
    *reinterpret_cast<uint2*>(a.out + ((long long)t * a.heads + h) * DV + c) =
        make_uint2(mma::pack_bf16(o[n][0], o[n][1]), mma::pack_bf16(o[n][2], o[n][3]));
  }
}

template <int DK, int DV, bool VINK, int WR, int WC, int KT, int STAGES, int MAPS>
struct Shape {
  static constexpr int kRows = 16 * WR, kThreads = 32 * WR * WC;
  static constexpr int kPairs = kRows / MAPS;       // (token, query head)s of a block
  static constexpr int kQStride = DK + 8, kKStride = MAPS * DK + 8;            // (elements; odd
  static constexpr int kVStride = VINK ? kKStride : DV + 8;                     //  times 16 bytes)
  static constexpr int kOStride = DV + 8, kPStride = KT + 8;
  static constexpr int kQBytes = kRows * kQStride * 2;
  static constexpr int kKBytes = KT * kKStride * 2;
  static constexpr int kStageBytes = kKBytes + (VINK ? 0 : KT * kVStride * 2);
  static constexpr int kPBytes = WC > 1 ? 3 * kRows * kPStride * 2 : 0;   // (a weight's three pieces)
  static constexpr int kSmall = (2 * WC + 2) * kRows * 4;        // maxima, sums, a row's m and l
  static constexpr int kMain = kQBytes + STAGES * kStageBytes + kPBytes;
  static constexpr int kOut = kRows * kOStride * 4;
  static constexpr int kBytes = (kMain > kOut ? kMain : kOut) + kSmall;
};

template <int DK, int DV, bool VINK, int WR, int WC, int KT, int STAGES, int MAPS>
__global__ void __launch_bounds__(32 * WR * WC)
attention_mma_kernel(const MmaAttention a) {
  using S = Shape<DK, DV, VINK, WR, WC, KT, STAGES, MAPS>;
  constexpr int NT = KT / WC / 8;            // tiles of 8 keys a warp scores
  constexpr int NV = DV / WC / 8;            // tiles of 8 value columns a warp sums
  constexpr int KS = DK / 16;
  static_assert(KT % (8 * WC) == 0 && DV % (16 * WC) == 0 && kCacheBlock % KT == 0, "");
  static_assert(WC > 1 || (KT % 16 == 0), "");
  static_assert(NT == 1 || NT % 2 == 0, "");
  static_assert(MAPS == 1 || (!VINK && S::kPairs % 16 == 0 && DV % 128 == 0), "a warp's rows are of one map");
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(smem);
  float* small = reinterpret_cast<float*>(smem + S::kBytes - S::kSmall);
  float* row_max = small;                    // [WC][rows]
  float* row_sum = small + WC * S::kRows;    // [WC][rows]
  float* row_m = small + 2 * WC * S::kRows;  // [rows]
  float* row_l = row_m + S::kRows;           // [rows]
  float* os = reinterpret_cast<float*>(smem);
  const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const uint32_t stage0 = base + S::kQBytes;
  const uint32_t p_base = stage0 + STAGES * S::kStageBytes;

  if (a.sums != nullptr && !a.ordered) let_next_kernel_start();   // (the fold waits for this kernel's end)
  wait_for_previous_kernel();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wr = warp / WC, wc = warp % WC;
  // The block's tokens. The longest rows of a prompt (its last tokens) start first.
  const int tile_at = (int)(gridDim.x - 1 - blockIdx.x);
  int t0 = tile_at * a.tokens_per_tile, t_end = min(t0 + a.tokens_per_tile, a.tokens);
  if (a.cu_seqlens != nullptr) {
    // tiles end where a sequence does: the sequence whose tiles hold this one
    t0 = -1;
    for (int b0 = 0, base = 0; b0 < a.sequences && t0 < 0; b0 += 32) {
      const int b = b0 + lane;
      const int begin = b < a.sequences ? a.cu_seqlens[b] : 0;
      const int end = b < a.sequences ? min(a.cu_seqlens[b + 1], a.tokens) : 0;
      const int mine = (end - begin + a.tokens_per_tile - 1) / a.tokens_per_tile;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      const int at = tile_at - (base + sum - mine);
      const unsigned here = __ballot_sync(0xffffffffu, at >= 0 && at < mine);
      if (here != 0) {
        const int from = __ffs(here) - 1;
        t0 = __shfl_sync(0xffffffffu, begin + at * a.tokens_per_tile, from);
        t_end = min(t0 + a.tokens_per_tile, __shfl_sync(0xffffffffu, end, from));
      }
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (t0 < 0) return;                      // (the grid has room for every cut into sequences)
  } else if (a.windows_shared) {
    // sequences not told: the block takes the z-th run of the window's tokens
    int run = -1, s1 = t0;
    for (; s1 < t_end && run < (int)blockIdx.z; ++run) {
      t0 = s1++;
      while (s1 < t_end && a.token_seq[s1] == a.token_seq[t0] &&
             a.positions[s1] == a.positions[s1 - 1] + 1) ++s1;
    }
    if (run != (int)blockIdx.z) return;
    t_end = s1;
  }
  const int hg = a.heads / a.kv_heads, hp = a.heads_per_tile;
  int y = blockIdx.y;
  const int head_tile = y % a.head_tiles;
  y /= a.head_tiles;
  // (MAPS 1: all rows are of one map; else rows from `kPairs` on are of the second)
  const int map0 = MAPS == 1 ? y % a.maps : 0, g = MAPS == 1 ? y / a.maps : y;
  const int h_base = g * hg + head_tile * hp;
  const int h_count = min(hp, hg - head_tile * hp);
  const int used = (t_end - t0) * hp;        // pairs beyond it belong to nobody

  // the queries
  constexpr int kPieces = DK / 8;
  for (int i = threadIdx.x; i < S::kRows * kPieces; i += S::kThreads) {
    const int r = i / kPieces, e = (i - r * kPieces) * 8;
    const int pair = r % S::kPairs;
    const int t = t0 + pair / hp, h = (h_base + pair % hp) * a.maps + map0 + r / S::kPairs;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (pair < used && pair % hp < h_count) {
      const __nv_bfloat16* src =
          e < a.q_split ? a.q + (long long)t * a.q_stride + (long long)h * a.q_head_stride + e
                        : a.q2 + (long long)t * a.q2_stride + (long long)h * a.q2_head_stride +
                              (e - a.q_split);
      v = *reinterpret_cast<const uint4*>(src);
    }
    *reinterpret_cast<uint4*>(qs + r * S::kQStride + e) = v;
  }

  // this thread's two rows
  int rt[2], rpos[2], rfirst[2];
  float rsl[2] = {0.f, 0.f}, rrt[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = (wr * 16 + (lane >> 2) + 8 * i) % S::kPairs;
    rt[i] = r < used && r % hp < h_count ? t0 + r / hp : -1;
    rpos[i] = rt[i] >= 0 ? a.positions[rt[i]] : -1;
    rfirst[i] = rt[i] >= 0 ? first_visible(rpos[i], a.window, a.chunk) : 0;
    if (rt[i] >= 0) {
      const int h = h_base + r % hp;
      if (a.slope != nullptr) {
        rsl[i] = a.slope[h];
        rrt[i] = a.rate[h];
      } else if (a.linear != nullptr) {
        rsl[i] = a.linear[h];
      }
    }
  }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float acc[NV][4];
#pragma unroll
  for (int n = 0; n < NV; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;

  const int split = a.windows_shared ? 0 : blockIdx.z;
  // The tile's tokens in runs of one sequence and consecutive positions (one run for what the engine
  // issues); rows outside the run see none of its keys.
  for (int s0 = t0; s0 < t_end;) {
    const int seq = a.token_seq[s0], p0 = a.positions[s0];
    // (its end: 32 tokens at a time; one by one they were 7.7 us of the 22.5 of a prompt of 64 tokens
    // with a head a key/value head)
    int s1 = t_end;
    for (int i0 = s0 + 1; i0 < t_end; i0 += 32) {
      const int i = i0 + lane;
      const unsigned ends = __ballot_sync(
          0xffffffffu, i < t_end && (a.token_seq[i] != seq || a.positions[i] != p0 + (i - s0)));
      if (ends != 0) {
        s1 = i0 + __ffs(ends) - 1;
        break;
      }
    }
    const int last = p0 + (s1 - s0) - 1;
    const int low = first_visible(p0, a.window, a.chunk);
    const int low_last = first_visible(last, a.window, a.chunk);
    const bool whole = s0 == t0 && s1 == t_end;
    const int32_t* table = a.block_table + (long long)seq * a.max_blocks;
    // tiles: those of the kept first tokens that lie before the first visible one's, then on
    const int from = low / KT;
    const int kept_all = (a.keep + KT - 1) / KT;
    const int kept = kept_all < from ? kept_all : from;
    const int count = kept + last / KT - from + 1;
    const int share = (count + a.key_splits - 1) / a.key_splits;
    const int lo = split * share, hi = min(count, lo + share);

    auto fetch = [&](int i) {
      const int tile = i < kept ? i : from + i - kept;
      const int j0 = tile * KT;
      const long long row0 = ((long long)table[j0 / kCacheBlock] * a.kv_heads + g) * kCacheBlock +
                             j0 % kCacheBlock;
      const uint32_t ks = stage0 + (i % STAGES) * S::kStageBytes;
      const __nv_bfloat16* kp = a.k_cache + row0 * a.k_row + map0 * DK;
      constexpr int kp16 = MAPS * DK / 8;
      for (int x = threadIdx.x; x < KT * kp16; x += S::kThreads) {
        const int r = x / kp16, e = (x - r * kp16) * 8;
        copy16(ks + (r * S::kKStride + e) * 2, kp + (long long)r * a.k_row + e, j0 + r <= last);
      }
      if constexpr (!VINK) {
        const __nv_bfloat16* vp = a.v_cache + row0 * a.v_row;
        constexpr int vp16 = DV / 8;
        for (int x = threadIdx.x; x < KT * vp16; x += S::kThreads) {
          const int r = x / vp16, e = (x - r * vp16) * 8;
          copy16(ks + S::kKBytes + (r * S::kVStride + e) * 2, vp + (long long)r * a.v_row + e,
                 j0 + r <= last);
        }
      }
    };

    __syncthreads();                 // (queries are there; the run before this one is done)
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) {
      if (lo + i < hi) fetch(lo + i);
      copies_commit();
    }
    for (int i = lo; i < hi; ++i) {
      copies_wait<STAGES - 2>();
      __syncthreads();               // tile i is there, and everybody has left tile i - 1
      if (i + STAGES - 1 < hi) fetch(i + STAGES - 1);
      copies_commit();
      const int tile = i < kept ? i : from + i - kept;
      const int j0 = tile * KT;
      const uint32_t ks = stage0 + (i % STAGES) * S::kStageBytes;
      const uint32_t vs = VINK ? ks : ks + S::kKBytes;

      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
      const uint32_t q_at = base + ((wr * 16 + (lane & 15)) * S::kQStride + (lane >> 4) * 8) * 2;
      if constexpr (NT == 1) {
        const uint32_t k_at =
            ks + ((wc * 8 + (lane & 7)) * S::kKStride + (lane >> 3) * 8) * 2;
#pragma unroll 4
        for (int kk = 0; kk < KS; kk += 2) {
          uint32_t b[4], q0[4], q1[4];
          mma::ldmatrix_x4(k_at + kk * 32, b[0], b[1], b[2], b[3]);
          mma::ldmatrix_x4(q_at + kk * 32, q0[0], q0[1], q0[2], q0[3]);
          mma::ldmatrix_x4(q_at + kk * 32 + 32, q1[0], q1[1], q1[2], q1[3]);
          mma::bf16_16816(s[0], q0, b[0], b[1]);
          mma::bf16_16816(s[0], q1, b[2], b[3]);
        }
      } else {
        const uint32_t k_at = ks + ((wc * NT * 8 + (lane & 7) + (lane >> 4) * 8) * S::kKStride +
                                    wr * 16 / S::kPairs * DK + ((lane >> 3) & 1) * 8) * 2;
#pragma unroll(KS <= 8 ? KS : 4)
        for (int kk = 0; kk < KS; ++kk) {
          uint32_t q[4];
          mma::ldmatrix_x4(q_at + kk * 32, q[0], q[1], q[2], q[3]);
#pragma unroll
          for (int n = 0; n < NT; n += 2) {
            uint32_t b[4];
            mma::ldmatrix_x4(k_at + (n * 8 * S::kKStride) * 2 + kk * 32, b[0], b[1], b[2], b[3]);
            mma::bf16_16816(s[n], q, b[0], b[1]);
            mma::bf16_16816(s[n + 1], q, b[2], b[3]);
          }
        }
      }

      // scores, masks, the tile's maxima
      const bool all_seen = whole && j0 + KT - 1 <= p0 && (j0 >= low_last || j0 + KT <= a.keep);
      float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = e >> 1;
          const int j = j0 + (wc * NT + n) * 8 + (lane & 3) * 2 + (e & 1);
          float v = score_of(a, s[n][e], (float)(rpos[r] - j), rsl[r], rrt[r]);
          if (!all_seen)
            v = rt[r] >= s0 && rt[r] < s1 && j <= rpos[r] && (j >= rfirst[r] || j < a.keep)
                    ? v : -INFINITY;
          s[n][e] = v;
          top[r] = fmaxf(top[r], v);
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
      }
      const int my_row = wr * 16 + (lane >> 2);
      if constexpr (WC > 1) {        // over the warps of these rows
        if ((lane & 3) == 0) {
          row_max[wc * S::kRows + my_row] = top[0];
          row_max[wc * S::kRows + my_row + 8] = top[1];
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + wr), "n"(32 * WC) : "memory");
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int w = 0; w < WC; ++w)
            top[r] = fmaxf(top[r], row_max[w * S::kRows + my_row + 8 * r]);
      }
      float corr[2], shift[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float next = fmaxf(m[r], top[r]);
        shift[r] = next == -INFINITY ? 0.f : next;     // (nothing seen yet: weights of 0)
        corr[r] = expf(m[r] - shift[r]);
        m[r] = next;
        l[r] *= corr[r];
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float p = expf(s[n][e] - shift[e >> 1]);
          s[n][e] = p;
          l[e >> 1] += p;
        }
      if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          mma::mul2(acc[n][0], acc[n][1], corr[0]);
          mma::mul2(acc[n][2], acc[n][3], corr[1]);
        }
      }

      // the weights as sums of three pieces (what a piece leaves of a number is exact), times the
      // values
      auto pieces = [](float x, float y, uint32_t& first, uint32_t& second, uint32_t& third) {
        auto take = [&] {
          uint32_t two = mma::pack_bf16(x, y);
          const float2 back = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&two));
          x -= back.x;
          y -= back.y;
          return two;
        };
        first = take();
        second = take();
        third = mma::pack_bf16(x, y);
      };
      constexpr int kPiece = S::kRows * S::kPStride;        // (elements between two pieces)
      if constexpr (WC > 1) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int at = (my_row + 8 * r) * S::kPStride + (wc * NT + n) * 8 + (lane & 3) * 2;
            uint32_t* ps = reinterpret_cast<uint32_t*>(smem + S::kQBytes + STAGES * S::kStageBytes);
            pieces(s[n][2 * r], s[n][2 * r + 1], ps[at / 2], ps[(kPiece + at) / 2],
                   ps[(2 * kPiece + at) / 2]);
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + wr), "n"(32 * WC) : "memory");
      }
      const uint32_t v_at = vs + (((lane & 7) + ((lane >> 3) & 1) * 8) * S::kVStride +
                                  wc * NV * 8 + (lane >> 4) * 8) * 2;
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk) {
        uint32_t p[3][4];
        if constexpr (WC > 1) {
          const uint32_t at =
              p_base + ((wr * 16 + (lane & 15)) * S::kPStride + kk * 16 + (lane >> 4) * 8) * 2;
#pragma unroll
          for (int i = 0; i < 3; ++i)
            mma::ldmatrix_x4(at + i * kPiece * 2, p[i][0], p[i][1], p[i][2], p[i][3]);
        } else {
          constexpr int kLast = NT > 1 ? NT - 1 : 0;
          const int n0 = 2 * kk, n1 = 2 * kk + 1 <= kLast ? 2 * kk + 1 : kLast;
          pieces(s[n0][0], s[n0][1], p[0][0], p[1][0], p[2][0]);
          pieces(s[n0][2], s[n0][3], p[0][1], p[1][1], p[2][1]);
          pieces(s[n1][0], s[n1][1], p[0][2], p[1][2], p[2][2]);
          pieces(s[n1][2], s[n1][3], p[0][3], p[1][3], p[2][3]);
        }
#pragma unroll
        for (int n = 0; n < NV; n += 2) {
          uint32_t b[4];
          mma::ldmatrix_x4_trans(v_at + (kk * 16 * S::kVStride + n * 8) * 2, b[0], b[1], b[2], b[3]);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            mma::bf16_16816(acc[n], p[i], b[0], b[1]);
            mma::bf16_16816(acc[n + 1], p[i], b[2], b[3]);
          }
        }
      }
    }
    copies_wait<0>();
    s0 = s1;
  }

  // the rows' sums and maxima, and their sums of values, into shared memory
  bool bad = false;
#pragma unroll
  for (int n = 0; n < NV; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) bad |= rt[e >> 1] >= 0 && !finite(acc[n][e]);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
  }
  const int any_bad = __syncthreads_or(bad);           // (and everybody has left the tiles)
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = wr * 16 + (lane >> 2) + 8 * r;
    if ((lane & 3) == 0) {
      row_sum[wc * S::kRows + row] = l[r];
      if (wc == 0) row_m[row] = m[r];
    }
#pragma unroll
    for (int n = 0; n < NV; ++n)
      *reinterpret_cast<float2*>(os + row * S::kOStride + (wc * NV + n) * 8 + (lane & 3) * 2) =
          make_float2(acc[n][2 * r], acc[n][2 * r + 1]);
  }
  __syncthreads();
  for (int row = threadIdx.x; row < S::kRows; row += S::kThreads) {
    float sum = row_sum[row];
    for (int w = 1; w < WC; ++w) sum += row_sum[w * S::kRows + row];
    row_l[row] = sum;
  }
  __syncthreads();
  // An infinity or a NaN among the values: a weight of 0 times it spoils rows that do not see it, and a
  // weight's pieces times it are not the weight times it. A warp of such a block walks a row's
  // keys one by one.
  auto walk = [&](int row, int t, int h) {
    float* acc_row = os + row * S::kOStride;
    const int pos = a.positions[t], first = first_visible(pos, a.window, a.chunk);
    const int32_t* table = a.block_table + (long long)a.token_seq[t] * a.max_blocks;
    // the same share of the run's tiles as above
    int s0 = t, s1 = t + 1;
    while (s0 > t0 && a.token_seq[s0 - 1] == a.token_seq[t] &&
           a.positions[s0 - 1] == a.positions[s0] - 1) --s0;
    while (s1 < t_end && a.token_seq[s1] == a.token_seq[t] &&
           a.positions[s1] == a.positions[s1 - 1] + 1) ++s1;
    const int last = a.positions[s1 - 1];
    const int from = first_visible(a.positions[s0], a.window, a.chunk) / KT;
    const int kept_all = (a.keep + KT - 1) / KT;
    const int kept = kept_all < from ? kept_all : from;
    const int count = kept + last / KT - from + 1;
    const int share = (count + a.key_splits - 1) / a.key_splits;
    const int lo = split * share, hi = min(count, lo + share);
    const int map = map0 + row / S::kPairs, vh = h * a.maps + map;
    const float sl = a.slope ? a.slope[h] : a.linear ? a.linear[h] : 0.f;
    const float rate = a.slope ? a.rate[h] : 0.f;
    float top = -INFINITY, sum = 0.f;
    for (int c = lane; c < DV; c += 32) acc_row[c] = 0.f;
    for (int i = lo; i < hi; ++i) {
      const int tile = i < kept ? i : from + i - kept;
      for (int j = tile * KT; j < tile * KT + KT; ++j) {
        if (j > pos || (j < first && j >= a.keep)) continue;
        const long long at = ((long long)table[j / kCacheBlock] * a.kv_heads + g) * kCacheBlock +
                             j % kCacheBlock;
        float part = 0.f;
        for (int e = lane; e < DK; e += 32) {
          const __nv_bfloat16 qv =
              e < a.q_split
                  ? a.q[(long long)t * a.q_stride + (long long)vh * a.q_head_stride + e]
                  : a.q2[(long long)t * a.q2_stride + (long long)vh * a.q2_head_stride + e - a.q_split];
          part = fmaf(widen(qv), widen(a.k_cache[at * a.k_row + map * DK + e]), part);
        }
        const float sc = score_of(a, warp_sum(part), (float)(pos - j), sl, rate);
        const float next = fmaxf(top, sc);
        const float shift = next == -INFINITY ? 0.f : next;      // (as above)
        const float f = expf(top - shift), p = expf(sc - shift);
        sum = fmaf(sum, f, p);
        const __nv_bfloat16* vr = VINK ? a.k_cache + at * a.k_row : a.v_cache + at * a.v_row;
        for (int c = lane; c < DV; c += 32) acc_row[c] = fmaf(acc_row[c], f, p * widen(vr[c]));
        top = next;
      }
    }
    __syncwarp();
    if (lane == 0) {
      row_m[row] = top;
      row_l[row] = sum;
    }
    __syncwarp();
  };
  for (int pair = warp; pair < used; pair += WR * WC) {
    if (pair % hp >= h_count) continue;
    const int t = t0 + pair / hp, h = h_base + pair % hp;
    if (any_bad)
      for (int m = 0; m < MAPS; ++m) walk(pair + m * S::kPairs, t, h);
    const float* acc_row = os + pair * S::kOStride;
    const float mm = row_m[pair], ll = row_l[pair];
    if constexpr (MAPS == 2) {
      constexpr int o = S::kPairs;
      write_pair<DV>(a, acc_row, acc_row + o * S::kOStride, make_float2(mm, row_m[pair + o]),
                     make_float2(ll, row_l[pair + o]), t, h, lane);
      continue;
    }
    if (a.sums == nullptr) {
      write_row<DV>(a, acc_row, mm, ll, t, h, lane);
      continue;
    }
    const long long part = ((long long)split * a.tokens + t) * a.heads * a.maps + h * a.maps + map0;
    for (int c = lane * 4; c < DV; c += 128)
      *reinterpret_cast<float4*>(a.sums + part * DV + c) = *reinterpret_cast<const float4*>(acc_row + c);
    if (lane == 0) *reinterpret_cast<float2*>(a.stats + part * 2) = make_float2(mm, ll);
  }
}

// Splits of a token's keys and maps of a head brought together: one block a token and head, a
// thread for four columns. A few hundred kilobytes of fresh sums in the L2: its time is its trip
// there (all splits asked for before the first is used) and the launch.
template <int DV>
__global__ void __launch_bounds__(DV / 4) attention_fold_kernel(const MmaAttention a) {
  wait_for_previous_kernel();
  const int t = blockIdx.x, h = blockIdx.y, c = threadIdx.x * 4;
  const long long vheads = (long long)a.heads * a.maps;
  float o[2][4];
#pragma unroll
  for (int map = 0; map < 2; ++map) {
    if (map >= a.maps) continue;
    const long long at = (long long)t * vheads + h * a.maps + map, step = a.tokens * vheads;
    float top = -INFINITY;
    for (int s = 0; s < a.key_splits; ++s) top = fmaxf(top, a.stats[(at + s * step) * 2]);
    if (a.sink != nullptr) top = fmaxf(top, a.sink[h]);
    float total = a.sink != nullptr ? expf(a.sink[h] - top) : 0.f;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int s = 0; s < a.key_splits; ++s) {
      const float2 ml = *reinterpret_cast<const float2*>(a.stats + (at + s * step) * 2);
      const float4 v = *reinterpret_cast<const float4*>(a.sums + (at + s * step) * DV + c);
      const float f = ml.x == -INFINITY ? 0.f : expf(ml.x - top);      // (a split without keys)
      total = fmaf(ml.y, f, total);
      sum[0] = fmaf(v.x, f, sum[0]);
      sum[1] = fmaf(v.y, f, sum[1]);
      sum[2] = fmaf(v.z, f, sum[2]);
      sum[3] = fmaf(v.w, f, sum[3]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) o[map][i] = sum[i] / total;
  }
  float r[4];
  if (a.maps == 2) {         // a1 - lambda a2, over its root mean square
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = o[0][i] - a.lambda * o[1][i];
      ss = fmaf(r[i], r[i], ss);
    }
    __shared__ float scratch[33];
    const float f = rsqrtf(block_sum(ss, scratch) / (float)DV + a.eps) * a.out_scale;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] *= f;
      if (a.map_gate != nullptr)
        r[i] *= 1.f / (1.f + expf(-widen(a.map_gate[(long long)t * a.map_gate_stride +
                                                   (long long)h * DV + c + i])));
    }
  } else {
    float f = a.out_scale;
    if (a.gate != nullptr)
      f *= 1.f / (1.f + expf(-widen(a.gate[(long long)t * a.gate_stride + h])));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = o[0][i] * f;
      if (a.elem_gate != nullptr)
        r[i] /= 1.f + expf(-a.elem_gate[(long long)t * a.elem_stride + (long long)h * DV + c + i]);
    }
  }
  *reinterpret_cast<uint2*>(a.out + ((long long)t * a.heads + h) * DV + c) =
      make_uint2(mma::pack_bf16(r[0], r[1]), mma::pack_bf16(r[2], r[3]));
}

template <int DK, int DV, bool VINK, int WR, int WC, int KT, int STAGES, int MAPS>
int launch_shape(MmaAttention& a, bool decode, cudaStream_t stream) {
  using S = Shape<DK, DV, VINK, WR, WC, KT, STAGES, MAPS>;
  static_assert(S::kBytes <= 227 * 1024, "shared memory of a block");
  auto kernel = attention_mma_kernel<DK, DV, VINK, WR, WC, KT, STAGES, MAPS>;
  static PerDeviceOnce configured;
  if (configured.needs()) {
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes);
    if (e != cudaSuccess) return (int)e;
    configured.done();
  }
  const int hg = a.heads / a.kv_heads;
  a.heads_per_tile = hg < S::kPairs ? hg : S::kPairs;
  a.head_tiles = (hg + a.heads_per_tile - 1) / a.heads_per_tile;
  a.tokens_per_tile = decode ? 1 : S::kPairs / a.heads_per_tile;
  // A tile of rows walks the keys of one sequence: a step's decoded tokens beside a prompt get blocks
  // of their own, where one tile would walk the keys of all of them in turn (one prompt of 512 tokens
  // beside 15 sequences of 2,000 keys, us a layer, general kernel / walked in turn / now: 128 columns, 8
  // heads of 2 key/value heads 1,228 / 2,161 / 144; two maps of 128 with 256 values, 4 of 2 heads 2,075 / 2,380 /
  // 146; latent rows, 16 heads 2,174 / 1,114 / 271). With `cu_seqlens` the tiles are counted sequence by
  // sequence on the device, so the grid has one more a sequence than the tokens alone need; without it
  // a window of consecutive tokens has as many blocks as it can have runs, most of which find none
  // and leave.
  long long tiles = (a.tokens + a.tokens_per_tile - 1) / a.tokens_per_tile;
  if (decode || a.sequences == 1) a.cu_seqlens = nullptr;
  if (a.cu_seqlens != nullptr) tiles = a.tokens / a.tokens_per_tile + (long long)a.sequences;
  a.windows_shared = !decode && a.sequences != 1 && a.cu_seqlens == nullptr;
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  const long long across = (long long)a.kv_heads * (MAPS == 1 ? a.maps : 1) * a.head_tiles;
  if (across > 65535) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)tiles, (unsigned)across,
                  a.windows_shared ? (unsigned)a.tokens_per_tile : (unsigned)a.key_splits),
      block(S::kThreads);
  const dim3 fold_grid((unsigned)a.tokens, (unsigned)a.heads), fold_block(DV / 4);
  // `ordered`: this attention stands between a library's products and kernels that read fresh
  // indices. An overlapped launch of the kernels there has once ended in a memory fault whose cause
  // is not known, so both kernels begin when the one before them has ended and neither lets its
  // successor start early.
  if (a.ordered) {
    const int code = launch_ordered(kernel, grid, block, S::kBytes, stream, a);
    if (code != 0 || a.sums == nullptr) return code;
    return launch_ordered(attention_fold_kernel<DV>, fold_grid, fold_block, 0, stream, a);
  }
  const int code = launch_overlapped(kernel, grid, block, S::kBytes, stream, 1, a);
  if (code != 0 || a.sums == nullptr) return code;
  return launch_overlapped(attention_fold_kernel<DV>, fold_grid, fold_block, 0, stream, 1, a);
}

}  // namespace

// Everything as in `sakv_cached_attention` (`csrc/attention_distance.cu`) with bfloat16 operands,
// plus slope and rate of the logarithmic penalty; gate: the pre-activations of a gate a head, map_gate:
// of two maps' gate element by element (first head's first column; rows *_stride apart). cu_seqlens
// (int32 [sequences + 1], or null: not known): which tokens each of `sequences` brings. decode 0:
// blocks of 64 rows of a prompt; 1: a block a token, key/value head, map and split. sums, stats: fp32
// scratch of key_splits * tokens * heads * maps * (vdim, 2) numbers, needed for decoded tokens with
// two maps or several splits, else null. ordered 1: both kernels in plain stream order. Refused (the
// caller's rule sends them elsewhere): other widths than (dim, vdim) = (64, 64), (128, 128), (128, 256)
// and, with v_cache null, (576, 512); rows that do not begin at multiples of 16 bytes.
SAKV_EXPORT int sakv_attention_mma(
    const void* q, long long q_stride, int q_head_stride, const void* q2, long long q2_stride,
    int q2_head_stride, int q_split, void* out, const void* k_cache, int k_row, const void* v_cache,
    int v_row, const int32_t* positions, const int32_t* token_seq, const int32_t* cu_seqlens,
    int sequences, const int32_t* block_table, int max_blocks, int tokens, int heads, int kv_heads,
    int maps, int dim, int vdim, float scale,
    int window, int chunk, int keep, const float* slope, const float* rate, float softcap,
    const float* linear, const float* sink, const void* gate, long long gate_stride,
    const float* elem_gate, long long elem_stride, const void* map_gate, long long map_gate_stride,
    float out_scale, float lambda, float eps, int decode, int key_splits, float* sums, float* stats,
    int ordered, cudaStream_t stream) {
  if (tokens < 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || (maps != 1 && maps != 2) ||
      window < 0 || chunk < 0 || keep < 0 || (window > 0 && chunk > 0) || softcap < 0.f ||
      max_blocks <= 0 || sequences < 0 || key_splits < 1 || key_splits > 64 || (!decode && key_splits > 1) ||
      k_row < maps * dim || (v_cache != nullptr ? v_row < vdim : k_row < vdim) ||
      (q2 != nullptr && (q_split < 0 || q_split > dim)) || heads > 65535)
    return cudaErrorInvalidValue;
  const bool two_step = (maps == 2 && decode) || key_splits > 1;
  if (two_step != (sums != nullptr) || two_step != (stats != nullptr)) return cudaErrorInvalidValue;
  if (maps == 2 && (gate != nullptr || elem_gate != nullptr)) return cudaErrorInvalidValue;
  if ((((uintptr_t)q | (uintptr_t)q2 | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) ||
      ((q_stride | q_head_stride | k_row) & 7) || (v_cache != nullptr && (v_row & 7)) ||
      (q2 != nullptr && ((q2_stride | q2_head_stride | q_split) & 7)))
    return cudaErrorInvalidValue;
  if (tokens == 0) return 0;
  MmaAttention a = {};
  a.q = (const __nv_bfloat16*)q;
  a.q_stride = q_stride;
  a.q_head_stride = q_head_stride;
  a.q2 = (const __nv_bfloat16*)q2;
  a.q2_stride = q2_stride;
  a.q2_head_stride = q2_head_stride;
  a.q_split = q2 != nullptr ? q_split : dim;
  a.k_cache = (const __nv_bfloat16*)k_cache;
  a.v_cache = (const __nv_bfloat16*)v_cache;
  a.k_row = k_row;
  a.v_row = v_row;
  a.positions = positions;
  a.token_seq = token_seq;
  a.cu_seqlens = cu_seqlens;
  a.sequences = sequences;
  a.block_table = block_table;
  a.max_blocks = max_blocks;
  a.tokens = tokens;
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.maps = maps;
  a.scale = scale;
  a.window = window;
  a.chunk = chunk;
  a.keep = window > 0 ? keep : 0;
  a.slope = slope;
  a.rate = rate;
  a.softcap = softcap;
  a.linear = linear;
  a.key_splits = key_splits;
  a.out = (__nv_bfloat16*)out;
  a.sums = sums;
  a.stats = stats;
  a.sink = sink;
  a.gate = (const __nv_bfloat16*)gate;
  a.gate_stride = gate_stride;
  a.elem_gate = elem_gate;
  a.elem_stride = elem_stride;
  a.map_gate = (const __nv_bfloat16*)map_gate;
  a.map_gate_stride = map_gate_stride;
  a.out_scale = out_scale;
  a.lambda = lambda;
  a.eps = eps;
  a.ordered = ordered;
  const bool in_key = v_cache == nullptr;
  if (in_key && dim == 576 && vdim == 512 && maps == 1)
    return decode ? launch_shape<576, 512, true, 1, 8, 64, 2, 1>(a, true, stream)
                  : launch_shape<576, 512, true, 4, 2, 32, 3, 1>(a, false, stream);
  if (in_key) return cudaErrorInvalidValue;
  if (dim == 128 && vdim == 128)
    return decode      ? launch_shape<128, 128, false, 1, 8, 64, 3, 1>(a, true, stream)
           : maps == 1 ? launch_shape<128, 128, false, 4, 1, 64, 2, 1>(a, false, stream)
                       : launch_shape<128, 128, false, 4, 1, 32, 2, 2>(a, false, stream);
  if (dim == 128 && vdim == 256)
    return decode      ? launch_shape<128, 256, false, 1, 8, 64, 3, 1>(a, true, stream)
           : maps == 1 ? launch_shape<128, 256, false, 4, 1, 32, 2, 1>(a, false, stream)
                       : launch_shape<128, 256, false, 4, 1, 32, 2, 2>(a, false, stream);
  if (dim == 64 && vdim == 64 && maps == 1)
    return decode ? launch_shape<64, 64, false, 1, 4, 64, 3, 1>(a, true, stream)
                  : launch_shape<64, 64, false, 4, 1, 64, 2, 1>(a, false, stream);
  return cudaErrorInvalidValue;
}
