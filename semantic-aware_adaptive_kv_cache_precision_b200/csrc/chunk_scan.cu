// A long prompt through the two recurrences whose state, a matrix a head, is faded by one number and
// added to by one outer product a token (the fading state and the state-space dual form; csrc/
// recurrent_scan.cu walks them token by token):
//
//     S <- f_t S + d_t k_t v_t^T;      o_t = S^T q_t              f_t = exp(g_t), d_t a step size or 1
//
// A sequence's part of the step is cut into runs of up to 64 tokens. With G_i the sum of the g up to
// token i of a run that starts from S0,
//
//     o_i = exp(G_i) S0^T q_i + sum_{j <= i} exp(G_i - G_j) d_j (q_i . k_j) v_j
//     S1  = exp(G_n) S0       + sum_j        exp(G_n - G_j) d_j k_j v_j^T
//
// so a run is four small matrix products, and three launches do a prompt: `run_states` leaves every
// run's S1 from S0 = 0, `carry` replaces it by the S0 of the run, going from run to run, `run_outputs`
// makes the outputs. Walked token by token, a thread's chain of multiply-adds through shared memory
// bound both passes.
//
// Nothing is rounded to 16 bits: an fp32 operand enters a product as the sum of three bfloat16 numbers,
// which hold its 24 bits (an operand that is bfloat16 enters as it is), all products of pieces down to
// 2^-16 of the largest are taken, and the sums are fp32 (mma.sync m16n8k16). The exponents G_i - G_j are
// differences of sums kept as two floats each, so they are as exact as if the steps between had been
// added. On mma.sync and not tcgen05: a run's products are 64 rows, half of what tcgen05's full rate
// takes, an operand of one is the accumulator of another, and the pieces are made in registers.
// All products of a step of 16 are added to a sum of their own, the smallest first, and that sum to the
// total: the tensor cores cut where they add, and a chain of them loses an ulp of the total a step.
//
// Measured (us; walked in runs -> as products): fading state, 3,001 tokens of 16 heads of 128 x 128: 593 +
// 292 + 26 -> 171 + 89 + 14; dual form, 16 prompts of 500 tokens, 32 heads of 128 x 64: 288 + 165 + 120 ->
// 135 + 54 + 33; 2,048 tokens of 64 heads: 275 + 157 + 64 -> 117 + 50 + 21. Error against 64 bits 1.6e-7
// and 1.1e-7 (2.9e-7 and 1.7e-7 walked). What bounds them now is the splitting of fp32 into pieces and the
// products of those, not memory.
//
// A run with an output that is not finite goes through its tokens one by one, in order, so that a value
// that is not finite (or beyond 3.3e38, whose first piece would not be) is not felt before its token.
#include "mma.cuh"
#include "scan.cuh"

#include <initializer_list>
#include <type_traits>

namespace {

using scan::FadeInput;
using scan::fade_act;
using scan::softplus;

constexpr int kTokens = 64;      // most tokens a run; 16 rows a warp
constexpr int kCols = 64;        // value columns a block
constexpr int kThreads = 128;
constexpr int kPitchV = kCols + 8;     // (rows 16 bytes apart modulo 128: ldmatrix without conflicts)

// One step's inputs of the fading state: columns of an fp32 projection, shaped on their way in.
// QUADS: everything in whole pieces of four numbers, so that a thread's loads are straight code.
template <bool QUADS>
struct FadeSource {
  static constexpr int kPieces = 3;
  static constexpr bool kQuads = QUADS;
  const float* proj;
  long long stride;
  int q_off, k_off, v_off;
  const float* less_one;          // [heads]: the decay less one
  int dim, vdim;
  FadeInput in;

  __device__ float turned(const float* head, int t, int i) const {
    const float x = fade_act(head[i], in.act);
    if (i >= in.rot) return x;
    const int half = in.rot >> 1, pair = i < half ? i : i - half;
    const float y = fade_act(head[i < half ? i + half : pair], in.act);
    const long long at = (long long)in.positions[t] * half + pair;
    const float c = in.cos_t[at], s = in.sin_t[at];
    return i < half ? x * c - y * s : x * c + y * s;
  }
  __device__ float4 acted(float4 v) const {
    return in.act ? make_float4(scan::silu(v.x), scan::silu(v.y), scan::silu(v.z), scan::silu(v.w)) : v;
  }
  // TURN: whether numbers i to i + 3 are turned (any value where they do not come as one quad)
  template <bool TURN>
  __device__ float4 turned4(const float* head, int t, int i) const {
    if constexpr (!QUADS) {
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = i + k < dim ? turned(head, t, i + k) : 0.f;
      return make_float4(v[0], v[1], v[2], v[3]);
    }
    const float4 x = acted(*reinterpret_cast<const float4*>(head + i));
    if constexpr (!TURN) return x;
    const int half = in.rot >> 1, pair = i < half ? i : i - half;
    const float4 y = acted(*reinterpret_cast<const float4*>(head + (i < half ? i + half : pair)));
    const long long at = (long long)in.positions[t] * half + pair;
    const float4 c = *reinterpret_cast<const float4*>(in.cos_t + at);
    float4 s = *reinterpret_cast<const float4*>(in.sin_t + at);
    if (i < half) s = make_float4(-s.x, -s.y, -s.z, -s.w);
    return make_float4(x.x * c.x + y.x * s.x, x.y * c.y + y.y * s.y, x.z * c.z + y.z * s.z,
                       x.w * c.w + y.w * s.w);
  }
  __device__ const float* head_of(int t, int h, int off) const {
    return proj + (long long)t * stride + off + (long long)h * dim;
  }
  __device__ float query(int t, int h, int i) const { return turned(head_of(t, h, q_off), t, i); }
  __device__ float key(int t, int h, int i) const {
    return turned(head_of(t, h, k_off), t, i) * in.k_scale;
  }
  __device__ float value(int t, int h, int c) const {
    return fade_act(proj[(long long)t * stride + v_off + (long long)h * vdim + c], in.act);
  }
  // four neighbouring numbers, 0 beyond the head's
  __device__ bool turns(int i) const { return i < in.rot; }
  template <bool TURN>
  __device__ float4 query4(int t, int h, int i) const {
    return turned4<TURN>(head_of(t, h, q_off), t, i);
  }
  template <bool TURN>
  __device__ float4 key4(int t, int h, int i) const {
    const float4 v = turned4<TURN>(head_of(t, h, k_off), t, i);
    return make_float4(v.x * in.k_scale, v.y * in.k_scale, v.z * in.k_scale, v.w * in.k_scale);
  }
  __device__ float4 value4(int t, int h, int c) const {
    if constexpr (QUADS)
      return acted(*reinterpret_cast<const float4*>(proj + (long long)t * stride + v_off +
                                                    (long long)h * vdim + c));
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = c + k < vdim ? value(t, h, c + k) : 0.f;
    return make_float4(v[0], v[1], v[2], v[3]);
  }
  __device__ float step(int, int) const { return 1.f; }
  // (of the decay's size; a decay below zero also changes the state's sign, every token)
  __device__ double rate(float, int h) const {
    return flips(h) ? log(-1.0 - (double)less_one[h]) : log1p((double)less_one[h]);
  }
  __device__ bool flips(int h) const { return less_one[h] < -1.f; }
  __device__ float change(float, int h) const { return less_one[h]; }      // the decay less one
  __device__ float skip(int) const { return 0.f; }
};

// One step's inputs of the dual form: x, B and C after the convolution, a step size a (token, head).
template <typename C, bool QUADS>
struct DualSource {
  static constexpr int kPieces = sizeof(C) == 2 ? 1 : 3;
  static constexpr bool kQuads = QUADS;
  const C* xbc;
  long long stride;
  int x_off, b_off, c_off;
  const float* dt;
  long long dt_stride;
  const float* dt_bias;
  const float* a;
  const float* d_skip;
  int dim, vdim, heads_a_group;

  __device__ float4 four(const C* row, int i, int size) const {
    if constexpr (QUADS) {
      if constexpr (sizeof(C) == 4) return *reinterpret_cast<const float4*>(row + i);
      const uint2 raw = *reinterpret_cast<const uint2*>(row + i);
      return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                         __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
    }
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k < size ? widen(row[i + k]) : 0.f;
    return make_float4(v[0], v[1], v[2], v[3]);
  }
  __device__ bool turns(int) const { return false; }
  template <bool TURN>
  __device__ float4 query4(int t, int h, int i) const {
    return four(xbc + (long long)t * stride + c_off + h / heads_a_group * dim, i, dim);
  }
  template <bool TURN>
  __device__ float4 key4(int t, int h, int i) const {
    return four(xbc + (long long)t * stride + b_off + h / heads_a_group * dim, i, dim);
  }
  __device__ float4 value4(int t, int h, int c) const {
    return four(xbc + (long long)t * stride + x_off + (long long)h * vdim, c, vdim);
  }
  __device__ float query(int t, int h, int i) const {
    return widen(xbc[(long long)t * stride + c_off + h / heads_a_group * dim + i]);
  }
  __device__ float key(int t, int h, int i) const {
    return widen(xbc[(long long)t * stride + b_off + h / heads_a_group * dim + i]);
  }
  __device__ float value(int t, int h, int c) const {
    return widen(xbc[(long long)t * stride + x_off + (long long)h * vdim + c]);
  }
  __device__ float step(int t, int h) const {
    return softplus(dt[(long long)t * dt_stride + h] + dt_bias[h]);
  }
  __device__ double rate(float step, int h) const { return (double)step * a[h]; }
  __device__ bool flips(int) const { return false; }
  __device__ float change(float step, int h) const { return (float)expm1(rate(step, h)); }
  __device__ float skip(int h) const { return d_skip[h]; }
};

struct Runs {
  float* scratch;                  // [rows, heads, vdim, dim], a row a run (`row_of`)
  float* logs;                     // [rows, heads]: the sum of a run's g
  const float* less_one;           // [heads]: the decay less one, where decays may be below zero (else null)
  const int32_t* cu_seqlens;
  int heads, dim, vdim, run_len, max_runs;
};

// The scratch row of a sequence's first run; its further runs follow. (Runs of the sequences before it: no
// more than their tokens / run_len, and one each that is not full.)
__device__ __forceinline__ long long row_of(const Runs& r, int b) {
  return r.cu_seqlens[b] / r.run_len + b;
}

__device__ __forceinline__ bool odd_value(float x) { return !(fabsf(x) < INFINITY); }

// Two neighbouring numbers as PIECES bfloat16 pairs, the pieces `apart` words from each other.
template <int PIECES>
__device__ __forceinline__ void put2(uint32_t* to, int apart, float x, float y) {
  uint32_t p = mma::pack_bf16(x, y);
  to[0] = p;
#pragma unroll
  for (int i = 1; i < PIECES; ++i) {
    x -= __uint_as_float(p << 16);
    y -= __uint_as_float(p & 0xffff0000u);
    p = mma::pack_bf16(x, y);
    to[i * apart] = p;
  }
}

// Four neighbouring numbers likewise, the pieces `apart` elements from each other.
template <int PIECES>
__device__ __forceinline__ void put4(__nv_bfloat16* to, int apart, float4 v) {
  uint32_t lo[PIECES], hi[PIECES];
  put2<PIECES>(lo, 1, v.x, v.y);
  put2<PIECES>(hi, 1, v.z, v.w);
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
    *reinterpret_cast<uint2*>(to + p * apart) = make_uint2(lo[p], hi[p]);
}

// A block's threads over rows of `wide` numbers, four a thread: `lanes` (a power of two) side by side.
struct Deal {
  int lanes, row, at, rows;        // threads a row; this thread's first row and number; rows at a time
};
__device__ __forceinline__ Deal deal(int wide) {
  int shift = 2;                                   // (rows of 16 numbers and more)
  while ((4 << shift) < wide) ++shift;
  Deal d;
  d.lanes = 1 << shift;
  d.at = (threadIdx.x & (d.lanes - 1)) * 4;
  d.row = threadIdx.x >> shift;
  d.rows = kThreads >> shift;
  return d;
}

// Rows `row`, `row` + `step`, ... below `whole` of a tile, four numbers of each a thread (from `to` on, rows
// `pitch` elements apart), from load(j), j below `n`, and zeros from there on. N rows are asked for before
// the first is split, whatever j: a load that waited for a branch would be a trip to memory a row, and
// sixteen of them were most of the kernels' time.
template <int PIECES, int N, class Load>
__device__ __forceinline__ void stage(__nv_bfloat16* to, int pitch, int apart, int row, int step, int whole,
                                      int n, Load load) {
  for (int j0 = row; j0 < whole; j0 += N * step) {
    float4 v[N];
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = load(min(j0 + q * step, n - 1));
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int j = j0 + q * step;
      if (j < whole) put4<PIECES>(to + j * pitch, apart, j < n ? v[q] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
  }
}
// The same of rows that are zeros.
template <int PIECES>
__device__ __forceinline__ void stage_zeros(__nv_bfloat16* to, int pitch, int apart, int row, int step,
                                            int whole) {
  for (int j = row; j < whole; j += step) put4<PIECES>(to + j * pitch, apart, make_float4(0.f, 0.f, 0.f, 0.f));
}

// d (two n-tiles) += the products of A's pieces and B's whose orders add up to no more than two.
// In a sum of their own, which then joins the total in fp32: see above.
template <int NA, int NB>
__device__ __forceinline__ void products(float (&d0)[4], float (&d1)[4], const uint32_t (&a)[NA][4],
                                         const uint32_t (&b)[NB][4]) {
  float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int order = 2; order >= 0; --order)
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int j = order - i;
      if (j < 0 || j >= NB) continue;
      mma::bf16_16816(s0, a[i], b[j][0], b[j][1]);
      mma::bf16_16816(s1, a[i], b[j][2], b[j][3]);
    }
  mma::add2(d0[0], d0[1], s0[0], s0[1]);
  mma::add2(d0[2], d0[3], s0[2], s0[3]);
  mma::add2(d1[0], d1[1], s1[0], s1[1]);
  mma::add2(d1[2], d1[3], s1[2], s1[3]);
}

// The run of this block: its first token and how many it has (0 or less: no such run).
struct Span {
  int b, run, first, n;
};
__device__ __forceinline__ Span span_of(const Runs& r) {
  Span s;
  s.b = blockIdx.z / r.max_runs;
  s.run = blockIdx.z % r.max_runs;
  s.first = r.cu_seqlens[s.b] + s.run * r.run_len;
  s.n = min(r.cu_seqlens[s.b + 1] - s.first, r.run_len);
  return s;
}

// Step sizes and G of the run's tokens (two floats each), by the first warp; lane l has tokens 2 l and
// 2 l + 1. A rate below -1e4 is as good as -1e4: nothing is left.
template <class Source>
__device__ __forceinline__ void sums_of(const Source& src, const Span& s, int h, float* steps,
                                        float* g_hi, float* g_lo, double* total) {
  const int lane = threadIdx.x;
  double sum[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = 2 * lane + k;
    const float d = i < s.n ? src.step(s.first + i, h) : 0.f;
    const double g = i < s.n ? src.rate(d, h) : 0.0;
    steps[i] = d;
    sum[k] = g < -1e4 ? -1e4 : g;
  }
  sum[1] += sum[0];
  double before = sum[1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += up;
  }
  *total = __shfl_sync(0xffffffffu, before, 31);
  before -= sum[1];                              // the sum before this lane's tokens
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double g = before + sum[k];
    g_hi[2 * lane + k] = (float)g;
    g_lo[2 * lane + k] = (float)(g - (double)(float)g);
  }
}

// The run token by token, for values that the products cannot take: a thread a column, its state in
// the scratch memory of the run.
template <class Source>
__device__ __noinline__ void walk(const Source& src, const Runs& r, const Span& s, int h, int col0,
                                  float* state, float* out) {
  for (int c = col0 + threadIdx.x; c < min(col0 + kCols, r.vdim); c += kThreads) {
    float* mine = state + (long long)c * r.dim;
    for (int t = s.first; t < s.first + s.n; ++t) {
      const float d = src.step(t, h), x = src.value(t, h, c), v = d * x;
      const float fade = src.change(d, h);
      float o = 0.f;
      for (int i = 0; i < r.dim; ++i) {
        const float m = fmaf(src.key(t, h, i), v, fmaf(fade, mine[i], mine[i]));
        mine[i] = m;
        if (out) o = fmaf(m, src.query(t, h, i), o);
      }
      if (out) out[((long long)t * r.heads + h) * r.vdim + c] = fmaf(src.skip(h), x, o);
    }
  }
}

// Where the four 8 x 8 pieces of a fragment lie that a lane's ldmatrix address chooses, in a tile of
// rows of the operand's outer index.
__device__ __forceinline__ int a_row(int lane) { return lane & 15; }
__device__ __forceinline__ int a_col(int lane) { return (lane >> 4) * 8; }
__device__ __forceinline__ int b_row(int lane) { return (lane & 7) + (lane >> 4) * 8; }
__device__ __forceinline__ int b_col(int lane) { return ((lane >> 3) & 1) * 8; }

// Every run's end state from nothing: U[c, i] = sum_j exp(G_n - G_j) d_j v_j[c] k_j[i]. Warp w makes 16
// columns c; the numbers i go by in groups of 64.
template <class Source>
__global__ void __launch_bounds__(kThreads) run_states(const Source src, const Runs r) {
  constexpr int NP = Source::kPieces;
  extern __shared__ __align__(16) uint32_t pool[];
  __shared__ float steps[kTokens], g_hi[kTokens], g_lo[kTokens], weight[kTokens];
  const Span s = span_of(r);
  if (s.n <= 0) return;                          // (the whole block)
  const int h = blockIdx.y, col0 = blockIdx.x * kCols;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wide = (r.dim + 15) / 16 * 16, pitch = wide + 8;
  __nv_bfloat16* ks = reinterpret_cast<__nv_bfloat16*>(pool);             // [NP][64][pitch]
  __nv_bfloat16* vs = ks + NP * kTokens * pitch;                          // [3][64][kPitchV]
  if (warp == 0) {
    double total;
    sums_of(src, s, h, steps, g_hi, g_lo, &total);
    __syncwarp();
    const float hi = (float)total, lo = (float)(total - (double)hi);
    for (int i = lane; i < kTokens; i += 32) {
      const float w = i < s.n ? steps[i] * expf((hi - g_hi[i]) + (lo - g_lo[i])) : 0.f;
      weight[i] = src.flips(h) && ((s.n - 1 - i) & 1) ? -w : w;
    }
    if (blockIdx.x == 0 && lane == 0)
      r.logs[(row_of(r, s.b) + s.run) * r.heads + h] = hi;
  }
  const int whole = (s.n + 15) & ~15;            // rows of the products
  const Deal d = deal(wide);
  if (d.at < r.dim) {
    if (src.turns(d.at))
      stage<NP, 8>(ks + d.at, pitch, kTokens * pitch, d.row, d.rows, whole, s.n,
                   [&](int j) { return src.template key4<true>(s.first + j, h, d.at); });
    else
      stage<NP, 8>(ks + d.at, pitch, kTokens * pitch, d.row, d.rows, whole, s.n,
                   [&](int j) { return src.template key4<false>(s.first + j, h, d.at); });
  } else if (d.at < wide) {
    stage_zeros<NP>(ks + d.at, pitch, kTokens * pitch, d.row, d.rows, whole);
  }
  __syncthreads();                               // (the weights)
  {
    const int c = (tid & 15) * 4;
    if (col0 + c < r.vdim)
      stage<3, 8>(vs + c, kPitchV, kTokens * kPitchV, tid >> 4, kThreads / 16, whole, s.n, [&](int j) {
        const float4 v = src.value4(s.first + j, h, col0 + c);
        const float w = weight[j];
        return make_float4(w * v.x, w * v.y, w * v.z, w * v.w);
      });
    else
      stage_zeros<3>(vs + c, kPitchV, kTokens * kPitchV, tid >> 4, kThreads / 16, whole);
  }
  float* state = r.scratch + ((row_of(r, s.b) + s.run) * r.heads + h) *
                                 ((long long)r.vdim * r.dim);
  __syncthreads();
  bool odd = false;
  const uint32_t ks_at = static_cast<uint32_t>(__cvta_generic_to_shared(ks));
  const uint32_t vs_at = static_cast<uint32_t>(__cvta_generic_to_shared(vs));
  const int steps16 = whole / 16;
  for (int i0 = 0; col0 + warp * 16 < r.vdim && i0 < wide; i0 += 64) {
    float acc[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
    for (int k = 0; k < steps16; ++k) {
      uint32_t a[3][4], b[NP][4];
      // A's rows are the columns c, its inner index the tokens: the tile lies turned
      const int arow = k * 16 + (lane & 7) + (lane >> 4) * 8;
      const int acol = warp * 16 + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int p = 0; p < 3; ++p)
        mma::ldmatrix_x4_trans(vs_at + ((p * kTokens + arow) * kPitchV + acol) * 2, a[p][0], a[p][1],
                               a[p][2], a[p][3]);
      const int brow = k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (i0 + n * 16 >= wide) continue;
#pragma unroll
        for (int p = 0; p < NP; ++p)
          mma::ldmatrix_x4_trans(
              ks_at + ((p * kTokens + brow) * pitch + i0 + n * 16 + (lane >> 4) * 8) * 2, b[p][0],
              b[p][1], b[p][2], b[p][3]);
        products(acc[2 * n], acc[2 * n + 1], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int i = i0 + n * 8 + (lane & 3) * 2;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int c = col0 + warp * 16 + (lane >> 2) + half * 8;
        if (c >= r.vdim || i >= r.dim) continue;
        odd |= odd_value(acc[n][2 * half]) || odd_value(acc[n][2 * half + 1]);
        float* to = state + (long long)c * r.dim + i;
        if (r.dim % 2 == 0) {
          *reinterpret_cast<float2*>(to) = make_float2(acc[n][2 * half], acc[n][2 * half + 1]);
        } else {
          to[0] = acc[n][2 * half];
          if (i + 1 < r.dim) to[1] = acc[n][2 * half + 1];
        }
      }
    }
  }
  if (__syncthreads_or(odd)) {
    for (int e = tid; e < min(kCols, r.vdim - col0) * r.dim; e += kThreads)
      state[(long long)col0 * r.dim + e] = 0.f;
    __syncthreads();
    walk(src, r, s, h, col0, state, nullptr);
  }
}

// From run to run: what run j left is replaced by what came before it, which fades by exp(log_j) over
// the run (`scan::Fade`). VEC neighbouring numbers of a (sequence, head) a thread, eight runs asked for before the
// first is used, since a store keeps the compiler from asking for what follows it.
template <int VEC>
__global__ void __launch_bounds__(256)
carry(const Runs r, float* __restrict__ states, const int32_t* __restrict__ slots, int keep_state) {
  constexpr int kAhead = 8;
  const int per_head = r.vdim * r.dim;
  const int e = (blockIdx.x * 256 + threadIdx.x) * VEC;
  if (e >= per_head) return;
  const int h = blockIdx.y, b = blockIdx.z;
  const int tokens = r.cu_seqlens[b + 1] - r.cu_seqlens[b];
  const int runs = (tokens + r.run_len - 1) / r.run_len;
  const bool flips = r.less_one && r.less_one[h] < -1.f;
  const long long apart = (long long)r.heads * per_head;
  float* p = r.scratch + (row_of(r, b) * r.heads + h) * per_head + e;
  const float* logs = r.logs + row_of(r, b) * r.heads + h;
  float* home = states + ((long long)slots[b] * r.heads + h) * per_head + e;
  float s[VEC];
  auto read = [](const float* at, float (&v)[VEC]) {
    if constexpr (VEC == 4) {
      const float4 x = *reinterpret_cast<const float4*>(at);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
      v[0] = at[0];
    }
  };
  auto write = [](float* at, const float (&v)[VEC]) {
    if constexpr (VEC == 4) *reinterpret_cast<float4*>(at) = make_float4(v[0], v[1], v[2], v[3]);
    else at[0] = v[0];
  };
  read(home, s);
  for (int j0 = 0; j0 < runs; j0 += kAhead) {
    float left[kAhead][VEC], log[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (j0 + k < runs) {
        read(p + (j0 + k) * apart, left[k]);
        log[k] = logs[(long long)(j0 + k) * r.heads];
      }
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (j0 + k < runs) {
        const scan::Fade fade(log[k]);
        write(p + (j0 + k) * apart, s);
        if (flips && (min(tokens - (j0 + k) * r.run_len, r.run_len) & 1)) {    // (an odd number of tokens)
          const float factor = -expf(log[k]);
#pragma unroll
          for (int i = 0; i < VEC; ++i) s[i] = fmaf(factor, s[i], left[k][i]);
          continue;
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) s[i] = fade.carried(s[i], left[k][i]);
      }
  }
  if (keep_state) write(home, s);
}

// The outputs of every run, its S0 in scratch memory. Warp w has rows (tokens) 16 w on and all of the
// block's columns; the scores never leave its registers. q stays in shared memory; k, then S0, then v
// take turns in one buffer, which leaves room for two blocks an SM at 128 numbers a head in three pieces.
template <class Source>
__global__ void __launch_bounds__(kThreads)
run_outputs(const Source src, const Runs r, float* __restrict__ out) {
  constexpr int NP = Source::kPieces;
  extern __shared__ __align__(16) uint32_t pool[];
  __shared__ float steps[kTokens], g_hi[kTokens], g_lo[kTokens];
  const Span s = span_of(r);
  if (s.n <= 0) return;
  const int h = blockIdx.y, col0 = blockIdx.x * kCols;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wide = (r.dim + 15) / 16 * 16, pitch = wide + 8;
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(pool);             // [NP][64][pitch]
  __nv_bfloat16* turn = qs + NP * kTokens * pitch;       // k [NP][64][pitch], S0 [3][64][pitch], v
  float* state = r.scratch + ((row_of(r, s.b) + s.run) * r.heads + h) *
                                 ((long long)r.vdim * r.dim);
  if (warp == 0) {
    double total;
    sums_of(src, s, h, steps, g_hi, g_lo, &total);
  }
  const int whole = (s.n + 15) & ~15;                    // rows of the products
  const Deal d = deal(wide);
  if (d.at < r.dim) {
    auto both = [&](auto turned) {
      constexpr bool T = decltype(turned)::value;
      stage<NP, 8>(qs + d.at, pitch, kTokens * pitch, d.row, d.rows, whole, s.n,
                   [&](int j) { return src.template query4<T>(s.first + j, h, d.at); });
      stage<NP, 8>(turn + d.at, pitch, kTokens * pitch, d.row, d.rows, whole, s.n,
                   [&](int j) { return src.template key4<T>(s.first + j, h, d.at); });
    };
    if (src.turns(d.at)) both(std::true_type());
    else both(std::false_type());
  } else if (d.at < wide) {
    stage_zeros<NP>(qs + d.at, pitch, kTokens * pitch, d.row, d.rows, whole);
    stage_zeros<NP>(turn + d.at, pitch, kTokens * pitch, d.row, d.rows, whole);
  }
  __syncthreads();
  const uint32_t qs_at = static_cast<uint32_t>(__cvta_generic_to_shared(qs));
  const uint32_t turn_at = static_cast<uint32_t>(__cvta_generic_to_shared(turn));
  const bool rows = warp * 16 < s.n;                     // (a warp without rows still fills buffers)
  const bool flips = src.flips(h);
  const uint32_t q_from = qs_at + ((warp * 16 + a_row(lane)) * pitch + a_col(lane)) * 2;
  const int piece = kTokens * pitch * 2;                 // bytes

  // scores: tokens j in groups of 16 up to the warp's own
  float sc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int k = 0; k < 4; ++k) sc[n][k] = 0.f;
  if (rows) {
    for (int k = 0; k < wide; k += 16) {
      uint32_t a[NP][4], b[NP][4];
#pragma unroll
      for (int p = 0; p < NP; ++p)
        mma::ldmatrix_x4(q_from + p * piece + k * 2, a[p][0], a[p][1], a[p][2], a[p][3]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (n > warp) continue;
#pragma unroll
        for (int p = 0; p < NP; ++p)
          mma::ldmatrix_x4(turn_at + p * piece + ((n * 16 + b_row(lane)) * pitch + k + b_col(lane)) * 2,
                           b[p][0], b[p][1], b[p][2], b[p][3]);
        products(sc[2 * n], sc[2 * n + 1], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (n > 2 * warp + 1) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = warp * 16 + (lane >> 2) + (k >> 1) * 8, j = n * 8 + (lane & 3) * 2 + (k & 1);
        const float w = sc[n][k] * steps[j] * expf((g_hi[i] - g_hi[j]) + (g_lo[i] - g_lo[j]));
        sc[n][k] = j > i ? 0.f : flips && ((i - j) & 1) ? -w : w;
      }
    }
  }

  // what the state brings
  __syncthreads();
  {
    const int columns = min(kCols, (r.vdim - col0 + 15) & ~15);
    if (d.at < r.dim)
      stage<3, 8>(turn + d.at, pitch, kTokens * pitch, d.row, d.rows, columns, min(kCols, r.vdim - col0),
                  [&](int c) {
                    const float* at = state + (long long)(col0 + c) * r.dim + d.at;
                    if constexpr (Source::kQuads) return *reinterpret_cast<const float4*>(at);
                    float4 v = make_float4(at[0], 0.f, 0.f, 0.f);
                    if (d.at + 1 < r.dim) v.y = at[1];
                    if (d.at + 2 < r.dim) v.z = at[2];
                    if (d.at + 3 < r.dim) v.w = at[3];
                    return v;
                  });
    else if (d.at < wide)
      stage_zeros<3>(turn + d.at, pitch, kTokens * pitch, d.row, d.rows, columns);
  }
  __syncthreads();
  float acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
  if (rows) {
    for (int k = 0; k < wide; k += 16) {
      uint32_t a[NP][4], b[3][4];
#pragma unroll
      for (int p = 0; p < NP; ++p)
        mma::ldmatrix_x4(q_from + p * piece + k * 2, a[p][0], a[p][1], a[p][2], a[p][3]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (col0 + n * 16 >= r.vdim) continue;
#pragma unroll
        for (int p = 0; p < 3; ++p)
          mma::ldmatrix_x4(turn_at + p * piece + ((n * 16 + b_row(lane)) * pitch + k + b_col(lane)) * 2,
                           b[p][0], b[p][1], b[p][2], b[p][3]);
        products(acc[2 * n], acc[2 * n + 1], a, b);
      }
    }
    float f[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = warp * 16 + (lane >> 2) + half * 8;
      f[half] = flips && !(i & 1) ? -expf(g_hi[i] + g_lo[i]) : expf(g_hi[i] + g_lo[i]);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[n][k] *= f[k >> 1];
  }

  // what the run's own tokens bring
  __syncthreads();
  {
    const int c = (tid & 15) * 4;
    if (col0 + c < r.vdim)
      stage<NP, 8>(turn + c, kPitchV, kTokens * kPitchV, tid >> 4, kThreads / 16, whole, s.n,
                   [&](int j) { return src.value4(s.first + j, h, col0 + c); });
    else
      stage_zeros<NP>(turn + c, kPitchV, kTokens * kPitchV, tid >> 4, kThreads / 16, whole);
  }
  __syncthreads();
  bool odd = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k > warp || !rows) continue;
    uint32_t a[3][4];
    uint32_t w[4][3];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      put2<3>(w[q], 1, sc[2 * k + (q >> 1)][2 * (q & 1)], sc[2 * k + (q >> 1)][2 * (q & 1) + 1]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) a[p][q] = w[q][p];
    const int brow = k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      if (col0 + n * 16 >= r.vdim) continue;
      uint32_t b[NP][4];
#pragma unroll
      for (int p = 0; p < NP; ++p)
        mma::ldmatrix_x4_trans(
            turn_at + ((p * kTokens + brow) * kPitchV + n * 16 + (lane >> 4) * 8) * 2, b[p][0],
            b[p][1], b[p][2], b[p][3]);
      products(acc[2 * n], acc[2 * n + 1], a, b);
    }
  }
  const float skip = src.skip(h);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = warp * 16 + (lane >> 2) + half * 8, t = s.first + i;
    if (!rows || i >= s.n) continue;
    float* row = out + ((long long)t * r.heads + h) * r.vdim;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int c = col0 + n * 8 + (lane & 3) * 2;
      if (c >= r.vdim) continue;
      float x = acc[n][2 * half], y = acc[n][2 * half + 1];
      if (skip != 0.f) {
        x = fmaf(skip, src.value(t, h, c), x);
        if (c + 1 < r.vdim) y = fmaf(skip, src.value(t, h, c + 1), y);
      }
      odd |= odd_value(x) || odd_value(y);
      if (r.vdim % 2 == 0) {
        *reinterpret_cast<float2*>(row + c) = make_float2(x, y);
      } else {
        row[c] = x;
        if (c + 1 < r.vdim) row[c + 1] = y;
      }
    }
  }
  if (__syncthreads_or(odd)) walk(src, r, s, h, col0, state, out);
}

bool multiples_of_4(std::initializer_list<long long> values) {
  for (const long long v : values)
    if (v % 4) return false;
  return true;
}

__device__ __noinline__ float plain_sum(const float* __restrict__ row, const __nv_bfloat16* __restrict__ w,
                                        int rank) {
  float sum = 0.f;
  for (int r = 0; r < rank; ++r) sum = fmaf(row[r], widen(w[r]), sum);
  return sum;
}

// Step sizes of the selective scan: dt[t, c] = softplus(sum_r low[t, r] W[c, r] + b[c]), low fp32 in three
// pieces, W bfloat16 as it is. A block has 64 tokens' rows of `low` and goes over `tiles` groups of 64
// channels; warp w makes 16 tokens. A sum that is not finite is made again number by number: the pieces of
// a value that is not finite (or beyond 3.3e38) are not, where the value times a weight may be.
// 3,400 tokens of 4,096 channels, rank 128: 85 us (on the CUDA cores 185), bound by the pieces and the softplus.
template <bool QUADS>
__global__ void __launch_bounds__(kThreads)
step_sizes(const float* __restrict__ low, long long stride, int rank,
           const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ bias,
           float* __restrict__ dt, int tokens, int channels, int tiles) {
  extern __shared__ __align__(16) uint32_t pool[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wide = (rank + 15) / 16 * 16, pitch = wide + 8;
  __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(pool);          // [3][64][pitch]
  __nv_bfloat16* ws = rows + 3 * kTokens * pitch;                        // [64][pitch]
  const int m0 = blockIdx.y * kTokens;
  const Deal d = deal(wide);
  if (d.at < rank)
    stage<3, 8>(rows + d.at, pitch, kTokens * pitch, d.row, d.rows, kTokens, min(kTokens, tokens - m0),
                [&](int j) {
                  const float* at = low + (long long)(m0 + j) * stride + d.at;
                  if constexpr (QUADS) return *reinterpret_cast<const float4*>(at);
                  float4 v = make_float4(at[0], 0.f, 0.f, 0.f);
                  if (d.at + 1 < rank) v.y = at[1];
                  if (d.at + 2 < rank) v.z = at[2];
                  if (d.at + 3 < rank) v.w = at[3];
                  return v;
                });
  else if (d.at < wide)
    stage_zeros<3>(rows + d.at, pitch, kTokens * pitch, d.row, d.rows, kTokens);
  const uint32_t rows_at = static_cast<uint32_t>(__cvta_generic_to_shared(rows));
  const uint32_t ws_at = static_cast<uint32_t>(__cvta_generic_to_shared(ws));
  const uint32_t from = rows_at + ((warp * 16 + a_row(lane)) * pitch + a_col(lane)) * 2;
  const int piece = kTokens * pitch * 2;
  for (int i = 0; i < tiles; ++i) {
    const int n0 = (blockIdx.x * tiles + i) * 64;
    if (n0 >= channels) break;
    if (i) __syncthreads();
    if (d.at < rank)
      stage<1, 8>(ws + d.at, pitch, 0, d.row, d.rows, 64, min(64, channels - n0), [&](int j) {
        const __nv_bfloat16* at = w + (long long)(n0 + j) * rank + d.at;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (QUADS) {
          read4(at, f);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (d.at + k < rank) f[k] = widen(at[k]);
        }
        return make_float4(f[0], f[1], f[2], f[3]);
      });
    else if (d.at < wide)
      stage_zeros<1>(ws + d.at, pitch, 0, d.row, d.rows, 64);
    __syncthreads();
    float acc[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
    for (int k = 0; k < wide; k += 16) {
      uint32_t a[3][4], b[1][4];
#pragma unroll
      for (int p = 0; p < 3; ++p)
        mma::ldmatrix_x4(from + p * piece + k * 2, a[p][0], a[p][1], a[p][2], a[p][3]);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        mma::ldmatrix_x4(ws_at + ((n * 16 + b_row(lane)) * pitch + k + b_col(lane)) * 2, b[0][0],
                         b[0][1], b[0][2], b[0][3]);
        products(acc[2 * n], acc[2 * n + 1], a, b);
      }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int c = n0 + n * 8 + (lane & 3) * 2;
      if (c >= channels) continue;
      const float b0 = bias ? widen(bias[c]) : 0.f;
      const float b1 = bias && c + 1 < channels ? widen(bias[c + 1]) : 0.f;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = m0 + warp * 16 + (lane >> 2) + half * 8;
        if (t >= tokens) continue;
        float x = acc[n][2 * half], y = acc[n][2 * half + 1];
        if (odd_value(x)) x = plain_sum(low + (long long)t * stride, w + (long long)c * rank, rank);
        if (odd_value(y) && c + 1 < channels)
          y = plain_sum(low + (long long)t * stride, w + (long long)(c + 1) * rank, rank);
        x = softplus(x + b0);
        y = softplus(y + b1);
        float* to = dt + (long long)t * channels + c;
        if (channels % 2 == 0) {
          *reinterpret_cast<float2*>(to) = make_float2(x, y);
        } else {
          to[0] = x;
          if (c + 1 < channels) to[1] = y;
        }
      }
    }
  }
}

template <class Source>
int launch_runs(const Source& src, const Runs& r, float* states, const int32_t* slots, float* out,
                int sequences, int keep_state, cudaStream_t stream) {
  constexpr size_t NP = Source::kPieces;
  const size_t pitch = (r.dim + 15) / 16 * 16 + 8;
  const size_t states_smem = kTokens * (NP * pitch + 3 * kPitchV) * 2;
  const size_t turn = 3 * pitch > NP * kPitchV ? 3 * pitch : NP * kPitchV;
  const size_t outputs_smem = kTokens * (NP * pitch + turn) * 2;
  static PerDeviceOnce once;
  if (once.needs()) {
    for (const void* kernel : {(const void*)run_states<Source>, (const void*)run_outputs<Source>}) {
      const cudaError_t e =
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    once.done();
  }
  const dim3 grid((unsigned)((r.vdim + kCols - 1) / kCols), (unsigned)r.heads,
                  (unsigned)(sequences * r.max_runs));
  int code = launch_ordered(run_states<Source>, grid, dim3(kThreads), states_smem, stream, src, r);
  if (code) return code;
  const long long per_head = (long long)r.vdim * r.dim;
  const bool wide = per_head % 4 == 0 && !(((uintptr_t)states | (uintptr_t)r.scratch) & 15);
  const long long threads = wide ? per_head / 4 : per_head;
  const dim3 across((unsigned)((threads + 255) / 256), (unsigned)r.heads, (unsigned)sequences);
  code = wide ? launch_ordered(carry<4>, across, dim3(256), 0, stream, r, states, slots, keep_state)
              : launch_ordered(carry<1>, across, dim3(256), 0, stream, r, states, slots, keep_state);
  if (code) return code;
  return launch_ordered(run_outputs<Source>, grid, dim3(kThreads), outputs_smem, stream, src, r, out);
}

bool takes(int tokens, int sequences, int heads, int dim, int vdim, int run_len, int max_runs,
           const void* scratch, const void* logs) {
  return tokens >= 0 && sequences >= 0 && heads > 0 && heads <= 65535 && dim > 0 && dim <= 256 &&
         vdim > 0 && run_len > 0 && run_len <= kTokens && max_runs > 0 && scratch && logs &&
         (long long)sequences * max_runs <= 65535;
}

}  // namespace

// As `sakv_step_size` (csrc/recurrent_scan.cu) with weights in bfloat16, for ranks of up to 256.
SAKV_EXPORT int sakv_chunk_step_size(const float* low, long long stride, int rank, const void* w,
                                     const void* bias, float* dt, int tokens, int channels,
                                     cudaStream_t stream) {
  if (tokens < 0 || channels <= 0 || rank <= 0 || rank > 256) return cudaErrorInvalidValue;
  if (tokens == 0) return 0;
  static PerDeviceOnce once;
  if (once.needs()) {
    for (const void* kernel : {(const void*)step_sizes<true>, (const void*)step_sizes<false>}) {
      const cudaError_t e =
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    once.done();
  }
  const size_t pitch = (rank + 15) / 16 * 16 + 8;
  const int groups = (channels + 63) / 64, down = (tokens + kTokens - 1) / kTokens;
  if (down > 65535) return cudaErrorInvalidValue;
  int tiles = 4;                             // (fewer while the blocks do not fill the GPU twice)
  while (tiles > 1 && (long long)((groups + tiles - 1) / tiles) * down < 4LL * sm_count()) tiles /= 2;
  const bool quads = multiples_of_4({stride, rank}) && !((uintptr_t)low & 15) && !((uintptr_t)w & 7);
  return launch_ordered(quads ? step_sizes<true> : step_sizes<false>,
                        dim3((unsigned)((groups + tiles - 1) / tiles), (unsigned)down), dim3(kThreads),
                        kTokens * pitch * 4 * 2, stream, low, stride, rank, (const __nv_bfloat16*)w,
                        (const __nv_bfloat16*)bias, dt, tokens, channels, tiles);
}

// As `sakv_decay_attention` (csrc/recurrent_scan.cu), a sequence's tokens in runs of run_len (up to 64):
// max_runs the most a sequence has. scratch: fp32 [tokens / run_len + sequences, heads, vdim, dim]; logs: fp32
// [tokens / run_len + sequences, heads].
SAKV_EXPORT int sakv_chunk_fade(const float* proj, long long stride, int q_off, int k_off, int v_off,
                                const float* decay, float* state, const int32_t* cu_seqlens,
                                const int32_t* slots, float* out, int tokens, int sequences, int heads,
                                int dim, int vdim, int keep_state, int run_len, int max_runs,
                                float* scratch, float* logs, int act, int rot,
                                const int32_t* positions, const float* cos_t, const float* sin_t,
                                float k_scale, cudaStream_t stream) {
  if (!takes(tokens, sequences, heads, dim, vdim, run_len, max_runs, scratch, logs) || rot < 0 ||
      rot % 2 || rot > dim || (rot > 0 && (!positions || !cos_t || !sin_t)))
    return cudaErrorInvalidValue;
  if (tokens == 0 || sequences == 0) return 0;
  const bool quads = multiples_of_4({stride, q_off, k_off, v_off, dim, vdim, rot / 2}) &&
                     !(((uintptr_t)proj | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15);
  const FadeInput in = {act, rot, positions, cos_t, sin_t, k_scale};
  const Runs r = {scratch, logs, decay, cu_seqlens, heads, dim, vdim, run_len, max_runs};
  if (quads)
    return launch_runs(FadeSource<true>{proj, stride, q_off, k_off, v_off, decay, dim, vdim, in}, r, state,
                       slots, out, sequences, keep_state, stream);
  return launch_runs(FadeSource<false>{proj, stride, q_off, k_off, v_off, decay, dim, vdim, in}, r, state,
                     slots, out, sequences, keep_state, stream);
}

// As `sakv_dual_scan`, likewise.
SAKV_EXPORT int sakv_chunk_dual(const void* xbc, int c_dtype, long long stride, int x_off, int b_off,
                                int c_off, const float* dt, long long dt_stride, const float* dt_bias,
                                const float* a, const float* d_skip, float* state,
                                const int32_t* cu_seqlens, const int32_t* slots, float* out, int tokens,
                                int sequences, int heads, int groups, int dim, int vdim, int keep_state,
                                int run_len, int max_runs, float* scratch, float* logs,
                                cudaStream_t stream) {
  if (!takes(tokens, sequences, heads, dim, vdim, run_len, max_runs, scratch, logs) || groups <= 0 ||
      heads % groups)
    return cudaErrorInvalidValue;
  if (tokens == 0 || sequences == 0) return 0;
  const Runs r = {scratch, logs, nullptr, cu_seqlens, heads, dim, vdim, run_len, max_runs};
  const bool quads = multiples_of_4({stride, x_off, b_off, c_off, dim, vdim}) &&
                     !((uintptr_t)xbc & (c_dtype == SAKV_F32 ? 15 : 7));
#define SAKV_DUAL(C, QUADS)                                                                      \
  return launch_runs(DualSource<C, QUADS>{(const C*)xbc, stride, x_off, b_off, c_off, dt,        \
                                          dt_stride, dt_bias, a, d_skip, dim, vdim,              \
                                          heads / groups},                                       \
                     r, state, slots, out, sequences, keep_state, stream)
  if (c_dtype == SAKV_F32) {
    if (quads) SAKV_DUAL(float, true);
    SAKV_DUAL(float, false);
  }
  if (c_dtype == SAKV_BF16) {
    if (quads) SAKV_DUAL(__nv_bfloat16, true);
    SAKV_DUAL(__nv_bfloat16, false);
  }
#undef SAKV_DUAL
  return cudaErrorInvalidValue;
}
