// The delta-rule recurrence with a decay and a removal rate for every key channel.
//
// For each head, with a state S of dim x dim (rows: key channels, columns: value channels)
// that is carried from token to token in fp32:
//
//   w = exp(-decay_scale * sigmoid(w0 + W2 tanh(l)))      l: the low-rank projection's output
//   a = sigmoid(a_pre + a_bias)
//   u = k / sqrt(sum(k^2) + key_eps)
//   S <- diag(w) S - (a * u)(u^T S) + k v^T                 (both terms read the old S)
//   o = S^T r;   out = o / sqrt(mean(o^2) + eps) * norm_w * sigmoid(g)
//
// Three kernels. `delta_prepare` works out what does not depend on the state, for all tokens
// side by side: w, u and a * u, fp32 [tokens, 3, heads * dim].
// `delta_scan` is the recurrence: a block has some neighbouring columns of one head's state
// for one sequence (columns never meet, so a head may be spread over several blocks when
// there are few heads and sequences) and walks the sequence's tokens of this step in chunks
// whose r, k, v, w, u, a * u are copied into shared memory one chunk ahead (cp.async, two
// buffers). The state is in registers: a column's rows are dealt to R neighbouring lanes, and
// the two sums over a column (u^T S and S^T r) are finished with shuffles among them.
// Block-wide barriers are paid per chunk, not per token. `delta_finish` norms and gates the
// raw outputs, a warp a token and head. The same kernels run a prompt, a piece of one and a
// single decoded token,
// and every sum has the same terms in the same order however the tokens are cut into steps
// and chunks, so a token's output does not depend on how the tokens came. r, k, v, g, a_pre
// and l are columns of one fp32 projection output [tokens, proj_stride].
#include "common.cuh"

namespace {

__device__ __forceinline__ float sigmoidf(float z) { return 1.f / (1.f + expf(-z)); }

constexpr int kPrepareThreads = 256;

// A warp's lanes share out a head's channels and a block takes `per_block` tokens: a channel's row of
// W2 (in shared memory) is read once for eight of them, whose factors lie side by side. 120 -> 87 us
// over 2,048 tokens of 32 heads of 64, rank 64 (with a warp a token every product read its weight
// and its factor from shared memory).
template <typename W>
__global__ void __launch_bounds__(kPrepareThreads)
delta_prepare_kernel(const float* __restrict__ proj, long long proj_stride, int off_k, int off_a,
                     int off_l, const W* __restrict__ w2, const W* __restrict__ w0,
                     const W* __restrict__ a_bias, float* __restrict__ prepared, int tokens,
                     int heads, int dim, int rank, int per_block, float decay_scale,
                     float key_eps) {
  extern __shared__ __align__(16) float shared[];
  float* s_l = shared;                              // [rank][tokens of the block]
  float* s_inv = s_l + rank * per_block;            // [tokens of the block]
  const int ld2 = rank + 1;                         // padded rows of W2: no bank conflicts
  float* s_w2 = s_inv + per_block;                  // [dim][rank + 1]
  let_next_kernel_start();
  const int head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kWarps = kPrepareThreads / 32;
  const int base = head * dim;
  for (int i = threadIdx.x; i < dim * rank; i += blockDim.x)
    s_w2[(i / rank) * ld2 + i % rank] = widen(w2[(long long)base * rank + i]);
  wait_for_previous_kernel();
  const long long t0 = (long long)blockIdx.x * per_block;
  const int count = tokens - t0 < per_block ? static_cast<int>(tokens - t0) : per_block;
  for (int i = threadIdx.x; i < per_block * rank; i += blockDim.x) {
    const int tt = i / rank, j = i - tt * rank;
    s_l[j * per_block + tt] = tt < count ? tanhf(proj[(t0 + tt) * proj_stride + off_l + j]) : 0.f;
  }
  for (int tt = warp; tt < count; tt += kWarps) {
    const float* row = proj + (t0 + tt) * proj_stride;
    float kk = 0.f;
    for (int c = lane; c < dim; c += 32) {
      const float k = row[off_k + base + c];
      kk = fmaf(k, k, kk);
    }
    kk = warp_sum(kk);
    if (lane == 0) s_inv[tt] = 1.f / sqrtf(kk + key_eps);
  }
  __syncthreads();
  const long long hd = (long long)heads * dim;
  constexpr int kTogether = 8;                      // (per_block is a multiple of it)
  const int runs = (dim + 31) / 32;                 // of 32 channels
  for (int job = warp; job < runs * (per_block / kTogether); job += kWarps) {
    const int c = job % runs * 32 + lane, tt0 = job / runs * kTogether;
    if (tt0 >= count || c >= dim) continue;
    float z[kTogether];
#pragma unroll
    for (int q = 0; q < kTogether; ++q) z[q] = widen(w0[base + c]);
    const float* w2row = s_w2 + c * ld2;
#pragma unroll 4
    for (int j = 0; j < rank; ++j) {
      const float w = w2row[j];
      const float4 l0 = *reinterpret_cast<const float4*>(s_l + j * per_block + tt0);
      const float4 l1 = *reinterpret_cast<const float4*>(s_l + j * per_block + tt0 + 4);
      z[0] = fmaf(w, l0.x, z[0]); z[1] = fmaf(w, l0.y, z[1]);
      z[2] = fmaf(w, l0.z, z[2]); z[3] = fmaf(w, l0.w, z[3]);
      z[4] = fmaf(w, l1.x, z[4]); z[5] = fmaf(w, l1.y, z[5]);
      z[6] = fmaf(w, l1.z, z[6]); z[7] = fmaf(w, l1.w, z[7]);
    }
    const float bias = widen(a_bias[base + c]);
    float k[kTogether], a[kTogether];
#pragma unroll
    for (int q = 0; q < kTogether; ++q) {           // (asked for together)
      const float* row = proj + (t0 + min(tt0 + q, count - 1)) * proj_stride + base + c;
      k[q] = row[off_k];
      a[q] = row[off_a];
    }
#pragma unroll
    for (int q = 0; q < kTogether; ++q) {
      if (tt0 + q >= count) break;
      float* dst = prepared + (t0 + tt0 + q) * 3 * hd + base;
      const float u = k[q] * s_inv[tt0 + q];
      dst[c] = expf(-decay_scale * sigmoidf(z[q]));
      dst[hd + c] = u;
      dst[2 * hd + c] = sigmoidf(a[q] + bias) * u;
    }
  }
}

template <int R>
__device__ __forceinline__ float sum_over_parts(float v) {
#pragma unroll
  for (int o = 1; o < R; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void copy16_async(float* dst, const float* src) {
  const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait_all_but_last() {
  asm volatile("cp.async.wait_group 1;" ::: "memory");
}

// Two fp32 numbers in one register pair, and the two-wide arithmetic on them.
typedef unsigned long long Two;
__device__ __forceinline__ Two two(float a, float b) {
  Two d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
  Two d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ Two mul2(Two a, Two b) {
  Two d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float both(Two v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}

constexpr size_t kScanBudget = 96 * 1024;      // shared memory of a scan's block
constexpr int kMostChunk = 16;                 // tokens that it takes at a time

// Bytes of two chunks of `n` tokens: five vectors in R parts of `rpt` rows, and `cols` values.
constexpr size_t scan_bytes(int n, int rpt, int R, int cols) {
  return (size_t)2 * n * (5 * R * (rpt + (R > 1 ? 4 : 0)) + cols) * sizeof(float);
}

// Tokens of a straight run in the WHOLE form: one a lane, four with 16 lanes. A chunk never holds 16 tokens
// of columns that long, and runs of the eight that it holds at 128 rows spill: 16 heads of 128,
// us, token by token / runs of 8 / of 4: 2,048 tokens 1,043 / 881 / 899, 8 sequences of 300 tokens 820 / 678 / 676,
// of 5 53 / 47 / 44; 8 heads of 256, 2,048 tokens 2,095 token by token, 1,477 in fours.
constexpr int scan_run(int R) { return R < 16 ? R : 4; }

// One block: `cols` neighbouring columns of one head's state for one sequence. A column's
// rows are dealt to R neighbouring lanes, dim / R <= RPT rows each. VEC: rows are read four
// at a time (dim / R a multiple of 4, everything 16-byte aligned); WHOLE: dim / R is RPT.
// The raw o = S^T r goes to `raw` [tokens, heads * dim] fp32 for `delta_finish`.
//
// What bounds it is the chain from token to token: the sum u^T S over a column's R lanes (a
// shuffle tree) and the update that waits for it. The WHOLE form keeps out of that chain what does
// not belong to it: `scan_run` tokens are one straight run of code,
// so that the next token's vectors can be read meanwhile; S is held in pairs for two-wide arithmetic;
// and the outputs' sums wait until a run's tokens have left theirs, when each lane finishes one token's
// (R - 1 exchanges instead of R log2 R in a run of R, the same tree of additions). One sequence of 2,048 tokens, 32 heads of 64, behind its
// prepare kernel: 842 us before, 373 now (of which the launch in plain order 206, see
// `launch_scan`). Tried and no faster (380 to 450): two columns a thread, bulk copies of the vectors
// (60 ns each), a copying warp of its own, vectors read by volatile loads a token ahead, 4 or 16
// lanes a column. Without its shuffles, copies and reads of shared memory, which lie in one chain
// each with the next, the bare arithmetic takes 118.
template <int RPT, int R, bool VEC, bool WHOLE>
__global__ void __launch_bounds__(512)
delta_scan_kernel(const float* __restrict__ proj, long long proj_stride, int off_r, int off_k,
                  int off_v, const float* __restrict__ prepared, float* __restrict__ state,
                  const int32_t* __restrict__ cu_seqlens, const int32_t* __restrict__ slots,
                  float* __restrict__ raw, int heads, int dim, int cols, int chunk,
                  int keep_state) {
  extern __shared__ __align__(16) float shared[];
  // a token's per-row vectors lie part by part with four floats between the parts, so that the
  // R lanes of a column read from different banks
  const int rpt = WHOLE ? RPT : dim / R;
  const int ldp = rpt + (R > 1 ? 4 : 0), ldt = R * ldp;      // a part's, a token's stride
  const int per_buffer = chunk * (5 * ldt + cols);
  let_next_kernel_start();
  const int head = blockIdx.x, seq = blockIdx.y, col0 = blockIdx.z * cols;
  const int tid = threadIdx.x, threads = blockDim.x;
  const int mycol = tid / R, part = tid % R, col = col0 + mycol;
  const bool mine = mycol < cols && col < dim;
  const int base = head * dim;
  const long long hd = (long long)heads * dim;
  wait_for_previous_kernel();
  const int begin = cu_seqlens[seq], end = cu_seqlens[seq + 1];
  float* my_state = state + (((long long)slots[seq] * heads + head) * dim + part * rpt) * dim + col;
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) S[i] = (mine && i < rpt) ? my_state[(long long)i * dim] : 0.f;
  Two S2[RPT / 2];                                 // (WHOLE: the same in pairs, instead of S)
#pragma unroll
  for (int i = 0; i < RPT / 2; ++i) S2[i] = two(S[2 * i], S[2 * i + 1]);

  const bool aligned = VEC && dim % 4 == 0 && cols % 4 == 0 && proj_stride % 4 == 0 &&
                       off_r % 4 == 0 && off_k % 4 == 0 && off_v % 4 == 0 &&
                       !((uintptr_t)proj & 15) && !((uintptr_t)prepared & 15);
  // the rows of a chunk: r, k (from proj) and w, u, a*u (prepared), part by part; then this
  // block's columns of v
  auto fetch = [&](int t0, int buffer) {
    const int count = min(chunk, end - t0);
    float* dst = shared + buffer * per_buffer;
    float* dst_v = dst + chunk * 5 * ldt;
    // (an item is four floats, or one, of one of the six vectors; its place in the token is
    // worked out once, then it is copied for every token of the chunk)
    if (aligned) {
      const int quads = dim / 4, vquads = cols / 4, per_token = 5 * quads + vquads;
      for (int j = tid; j < per_token; j += threads) {
        const float* src;
        float* to;
        long long src_step = proj_stride;
        int to_step = 5 * ldt;
        if (j >= 5 * quads) {
          const int c = (j - 5 * quads) * 4;
          src = proj + (long long)t0 * proj_stride + off_v + base + col0 + c;
          to = dst_v + c;
          to_step = cols;
        } else {
          const int which = j / quads, c = (j - which * quads) * 4;
          to = dst + which * ldt + (c / rpt) * ldp + c % rpt;
          if (which < 2) {
            src = proj + (long long)t0 * proj_stride + (which == 0 ? off_r : off_k) + base + c;
          } else {
            src = prepared + ((long long)t0 * 3 + (which - 2)) * hd + base + c;
            src_step = 3 * hd;
          }
        }
        for (int tt = 0; tt < count; ++tt) copy16_async(to + tt * to_step, src + tt * src_step);
      }
    } else {
      const int per_token = 5 * dim + cols;
      for (int j = tid; j < per_token; j += threads) {
        const float* src;
        float* to;
        long long src_step = proj_stride;
        int to_step = 5 * ldt;
        bool real = true;
        if (j >= 5 * dim) {
          const int c = j - 5 * dim;
          real = col0 + c < dim;
          src = proj + (long long)t0 * proj_stride + off_v + base + col0 + c;
          to = dst_v + c;
          to_step = cols;
        } else {
          const int which = j / dim, c = j - which * dim;
          to = dst + which * ldt + (c / rpt) * ldp + c % rpt;
          if (which < 2) {
            src = proj + (long long)t0 * proj_stride + (which == 0 ? off_r : off_k) + base + c;
          } else {
            src = prepared + ((long long)t0 * 3 + (which - 2)) * hd + base + c;
            src_step = 3 * hd;
          }
        }
        for (int tt = 0; tt < count; ++tt) to[tt * to_step] = real ? src[tt * src_step] : 0.f;
      }
    }
    copies_commit();
  };

  int buffer = 0;
  if (begin < end) fetch(begin, 0);
  for (int t0 = begin; t0 < end; t0 += chunk, buffer ^= 1) {
    const int count = min(chunk, end - t0);
    if (t0 + chunk < end) fetch(t0 + chunk, buffer ^ 1);
    else copies_commit();
    copies_wait_all_but_last();
    __syncthreads();                                 // the chunk has landed, for everyone
    const float* rows = shared + buffer * per_buffer + part * ldp;
    const float* vals = shared + buffer * per_buffer + chunk * 5 * ldt + (mine ? mycol : 0);
    if constexpr (WHOLE) {
      // a token: the lane's share of its o, before the sum over the lanes
      auto token = [&](int tt) {
        const float* x = rows + tt * 5 * ldt;
        Two r[RPT / 2], k[RPT / 2], w[RPT / 2], u[RPT / 2], b[RPT / 2];
        auto read = [&](Two (&to)[RPT / 2], const float* from) {
#pragma unroll
          for (int i = 0; i < RPT / 2; i += 2) {
            const ulonglong2 got = *reinterpret_cast<const ulonglong2*>(from + 2 * i);
            to[i] = got.x;
            to[i + 1] = got.y;
          }
        };
        read(u, x + 3 * ldt);
        read(b, x + 4 * ldt);
        read(k, x + ldt);
        read(w, x + 2 * ldt);
        read(r, x);
        const float v = vals[tt * cols];
        Two sum = mul2(u[0], S2[0]);
#pragma unroll
        for (int i = 1; i < RPT / 2; ++i) sum = fma2(u[i], S2[i], sum);
        const float sa = sum_over_parts<R>(both(sum));
        const Two taken = two(-sa, -sa), put = two(v, v);
        Two o = two(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < RPT / 2; ++i) {
          S2[i] = fma2(w[i], S2[i], fma2(b[i], taken, mul2(k[i], put)));
          o = fma2(S2[i], r[i], o);
        }
        return both(o);
      };
      constexpr int kRun = scan_run(R);
      static_assert(kRun > 1 && scan_bytes(kRun, RPT, R, 512 / R) <= kScanBudget, "a chunk holds a run");
      int tt = 0;
      for (; tt + kRun <= count; tt += kRun) {
        float o[kRun];
#pragma unroll
        for (int q = 0; q < kRun; ++q) o[q] = token(tt + q);
#pragma unroll
        for (int step = 1, n = kRun / 2; step < kRun; step <<= 1, n >>= 1) {
          const bool odd = (part & step) != 0;
#pragma unroll
          for (int i = 0; i < kRun / 2; ++i)
            if (i < n) {
              const float keep = odd ? o[2 * i + 1] : o[2 * i], give = odd ? o[2 * i] : o[2 * i + 1];
              o[i] = keep + __shfl_xor_sync(0xffffffffu, give, step);
            }
        }
#pragma unroll
        for (int step = kRun; step < R; step <<= 1) o[0] += __shfl_xor_sync(0xffffffffu, o[0], step);
        if (mine && part < kRun) raw[(long long)(t0 + tt + part) * hd + base + col] = o[0];
      }
      for (; tt < count; ++tt) {
        const float o = sum_over_parts<R>(token(tt));
        if (mine && part == 0) raw[(long long)(t0 + tt) * hd + base + col] = o;
      }
    }
    for (int tt = 0; !WHOLE && tt < count; ++tt) {   // the recurrence
      const float* x = rows + tt * 5 * ldt;          // r, k, w, u, a*u: ldt apart
      const float v = vals[tt * cols];
      float sa = 0.f, o = 0.f;
      if constexpr (VEC) {
        float r[RPT], k[RPT], w[RPT], u[RPT], b[RPT];
#pragma unroll
        for (int i = 0; i < RPT; i += 4)
          if (i < rpt) {
            *reinterpret_cast<float4*>(u + i) = *reinterpret_cast<const float4*>(x + 3 * ldt + i);
            *reinterpret_cast<float4*>(r + i) = *reinterpret_cast<const float4*>(x + i);
            *reinterpret_cast<float4*>(k + i) = *reinterpret_cast<const float4*>(x + ldt + i);
            *reinterpret_cast<float4*>(w + i) = *reinterpret_cast<const float4*>(x + 2 * ldt + i);
            *reinterpret_cast<float4*>(b + i) = *reinterpret_cast<const float4*>(x + 4 * ldt + i);
          }
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i < rpt) sa = fmaf(u[i], S[i], sa);
        sa = sum_over_parts<R>(sa);
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i < rpt) {
            S[i] = fmaf(w[i], S[i], fmaf(-b[i], sa, k[i] * v));
            o = fmaf(S[i], r[i], o);
          }
      } else {
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i < rpt) sa = fmaf(x[3 * ldt + i], S[i], sa);
        sa = sum_over_parts<R>(sa);
#pragma unroll
        for (int i = 0; i < RPT; ++i)
          if (i < rpt) {
            S[i] = fmaf(x[2 * ldt + i], S[i], fmaf(-x[4 * ldt + i], sa, x[ldt + i] * v));
            o = fmaf(S[i], x[i], o);
          }
      }
      o = sum_over_parts<R>(o);
      if (mine && part == 0) raw[(long long)(t0 + tt) * hd + base + col] = o;
    }
    __syncthreads();                                 // everyone is done with this buffer
  }
  if constexpr (WHOLE) {
#pragma unroll
    for (int i = 0; i < RPT / 2; ++i)
      asm("mov.b64 {%0, %1}, %2;" : "=f"(S[2 * i]), "=f"(S[2 * i + 1]) : "l"(S2[i]));
  }
  if (keep_state && mine) {
#pragma unroll
    for (int i = 0; i < RPT; ++i)
      if (i < rpt) my_state[(long long)i * dim] = S[i];
  }
}

// out = raw / sqrt(mean(raw^2) + eps) * norm_w * sigmoid(g), head by head: a warp for each
// (token, head).
template <typename W, typename Out>
__global__ void delta_finish_kernel(const float* __restrict__ raw, const float* __restrict__ proj,
                                    long long proj_stride, int off_g,
                                    const W* __restrict__ norm_w, Out* __restrict__ out,
                                    long long items, int heads, int dim, float eps) {
  let_next_kernel_start();
  wait_for_previous_kernel();
  const long long item = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (item >= items) return;
  const long long t = item / heads;
  const int base = static_cast<int>(item - t * heads) * dim;
  const float* o = raw + t * heads * dim + base;
  float oo = 0.f;
  for (int c = lane; c < dim; c += 32) oo = fmaf(o[c], o[c], oo);
  const float inv = 1.f / sqrtf(warp_sum(oo) / (float)dim + eps);
  for (int c = lane; c < dim; c += 32)
    out[t * heads * dim + base + c] = narrow<Out>(
        o[c] * inv * widen(norm_w[base + c]) * sigmoidf(proj[t * proj_stride + off_g + base + c]));
}

template <int RPT, int R, bool VEC, bool WHOLE>
int launch_scan(const float* proj, long long proj_stride, const int* off, const float* prepared,
                float* state, const int32_t* cu_seqlens, const int32_t* slots, float* raw,
                int sequences, int heads, int dim, int chunk, int keep_state,
                cudaStream_t stream) {
  // columns a block: few enough that the blocks fill the GPU, at least 128 threads' worth
  int cols = dim;
  if (VEC) {
    const int least = 128 / R > 4 ? 128 / R : 4;
    while (cols % 8 == 0 && cols / 2 >= least &&
           (long long)heads * sequences * (dim / cols) * 2 <= sm_count() * 2)
      cols /= 2;
    while (cols * R > 512 && cols % 8 == 0) cols /= 2;
  }
  if (cols * R > 512) return cudaErrorInvalidValue;
  auto bytes = [&](int n) { return scan_bytes(n, dim / R, R, cols); };
  const bool prompt = chunk >= 8;            // (what a sequence brings, not what fits)
  if (chunk < 1) chunk = 1;
  if (chunk > kMostChunk) chunk = kMostChunk;
  while (chunk > 1 && bytes(chunk) > kScanBudget) chunk /= 2;
  if (bytes(chunk) > kScanBudget) return cudaErrorInvalidValue;
  const int threads = ((cols * R + 31) / 32) * 32;
  static PerDeviceOnce configured;
  auto kernel = delta_scan_kernel<RPT, R, VEC, WHOLE>;
  if (configured.needs()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kScanBudget);
    if (e != cudaSuccess) return (int)e;
    configured.done();
  }
  // A prompt's blocks begin when the kernel before them has left the SMs, so that each finds one
  // of its own: begun while it drains, two or three of them share an SM, and the longest decides
  // (2,048 tokens, 32 heads of 64: 585 us a scan behind its prepare kernel, 379 in plain order).
  // For a few tokens the early start is worth more.
  const dim3 grid(heads, sequences, (dim + cols - 1) / cols);
  if (prompt)
    return launch_ordered(kernel, grid, dim3(threads), bytes(chunk), stream, proj, proj_stride, off[0],
                          off[1], off[2], prepared, state, cu_seqlens, slots, raw, heads, dim, cols,
                          chunk, keep_state);
  return launch_overlapped(kernel, grid, dim3(threads), bytes(chunk), stream, 1, proj, proj_stride,
                           off[0], off[1], off[2], prepared, state, cu_seqlens, slots, raw, heads, dim,
                           cols, chunk, keep_state);
}

int pick_scan(const float* proj, long long proj_stride, const int* off, const float* prepared,
              float* state, const int32_t* cu_seqlens, const int32_t* slots, float* raw,
              int sequences, int heads, int dim, int chunk, int keep_state, cudaStream_t stream) {
#define SAKV_SCAN_AS(RPT, R, VEC, WHOLE)                                                        \
  return launch_scan<RPT, R, VEC, WHOLE>(proj, proj_stride, off, prepared, state, cu_seqlens,   \
                                         slots, raw, sequences, heads, dim, chunk, keep_state,  \
                                         stream)
#define SAKV_SCAN(RPT, R, VEC) SAKV_SCAN_AS(RPT, R, VEC, false)
#define SAKV_SCAN_WHOLE(RPT, R)                                \
  do {                                                         \
    if (dim == RPT * R) SAKV_SCAN_AS(RPT, R, true, true);      \
    SAKV_SCAN_AS(RPT, R, true, false);                         \
  } while (0)
  // a column's rows over R lanes, four rows at a time: the most lanes (up to 16) that leave
  // a lane 8 rows, or 4 where dim is small; dims that 16 does not divide: one lane a column
  if (dim % 16 == 0) {
    int lanes = 4;
    while (lanes < 16 && dim % (8 * lanes) == 0 && dim / (2 * lanes) >= 8) lanes *= 2;
    const int rpt = dim / lanes;
    if (lanes == 4 && rpt <= 4) SAKV_SCAN_WHOLE(4, 4);
    if (lanes == 4 && rpt <= 8) SAKV_SCAN_WHOLE(8, 4);
    if (lanes == 4 && rpt <= 16) SAKV_SCAN(16, 4, true);
    if (lanes == 8 && rpt <= 8) SAKV_SCAN_WHOLE(8, 8);
    if (lanes == 8 && rpt <= 16) SAKV_SCAN(16, 8, true);
    if (lanes == 16 && rpt <= 8) SAKV_SCAN_WHOLE(8, 16);
    if (lanes == 16 && rpt <= 16) SAKV_SCAN_WHOLE(16, 16);
  }
  if (dim <= 32) SAKV_SCAN(32, 1, false);
  if (dim <= 64) SAKV_SCAN(64, 1, false);
  if (dim <= 128) SAKV_SCAN(128, 1, false);
  SAKV_SCAN(256, 1, false);
#undef SAKV_SCAN
#undef SAKV_SCAN_WHOLE
#undef SAKV_SCAN_AS
}

template <typename W>
int run(const float* proj, long long proj_stride, const int* off, const void* w2, const void* w0,
        const void* a_bias, const void* norm_w, float* prepared, float* raw, float* state,
        const int32_t* cu_seqlens, const int32_t* slots, void* out, int out_dtype, int tokens,
        int sequences, int heads, int dim, int rank, int chunk, float decay_scale, float key_eps,
        float eps, int keep_state, cudaStream_t stream) {
  constexpr size_t kPrepareBudget = 227 * 1024;
  // tokens of a block of `delta_prepare`: 32, fewer where there are few or the weights leave no room
  auto prepare_bytes = [&](int n) { return (size_t)(dim + n) * (rank + 1) * sizeof(float); };
  int per_block = 32;
  while (per_block > 8 && (per_block / 2 >= tokens || prepare_bytes(per_block) > kPrepareBudget))
    per_block /= 2;
  const size_t smem = prepare_bytes(per_block);
  if (smem > kPrepareBudget) return cudaErrorInvalidValue;
  static PerDeviceOnce configured;
  if (configured.needs()) {
    const cudaError_t e = cudaFuncSetAttribute(delta_prepare_kernel<W>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kPrepareBudget);
    if (e != cudaSuccess) return (int)e;
    configured.done();
  }
  int code = launch_overlapped(
      delta_prepare_kernel<W>, dim3((tokens + per_block - 1) / per_block, heads),
      dim3(kPrepareThreads), smem, stream, 1, proj, proj_stride, off[1], off[4], off[5],
      (const W*)w2, (const W*)w0, (const W*)a_bias, prepared, tokens, heads, dim, rank,
      per_block, decay_scale, key_eps);
  if (code != 0) return code;
  code = pick_scan(proj, proj_stride, off, prepared, state, cu_seqlens, slots, raw, sequences,
                   heads, dim, chunk, keep_state, stream);
  if (code != 0) return code;
  const long long items = (long long)tokens * heads;
  const long long blocks = (items * 32 + 255) / 256;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  if (out_dtype == SAKV_F32)
    return launch_overlapped(delta_finish_kernel<W, float>, dim3((unsigned)blocks), dim3(256), 0,
                             stream, 1, (const float*)raw, proj, proj_stride, off[3],
                             (const W*)norm_w, (float*)out, items, heads, dim, eps);
  if (out_dtype == SAKV_BF16)
    return launch_overlapped(delta_finish_kernel<W, __nv_bfloat16>, dim3((unsigned)blocks),
                             dim3(256), 0, stream, 1, (const float*)raw, proj, proj_stride, off[3],
                             (const W*)norm_w, (__nv_bfloat16*)out, items, heads, dim, eps);
  return cudaErrorInvalidValue;
}

}  // namespace

// proj: fp32 [tokens, proj_stride]; the first columns of r, k, v, g, a_pre (each heads * dim
// wide) and of l (rank wide) are given. w2 [heads * dim, rank], w0, a_bias, norm_w [heads *
// dim] of type `w_dtype`. prepared, raw: fp32 scratch [tokens, 3, heads * dim] and [tokens,
// heads * dim]. state: fp32 [slots,
// heads, dim, dim]. out: [tokens, heads * dim] of `out_dtype`. Sequence i of the step owns the
// tokens cu_seqlens[i] .. cu_seqlens[i + 1] - 1 and the state of slot slots[i]. `chunk`: how
// many tokens a block takes into shared memory at a time (the most a sequence brings in this
// step is enough; at most 16).
SAKV_EXPORT int sakv_delta_rule(const float* proj, long long proj_stride, int off_r, int off_k,
                                int off_v, int off_g, int off_a, int off_l, const void* w2,
                                const void* w0, const void* a_bias, const void* norm_w,
                                int w_dtype, float* prepared, float* raw, float* state,
                                const int32_t* cu_seqlens, const int32_t* slots, void* out,
                                int out_dtype, int tokens, int sequences, int heads, int dim,
                                int rank, int chunk, float decay_scale, float key_eps, float eps,
                                int keep_state, cudaStream_t stream) {
  if (tokens < 0 || sequences < 0 || heads <= 0 || heads > 65535 || dim <= 0 || dim > 256 ||
      rank <= 0 || sequences > 65535)
    return cudaErrorInvalidValue;
  if (sequences == 0 || tokens == 0) return 0;
  const int off[6] = {off_r, off_k, off_v, off_g, off_a, off_l};
  if (w_dtype == SAKV_F32)
    return run<float>(proj, proj_stride, off, w2, w0, a_bias, norm_w, prepared, raw, state,
                      cu_seqlens, slots, out, out_dtype, tokens, sequences, heads, dim, rank, chunk,
                      decay_scale, key_eps, eps, keep_state, stream);
  if (w_dtype == SAKV_BF16)
    return run<__nv_bfloat16>(proj, proj_stride, off, w2, w0, a_bias, norm_w, prepared, raw,
                              state, cu_seqlens, slots, out, out_dtype, tokens, sequences, heads, dim,
                              rank, chunk, decay_scale, key_eps, eps, keep_state, stream);
  return cudaErrorInvalidValue;
}
