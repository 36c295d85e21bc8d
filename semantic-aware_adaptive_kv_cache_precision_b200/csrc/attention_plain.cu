// The plain attention kernel: one warp for each (token, query head), every key
// of the cache taken one after the other with a running maximum and sum.
//
//   s_j = (q * scale) . k_j      for the keys j the query may see: j <= pos, and
//                                 pos - j < window where the layer has a window
//   out = sum_j exp(s_j - m) v_j / sum_j exp(s_j - m)
//
// q * scale, the scores, exp, the sums and the output are fp32; k and v are
// widened from their stored type (`src/core_kernels/attention.cu:541-657`).
// Keys are visited in the order of their positions, so the result for a token
// is the same to the bit whether the token came in a whole prompt, alone in a
// decode step or beside other sequences in a batch. It serves the fp32 path for
// prefill and for decode, and is what the tensor-core kernels are tested
// against.
//
// Keys and values of cache entry: [block, kv_head, 64, head_dim]; a sequence's
// blocks are block_table[seq, :]. Queries are read from the fused projection
// buffer with row stride `q_stride`; the output is [token, heads * head_dim].
#include "common.cuh"

namespace {

constexpr int kMaxPerLane = 8;  // head_dim <= 256
constexpr int kTogether = 8;    // keys taken at a time

// A warp a (token, head). Bound by the chain from key to key (a trip to memory, a sum over the lanes,
// the running maximum): keys are taken eight at a time, from multiples of eight on, so their rows
// and their values' rows are asked for together, their scores are summed side by side and the
// maximum moves once for the eight. PER: elements a lane.
template <typename T, int PER>
__global__ void __launch_bounds__(128)
attention_plain_kernel(const T* __restrict__ q, long long q_stride, T* __restrict__ out,
                       const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                       const int32_t* __restrict__ positions,
                       const int32_t* __restrict__ token_seq,
                       const int32_t* __restrict__ block_table, int max_blocks, int tokens,
                       int heads, int kv_heads, int head_dim, float scale, int window) {
  const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= (long long)tokens * heads) return;
  const int t = static_cast<int>(warp / heads);
  const int h = static_cast<int>(warp - (long long)t * heads);
  const int g = h / (heads / kv_heads);
  const int pos = positions[t];
  const int32_t* table = block_table + (long long)token_seq[t] * max_blocks;

  float qr[PER], acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    qr[i] = e < head_dim ? widen(q[(long long)t * q_stride + (long long)h * head_dim + e]) * scale : 0.f;
    acc[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int first = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  for (int j0 = first / kTogether * kTogether; j0 <= pos; j0 += kTogether) {
    const int block = table[j0 / kCacheBlock];
    const long long base =
        (((long long)block * kv_heads + g) * kCacheBlock + j0 % kCacheBlock) * head_dim + lane;
    float k[kTogether][PER], v[kTogether][PER], s[kTogether];
#pragma unroll
    for (int n = 0; n < kTogether; ++n) {
      const bool seen = j0 + n >= first && j0 + n <= pos;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const bool real = seen && lane + 32 * i < head_dim;
        k[n][i] = real ? widen(k_cache[base + (long long)n * head_dim + 32 * i]) : 0.f;
        v[n][i] = real ? widen(v_cache[base + (long long)n * head_dim + 32 * i]) : 0.f;
      }
    }
#pragma unroll
    for (int n = 0; n < kTogether; ++n) {
      s[n] = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) s[n] += qr[i] * k[n][i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int n = 0; n < kTogether; ++n) s[n] += __shfl_xor_sync(0xffffffffu, s[n], o);
    float m_new = m;
#pragma unroll
    for (int n = 0; n < kTogether; ++n)
      if (j0 + n >= first && j0 + n <= pos) m_new = fmaxf(m_new, s[n]);
    const float corr = expf(m - m_new);
    l *= corr;
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] *= corr;
#pragma unroll
    for (int n = 0; n < kTogether; ++n) {
      if (j0 + n < first || j0 + n > pos) continue;
      const float p = expf(s[n] - m_new);
      l += p;
#pragma unroll
      for (int i = 0; i < PER; ++i) acc[i] = acc[i] + p * v[n][i];
    }
    m = m_new;
  }
  const float inv = 1.f / l;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    if (e < head_dim) out[((long long)t * heads + h) * head_dim + e] = narrow<T>(acc[i] * inv);
  }
}

template <typename T>
int launch_plain(const void* q, long long q_stride, void* out, const void* k_cache,
                 const void* v_cache, const int32_t* positions, const int32_t* token_seq,
                 const int32_t* block_table, int max_blocks, int tokens, int heads, int kv_heads,
                 int head_dim, float scale, int window, cudaStream_t stream) {
  const int threads = 128;
  const long long warps = (long long)tokens * heads;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
#define SAKV_PLAIN(PER)                                                                           \
  attention_plain_kernel<T, PER><<<(unsigned)blocks, threads, 0, stream>>>(                       \
      (const T*)q, q_stride, (T*)out, (const T*)k_cache, (const T*)v_cache, positions, token_seq, \
      block_table, max_blocks, tokens, heads, kv_heads, head_dim, scale, window)
  if (head_dim <= 32) SAKV_PLAIN(1);
  else if (head_dim <= 64) SAKV_PLAIN(2);
  else if (head_dim <= 128) SAKV_PLAIN(4);
  else SAKV_PLAIN(8);
#undef SAKV_PLAIN
  return launch_status();
}

}  // namespace

SAKV_EXPORT int sakv_attention_plain(const void* q, int dtype, long long q_stride, void* out,
                                     const void* k_cache, const void* v_cache,
                                     const int32_t* positions, const int32_t* token_seq,
                                     const int32_t* block_table, int max_blocks, int tokens,
                                     int heads, int kv_heads, int head_dim, float scale, int window,
                                     cudaStream_t stream) {
  if (tokens < 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || head_dim <= 0 ||
      head_dim > 32 * kMaxPerLane || max_blocks <= 0)
    return cudaErrorInvalidValue;
  if (tokens == 0) return 0;
  if (dtype == SAKV_F32)
    return launch_plain<float>(q, q_stride, out, k_cache, v_cache, positions, token_seq, block_table,
                               max_blocks, tokens, heads, kv_heads, head_dim, scale, window, stream);
  if (dtype == SAKV_BF16)
    return launch_plain<__nv_bfloat16>(q, q_stride, out, k_cache, v_cache, positions, token_seq,
                                       block_table, max_blocks, tokens, heads, kv_heads, head_dim,
                                       scale, window, stream);
  return cudaErrorInvalidValue;
}
