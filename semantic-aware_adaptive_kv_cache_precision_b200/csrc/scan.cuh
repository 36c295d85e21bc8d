// Pieces shared by the kernels of the recurrent mixers: activations, what shapes q, k and v of the
// fading state on their way in, and two-wide arithmetic.
#pragma once

#include "common.cuh"

namespace scan {

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// `act` 1 is silu of each element (0: as projected); `rot` > 0 turns the first `rot` numbers of
// every head of q and k by the token's position (pairs (i, i + rot / 2), tables [positions, rot / 2]
// that carry the rotation's magnitude), after the activation; `k_scale` multiplies k after that.
struct FadeInput {
  int act;
  int rot;
  const int32_t* positions;
  const float* cos_t;
  const float* sin_t;
  float k_scale;
};

__device__ __forceinline__ float fade_act(float x, int act) { return act ? silu(x) : x; }

// Two fp32 numbers in one register pair, for the two-wide arithmetic of sm_100.
using Two = unsigned long long;
__device__ __forceinline__ Two two(float x, float y) {
  Two d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 apart(Two v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
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
__device__ __forceinline__ Two add2(Two a, Two b) {
  Two d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

}  // namespace scan
