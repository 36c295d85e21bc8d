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

// What is left over a run whose decays' logarithms add up to `log`: a state s becomes exp(log) s + left.
// Near 1 by its change, so that a decay keeps its distance from 1; where the run forgets, by the product: the
// change would take the state off itself, and half a unit of the last place of the OLD state stayed in the
// new one (s = 1e4, log = -18.4, left = 1e-2: 3 % of the new one).
struct Fade {
  bool change;
  float factor;
  __device__ __forceinline__ explicit Fade(float log)
      : change(log > -0.5f), factor(change ? expm1f(log) : expf(log)) {}
  __device__ __forceinline__ float carried(float s, float left) const {
    const float moved = fmaf(factor, s, left);
    return change ? s + moved : moved;
  }
};

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
