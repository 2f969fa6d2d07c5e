// Activations of the GEMM epilogues (NFK_ACT_*, NFK_LIN_*), shared by the dense and the grouped products.
#pragma once
#include "kernels.h"

namespace nf {

struct GatedAct {
  int kind;
  float limit, alpha, shift;
};

template <bool PRECISE>
__device__ __forceinline__ float gated_act_of(float g, float u, const GatedAct& a) {
  if (a.kind == NFK_ACT_RELU) return fmaxf(g, 0.f) * u;
  if (a.kind == NFK_ACT_GELU_TANH) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
  if (a.kind == NFK_ACT_CAPPED) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
    const float z = -a.alpha * g;
    return g / (1.f + (PRECISE ? expf(z) : __expf(z))) * (u + a.shift);
  }
  return g / (1.f + (PRECISE ? expf(-g) : __expf(-g))) * u;
}

// x sigmoid(z). A division per element is a chain of some 300 cycles in which the compiler cannot interleave elements (its
// slow path is a branch): 128 x 128 gated outputs of a CTA took 22 us to leave tensor memory. Here the quotient q = x r with
// r ~ 1/d is corrected once by its remainder x - d q (Markstein's step), which leaves it within an ulp of the division and
// has no branch, so the elements' chains overlap. Where the remainder is no number (d or x infinite), q is what counts.
__device__ __forceinline__ float mul_sigmoid(float x, float z) {
  const float d = 1.f + __expf(-z);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = x * r, rest = fmaf(-d, q, x);
  return fabsf(rest) <= 3.402823466e38f ? fmaf(r, rest, q) : q;
}

// g[j] = act(g[j], u[j]): the kind is looked at once, not per element.
template <int N>
__device__ __forceinline__ void gated_acts(float* g, const float* u, const GatedAct& a) {
  if (a.kind == NFK_ACT_SILU) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = mul_sigmoid(g[j], g[j]) * u[j];
  } else if (a.kind == NFK_ACT_CAPPED) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float x = fminf(g[j], a.limit);
      g[j] = mul_sigmoid(x, a.alpha * x) * (fminf(fmaxf(u[j], -a.limit), a.limit) + a.shift);
    }
  } else if (a.kind == NFK_ACT_RELU) {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = fmaxf(g[j], 0.f) * u[j];
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) g[j] = gated_act_of<false>(g[j], u[j], GatedAct{NFK_ACT_GELU_TANH, 0.f, 0.f, 0.f});
  }
}

__device__ __forceinline__ float lin_act_of(float v, int kind) {
  if (kind == NFK_LIN_TANH) return tanhf(v);
  if (kind == NFK_LIN_GELU) return 0.5f * v * (1.f + erff(v * 0.7071067811865476f));
  if (kind == NFK_LIN_RELU2) {
    const float r = fmaxf(v, 0.f);
    return r * r;
  }
  return v;
}

}  // namespace nf
