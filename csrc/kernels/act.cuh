// Activation functions and their derivatives, shared by the GEMM epilogues and the standalone
// elementwise kernels. Semantics follow machine_learning/src/arch/layers/{relu,sigmoid,tanh}.rs of
// the reference: derivatives are expressed in terms of the stored *activation* a (not the
// pre-activation), except GELU (not in the reference) whose derivative needs the pre-activation z.
#pragma once
#include <cuda_runtime.h>

namespace ono {

enum ActKind : int { ACT_NONE = 0, ACT_RELU = 1, ACT_SIGMOID = 2, ACT_TANH = 3, ACT_GELU = 4 };

// GELU's derivative Phi(x) + x phi(x) without a branch, so that the values of a group overlap in the pipeline (erff has two sides, and
// a warp walks both). The tail is taken in the form of C. Hastings (Approximations for Digital Computers, 1955), exp(-x^2/2) times a
// polynomial in 1 / (1 + p |x|), here around its value at zero: Phi(-z) = exp(-z^2/2) (1/2 - z w(t)), t = 1 / (1 + 0.3 z), w of degree 5
// fitted to the exact ratio for the smallest largest error of Phi (2.2e-9 before rounding); x phi(x) adds 0.39894 to w. Error against 64
// bits, relative in the 2-norm, of N(0, 0.3), N(0, 1), N(0, 3): 3.8e-8, 3.5e-8, 3.4e-8 (with erff and expf 3.8e-8, 3.9e-8, 4.1e-8); the
// activation itself has no such margin near zero and stays with erff. 512 x 8192 x 8192 bf16 with it in the epilogue: 66.4 -> 62.1 us.
__host__ __device__ __forceinline__ float gelu_slope(float x) {
  const float z = fminf(fabsf(x), 1e4f);      // (finite, so that the tail of an infinite x is zero)
#ifdef __CUDA_ARCH__
  const float t = __fdividef(1.0f, fmaf(0.3f, z, 1.0f));
#else
  const float t = 1.0f / fmaf(0.3f, z, 1.0f);
#endif
  float w = fmaf(-0.051896318793296814f, t, 0.19135144352912903f);
  w = fmaf(w, t, -0.05476323515176773f);
  w = fmaf(w, t, 0.17923074960708618f);
  w = fmaf(w, t, 0.1332300901412964f);
  w = fmaf(w, t, 0.4007317125797272f);
  const float r = fmaf(-z, w, 0.5f), e = expf(-0.5f * x * x);
  return x > 0.0f ? fmaf(-e, r, 1.0f) : e * r;
}

__host__ __device__ __forceinline__ float act_fwd(int kind, float param, float x) {
  switch (kind) {
    case ACT_RELU: {
      // relu.rs:30-32: max(x, slope*x)
      float sx = param * x;
      return x > sx ? x : sx;
    }
    case ACT_SIGMOID:
      return param / (1.0f + expf(-x));  // sigmoid.rs:28-36
    case ACT_TANH:
      return param * tanhf(x);  // tanh.rs:28-38
    case ACT_GELU:
      return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
    default:
      return x;
  }
}

// d * act'(.) given the stored value s (activation a; for GELU the pre-activation z).
// relu_quirk reproduces relu.rs:41-45, which overwrites d with slope*a where a <= 0.
__host__ __device__ __forceinline__ float act_bwd(int kind, float param, int relu_quirk, float s,
                                                  float d) {
  switch (kind) {
    case ACT_RELU:
      if (s > 0.0f) return d;
      return relu_quirk ? param * s : param * d;
    case ACT_SIGMOID:
      return d * s * (1.0f - s / param);  // sigmoid.rs:38-49
    case ACT_TANH:
      return d * (param - s * s / param);  // tanh.rs:40-51
    case ACT_GELU:
      return d * gelu_slope(s);
    default:
      return d;
  }
}

// N values, the kind chosen once: chosen value by value, unrolled, the code of every kind is walked around for each.
template <int N>
__device__ __forceinline__ void act_fwd_n(int kind, float param, float (&v)[N]) {
  switch (kind) {
    case ACT_RELU:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_fwd(ACT_RELU, param, v[k]);
      break;
    case ACT_SIGMOID:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_fwd(ACT_SIGMOID, param, v[k]);
      break;
    case ACT_TANH:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_fwd(ACT_TANH, param, v[k]);
      break;
    case ACT_GELU:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_fwd(ACT_GELU, param, v[k]);
      break;
    default: break;
  }
}

// N gradients through the derivative, likewise.
template <int N>
__device__ __forceinline__ void act_bwd_n(int kind, float param, int relu_quirk, const float (&s)[N], float (&v)[N]) {
  switch (kind) {
    case ACT_RELU:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_bwd(ACT_RELU, param, relu_quirk, s[k], v[k]);
      break;
    case ACT_SIGMOID:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_bwd(ACT_SIGMOID, param, relu_quirk, s[k], v[k]);
      break;
    case ACT_TANH:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_bwd(ACT_TANH, param, relu_quirk, s[k], v[k]);
      break;
    case ACT_GELU:
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = act_bwd(ACT_GELU, param, relu_quirk, s[k], v[k]);
      break;
    default: break;
  }
}

}  // namespace ono
