// One row of a loss, by a warp: softmax where it is fused, the loss, whether the largest output is the largest label, and the gradient
// with respect to the last layer's pre-activation. Reference semantics: machine_learning/src/arch/loss/{mse,cross_entropy}.rs,
// arch/layers/softmax.rs.
#pragma once
#include <cuda_runtime.h>

#include "act.cuh"
#include "ono_kernels.h"

namespace ono {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct LossRow {
  float loss;         // not yet divided by B * C
  int correct;
};

// a, y, aux (null: the outputs themselves): the row's outputs, labels and what act' is evaluated on. `put(j, p, d)` gets every output and
// gradient. NV > 0: a lane keeps its values in registers, NV of each (at least ceil(C / 32)); otherwise they are read again on every
// pass, NV < 0: with `ex` (shared memory, may be `a`) holding the exponentials. The additions are in the same order in every form.
template <int NV, class Put>
__device__ __forceinline__ LossRow loss_row(const OnoLoss& l, const float* a, const float* y, const float* aux, float* ex, int lane, Put put) {
  constexpr int R = NV > 0 ? NV : 1;
  const float inv_n = 1.0f / ((float)l.B * (float)l.C);
  float pr[R], yr[R];
  if (NV > 0) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int j = lane + 32 * i;
      pr[i] = j < l.C ? a[j] : -INFINITY;
      yr[i] = j < l.C ? y[j] : 0.0f;
    }
  }
  float mx = -INFINITY, inv_z = 1.0f;
  if (l.softmax) {
    if (NV > 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) mx = fmaxf(mx, pr[i]);
    } else {
      for (int j = lane; j < l.C; j += 32) mx = fmaxf(mx, a[j]);
    }
    mx = warp_max(mx);
    float z = 0.0f;
    if (NV > 0) {
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (lane + 32 * i < l.C) { pr[i] = expf(pr[i] - mx); z += pr[i]; }
    } else {
      for (int j = lane; j < l.C; j += 32) {
        const float e = expf(a[j] - mx);
        if (NV < 0) ex[j] = e;
        z += e;
      }
    }
    inv_z = 1.0f / warp_sum(z);
    if (NV > 0) {
#pragma unroll
      for (int i = 0; i < R; ++i) pr[i] *= inv_z;
    }
  }
  // pass 1: loss, dot = sum_k p_k g_k, argmax bookkeeping
  float loss = 0.0f, dot = 0.0f;
  float best_p = -INFINITY, best_y = -INFINITY;
  int arg_p = 0, arg_y = 0;
  auto first = [&](int j, float p, float yt) {
    float g;
    if (l.kind == 1) {
      g = -0.0f;
      const float ps = fmaxf(p, l.eps);
      if (yt != 0.0f || isinf(p) || !(ps > 0.0f)) {      // most labels of a row are zero: no logarithm and no division for those
        loss -= yt * logf(ps);
        g = -(yt / ps) * inv_n;
      }
    } else {
      const float diff = p - yt;
      loss += diff * diff;
      g = 2.0f * diff * inv_n;
    }
    dot += p * g;
    if (p > best_p) { best_p = p; arg_p = j; }
    if (yt > best_y) { best_y = yt; arg_y = j; }
  };
  if (NV > 0) {
#pragma unroll
    for (int i = 0; i < R; ++i) if (lane + 32 * i < l.C) first(lane + 32 * i, pr[i], yr[i]);
  } else {
    for (int j = lane; j < l.C; j += 32) first(j, l.softmax ? (NV < 0 ? ex[j] : expf(a[j] - mx)) * inv_z : a[j], y[j]);
  }
  loss = warp_sum(loss);
  dot = warp_sum(dot);
  int correct = 0;
  if (l.correct) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float op = __shfl_xor_sync(0xffffffffu, best_p, o);
      int oa = __shfl_xor_sync(0xffffffffu, arg_p, o);
      if (op > best_p || (op == best_p && oa < arg_p)) { best_p = op; arg_p = oa; }
      float oy = __shfl_xor_sync(0xffffffffu, best_y, o);
      int ob = __shfl_xor_sync(0xffffffffu, arg_y, o);
      if (oy > best_y || (oy == best_y && ob < arg_y)) { best_y = oy; arg_y = ob; }
    }
    correct = arg_p == arg_y;
  }
  // pass 2: gradient wrt the last layer's pre-activation
  auto second = [&](int j, float p, float yt) {
    float g = -0.0f;
    if (l.kind != 1) g = 2.0f * (p - yt) * inv_n;
    else if (yt != 0.0f || isinf(p) || !(fmaxf(p, l.eps) > 0.0f)) g = -(yt / fmaxf(p, l.eps)) * inv_n;
    float d;
    if (l.softmax) d = p * (g - dot);
    else if (l.dact != ACT_NONE) {
      const float s = aux ? aux[j] : p;
      d = act_bwd(l.dact, l.dact_param, l.relu_quirk, s, g);
    } else d = g;
    put(j, p, d);
  };
  if (NV > 0) {
#pragma unroll
    for (int i = 0; i < R; ++i) if (lane + 32 * i < l.C) second(lane + 32 * i, pr[i], yr[i]);
  } else {
    for (int j = lane; j < l.C; j += 32) second(j, l.softmax ? (NV < 0 ? ex[j] : expf(a[j] - mx)) * inv_z : a[j], y[j]);
  }
  return LossRow{loss, correct};
}

}  // namespace ono
