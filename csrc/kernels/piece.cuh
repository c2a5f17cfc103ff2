// Runs of consecutive channels of a pixel, moved with one access and worked on as f32.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ono {

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

// A piece: consecutive channels moved with one access of type P (16, 8, 4 or 2 bytes), the widest that divides the channel count
// and that the rows are aligned for.
template <typename T, typename P>
__device__ __forceinline__ void unpack_piece(const P& w, float (&f)[sizeof(P) / sizeof(T)]) {
  const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(P) / sizeof(T)); ++i) f[i] = to_f32(e[i]);
}
template <typename T, typename P>
__device__ __forceinline__ P pack_piece(const float (&f)[sizeof(P) / sizeof(T)]) {
  P w;
  T* e = reinterpret_cast<T*>(&w);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(P) / sizeof(T)); ++i) e[i] = from_f32<T>(f[i]);
  return w;
}

// acc += a * b on two values at once: one instruction, each half rounded like fmaf.
__device__ __forceinline__ void fma2(float2& acc, float2 a, float2 b) {
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\tfma.rn.f32x2 z, x, y, z;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "+f"(acc.x), "+f"(acc.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

}  // namespace ono
