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

// acc += a piece's values: f32 by twos, bf16 by the addition that takes it as it is (the values are converted exactly, so each sum is
// that of the unpacked value).
__device__ __forceinline__ void add_f32x2(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}
__device__ __forceinline__ void add_bf16x2(float& a0, float& a1, uint32_t w) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tadd.rn.f32.bf16 %0, l, %0;\n\tadd.rn.f32.bf16 %1, h, %1;\n\t}" : "+f"(a0), "+f"(a1) : "r"(w));
}
template <typename T, int V>
__device__ __forceinline__ void add_piece(float (&acc)[V], const uint4& w) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
  if constexpr (sizeof(T) == 4) {
    add_f32x2(acc[0], acc[1], __uint_as_float(u[0]), __uint_as_float(u[1]));
    add_f32x2(acc[2], acc[3], __uint_as_float(u[2]), __uint_as_float(u[3]));
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) add_bf16x2(acc[2 * k], acc[2 * k + 1], u[k]);
  }
}

// acc += a * b on two values at once: one instruction, each half rounded like fmaf.
__device__ __forceinline__ void fma2(float2& acc, float2 a, float2 b) {
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%0, %1};\n\tfma.rn.f32x2 z, x, y, z;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "+f"(acc.x), "+f"(acc.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

}  // namespace ono
