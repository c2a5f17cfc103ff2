// Convolution and pooling around the tcgen05 GEMM: the gather / scatter halves of the reference's
// im2col convolution (machine_learning/src/arch/layers/conv/conv2d.rs:84-104,202-266) and its max
// pooling (arch/layers/max_pooling.rs:47-157), on pixel-major activations.
//
// Activations of image layers are 2-D matrices [B*H*W, ldc] (one row per pixel, channels contiguous),
// which is exactly what the GEMM epilogue writes for Y = cols * K^T; the column order of `cols` is
// (ky, kx, c) (channels fastest: coalesced gathers), so the reference's kernel layout K[F][C][k][k] is permuted
// into that order when parameters are refreshed.
// Semantics kept from the reference: zero padding, output size floor((H+2p-k)/s)+1 (trailing rows and
// columns the strided window never reaches are dropped), zero padding competes in the max, and a
// pooling gradient whose arg-max lies in the padding is dropped.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "act.cuh"
#include "ono_kernels.h"
#include "opt.cuh"
#include "piece.cuh"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);

// Column order of `cols` is q = (ky, kx, c): channels fastest, so that both the gather below and the GEMM
// operand rows are contiguous runs of the pixel-major input. The kernel tensor K[F][C][k][k] is permuted to
// that order once per parameter refresh (kperm_kernel), and the weight gradient is permuted back.
//
// cols[r, q] = x[(b, oy*s+ky-p, ox*s+kx-p), c]  with r = (b, oy, ox); optional transposed copy colsT[q, r].
// One block handles a 32 x 32 tile of (r, q): reads and the row-major write are coalesced along q, the
// transposed write goes through shared memory and is coalesced along r.
template <typename T>
__global__ void im2col_kernel(const OnoConvGeom g, const T* x, int ldx, T* cols, int ld_cols, T* colsT, int ld_colsT) {
  __shared__ float tile[32][33];
  __shared__ int s_iy0[32], s_ix0[32], s_img[32];   // per tile row: window origin and image index (divisions once per row)
  const int ckk = g.C * g.K * g.K;
  const long long rows = (long long)g.B * g.OH * g.OW;
  const int qtiles = (ckk + 31) / 32;
  const long long ntiles = ((rows + 31) / 32) * qtiles;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const long long r0 = (t / qtiles) * 32;
    const int q0 = (int)(t % qtiles) * 32;
    const int q = q0 + threadIdx.x;
    const int c = q % g.C, kx = (q / g.C) % g.K, ky = q / (g.C * g.K);
    if (threadIdx.y == 0) {
      const long long r = r0 + threadIdx.x;
      const int ox = (int)(r % g.OW), oy = (int)((r / g.OW) % g.OH);
      s_iy0[threadIdx.x] = oy * g.S - g.P;
      s_ix0[threadIdx.x] = ox * g.S - g.P;
      s_img[threadIdx.x] = (int)(r / ((long long)g.OW * g.OH));
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = threadIdx.y + 8 * j;
      const long long r = r0 + rr;
      float v = 0.f;
      if (r < rows && q < ckk) {
        const int iy = s_iy0[rr] + ky, ix = s_ix0[rr] + kx;
        if (iy >= 0 && iy < g.H && ix >= 0 && ix < g.W)
          v = to_f32(x[((long long)(s_img[rr] * g.H + iy) * g.W + ix) * ldx + c]);
        cols[r * ld_cols + q] = from_f32<T>(v);
      }
      tile[rr][threadIdx.x] = v;
    }
    if (colsT) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int qq = threadIdx.y + 8 * j;
        const long long r = r0 + threadIdx.x;
        if (r < rows && q0 + qq < ckk) colsT[(long long)(q0 + qq) * ld_colsT + r] = from_f32<T>(tile[threadIdx.x][qq]);
      }
      __syncthreads();
    } else {
      __syncthreads();   // s_* are rewritten by the next tile
    }
  }
}

// dx[(b,iy,ix), c] = act'(aux) * sum_{ky,kx} dcols[(b,oy,ox), (ky,kx,c)] over the windows covering the pixel
// (gather form: no atomics). One block handles 32 pixels x 32 channels; the optional transposed copy
// dxT[c, pix] goes through shared memory.
template <typename T>
__global__ void col2im_kernel(const OnoConvGeom g, const T* dcols, int ld_dcols, const T* aux, int ld_aux, int dact,
                              float dact_param, int relu_quirk, T* dx, int ld_dx, T* dxT, int ld_dxT) {
  __shared__ float tile[32][33];
  __shared__ int s_iy[32], s_ix[32], s_img[32];
  const long long npix = (long long)g.B * g.H * g.W;
  const int ctiles = (g.C + 31) / 32;
  const long long ntiles = ((npix + 31) / 32) * ctiles;
  const int shift = g.S == 1 ? 0 : g.S == 2 ? 1 : g.S == 4 ? 2 : -1;   // power-of-two strides avoid the divisions
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const long long p0 = (t / ctiles) * 32;
    const int c0 = (int)(t % ctiles) * 32;
    const int c = c0 + threadIdx.x;
    if (threadIdx.y == 0) {
      const long long pix = p0 + threadIdx.x;
      s_ix[threadIdx.x] = (int)(pix % g.W) + g.P;
      s_iy[threadIdx.x] = (int)((pix / g.W) % g.H) + g.P;
      s_img[threadIdx.x] = (int)(pix / ((long long)g.W * g.H));
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int pp = threadIdx.y + 8 * j;
      const long long pix = p0 + pp;
      float acc = 0.f;
      if (pix < npix && c < g.C) {
        const int ixp = s_ix[pp], iyp = s_iy[pp];
        const long long img_row = (long long)s_img[pp] * g.OH;
        for (int ky = 0; ky < g.K; ++ky) {
          const int ty = iyp - ky;
          if (ty < 0) break;
          int oy;
          if (shift >= 0) { if (ty & (g.S - 1)) continue; oy = ty >> shift; }
          else { if (ty % g.S) continue; oy = ty / g.S; }
          if (oy >= g.OH) continue;
          const T* rowp = dcols + (img_row + oy) * g.OW * (long long)ld_dcols + (ky * g.K) * g.C + c;
          for (int kx = 0; kx < g.K; ++kx) {
            const int tx = ixp - kx;
            if (tx < 0) break;
            int ox;
            if (shift >= 0) { if (tx & (g.S - 1)) continue; ox = tx >> shift; }
            else { if (tx % g.S) continue; ox = tx / g.S; }
            if (ox >= g.OW) continue;
            acc += to_f32(rowp[(long long)ox * ld_dcols + kx * g.C]);
          }
        }
        if (dact != ACT_NONE) acc = act_bwd(dact, dact_param, relu_quirk, to_f32(aux[pix * ld_aux + c]), acc);
        dx[pix * ld_dx + c] = from_f32<T>(acc);
      }
      tile[pp][threadIdx.x] = acc;
    }
    if (dxT) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int cc = threadIdx.y + 8 * j;
        const long long pix = p0 + threadIdx.x;
        if (pix < npix && c0 + cc < g.C) dxT[(long long)(c0 + cc) * ld_dxT + pix] = from_f32<T>(tile[threadIdx.x][cc]);
      }
      __syncthreads();
    } else {
      __syncthreads();
    }
  }
}

// Four consecutive channels at once (16-byte loads of f32, 8-byte loads of bf16).
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<const uint32_t*>(&a);
  u.y = *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// Elements of the widest piece for C channels: `lds` is the bitwise or of the leading dimensions, `ptrs` of the addresses.
static int piece_width(int esz, int C, int lds, uintptr_t ptrs) {
  int v = 16 / esz;
  while (v > 1 && (C % v != 0 || lds % v != 0 || (ptrs & (uintptr_t)(v * esz - 1)) != 0)) v /= 2;
  return v;
}

// im2col in pieces (C is a multiple of the piece, so that a piece lies within one tap): a block takes IM_ROWS output
// pixels. Window origins (one per pixel) and tap offsets (one per piece of a row) are worked out once into shared memory, and a
// thread walks its pieces by adding, four copies in flight. With the divisions made per 8-byte piece the kernel was bound by
// issue: 401408 x 288 bf16 out of 32 channels took 189 us beside the batch copy of the next step, now 56 alone (334 MB, 51 us at the copy
// rate); 100352 x 576: 94 us, now 30.
constexpr int IM_ROWS = 64;
constexpr int IM_MAX_PIECES = 1024;
template <typename T, typename P>
__global__ void __launch_bounds__(256) im2col_vec_kernel(const OnoConvGeom g, const T* x, int ldx, T* cols, int ld_cols, int rows) {
  constexpr int V = (int)(sizeof(P) / sizeof(T)), U = 4;
  __shared__ int s_iy0[IM_ROWS], s_ix0[IM_ROWS], s_base[IM_ROWS];
  __shared__ int s_tap[IM_MAX_PIECES], s_off[IM_MAX_PIECES];
  const int np = g.C * g.K * g.K / V;          // pieces of a row
  const int r0 = blockIdx.x * IM_ROWS;
  const int nr = min(IM_ROWS, rows - r0);
  for (int i = threadIdx.x; i < np; i += 256) {
    const int q = i * V, tap = q / g.C, c = q - tap * g.C, ky = tap / g.K, kx = tap - ky * g.K;
    s_tap[i] = (ky << 16) | kx;
    s_off[i] = (ky * g.W + kx) * ldx + c;
  }
  if ((int)threadIdx.x < nr) {
    const int r = r0 + threadIdx.x, rest = r / g.OW, ox = r - rest * g.OW, img = rest / g.OH, oy = rest - img * g.OH;
    const int iy0 = oy * g.S - g.P, ix0 = ox * g.S - g.P;
    s_iy0[threadIdx.x] = iy0;
    s_ix0[threadIdx.x] = ix0;
    s_base[threadIdx.x] = (img * g.H + iy0) * g.W + ix0;      // pixel index of the window's origin, may lie outside the image
  }
  __syncthreads();
  const int total = nr * np, drow = 256 / np, dpc = 256 - drow * np;
  int row = threadIdx.x / np, pc = threadIdx.x - row * np;
  for (int e = threadIdx.x; e < total; e += 256 * U) {
    P v[U];
    long long at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      v[u] = P{};
      at[u] = -1;
      if (e + 256 * u < total) {
        const int tap = s_tap[pc], iy = s_iy0[row] + (tap >> 16), ix = s_ix0[row] + (tap & 0xffff);
        if ((unsigned)iy < (unsigned)g.H && (unsigned)ix < (unsigned)g.W)
          v[u] = *reinterpret_cast<const P*>(x + (long long)s_base[row] * ldx + s_off[pc]);
        at[u] = (long long)(r0 + row) * ld_cols + pc * V;
      }
      row += drow;
      pc += dpc;
      if (pc >= np) { pc -= np; ++row; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) *reinterpret_cast<P*>(cols + at[u]) = v[u];
  }
}

// col2im in pieces with compile-time kernel size and stride: thread = pixel x piece. Of the K x K taps only those whose
// offset from the pixel is a multiple of the stride exist, ceil(K / S) per axis: these unroll into independent predicated loads.
// The sums are f32, in tap order. With 8-byte pieces and a test per tap:
// 1605632 pixels x 32 channels bf16, stride 2, took 219 us (now 80, 437 MB), 401408 x 64 took 126 us (now 41);
// 12544 pixels x 6 channels f32, 5 x 5, through the generic kernel 25.4 us (now 2.9).
template <typename T, typename P, int K, int S>
__global__ void __launch_bounds__(256) col2im_vec_kernel(const OnoConvGeom g, const T* dcols, int ld_dcols, const T* aux, int ld_aux,
                                                         int dact, float dact_param, int relu_quirk, T* dx, int ld_dx, unsigned total) {
  constexpr int V = (int)(sizeof(P) / sizeof(T)), KT = (K + S - 1) / S;
  const unsigned np = (unsigned)(g.C / V);
  for (unsigned e = blockIdx.x * 256u + threadIdx.x; e < total; e += gridDim.x * 256u) {
    const unsigned pix = e / np, c = (e - pix * np) * V;
    const unsigned rest = pix / (unsigned)g.W, img = rest / (unsigned)g.H;
    const int ixp = (int)(pix - rest * (unsigned)g.W) + g.P, iyp = (int)(rest - img * (unsigned)g.H) + g.P;
    P av{};
    if (dact != ACT_NONE) av = *reinterpret_cast<const P*>(aux + (long long)pix * ld_aux + c);
    P w[KT * KT];
    const int ky0 = iyp % S, kx0 = ixp % S;
    const int oy0 = (iyp - ky0) / S, ox0 = (ixp - kx0) / S;      // tap (ky0 + S i, kx0 + S j) belongs to window (oy0 - i, ox0 - j)
#pragma unroll
    for (int i = 0; i < KT; ++i)
#pragma unroll
      for (int j = 0; j < KT; ++j) {
        const int ky = ky0 + S * i, kx = kx0 + S * j, oy = oy0 - i, ox = ox0 - j;
        w[i * KT + j] = P{};
        if (ky < K && kx < K && oy >= 0 && ox >= 0 && oy < g.OH && ox < g.OW)
          w[i * KT + j] = *reinterpret_cast<const P*>(dcols + ((long long)((int)img * g.OH + oy) * g.OW + ox) * ld_dcols + (ky * K + kx) * g.C + c);
      }
    float acc[V];
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = 0.f;
#pragma unroll
    for (int i = 0; i < KT * KT; ++i) {
      float f[V];
      unpack_piece<T, P>(w[i], f);
#pragma unroll
      for (int k = 0; k < V; ++k) acc[k] += f[k];
    }
    if (dact != ACT_NONE) {
      float a[V];
      unpack_piece<T, P>(av, a);
      act_bwd_n<V>(dact, dact_param, relu_quirk, a, acc);
    }
    *reinterpret_cast<P*>(dx + (long long)pix * ld_dx + c) = pack_piece<T, P>(acc);
  }
}

// Kernel tensor between the parameter layout K[F][C][k][k] (f32, contiguous) and the operand layout
// [F][(ky,kx,c)] used by the GEMMs. dir 0: parameters -> operand (dst, dtype T, leading dimension ld_dst) and
// optionally its transpose dstT[(ky,kx,c)][F]; dir 1: f32 operand-ordered gradient (src, ld_src) -> parameter
// order, dst = beta * dst + src.
template <typename T>
__global__ void kperm_kernel(int F, int C, int K, int dir, const float* src, int ld_src, void* dst_, int ld_dst, T* dstT,
                             int ld_dstT, float beta) {
  const int ckk = C * K * K;
  const long long total = (long long)F * ckk;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int f = (int)(i / ckk), q = (int)(i % ckk);                   // q in operand order (ky, kx, c)
    const int c = q % C, kx = (q / C) % K, ky = q / (C * K);
    const long long pidx = ((long long)(f * C + c) * K + ky) * K + kx;    // parameter order
    if (dir == 0) {
      const float v = src[pidx];
      reinterpret_cast<T*>(dst_)[(long long)f * ld_dst + q] = from_f32<T>(v);
      if (dstT) dstT[(long long)q * ld_dstT + f] = from_f32<T>(v);
    } else {
      float* d = reinterpret_cast<float*>(dst_);
      const float v = src[(long long)f * ld_src + q];
      d[pidx] = beta != 0.f ? beta * d[pidx] + v : v;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Single-input-channel convolution (the first layer of every image model of the reference), computed
// directly on CUDA cores: with C = 1 the GEMM would have K = k*k <= 25, far too short for the tensor
// cores, and im2col would write k*k times the input. Thread x = filter, thread y strides over output
// pixels; the k*k taps of a pixel are broadcast loads, the filter's weights live in registers.
// ------------------------------------------------------------------------------------------------
constexpr int C1_MAXKK = 25;  // up to 5 x 5 kernels

template <typename T>
__global__ void conv1_fwd_kernel(const OnoConvGeom g, int F, const T* x, int ldx, const float* kparams, const float* bias,
                                 int act, float act_param, T* y, int ldy) {
  const int kk = g.K * g.K;
  const int f = blockIdx.y * 32 + threadIdx.x;
  float w[C1_MAXKK];
#pragma unroll
  for (int i = 0; i < C1_MAXKK; ++i) w[i] = (i < kk && f < F) ? kparams[(long long)f * kk + i] : 0.f;
  const float bv = (bias && f < F) ? bias[f] : 0.f;
  // A warp takes 32 consecutive output pixels: lane l works out the window origin of pixel r0 + l once (the
  // divisions), then the warp walks the 32 pixels with the coordinates broadcast by shuffles.
  const int rows = g.B * g.OH * g.OW;
  const int ohw = g.OH * g.OW;
  for (int r0 = (blockIdx.x * blockDim.y + threadIdx.y) * 32; r0 < rows; r0 += gridDim.x * blockDim.y * 32) {
    const int rl = min(r0 + (int)threadIdx.x, rows - 1);
    const int img_l = rl / ohw, rem = rl - img_l * ohw;
    const int oy_l = rem / g.OW, ox_l = rem - oy_l * g.OW;
    const int my_iy0 = oy_l * g.S - g.P, my_ix0 = ox_l * g.S - g.P, my_base = img_l * g.H;
    const int np = min(32, rows - r0);
    for (int pp = 0; pp < np; ++pp) {
      const int iy0 = __shfl_sync(0xffffffffu, my_iy0, pp), ix0 = __shfl_sync(0xffffffffu, my_ix0, pp);
      const int base = __shfl_sync(0xffffffffu, my_base, pp);
      float acc = bv;
#pragma unroll
      for (int i = 0; i < C1_MAXKK; ++i) {
        if (i >= kk) break;
        const int ky = i / g.K, kx = i - ky * g.K;
        const int iy = iy0 + ky, ix = ix0 + kx;
        if (iy >= 0 && iy < g.H && ix >= 0 && ix < g.W) acc += w[i] * to_f32(x[(long long)((base + iy) * g.W + ix) * ldx]);
      }
      if (f < F) y[(long long)(r0 + pp) * ldy + f] = from_f32<T>(act_fwd(act, act_param, acc));
    }
  }
}

// dK[f][ky][kx] = sum over output pixels dy[r][f] * x[tap], db[f] = sum dy[r][f]. Every block writes one row of
// partial sums to a scratch array; the last block to finish (atomic ticket) adds the rows in block order, so the
// result does not depend on scheduling. Calls must not overlap on the device (one training stream).
constexpr int C1_MAXBLOCKS = 592;
constexpr int C1_MAXF = 128;
__device__ float g_c1_part[C1_MAXBLOCKS * C1_MAXF * (C1_MAXKK + 1)];
__device__ unsigned int g_c1_ticket;

template <typename T>
__global__ void conv1_wgrad_kernel(const OnoConvGeom g, int F, const T* x, int ldx, const T* dy, int ld_dy, float* gk,
                                   float* gb, float beta) {
  __shared__ float red[8][32][C1_MAXKK + 2];
  __shared__ int s_last;
  const int kk = g.K * g.K;
  const int nfb = (F + 31) / 32;
  float acc[C1_MAXKK + 1];
  const int rows = g.B * g.OH * g.OW;
  const int ohw = g.OH * g.OW;
  for (int fb = 0; fb < nfb; ++fb) {
    const int f = fb * 32 + threadIdx.x;
#pragma unroll
    for (int i = 0; i <= C1_MAXKK; ++i) acc[i] = 0.f;
    for (int r0 = (blockIdx.x * blockDim.y + threadIdx.y) * 32; r0 < rows; r0 += gridDim.x * blockDim.y * 32) {
      const int rl = min(r0 + (int)threadIdx.x, rows - 1);
      const int img_l = rl / ohw, rem = rl - img_l * ohw;
      const int oy_l = rem / g.OW, ox_l = rem - oy_l * g.OW;
      const int my_iy0 = oy_l * g.S - g.P, my_ix0 = ox_l * g.S - g.P, my_base = img_l * g.H;
      const int np = min(32, rows - r0);
      for (int pp = 0; pp < np; ++pp) {
        const int iy0 = __shfl_sync(0xffffffffu, my_iy0, pp), ix0 = __shfl_sync(0xffffffffu, my_ix0, pp);
        const int base = __shfl_sync(0xffffffffu, my_base, pp);
        const float d = f < F ? to_f32(dy[(long long)(r0 + pp) * ld_dy + f]) : 0.f;
#pragma unroll
        for (int i = 0; i < C1_MAXKK; ++i) {
          if (i >= kk) break;
          const int ky = i / g.K, kx = i - ky * g.K;
          const int iy = iy0 + ky, ix = ix0 + kx;
          if (iy >= 0 && iy < g.H && ix >= 0 && ix < g.W) acc[i] += d * to_f32(x[(long long)((base + iy) * g.W + ix) * ldx]);
        }
        acc[C1_MAXKK] += d;
      }
    }
#pragma unroll
    for (int i = 0; i <= C1_MAXKK; ++i) red[threadIdx.y][threadIdx.x][i] = acc[i];
    __syncthreads();
    if (threadIdx.y == 0 && f < F) {
      float* out = g_c1_part + ((size_t)blockIdx.x * C1_MAXF + f) * (C1_MAXKK + 1);
      for (int i = 0; i <= C1_MAXKK; ++i) {
        if (i >= kk && i != C1_MAXKK) continue;
        float t = 0.f;
#pragma unroll
        for (int yy = 0; yy < 8; ++yy) t += red[yy][threadIdx.x][i];
        out[i] = t;
      }
    }
    __syncthreads();
  }
  __threadfence();
  if (threadIdx.x == 0 && threadIdx.y == 0) s_last = atomicAdd(&g_c1_ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int per = kk + 1;
  for (int idx = threadIdx.y * 32 + threadIdx.x; idx < F * per; idx += 256) {
    const int f = idx / per, i = idx % per;
    const int slot = i < kk ? i : C1_MAXKK;
    float t = 0.f;
    for (unsigned b = 0; b < gridDim.x; ++b) t += __ldcg(&g_c1_part[((size_t)b * C1_MAXF + f) * (C1_MAXKK + 1) + slot]);
    float* dst = i < kk ? gk + (long long)f * kk + i : gb + f;
    *dst = beta != 0.f ? beta * (*dst) + t : t;
  }
  if (threadIdx.x == 0 && threadIdx.y == 0) g_c1_ticket = 0u;
}

// Image-tiled variants of the two kernels above for k = 3 and k = 5 (compile-time taps): a block keeps the rows of one image that
// it needs, zero-padded, in shared memory (with C1_PX * stride further zero columns on the right where a group of pixels may
// reach past the end of a row), with no bounds test and no division in the pixel loop.
constexpr int C1_PX = 4;      // output pixels of a row that a thread works on at a time
constexpr int C1_FC = 32;     // filters of a block (forward) or of a pass (weight gradient)

// Rows [row0, row0 + nrow) of the padded image.
template <typename T>
__device__ __forceinline__ void c1_stage_rows(const OnoConvGeom& g, const T* x, int ldx, int img, int row0, int nrow, float* tile, int pitch) {
  const int n = nrow * pitch, drow = 256 / pitch, dcol = 256 - drow * pitch;
  int ty = threadIdx.x / pitch, tx = threadIdx.x - ty * pitch;
  for (int i = threadIdx.x; i < n; i += 256) {
    const int iy = row0 + ty - g.P, ix = tx - g.P;
    tile[i] = (iy >= 0 && iy < g.H && ix >= 0 && ix < g.W) ? to_f32(x[(long long)((img * g.H + iy) * g.W + ix) * ldx]) : 0.f;
    ty += drow;
    tx += dcol;
    if (tx >= pitch) { tx -= pitch; ++ty; }
  }
}

// Forward: a thread computes C1_PX pixels of a row x four filters. Per kernel row it reads the pixels' taps once (K + 3 S values
// for 4 K products each) and one 16-byte word of weights per tap for 16 products, all from shared memory; neighbouring threads
// take neighbouring filters, so the stores of a pixel are contiguous. Bound by issue. With one or four pixels of a filter per
// thread and a tap load per product or per four: 64 images, 6 filters, 5 x 5: 22.3 us (now 5.7); 256 images, 20 filters: 18.3 us (now 9.2);
// 2048 images, 32 filters, 3 x 3, bf16: 58.6 us (49.7; now, with two products an instruction, 46.0). Row chunks (grid.x = images x chunks) fill the SMs when images are few and
// keep the rows of a large image within shared memory. S = 0: any stride, known at run time; neighbouring pixels then share no
// taps, and each reads its own (256 images, 64 x 64, 64 filters, 5 x 5, stride 3: 274 us through the generic kernel, 33 so; events around a cold call).
template <typename T, int K, int S>
__global__ void __launch_bounds__(256) conv1_fwd_img_kernel(const OnoConvGeom g, int F, const T* x, int ldx, const float* kparams,
                                                            const float* bias, int act, float act_param, T* y, int ldy, int vec, int chunks) {
  extern __shared__ __align__(16) float c1_smem[];
  constexpr int KK = K * K, NT = S ? K + (C1_PX - 1) * S : K * C1_PX;
  const int stride = S ? S : g.S, pitch = g.W + 2 * g.P + C1_PX * stride;
  float* sw = c1_smem;                          // [tap][filter of the chunk]
  float* sb = sw + KK * C1_FC;
  float* tile = sb + C1_FC;
  const int img = (int)(blockIdx.x / chunks), ch = (int)(blockIdx.x - img * chunks);
  const int oy0 = (int)((long long)g.OH * ch / chunks), oy1 = (int)((long long)g.OH * (ch + 1) / chunks);
  const int f0 = blockIdx.y * C1_FC, nf = min(C1_FC, F - f0), nfg = (nf + 3) / 4;
  for (int i = threadIdx.x; i < KK * C1_FC; i += 256) {
    const int tap = i / C1_FC, f = i % C1_FC;
    sw[i] = f < nf ? kparams[(long long)(f0 + f) * KK + tap] : 0.f;
  }
  if (threadIdx.x < C1_FC) sb[threadIdx.x] = (bias && (int)threadIdx.x < nf) ? bias[f0 + threadIdx.x] : 0.f;
  c1_stage_rows(g, x, ldx, img, oy0 * stride, (oy1 - oy0 - 1) * stride + K, tile, pitch);
  __syncthreads();
  const int pgs = (g.OW + C1_PX - 1) / C1_PX, items = (oy1 - oy0) * pgs * nfg;
  for (int it = threadIdx.x; it < items; it += 256) {
    const int pos = it / nfg, fg = it - pos * nfg, ry = pos / pgs, ox = (pos - ry * pgs) * C1_PX;
    const float* t0 = tile + ry * stride * pitch + ox * stride;
    const float4 b4 = *reinterpret_cast<const float4*>(sb + 4 * fg);
    float2 acc2[C1_PX * 2];
#pragma unroll
    for (int q = 0; q < C1_PX; ++q) { acc2[2 * q] = make_float2(b4.x, b4.y); acc2[2 * q + 1] = make_float2(b4.z, b4.w); }
#pragma unroll
    for (int ky = 0; ky < K; ++ky) {
      float t[NT];
#pragma unroll
      for (int i = 0; i < NT; ++i) t[i] = t0[ky * pitch + (S ? i : (i / K) * stride + i % K)];
#pragma unroll
      for (int kx = 0; kx < K; ++kx) {
        const float4 w = *reinterpret_cast<const float4*>(sw + (ky * K + kx) * C1_FC + 4 * fg);
#pragma unroll
        for (int q = 0; q < C1_PX; ++q) {
          const float tv = t[q * (S ? S : K) + kx];
          fma2(acc2[2 * q], make_float2(w.x, w.y), make_float2(tv, tv));
          fma2(acc2[2 * q + 1], make_float2(w.z, w.w), make_float2(tv, tv));
        }
      }
    }
    float acc[C1_PX * 4];
#pragma unroll
    for (int q = 0; q < C1_PX * 2; ++q) { acc[2 * q] = acc2[q].x; acc[2 * q + 1] = acc2[q].y; }
    act_fwd_n(act, act_param, acc);
    T* yp = y + ((long long)(img * g.OH + oy0 + ry) * g.OW + ox) * ldy + f0 + 4 * fg;
#pragma unroll
    for (int q = 0; q < C1_PX; ++q) {
      if (ox + q >= g.OW) break;
      if (vec) store4(yp + (long long)q * ldy, make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]));
      else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (4 * fg + c < nf) yp[(long long)q * ldy + c] = from_f32<T>(acc[4 * q + c]);
      }
    }
  }
}

// Weight and bias gradient: a thread owns four filters and c1_ky(K) kernel rows (K x 4 sums each, 4 more for the bias) over the
// pixels of its row group; four pixels at a time their dy come in with four loads in flight and their taps are read once. All
// three rows of a 3 x 3 kernel fit one thread, which then reads dy once; of a 5 x 5 kernel a thread takes one row, for the
// registers. The threads of a block are kernel rows x filter groups x row groups, whose sums are folded through shared memory in row-group order; block b's
// sums go to g_c1_part[(f * (K*K+1) + i) * gridDim.x + b] (slot K*K = bias) and conv1_wgrad_reduce_kernel adds them with one warp
// in a fixed order. A block takes every gridDim.x-th (image, row chunk). With K*K sums per thread (one block of 256 threads per
// SM for K = 5, and a tap load per product): 64 images, 6 filters, 5 x 5: 20.6 us (now 7.9); 256 images, 20 filters: 22.6 us (now 15.3);
// 2048 images, 32 filters, 3 x 3, bf16: 84.5 us (61.0 here; bf16 images that fit shared memory keep the order of the kernel below).
__host__ __device__ constexpr int c1_ky(int K) { return K == 3 ? 3 : 1; }
template <typename T, int K, int S>
__global__ void __launch_bounds__(256) conv1_wgrad_img_kernel(const OnoConvGeom g, int F, const T* x, int ldx, const T* dy, int ld_dy,
                                                              int vec, int chunks) {
  extern __shared__ __align__(16) float c1_smem[];   // the padded rows; afterwards the sums of the row groups
  constexpr int KK = K * K, NT = K + (C1_PX - 1) * S, KY = c1_ky(K), BIAS = 4 * K * KY, SUMS = BIAS + 4;
  const int pitch = g.W + 2 * g.P + C1_PX * S;
  const int units_total = g.B * chunks;
  for (int f0 = 0; f0 < F; f0 += C1_FC) {
    const int nf = min(C1_FC, F - f0), nfg = (nf + 3) / 4, per = nfg * (K / KY), groups = 256 / per;
    const int u = threadIdx.x % per, grp = threadIdx.x / per, fg = u % nfg, ky = (u / nfg) * KY;
    const int nlive = min(4, nf - 4 * fg);             // filters of this thread that exist
    float acc[SUMS];
#pragma unroll
    for (int i = 0; i < SUMS; ++i) acc[i] = 0.f;
    for (int un = blockIdx.x; un < units_total; un += gridDim.x) {
      const int img = un / chunks, ch = un - img * chunks;
      const int oy0 = (int)((long long)g.OH * ch / chunks), oy1 = (int)((long long)g.OH * (ch + 1) / chunks);
      __syncthreads();
      c1_stage_rows(g, x, ldx, img, oy0 * S, (oy1 - oy0 - 1) * S + K, c1_smem, pitch);
      __syncthreads();
      if (grp >= groups) continue;
      // groups of four pixels, numbered row after row, are dealt out to the thread groups
      const int pgs = (g.OW + C1_PX - 1) / C1_PX, npos = (oy1 - oy0) * pgs, dr = groups / pgs, dp = groups - dr * pgs;
      int ry = grp / pgs, pg = grp - ry * pgs;
      for (int pos = grp; pos < npos; pos += groups) {
        const int ox = pg * C1_PX;
        const float* trow = c1_smem + (ry * S + ky) * pitch;
        const T* drow = dy + (long long)(img * g.OH + oy0 + ry) * g.OW * ld_dy + f0 + 4 * fg;
        ry += dr;
        pg += dp;
        if (pg >= pgs) { pg -= pgs; ++ry; }
        float4 d[C1_PX];
#pragma unroll
        for (int q = 0; q < C1_PX; ++q) {
          d[q] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (ox + q < g.OW) {
            const T* dp = drow + (long long)(ox + q) * ld_dy;
            if (vec) d[q] = load4(dp);
            else {
              d[q].x = to_f32(dp[0]);
              if (nlive > 1) d[q].y = to_f32(dp[1]);
              if (nlive > 2) d[q].z = to_f32(dp[2]);
              if (nlive > 3) d[q].w = to_f32(dp[3]);
            }
          }
        }
        // past the end of a row there is no pixel: its taps may be infinite, and zero times that is no zero
        auto products = [&](auto whole) {
#pragma unroll
          for (int r = 0; r < KY; ++r) {
            float t[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) t[i] = trow[r * pitch + ox * S + i];
#pragma unroll
            for (int q = 0; q < C1_PX; ++q) {
              if (!decltype(whole)::value && ox + q >= g.OW) continue;
#pragma unroll
              for (int kx = 0; kx < K; ++kx) {
                const float tv = t[q * S + kx];
                float* a = acc + 4 * (r * K + kx);
                a[0] += d[q].x * tv; a[1] += d[q].y * tv; a[2] += d[q].z * tv; a[3] += d[q].w * tv;
              }
            }
          }
        };
        if (ox + C1_PX <= g.OW) products(std::true_type{});
        else products(std::false_type{});
#pragma unroll
        for (int q = 0; q < C1_PX; ++q) {
          acc[BIAS] += d[q].x; acc[BIAS + 1] += d[q].y; acc[BIAS + 2] += d[q].z; acc[BIAS + 3] += d[q].w;
        }
      }
    }
    __syncthreads();   // the image is no longer needed: its space takes the row groups' sums, [sum][thread]
#pragma unroll
    for (int i = 0; i < SUMS; ++i) c1_smem[i * 256 + threadIdx.x] = acc[i];
    __syncthreads();
    for (int o = threadIdx.x; o < per * SUMS; o += 256) {
      const int uu = o % per, i = o / per, fo = 4 * (uu % nfg) + (i & 3), kyo = (uu / nfg) * KY;
      const bool is_bias = i >= BIAS;
      if (fo >= nf || (is_bias && kyo != 0)) continue;
      float t = 0.f;
      for (int gq = 0; gq < groups; ++gq) t += c1_smem[i * 256 + gq * per + uu];
      const int slot = is_bias ? KK : kyo * K + (i >> 2);      // i >> 2 counts (row, column) pairs of this thread
      g_c1_part[((size_t)(f0 + fo) * (KK + 1) + slot) * gridDim.x + blockIdx.x] = t;
    }
  }
}

// Weight and bias gradient in the order that a network with bf16 tiles keeps from version to version (see fixed_order in the
// engine): block b takes the images b, b + grid, ...; warp w their output rows w, w + 8, ...; a lane holds V filters and adds the
// pixels of such a row one after the other, every V-th of them (V = 4: four pixel groups a warp, folded with shuffles); the eight
// warps' sums are added in warp order. The order leaves each lane one chain of sums, so what bounds it is the latency of dy: up to
// eight pixels' loads are in flight. 2048 images, 32 filters, 3 x 3: 91.2 us (events around a cold call, which adds about 8; the
// register-tiled kernel of f32 below 76.8). Two blocks per SM, so that its up to 592 make two full waves: with three 97.3.
// Also what f32 takes at strides above 2, where neighbouring windows share too little to be tiled (256 images, 64 x 64, 64 filters,
// 5 x 5, stride 3: 436 us through the generic kernel, 54 so).
template <typename T, int V> struct C1Raw;
template <> struct C1Raw<float, 4> { using type = float4; };
template <> struct C1Raw<float, 1> { using type = float; };
template <> struct C1Raw<__nv_bfloat16, 4> { using type = uint2; };
template <> struct C1Raw<__nv_bfloat16, 1> { using type = unsigned short; };

template <typename T, int K, int V>
__global__ void __launch_bounds__(256, V == 1 ? 4 : 2) conv1_wgrad_walk_kernel(const OnoConvGeom g, int F, const T* x, int ldx, const T* dy, int ld_dy) {
  extern __shared__ __align__(16) float c1_smem[];   // the padded image; afterwards the warps' sums, [warp][filter][slot]
  using Raw = typename C1Raw<T, V>::type;
  constexpr int KK = K * K, LPP = 32 / V, U = V == 1 ? 8 : (K == 5 ? 16 : 32) / (int)sizeof(T) / 2;      // lanes of a pixel, loads in flight (as registers allow)
  const int pitch = g.W + 2 * g.P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fq = lane % LPP, pg = lane / LPP;
  for (int f0 = 0; f0 < F; f0 += 32) {
    const int fl = f0 + V * fq;                       // first of this lane's filters
    const bool live = fl < F;
    float acc[KK + 1][V];
#pragma unroll
    for (int i = 0; i <= KK; ++i)
#pragma unroll
      for (int c = 0; c < V; ++c) acc[i][c] = 0.f;
    for (int img = blockIdx.x; img < g.B; img += gridDim.x) {
      __syncthreads();
      c1_stage_rows(g, x, ldx, img, 0, g.H + 2 * g.P, c1_smem, pitch);
      __syncthreads();
      for (int oy = warp; oy < g.OH; oy += 8) {
        const float* trow = c1_smem + oy * g.S * pitch;
        const T* drow = dy + (long long)(img * g.OH + oy) * g.OW * ld_dy + fl;
        for (int ox0 = pg; ox0 < g.OW; ox0 += V * U) {
          Raw raw[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            raw[u] = Raw{};
            if (live && ox0 + V * u < g.OW) raw[u] = *reinterpret_cast<const Raw*>(drow + (long long)(ox0 + V * u) * ld_dy);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int ox = ox0 + V * u;
            if (ox >= g.OW) break;
            const float* t0 = trow + ox * g.S;
            float d[V];
            unpack_piece<T, Raw>(raw[u], d);
#pragma unroll
            for (int ky = 0; ky < K; ++ky)
#pragma unroll
              for (int kx = 0; kx < K; ++kx) {
                const float t = t0[ky * pitch + kx];
#pragma unroll
                for (int c = 0; c < V; ++c) acc[ky * K + kx][c] += d[c] * t;
              }
#pragma unroll
            for (int c = 0; c < V; ++c) acc[KK][c] += d[c];
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i <= KK; ++i)
#pragma unroll
      for (int c = 0; c < V; ++c)
#pragma unroll
        for (int o = LPP; o < 32; o *= 2) acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], o);
    __syncthreads();   // the image is no longer needed
    if (pg == 0) {
#pragma unroll
      for (int c = 0; c < V; ++c)
#pragma unroll
        for (int i = 0; i <= KK; ++i) c1_smem[(warp * 32 + V * fq + c) * (KK + 1) + i] = acc[i][c];
    }
    __syncthreads();
    for (int o = threadIdx.x; o < min(32, F - f0) * (KK + 1); o += 256) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += c1_smem[w * 32 * (KK + 1) + o];
      g_c1_part[((size_t)f0 * (KK + 1) + o) * gridDim.x + blockIdx.x] = t;
    }
  }
}

__global__ void __launch_bounds__(256) conv1_wgrad_reduce_kernel(int F, int kk, int nblocks, float* gk, float* gb, float beta) {
  const int lane = threadIdx.x & 31;
  const int pair = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (pair >= F * (kk + 1)) return;
  const float* p = g_c1_part + (size_t)pair * nblocks;
  float t = 0.f;
  for (int b = lane; b < nblocks; b += 32) t += p[b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) {
    const int f = pair / (kk + 1), i = pair - f * (kk + 1);
    float* dst = i < kk ? gk + (long long)f * kk + i : gb + f;
    *dst = beta != 0.f ? beta * (*dst) + t : t;
  }
}

static size_t c1_img_smem(const OnoConvGeom* g, int chunks, bool wgrad);
// Row chunks per image, so that few images still make about two blocks per SM; at least four output rows a chunk, or as few as the
// shared memory asks for.
static int c1_chunks(const OnoConvGeom* g) {
  int c = std::max(1, std::min({g->OH / 4, (2 * 148 + g->B - 1) / g->B}));
  while (c < g->OH && !c1_img_smem(g, c, false)) c = std::min(2 * c, g->OH);
  return c;
}
// Weight gradient: blocks that are resident together (registers: two per SM for K = 3, three for K = 5) and the row chunks that
// give the shortest sequence of pixel groups per thread on them (342 images of 28 rows in halves: 3 x 4 groups instead of 2 x 7).
static int c1_wgrad_blocks(const OnoConvGeom* g) { return std::min(C1_MAXBLOCKS, 148 * (g->K == 3 ? 2 : 3)); }
static int c1_wgrad_chunks(const OnoConvGeom* g, int F) {
  const int per = (std::min(F, C1_FC) + 3) / 4 * (g->K / c1_ky(g->K)), groups = 256 / per, pgs = (g->OW + C1_PX - 1) / C1_PX;
  const int slots = c1_wgrad_blocks(g);
  int best = 1;
  double best_cost = 1e30;
  for (int c = 1; c <= g->OH; c *= 2) {
    if ((c > 1 && c > g->OH / 4 && best_cost < 1e30) || !c1_img_smem(g, c, true)) continue;
    const double waves = (double)(((long long)g->B * c + slots - 1) / slots);
    const double cost = waves * (2.0 + (double)(((g->OH + c - 1) / c * pgs + groups - 1) / groups));   // 2: staging a chunk
    if (cost < best_cost) { best_cost = cost; best = c; }
  }
  return best;
}
// Shared memory of conv1_wgrad_walk_kernel (whole images), or 0 when the shape has to take the generic kernel.
static size_t c1_walk_smem(const OnoConvGeom* g) {
  if (g->K != 3 && g->K != 5) return 0;
  const size_t floats = std::max((size_t)(g->H + 2 * g->P) * (g->W + 2 * g->P), (size_t)256 * (g->K * g->K + 1));
  return floats * sizeof(float) <= 48 * 1024 ? floats * sizeof(float) : 0;
}
// Shared memory of the image-tiled kernels (forward, weight gradient), or 0 when the shape has to take the generic kernels.
static size_t c1_img_smem(const OnoConvGeom* g, int chunks, bool wgrad) {
  if ((g->K != 3 && g->K != 5) || (wgrad && g->S != 1 && g->S != 2)) return 0;
  const size_t rows = (size_t)((g->OH + chunks - 1) / chunks - 1) * g->S + g->K;
  const size_t tile = rows * (g->W + 2 * g->P + C1_PX * g->S);
  const size_t floats = wgrad ? std::max(tile, (size_t)256 * (4 * g->K * c1_ky(g->K) + 4)) : tile + (size_t)(g->K * g->K + 1) * C1_FC;
  return floats * sizeof(float) <= 48 * 1024 ? floats * sizeof(float) : 0;
}

// Division of an index by a number fixed at launch. 32-bit indexes: multiplication by the rounded-up reciprocal 2^p / d with
// p = 31 + ceil(log2 d), exact for every index below 2^31 (T. Granlund, P. Montgomery, "Division by invariant integers using
// multiplication", PLDI 1994); a division by a run-time value is about ten times the instructions. 64-bit indexes divide.
template <typename I>
struct FastDiv {
  I d;
  __host__ explicit FastDiv(int v) : d(v) {}
  __device__ __forceinline__ I operator()(I n) const { return n / d; }
};
template <>
struct FastDiv<unsigned> {
  unsigned d, m, sh;
  __host__ explicit FastDiv(int v) : d((unsigned)v), m(0), sh(0) {
    unsigned l = 0;
    while ((1u << l) < d) ++l;
    if (d > 1) { m = (unsigned)(((1ull << (31 + l)) + d - 1) / d); sh = l - 1; }
  }
  __device__ __forceinline__ unsigned operator()(unsigned n) const { return d == 1 ? n : __umulhi(n, m) >> sh; }
};
template <typename I>
struct PoolDiv {
  FastDiv<I> C, W, H, S;
  PoolDiv(int c, int w, int h, int s) : C(c), W(w), H(h), S(s) {}
};

// y[(b,oy,ox), c] = max over the window of the zero-padded input; arg[...] = input pixel (iy*W+ix) of the
// maximum or -1 when the maximum is a padding zero. Ties: the last element in scan order.
// I: 32-bit indexes where they suffice, 64-bit ones for larger images. A thread takes one piece of channels.
template <typename T, typename P, typename I>
__global__ void pool_fwd_kernel(const OnoConvGeom g, const T* x, int ldx, T* y, int ldy, T* yT, int ld_yT, int* arg,
                                int act, float act_param, const PoolDiv<I> by, I total) {
  constexpr int V = (int)(sizeof(P) / sizeof(T));
  for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const I r = by.C(i), c = (i - r * by.C.d) * V;
    const I rest = by.W(r), b = by.H(rest);
    const int ox = (int)(r - rest * (I)g.OW), oy = (int)(rest - b * (I)g.OH);
    float best[V];
    int where[V];
#pragma unroll
    for (int k = 0; k < V; ++k) { best[k] = -INFINITY; where[k] = -1; }
    for (int ky = 0; ky < g.K; ++ky)
      for (int kx = 0; kx < g.K; ++kx) {
        const int iy = oy * g.S + ky - g.P, ix = ox * g.S + kx - g.P;
        const bool in = iy >= 0 && iy < g.H && ix >= 0 && ix < g.W;
        P w{};
        if (in) w = *reinterpret_cast<const P*>(x + (((long long)b * g.H + iy) * g.W + ix) * ldx + c);
        float v[V];
        unpack_piece<T, P>(w, v);
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (v[k] >= best[k]) { best[k] = v[k]; where[k] = in ? iy * g.W + ix : -1; }
      }
    int* ap = arg + (long long)r * g.C + c;
#pragma unroll
    for (int k = 0; k < V; ++k) ap[k] = where[k];
    act_fwd_n<V>(act, act_param, best);
    *reinterpret_cast<P*>(y + (long long)r * ldy + c) = pack_piece<T, P>(best);
    if (yT) {
#pragma unroll
      for (int k = 0; k < V; ++k) yT[(long long)(c + k) * ld_yT + r] = from_f32<T>(best[k]);
    }
  }
}

// Gradient of the pooling layer and of the activation below it in one pass over the input pixels: a pixel looks up the windows
// that cover it (one where windows do not overlap) and adds the gradients of those whose maximum it is, in window order, each
// taken through the pooling layer's own activation (on y); the sum goes through the previous layer's derivative (on aux) and out
// in the tile dtype. It was a zero fill, a scatter with atomics into an f32 image and a conversion: 23.2 us for 256 x 24 x 24 x 20,
// now 7.4.
template <typename T, typename P, typename I>
__global__ void pool_bwd_kernel(const OnoConvGeom g, const T* d, int ldd, const T* y, int ldy, const int* arg, int act,
                                float act_param, int relu_quirk, const T* aux, int ld_aux, int dact, float dact_param, T* dx,
                                int ld_dx, T* dxT, int ld_dxT, const PoolDiv<I> by, I total) {
  constexpr int V = (int)(sizeof(P) / sizeof(T));
  for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const I pix = by.C(i), c = (i - pix * by.C.d) * V;
    const I rest = by.W(pix), b = by.H(rest);
    const int ix = (int)(pix - rest * (I)g.W), iy = (int)(rest - b * (I)g.H);
    const int want = iy * g.W + ix;
    P av{};
    if (dact != ACT_NONE) av = *reinterpret_cast<const P*>(aux + (long long)pix * ld_aux + c);
    // windows oy with oy * S <= iy + P < oy * S + K
    const int oy1 = min(g.OH - 1, (int)by.S(iy + g.P)), ox1 = min(g.OW - 1, (int)by.S(ix + g.P));
    const int oy0 = iy + g.P < g.K ? 0 : (int)by.S(iy + g.P - g.K + g.S), ox0 = ix + g.P < g.K ? 0 : (int)by.S(ix + g.P - g.K + g.S);
    float v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = 0.f;
    for (int oy = oy0; oy <= oy1; ++oy)
      for (int ox = ox0; ox <= ox1; ++ox) {
        const long long r = ((long long)b * g.OH + oy) * g.OW + ox;
        const int* ap = arg + r * g.C + c;
        const P dw = *reinterpret_cast<const P*>(d + r * ldd + c);
        int w[V];
#pragma unroll
        for (int k = 0; k < V; ++k) w[k] = ap[k];
        float t[V];
        unpack_piece<T, P>(dw, t);
        if (act != ACT_NONE) {
          float yv[V];
          unpack_piece<T, P>(*reinterpret_cast<const P*>(y + r * ldy + c), yv);
          act_bwd_n<V>(act, act_param, relu_quirk, yv, t);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] += w[k] == want ? t[k] : 0.f;
      }
    if (dact != ACT_NONE) {
      float a[V];
      unpack_piece<T, P>(av, a);
      act_bwd_n<V>(dact, dact_param, relu_quirk, a, v);
    }
    *reinterpret_cast<P*>(dx + (long long)pix * ld_dx + c) = pack_piece<T, P>(v);
    if (dxT) {
#pragma unroll
      for (int k = 0; k < V; ++k) dxT[(long long)(c + k) * ld_dxT + pix] = from_f32<T>(v[k]);
    }
  }
}

// A block moves a 32 x 32 tile of one image's HW x C matrix through shared memory, so that both sides are read and written along
// their contiguous dimension. With a thread per element, one side a stride of HW or C apart, 2048 x 64 x 49 bf16 (13 MB) took
// 53 us there and 30 us back (17 and 27 in tiles; 6.0 and 9.8 as whole images, below).
template <typename T>
__global__ void __launch_bounds__(256) nchw_flat_kernel(int B, int C, int HW, int to_flat, T* img, int ld_img, T* flat, int ld_flat,
                                                        T* outT, int ld_outT, const T* aux, int ld_aux, int dact, float dact_param,
                                                        int relu_quirk) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int ptiles = (HW + 31) / 32;
  const int p0 = (int)(blockIdx.x % ptiles) * 32, c0 = (int)(blockIdx.x / ptiles) * 32;
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    const long long pb = (long long)b * HW;
    __syncthreads();                       // the previous image's tile has been read
    if (to_flat) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = p0 + ty + 8 * j, c = c0 + tx;
        if (p < HW && c < C) tile[ty + 8 * j][tx] = to_f32(img[(pb + p) * ld_img + c]);
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = p0 + tx, c = c0 + ty + 8 * j;
        if (p < HW && c < C) {
          const T v = from_f32<T>(tile[tx][ty + 8 * j]);
          const long long f = (long long)c * HW + p;
          flat[(long long)b * ld_flat + f] = v;
          if (outT) outT[f * ld_outT + b] = v;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = p0 + tx, c = c0 + ty + 8 * j;
        if (p < HW && c < C) tile[tx][ty + 8 * j] = to_f32(flat[(long long)b * ld_flat + (long long)c * HW + p]);
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int p = p0 + ty + 8 * j, c = c0 + tx;
        if (p < HW && c < C) {
          float v = tile[ty + 8 * j][tx];
          if (dact != ACT_NONE) v = act_bwd(dact, dact_param, relu_quirk, to_f32(aux[(pb + p) * ld_aux + c]), v);
          img[(pb + p) * ld_img + c] = from_f32<T>(v);
          if (outT) outT[(long long)c * ld_outT + pb + p] = from_f32<T>(v);
        }
      }
    }
  }
}

// The same for whole images in shared memory: an image's HW x C block and its row of the flattened matrix are both contiguous, so
// both sides move in pieces (P: channels of a pixel, Q: a run of the row), and only shared memory is walked with a stride.
template <typename T, typename P, typename Q>
__global__ void __launch_bounds__(256) nchw_image_kernel(int B, int C, int HW, int to_flat, T* img, int ld_img, T* flat, int ld_flat,
                                                         const T* aux, int ld_aux, int dact, float dact_param, int relu_quirk) {
  extern __shared__ __align__(16) unsigned char nchw_smem[];
  T* s = reinterpret_cast<T*>(nchw_smem);                     // [c * HW + p]
  constexpr int V = (int)(sizeof(P) / sizeof(T)), VQ = (int)(sizeof(Q) / sizeof(T));
  const int np = C / V, pieces = HW * np, runs = C * HW / VQ;
  for (int b = blockIdx.x; b < B; b += gridDim.x) {
    T* const row = flat + (long long)b * ld_flat;
    const long long pb = (long long)b * HW;
    __syncthreads();                                          // the previous image has been read
    if (to_flat) {
      for (int e = threadIdx.x; e < pieces; e += 256) {
        const int p = e / np, c = (e - p * np) * V;
        const P w = *reinterpret_cast<const P*>(img + (pb + p) * ld_img + c);
        const T* v = reinterpret_cast<const T*>(&w);
#pragma unroll
        for (int k = 0; k < V; ++k) s[(c + k) * HW + p] = v[k];
      }
      __syncthreads();
      for (int e = threadIdx.x; e < runs; e += 256) reinterpret_cast<Q*>(row)[e] = reinterpret_cast<const Q*>(s)[e];
    } else {
      for (int e = threadIdx.x; e < runs; e += 256) reinterpret_cast<Q*>(s)[e] = reinterpret_cast<const Q*>(row)[e];
      __syncthreads();
      for (int e = threadIdx.x; e < pieces; e += 256) {
        const int p = e / np, c = (e - p * np) * V;
        float f[V];
#pragma unroll
        for (int k = 0; k < V; ++k) f[k] = to_f32(s[(c + k) * HW + p]);
        if (dact != ACT_NONE) {
          float a[V];
          unpack_piece<T, P>(*reinterpret_cast<const P*>(aux + (pb + p) * ld_aux + c), a);
          act_bwd_n<V>(dact, dact_param, relu_quirk, a, f);
        }
        *reinterpret_cast<P*>(img + (pb + p) * ld_img + c) = pack_piece<T, P>(f);
      }
    }
  }
}

// Pooling at the end of the image layers, together with the change to the flattened rows the dense layers read (fwd) and back (bwd): a block
// takes an image, whose pooled values lie in shared memory channel by channel (`step` floats apart, an odd number: a warp's channels fall into
// different banks). Values and places of the maxima are those of pool_*_kernel and nchw_*_kernel. What bounds both is the latency of an
// image's loads, so blocks are large and a thread's loads are issued together. 256 images of 24 x 24 x 20,
// f32: forward 7.4 us as two kernels, 5.9 so, backward 10.7 and 8.9; 64 of 8 x 8 x 16 4.6 and 3.0, 4.0 and 2.7.
constexpr int PF_THREADS = 512;
template <typename T>
__device__ __forceinline__ void flat_row_move(T* row, T* s, int C, int HW, int step, bool wide, bool out, const FastDiv<unsigned>& by_hw) {
  constexpr int VQ = 16 / (int)sizeof(T);
  const int n = C * HW;
  if (!wide) {
    for (int e = threadIdx.x; e < n; e += PF_THREADS) {
      const int c = (int)by_hw(e), at = e + c * (step - HW);
      if (out) row[e] = s[at];
      else s[at] = row[e];
    }
    return;
  }
  for (int e = threadIdx.x * VQ; e < n; e += PF_THREADS * VQ) {
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (!out) w = *reinterpret_cast<const uint4*>(row + e);
    T* const v = reinterpret_cast<T*>(&w);
    int c = (int)by_hw(e), p = e - c * HW;
#pragma unroll
    for (int k = 0; k < VQ; ++k) {
      if (out) v[k] = s[c * step + p];
      else s[c * step + p] = v[k];
      if (++p == HW) { p = 0; ++c; }
    }
    if (out) *reinterpret_cast<uint4*>(row + e) = w;
  }
}
struct PoolFlat {
  FastDiv<unsigned> C, OW, W, S, HW;      // pieces of a pixel; the pooled image's pixels
  int step, wide;
};
template <typename T, typename P>
__global__ void __launch_bounds__(PF_THREADS) pool_flat_fwd_kernel(const OnoConvGeom g, const T* x, int ldx, T* y, int ldy, int* arg, int act,
                                                                   float act_param, T* flat, int ld_flat, const PoolFlat by) {
  extern __shared__ __align__(16) unsigned char pool_smem[];
  T* const s = reinterpret_cast<T*>(pool_smem);
  constexpr int V = (int)(sizeof(P) / sizeof(T));
  const int HWo = g.OH * g.OW, pieces = HWo * (int)by.C.d;
  const int b = blockIdx.x;
  const T* const xb = x + (long long)b * g.H * g.W * ldx;
  for (int e = threadIdx.x; e < pieces; e += PF_THREADS) {
    const int r = (int)by.C(e), c = (e - r * (int)by.C.d) * V, oy = (int)by.OW(r), ox = r - oy * g.OW;
    float best[V];
    int where[V];
#pragma unroll
    for (int k = 0; k < V; ++k) { best[k] = -INFINITY; where[k] = -1; }
    for (int ky = 0; ky < g.K; ++ky)
#pragma unroll 2
      for (int kx = 0; kx < g.K; ++kx) {
        const int iy = oy * g.S + ky - g.P, ix = ox * g.S + kx - g.P;
        const bool in = iy >= 0 && iy < g.H && ix >= 0 && ix < g.W;
        P w{};
        if (in) w = *reinterpret_cast<const P*>(xb + (long long)(iy * g.W + ix) * ldx + c);
        float v[V];
        unpack_piece<T, P>(w, v);
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (v[k] >= best[k]) { best[k] = v[k]; where[k] = in ? iy * g.W + ix : -1; }
      }
    const long long pix = (long long)b * HWo + r;
#pragma unroll
    for (int k = 0; k < V; ++k) arg[pix * g.C + c + k] = where[k];
    act_fwd_n<V>(act, act_param, best);
    const P out = pack_piece<T, P>(best);
    *reinterpret_cast<P*>(y + pix * ldy + c) = out;
    const T* const o = reinterpret_cast<const T*>(&out);
#pragma unroll
    for (int k = 0; k < V; ++k) s[(c + k) * by.step + r] = o[k];
  }
  __syncthreads();
  flat_row_move<T>(flat + (long long)b * ld_flat, s, g.C, HWo, by.step, by.wide, true, by.HW);
}
template <typename T, typename P>
__global__ void __launch_bounds__(PF_THREADS) pool_flat_bwd_kernel(const OnoConvGeom g, T* flat, int ld_flat, const T* y, int ldy, const int* arg,
                                                                   int act, float act_param, int relu_quirk, const T* aux, int ld_aux, int dact,
                                                                   float dact_param, T* dx, int ld_dx, const PoolFlat by) {
  extern __shared__ __align__(16) unsigned char pool_smem[];
  T* const s = reinterpret_cast<T*>(pool_smem);
  constexpr int V = (int)(sizeof(P) / sizeof(T));
  const int HWo = g.OH * g.OW, pieces = g.H * g.W * (int)by.C.d;
  const int b = blockIdx.x;
  const long long pix0 = (long long)b * g.H * g.W, out0 = (long long)b * HWo;
  flat_row_move<T>(flat + (long long)b * ld_flat, s, g.C, HWo, by.step, by.wide, false, by.HW);
  __syncthreads();
  for (int e = threadIdx.x; e < pieces; e += PF_THREADS) {
    const int pix = (int)by.C(e), c = (e - pix * (int)by.C.d) * V, iy = (int)by.W(pix), ix = pix - iy * g.W;
    P av{};
    if (dact != ACT_NONE) av = *reinterpret_cast<const P*>(aux + (pix0 + pix) * ld_aux + c);
    // windows oy with oy * S <= iy + P < oy * S + K
    const int oy1 = min(g.OH - 1, (int)by.S(iy + g.P)), ox1 = min(g.OW - 1, (int)by.S(ix + g.P));
    const int oy0 = iy + g.P < g.K ? 0 : (int)by.S(iy + g.P - g.K + g.S), ox0 = ix + g.P < g.K ? 0 : (int)by.S(ix + g.P - g.K + g.S);
    float v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = 0.f;
    for (int oy = oy0; oy <= oy1; ++oy)
      for (int ox = ox0; ox <= ox1; ++ox) {
        const int r = oy * g.OW + ox;
        const int* const ap = arg + (out0 + r) * g.C + c;
        int w[V];
        if constexpr (V >= 4) {
#pragma unroll
          for (int k = 0; k < V; k += 4) *reinterpret_cast<int4*>(w + k) = *reinterpret_cast<const int4*>(ap + k);
        } else {
          w[0] = ap[0];
        }
        float t[V];
#pragma unroll
        for (int k = 0; k < V; ++k) t[k] = to_f32(s[(c + k) * by.step + r]);
        if (act != ACT_NONE) {
          float yv[V];
          unpack_piece<T, P>(*reinterpret_cast<const P*>(y + (out0 + r) * ldy + c), yv);
          act_bwd_n<V>(act, act_param, relu_quirk, yv, t);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] += w[k] == pix ? t[k] : 0.f;
      }
    if (dact != ACT_NONE) {
      float a[V];
      unpack_piece<T, P>(av, a);
      act_bwd_n<V>(dact, dact_param, relu_quirk, a, v);
    }
    *reinterpret_cast<P*>(dx + (pix0 + pix) * ld_dx + c) = pack_piece<T, P>(v);
  }
}

static int grid_of(long long n) {
  long long g = (n + 255) / 256;
  if (g < 1) g = 1;
  if (g > 148 * 32) g = 148 * 32;
  return (int)g;
}
static int done(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("%s launch failed (%lld)", what, (long long)e, 0); return -7; }
  return 0;
}

}  // namespace ono

using namespace ono;
typedef __nv_bfloat16 bf16;

#define ONO_DISPATCH(dtype, CALL_F32, CALL_BF16) \
  if ((dtype) == 0) { CALL_F32; } else { CALL_BF16; }

extern "C" int ono_im2col(const OnoConvGeom* g, int dtype, const void* x, int ldx, void* cols, int ld_cols, void* colsT,
                          int ld_colsT, ono_stream_t st) {
  const long long n = (long long)g->B * g->OH * g->OW * g->C * g->K * g->K, rows = (long long)g->B * g->OH * g->OW;
  const dim3 blk(32, 8);
  const int grid = grid_of(n / 4);
  const int V = piece_width(dtype == 0 ? 4 : 2, g->C, ldx | ld_cols, (uintptr_t)x | (uintptr_t)cols);
  // no transposed copy, 32-bit pixel indexes, a piece table that fits
  if (!colsT && g->C * g->K * g->K / V <= IM_MAX_PIECES && g->K < (1 << 15) && (long long)g->B * g->H * g->W < (1ll << 30) &&
      rows < (1ll << 30) && (long long)(g->K + 1) * g->W * ldx < (1ll << 30)) {
    const unsigned nb = (unsigned)((rows + IM_ROWS - 1) / IM_ROWS);
    const cudaStream_t s = (cudaStream_t)st;
#define ONO_IM2COL(T, P) im2col_vec_kernel<T, P><<<nb, 256, 0, s>>>(*g, (const T*)x, ldx, (T*)cols, ld_cols, (int)rows)
    if (dtype == 0) {
      if (V == 4) ONO_IM2COL(float, uint4);
      else if (V == 2) ONO_IM2COL(float, uint2);
      else ONO_IM2COL(float, unsigned);
    } else {
      if (V == 8) ONO_IM2COL(bf16, uint4);
      else if (V == 4) ONO_IM2COL(bf16, uint2);
      else if (V == 2) ONO_IM2COL(bf16, unsigned);
      else ONO_IM2COL(bf16, unsigned short);
    }
#undef ONO_IM2COL
    return done("im2col");
  }
  ONO_DISPATCH(dtype,
               (im2col_kernel<float><<<grid, blk, 0, (cudaStream_t)st>>>(*g, (const float*)x, ldx, (float*)cols, ld_cols, (float*)colsT, ld_colsT)),
               (im2col_kernel<bf16><<<grid, blk, 0, (cudaStream_t)st>>>(*g, (const bf16*)x, ldx, (bf16*)cols, ld_cols, (bf16*)colsT, ld_colsT)))
  return done("im2col");
}

extern "C" int ono_col2im(const OnoConvGeom* g, int dtype, const void* dcols, int ld_dcols, const void* aux, int ld_aux,
                          int dact, float dact_param, int relu_quirk, void* dx, int ld_dx, void* dxT, int ld_dxT, ono_stream_t st) {
  const long long n = (long long)g->B * g->H * g->W * ((g->C + 31) / 32 * 32);
  const dim3 blk(32, 8);
  const int grid = grid_of(n / 4);
  const int V = piece_width(dtype == 0 ? 4 : 2, g->C, ld_dcols | ld_dx | (aux ? ld_aux : 0), (uintptr_t)dcols | (uintptr_t)dx | (uintptr_t)aux);
  const long long pieces = (long long)g->B * g->H * g->W * (g->C / V);
  const bool vec = !dxT && pieces < (1ll << 31) && (long long)g->B * g->OH * g->OW < (1ll << 31) && (aux || dact == ACT_NONE);
#define ONO_COL2IM_RUN(T, P, KK, SS)                                                                                              \
  (col2im_vec_kernel<T, P, KK, SS><<<grid_of(pieces), 256, 0, (cudaStream_t)st>>>(*g, (const T*)dcols, ld_dcols, (const T*)aux,    \
                                                                                 ld_aux, dact, dact_param, relu_quirk, (T*)dx,    \
                                                                                 ld_dx, (unsigned)pieces))
#define ONO_COL2IM_VEC(KK, SS)                                                                                                    \
  if (vec && g->K == KK && g->S == SS) {                                                                                          \
    if (dtype == 0) {                                                                                                             \
      if (V == 4) ONO_COL2IM_RUN(float, uint4, KK, SS);                                                                           \
      else if (V == 2) ONO_COL2IM_RUN(float, uint2, KK, SS);                                                                      \
      else ONO_COL2IM_RUN(float, unsigned, KK, SS);                                                                               \
    } else {                                                                                                                      \
      if (V == 8) ONO_COL2IM_RUN(bf16, uint4, KK, SS);                                                                            \
      else if (V == 4) ONO_COL2IM_RUN(bf16, uint2, KK, SS);                                                                       \
      else if (V == 2) ONO_COL2IM_RUN(bf16, unsigned, KK, SS);                                                                    \
      else ONO_COL2IM_RUN(bf16, unsigned short, KK, SS);                                                                          \
    }                                                                                                                             \
    return done("col2im");                                                                                                        \
  }
  ONO_COL2IM_VEC(3, 1)
  ONO_COL2IM_VEC(3, 2)
  ONO_COL2IM_VEC(5, 1)
  ONO_COL2IM_VEC(5, 2)
#undef ONO_COL2IM_VEC
#undef ONO_COL2IM_RUN
  ONO_DISPATCH(dtype,
               (col2im_kernel<float><<<grid, blk, 0, (cudaStream_t)st>>>(*g, (const float*)dcols, ld_dcols, (const float*)aux, ld_aux, dact, dact_param, relu_quirk, (float*)dx, ld_dx, (float*)dxT, ld_dxT)),
               (col2im_kernel<bf16><<<grid, blk, 0, (cudaStream_t)st>>>(*g, (const bf16*)dcols, ld_dcols, (const bf16*)aux, ld_aux, dact, dact_param, relu_quirk, (bf16*)dx, ld_dx, (bf16*)dxT, ld_dxT)))
  return done("col2im");
}

extern "C" int ono_conv1_fwd(const OnoConvGeom* g, int F, int dtype, const void* x, int ldx, const float* kparams, const float* bias,
                             int act, float act_param, void* y, int ldy, ono_stream_t st) {
  if (!g || g->C != 1 || g->K * g->K > C1_MAXKK || F <= 0) { set_error("conv1_fwd: needs one input channel and k <= 5%s", "", 0, 0); return -1; }
  const long long rows = (long long)g->B * g->OH * g->OW;
  if (rows >= (1ll << 31)) { set_error("conv1_fwd: too many output pixels%s", "", 0, 0); return -1; }
  const int chunks = c1_chunks(g);
  const size_t sm = c1_img_smem(g, chunks, false);
  if (sm && (long long)g->B * chunks < (1ll << 31)) {
    const dim3 grid((unsigned)(g->B * chunks), (F + C1_FC - 1) / C1_FC);
    const cudaStream_t s = (cudaStream_t)st;
    const int esz = dtype == 0 ? 4 : 2;
    const int vec = F % 4 == 0 && ldy % 4 == 0 && ((uintptr_t)y & (uintptr_t)(4 * esz - 1)) == 0;
#define ONO_C1_FWD(T, KK, SS) conv1_fwd_img_kernel<T, KK, SS><<<grid, 256, sm, s>>>(*g, F, (const T*)x, ldx, kparams, bias, act, act_param, (T*)y, ldy, vec, chunks)
    if (g->S > 2 && g->K == 3) { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 3, 0), ONO_C1_FWD(bf16, 3, 0)) }
    else if (g->S > 2) { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 5, 0), ONO_C1_FWD(bf16, 5, 0)) }
    else if (g->K == 3 && g->S == 1) { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 3, 1), ONO_C1_FWD(bf16, 3, 1)) }
    else if (g->K == 3) { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 3, 2), ONO_C1_FWD(bf16, 3, 2)) }
    else if (g->S == 1) { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 5, 1), ONO_C1_FWD(bf16, 5, 1)) }
    else { ONO_DISPATCH(dtype, ONO_C1_FWD(float, 5, 2), ONO_C1_FWD(bf16, 5, 2)) }
#undef ONO_C1_FWD
    return done("conv1_fwd");
  }
  const dim3 blk(32, 8), grid((unsigned)std::min<long long>((rows + 255) / 256, 148 * 8), (F + 31) / 32);
  ONO_DISPATCH(dtype,
               (conv1_fwd_kernel<float><<<grid, blk, 0, (cudaStream_t)st>>>(*g, F, (const float*)x, ldx, kparams, bias, act, act_param, (float*)y, ldy)),
               (conv1_fwd_kernel<bf16><<<grid, blk, 0, (cudaStream_t)st>>>(*g, F, (const bf16*)x, ldx, kparams, bias, act, act_param, (bf16*)y, ldy)))
  return done("conv1_fwd");
}

extern "C" int ono_conv1_wgrad(const OnoConvGeom* g, int F, int dtype, const void* x, int ldx, const void* dy, int ld_dy, float* gk,
                               float* gb, float beta, ono_stream_t st) {
  if (!g || g->C != 1 || g->K * g->K > C1_MAXKK || F <= 0 || F > C1_MAXF) { set_error("conv1_wgrad: needs one input channel, k <= 5, F <= 128%s", "", 0, 0); return -1; }
  const long long rows = (long long)g->B * g->OH * g->OW;
  const dim3 blk(32, 8);
  if (rows >= (1ll << 31)) { set_error("conv1_wgrad: too many output pixels%s", "", 0, 0); return -1; }
  const int esz = dtype == 0 ? 4 : 2;
  const int vec = F % 4 == 0 && ld_dy % 4 == 0 && ((uintptr_t)dy & (uintptr_t)(4 * esz - 1)) == 0;
  // bf16: the fixed order wherever an image fits. f32: where the tiled kernel has no form.
  if (const size_t sm = dtype != 0 || g->S > 2 ? c1_walk_smem(g) : 0) {
    const int nb = std::min(g->B, C1_MAXBLOCKS);
    const cudaStream_t s = (cudaStream_t)st;
#define ONO_C1_WALK(T, KK, V) conv1_wgrad_walk_kernel<T, KK, V><<<nb, 256, sm, s>>>(*g, F, (const T*)x, ldx, (const T*)dy, ld_dy)
    if (vec && g->K == 3) { ONO_DISPATCH(dtype, ONO_C1_WALK(float, 3, 4), ONO_C1_WALK(bf16, 3, 4)) }
    else if (vec) { ONO_DISPATCH(dtype, ONO_C1_WALK(float, 5, 4), ONO_C1_WALK(bf16, 5, 4)) }
    else if (g->K == 3) { ONO_DISPATCH(dtype, ONO_C1_WALK(float, 3, 1), ONO_C1_WALK(bf16, 3, 1)) }
    else { ONO_DISPATCH(dtype, ONO_C1_WALK(float, 5, 1), ONO_C1_WALK(bf16, 5, 1)) }
#undef ONO_C1_WALK
    const int pairs = F * (g->K * g->K + 1);
    conv1_wgrad_reduce_kernel<<<(pairs + 7) / 8, 256, 0, s>>>(F, g->K * g->K, nb, gk, gb, beta);
    return done("conv1_wgrad");
  }
  const int chunks = c1_wgrad_chunks(g, F);
  const size_t sm = c1_img_smem(g, chunks, true);
  if (sm && (long long)g->B * chunks < (1ll << 31)) {
    const int nb = std::min(g->B * chunks, c1_wgrad_blocks(g));
    const cudaStream_t s = (cudaStream_t)st;
#define ONO_C1_WGRAD(T, KK, SS) conv1_wgrad_img_kernel<T, KK, SS><<<nb, 256, sm, s>>>(*g, F, (const T*)x, ldx, (const T*)dy, ld_dy, vec, chunks)
    if (g->K == 3 && g->S == 1) { ONO_DISPATCH(dtype, ONO_C1_WGRAD(float, 3, 1), ONO_C1_WGRAD(bf16, 3, 1)) }
    else if (g->K == 3) { ONO_DISPATCH(dtype, ONO_C1_WGRAD(float, 3, 2), ONO_C1_WGRAD(bf16, 3, 2)) }
    else if (g->S == 1) { ONO_DISPATCH(dtype, ONO_C1_WGRAD(float, 5, 1), ONO_C1_WGRAD(bf16, 5, 1)) }
    else { ONO_DISPATCH(dtype, ONO_C1_WGRAD(float, 5, 2), ONO_C1_WGRAD(bf16, 5, 2)) }
#undef ONO_C1_WGRAD
    const int pairs = F * (g->K * g->K + 1);
    conv1_wgrad_reduce_kernel<<<(pairs + 7) / 8, 256, 0, s>>>(F, g->K * g->K, nb, gk, gb, beta);
    return done("conv1_wgrad");
  }
  const int grid = (int)std::min<long long>((rows + 255) / 256, C1_MAXBLOCKS);
  ONO_DISPATCH(dtype,
               (conv1_wgrad_kernel<float><<<grid, blk, 0, (cudaStream_t)st>>>(*g, F, (const float*)x, ldx, (const float*)dy, ld_dy, gk, gb, beta)),
               (conv1_wgrad_kernel<bf16><<<grid, blk, 0, (cudaStream_t)st>>>(*g, F, (const bf16*)x, ldx, (const bf16*)dy, ld_dy, gk, gb, beta)))
  return done("conv1_wgrad");
}

extern "C" int ono_conv_kperm(int F, int C, int K, int dir, int dtype, const float* src, int ld_src, void* dst, int ld_dst,
                              void* dstT, int ld_dstT, float beta, ono_stream_t st) {
  if (F <= 0 || C <= 0 || K <= 0 || !src || !dst) { set_error("bad kperm args%s", "", 0, 0); return -1; }
  const long long n = (long long)F * C * K * K;
  ONO_DISPATCH(dtype,
               (kperm_kernel<float><<<grid_of(n), 256, 0, (cudaStream_t)st>>>(F, C, K, dir, src, ld_src, dst, ld_dst, (float*)dstT, ld_dstT, beta)),
               (kperm_kernel<bf16><<<grid_of(n), 256, 0, (cudaStream_t)st>>>(F, C, K, dir, src, ld_src, dst, ld_dst, (bf16*)dstT, ld_dstT, beta)))
  return done("conv_kperm");
}

constexpr long long POOL_MAX_32 = (1ll << 31) - (1ll << 24);      // an index one grid past the end still fits
// The pieces the pooling kernels exist for: 16 and 8 bytes and single values; 64-bit indexes with single values only.
static int pool_width(int dtype, int C, long long pixels, int lds, uintptr_t ptrs) {
  const int v = piece_width(dtype == 0 ? 4 : 2, C, lds, ptrs);
  return v == 2 || pixels * C >= POOL_MAX_32 ? 1 : v;
}
#define ONO_POOL_PIECES(RUN)                                                                             \
  if (!small) { if (dtype == 0) RUN(float, float, long long); else RUN(bf16, bf16, long long); }         \
  else if (dtype == 0) { if (V == 4) RUN(float, uint4, unsigned); else RUN(float, float, unsigned); }    \
  else if (V == 8) RUN(bf16, uint4, unsigned);                                                           \
  else if (V == 4) RUN(bf16, uint2, unsigned);                                                           \
  else RUN(bf16, bf16, unsigned);

extern "C" int ono_pool_fwd(const OnoConvGeom* g, int dtype, const void* x, int ldx, void* y, int ldy, void* yT, int ld_yT,
                            int* arg, int act, float act_param, ono_stream_t st) {
  const int V = pool_width(dtype, g->C, (long long)g->B * g->OH * g->OW, ldx | ldy, (uintptr_t)x | (uintptr_t)y);
  const long long n = (long long)g->B * g->OH * g->OW * (g->C / V);
  const bool small = n < POOL_MAX_32;
#define ONO_POOL_FWD(T, P, I) (pool_fwd_kernel<T, P, I><<<grid_of(n), 256, 0, (cudaStream_t)st>>>(*g, (const T*)x, ldx, (T*)y, ldy, (T*)yT, ld_yT, arg, act, act_param, PoolDiv<I>(g->C / V, g->OW, g->OH, g->S), (I)n))
  ONO_POOL_PIECES(ONO_POOL_FWD)
#undef ONO_POOL_FWD
  return done("pool_fwd");
}

extern "C" int ono_pool_bwd(const OnoConvGeom* g, int dtype, const void* d, int ldd, const void* y, int ldy, const int* arg,
                            int act, float act_param, int relu_quirk, const void* aux, int ld_aux, int dact, float dact_param,
                            void* dx, int ld_dx, void* dxT, int ld_dxT, ono_stream_t st) {
  if (dact != ACT_NONE && !aux) { set_error("pool_bwd: a derivative needs the stored activation%s", "", 0, 0); return -1; }
  const int V = pool_width(dtype, g->C, (long long)g->B * g->H * g->W, ldd | ldy | ld_dx | (aux ? ld_aux : 0),
                           (uintptr_t)d | (uintptr_t)y | (uintptr_t)aux | (uintptr_t)dx);
  const long long n = (long long)g->B * g->H * g->W * (g->C / V);
  const bool small = n < POOL_MAX_32;
#define ONO_POOL_BWD(T, P, I)                                                                                                      \
  (pool_bwd_kernel<T, P, I><<<grid_of(n), 256, 0, (cudaStream_t)st>>>(*g, (const T*)d, ldd, (const T*)y, ldy, arg, act, act_param,  \
                                                                     relu_quirk, (const T*)aux, ld_aux, dact, dact_param, (T*)dx,  \
                                                                     ld_dx, (T*)dxT, ld_dxT, PoolDiv<I>(g->C / V, g->W, g->H, g->S), (I)n))
  ONO_POOL_PIECES(ONO_POOL_BWD)
#undef ONO_POOL_BWD
  return done("pool_bwd");
}

static size_t pool_flat_smem(const OnoConvGeom* g, int dtype) { return (size_t)g->C * ((g->OH * g->OW) | 1) * (dtype == 0 ? 4 : 2); }
// Images whose pooled values fit the default shared memory. A block goes through its image in rounds of PF_THREADS pieces, with a trip to memory for
// each, so an image has at most twelve of them; where the images fill less than half of the SMs, and the separate kernels spread the few there are
// over the idle ones, two, or four where no windows overlap (each piece is then read once, and an input pixel has one window). More images
// keep those kernels busy all the time (2048 of 24 x 24 x 16: 30.6 us forward as two kernels, 37.3 so; 512 of 16 x 16 x 40, bf16, 10.9 and 8.4).
// There and back, as four kernels and as two, us: 64 of 24 x 24 x 20 12.0 and 11.5, 16 of 12 x 12 x 16 8.9 and 7.0; beyond the line, windows of 2 with
// stride 1, 6 of 24 x 24 x 6 bf16 8.9 and 18.7, 2 of 21 x 21 x 24 bf16 10.5 and 15.8; 388 of 27 x 27 x 64, 4 x 4, 61.6 and 72.9. Of 250 drawn
// layers below 48 KB and 592 images 225 are on this side, 8 of them slower by more than 5 % (at most 1.22 times), 3 beyond it would be faster by as much.
// Of 250 more on this side 9 are slower by more than 5 %, at most 1.19 times.
extern "C" int ono_pool_flat_fits(const OnoConvGeom* g, int dtype) {
  if (!g || g->B <= 0 || pool_flat_smem(g, dtype) > 48 * 1024 || (long long)g->H * g->W >= (1 << 20) || (long long)g->H * g->W * g->C >= (1ll << 30)) return 0;
  const long long pieces = (long long)g->H * g->W * (g->C / pool_width(dtype, g->C, 0, 0, 0)), rounds = (pieces + PF_THREADS - 1) / PF_THREADS;
  return g->B <= 4 * ono_num_sms() && rounds <= (g->B >= 64 ? 12 : g->K <= g->S ? 4 : 2);
}
static PoolFlat pool_flat_of(const OnoConvGeom* g, int dtype, int V, const void* flat, int ld_flat) {
  const int HWo = g->OH * g->OW, per = dtype == 0 ? 4 : 8;
  return PoolFlat{FastDiv<unsigned>(g->C / V), FastDiv<unsigned>(g->OW), FastDiv<unsigned>(g->W), FastDiv<unsigned>(g->S), FastDiv<unsigned>(HWo),
                  HWo | 1, (g->C * HWo) % per == 0 && ld_flat % per == 0 && ((uintptr_t)flat & 15) == 0};
}
#define ONO_POOL_FLAT_PIECES(RUN)                                        \
  if (dtype == 0) { if (V == 4) RUN(float, uint4); else RUN(float, float); } \
  else if (V == 8) RUN(bf16, uint4);                                     \
  else if (V == 4) RUN(bf16, uint2);                                     \
  else RUN(bf16, bf16);

extern "C" int ono_pool_flat_fwd(const OnoConvGeom* g, int dtype, const void* x, int ldx, void* y, int ldy, int* arg, int act, float act_param,
                                 void* flat, int ld_flat, ono_stream_t st) {
  if (!ono_pool_flat_fits(g, dtype)) { set_error("pool_flat_fwd: sizes it does not take%s", "", 0, 0); return -1; }
  const int V = pool_width(dtype, g->C, 0, ldx | ldy, (uintptr_t)x | (uintptr_t)y);
  const PoolFlat by = pool_flat_of(g, dtype, V, flat, ld_flat);
#define ONO_POOL_FLAT_FWD(T, P) (pool_flat_fwd_kernel<T, P><<<g->B, PF_THREADS, pool_flat_smem(g, dtype), (cudaStream_t)st>>>(*g, (const T*)x, ldx, (T*)y, ldy, arg, act, act_param, (T*)flat, ld_flat, by))
  ONO_POOL_FLAT_PIECES(ONO_POOL_FLAT_FWD)
#undef ONO_POOL_FLAT_FWD
  return done("pool_flat_fwd");
}

extern "C" int ono_pool_flat_bwd(const OnoConvGeom* g, int dtype, const void* flat, int ld_flat, const void* y, int ldy, const int* arg, int act,
                                 float act_param, int relu_quirk, const void* aux, int ld_aux, int dact, float dact_param, void* dx, int ld_dx,
                                 ono_stream_t st) {
  if (dact != ACT_NONE && !aux) { set_error("pool_flat_bwd: a derivative needs the stored activation%s", "", 0, 0); return -1; }
  if (!ono_pool_flat_fits(g, dtype)) { set_error("pool_flat_bwd: sizes it does not take%s", "", 0, 0); return -1; }
  const int V = (uintptr_t)arg & 15 ? 1 : pool_width(dtype, g->C, 0, ldy | ld_dx | (aux ? ld_aux : 0), (uintptr_t)y | (uintptr_t)aux | (uintptr_t)dx);
  const PoolFlat by = pool_flat_of(g, dtype, V, flat, ld_flat);
#define ONO_POOL_FLAT_BWD(T, P)                                                                                                              \
  (pool_flat_bwd_kernel<T, P><<<g->B, PF_THREADS, pool_flat_smem(g, dtype), (cudaStream_t)st>>>(*g, (T*)flat, ld_flat, (const T*)y, ldy, arg, \
                                                                                             act, act_param, relu_quirk, (const T*)aux, \
                                                                                             ld_aux, dact, dact_param, (T*)dx, ld_dx, by))
  ONO_POOL_FLAT_PIECES(ONO_POOL_FLAT_BWD)
#undef ONO_POOL_FLAT_BWD
  return done("pool_flat_bwd");
}

extern "C" int ono_nchw_flat(int dtype, int B, int C, int HW, int to_flat, void* img, int ld_img, void* flat, int ld_flat,
                             void* outT, int ld_outT, const void* aux, int ld_aux, int dact, float dact_param, int relu_quirk,
                             ono_stream_t st) {
  const int esz = dtype == 0 ? 4 : 2;
  const size_t image = (size_t)C * HW * esz;
  // Whole images where one fits the default shared memory, nobody wants the transposed copy and a channel is not all there is;
  // from a few images on (below that the tiles fill more SMs).
  if (!outT && image <= 48 * 1024 && C > 1 && B >= 16) {
    const int V = piece_width(esz, C, ld_img | (aux ? ld_aux : 0), (uintptr_t)img | (uintptr_t)aux);
    const bool wide = piece_width(esz, C * HW, ld_flat, (uintptr_t)flat) * esz == 16;
    const cudaStream_t s = (cudaStream_t)st;
    const int nb = std::min(B, 148 * 8);
#define ONO_NCHW(T, P, Q) nchw_image_kernel<T, P, Q><<<nb, 256, image, s>>>(B, C, HW, to_flat, (T*)img, ld_img, (T*)flat, ld_flat, (const T*)aux, ld_aux, dact, dact_param, relu_quirk)
    if (dtype == 0) {
      if (V == 4 && wide) ONO_NCHW(float, uint4, uint4);
      else if (wide) ONO_NCHW(float, float, uint4);
      else ONO_NCHW(float, float, float);
    } else {
      if (V == 8 && wide) ONO_NCHW(bf16, uint4, uint4);
      else if (V >= 4 && wide) ONO_NCHW(bf16, uint2, uint4);
      else if (wide) ONO_NCHW(bf16, bf16, uint4);
      else ONO_NCHW(bf16, bf16, bf16);
    }
#undef ONO_NCHW
    return done("nchw_flat");
  }
  const dim3 grid((unsigned)((HW + 31) / 32) * (unsigned)((C + 31) / 32), (unsigned)std::min(B, 65535));
  ONO_DISPATCH(dtype,
               (nchw_flat_kernel<float><<<grid, 256, 0, (cudaStream_t)st>>>(B, C, HW, to_flat, (float*)img, ld_img, (float*)flat, ld_flat, (float*)outT, ld_outT, (const float*)aux, ld_aux, dact, dact_param, relu_quirk)),
               (nchw_flat_kernel<bf16><<<grid, 256, 0, (cudaStream_t)st>>>(B, C, HW, to_flat, (bf16*)img, ld_img, (bf16*)flat, ld_flat, (bf16*)outT, ld_outT, (const bf16*)aux, ld_aux, dact, dact_param, relu_quirk)))
  return done("nchw_flat");
}
