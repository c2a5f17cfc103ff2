// Bandwidth-bound kernels around the GEMMs: fused softmax + loss + first backward step, bias
// gradient, optimizers on flat shards, round-cadence local SGD, Philox initialisers and the
// gather / cast / transpose that feeds the tensor-core operands.
// Reference semantics: machine_learning/src/arch/loss/{mse,cross_entropy}.rs, arch/layers/softmax.rs,
// optimization/{gradient_descent,gradient_descent_with_momentum,adam}.rs, param_manager.rs:168-197.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "../core/philox.h"
#include "act.cuh"
#include "loss.cuh"
#include "ono_kernels.h"
#include "opt.cuh"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);

static int launch_ok(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s launch failed (%lld)", what, (long long)e, 0);
    return -7;
  }
  return 0;
}

// ------------------------------------------------------------------------------------------------
// Loss: one warp per row.
// ------------------------------------------------------------------------------------------------
// NV > 0: a lane keeps its logits and labels in registers, NV of each (at least ceil(C / 32)); NV < 0: the warp keeps them in shared memory
// (above 128 classes, LOSS_ROW at most; unrolled over more registers the code would cost more to fetch than it saves). Either way all of a
// row's loads are in flight at once and the exponentials are taken once. With the passes over memory (NV = 0, longer rows)
// 512 x 1000 took 29.0 us (now 10.5), every pass a chain of 32 dependent round trips. The additions are in the same order in every form.
constexpr int LOSS_ROW = 1024;
template <int NV>
__global__ void __launch_bounds__(128) loss_kernel(const OnoLoss l) {
  __shared__ float s_row[NV < 0 ? 2 * 4 * LOSS_ROW : 1];
  const int warps_per_block = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_n = 1.0f / ((float)l.B * (float)l.C);
  double block_loss = 0.0;
  int block_correct = 0;
  for (int row = blockIdx.x * warps_per_block + warp; row < l.B; row += gridDim.x * warps_per_block) {
    const float* a = l.a + (size_t)row * l.ld;
    const float* y = l.y + (size_t)row * l.ldy;
    float* sp = s_row;
    if (NV < 0) {
      sp = s_row + 2 * LOSS_ROW * warp;
      __syncwarp();                   // the previous row has been read
      for (int j0 = lane; j0 < l.C; j0 += 256) {
        float ta[8], ty[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (j0 + 32 * u < l.C) { ta[u] = a[j0 + 32 * u]; ty[u] = y[j0 + 32 * u]; }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (j0 + 32 * u < l.C) { sp[j0 + 32 * u] = ta[u]; sp[LOSS_ROW + j0 + 32 * u] = ty[u]; }
      }
      a = sp;                         // a lane reads only what it has written itself
      y = sp + LOSS_ROW;
    }
    auto put = [&](int j, float p, float d) {
      if (l.probs) l.probs[(size_t)row * l.ld + j] = p;
      if (l.d_f32) l.d_f32[(size_t)row * l.ld_d + j] = d;
      if (l.d_bf16) reinterpret_cast<__nv_bfloat16*>(l.d_bf16)[(size_t)row * l.ld_d + j] = __float2bfloat16_rn(d);
      if (l.dT_f32) l.dT_f32[(size_t)j * l.ld_dT + row] = d;
      if (l.dT_bf16) reinterpret_cast<__nv_bfloat16*>(l.dT_bf16)[(size_t)j * l.ld_dT + row] = __float2bfloat16_rn(d);
    };
    const LossRow r = loss_row<NV>(l, a, y, l.aux ? l.aux + (size_t)row * l.ld : nullptr, sp, lane, put);
    if (lane == 0) { block_loss += (double)r.loss; block_correct += r.correct; }
  }
  __shared__ double s_loss[32];
  __shared__ int s_correct[32];
  if (lane == 0) { s_loss[warp] = block_loss; s_correct[warp] = block_correct; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    int c = 0;
    for (int w = 0; w < warps_per_block; ++w) { t += s_loss[w]; c += s_correct[w]; }
    if (l.loss_sum) atomicAdd(l.loss_sum, t * (double)inv_n);
    if (l.correct && c) atomicAdd(l.correct, c);
  }
}

// ------------------------------------------------------------------------------------------------
// Softmax layer (forward and Jacobian-vector product): one warp per row, three passes over the row.
// ------------------------------------------------------------------------------------------------
__global__ void softmax_kernel(const OnoSoftmax a) {
  const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(a.out_bf16);
  __nv_bfloat16* otb = reinterpret_cast<__nv_bfloat16*>(a.outT_bf16);
  const __nv_bfloat16* pb = reinterpret_cast<const __nv_bfloat16*>(a.p_bf16);
  for (int row = blockIdx.x * wpb + warp; row < a.B; row += gridDim.x * wpb) {
    const float* x = a.x + (size_t)row * a.ld_x;
    float mx = -INFINITY, inv_z = 1.0f, dot = 0.0f;
    if (!a.backward) {
      for (int j = lane; j < a.C; j += 32) mx = fmaxf(mx, x[j]);
      mx = warp_max(mx);
      float z = 0.0f;
      for (int j = lane; j < a.C; j += 32) z += expf(x[j] - mx);
      inv_z = 1.0f / warp_sum(z);
    } else {
      for (int j = lane; j < a.C; j += 32) {
        const float p = a.p_f32 ? a.p_f32[(size_t)row * a.ld_p + j] : __bfloat162float(pb[(size_t)row * a.ld_p + j]);
        dot += p * x[j];
      }
      dot = warp_sum(dot);
    }
    for (int j = lane; j < a.C; j += 32) {
      float v;
      if (!a.backward) v = expf(x[j] - mx) * inv_z;
      else {
        const float p = a.p_f32 ? a.p_f32[(size_t)row * a.ld_p + j] : __bfloat162float(pb[(size_t)row * a.ld_p + j]);
        v = p * (x[j] - dot);      // softmax.rs:44-64
      }
      if (a.out_f32) a.out_f32[(size_t)row * a.ld_out + j] = v;
      if (ob) ob[(size_t)row * a.ld_out + j] = __float2bfloat16_rn(v);
      if (a.outT_f32) a.outT_f32[(size_t)j * a.ld_outT + row] = v;
      if (otb) otb[(size_t)j * a.ld_outT + row] = __float2bfloat16_rn(v);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Column sums (bias gradient).
// ------------------------------------------------------------------------------------------------
// Rows are split into `nchunks` slabs (grid.y) so that a tall, narrow matrix (the bias gradient of a
// convolution: hundreds of thousands of rows, 32 columns) still fills the GPU. Every slab writes its
// partial column sums to a scratch array; the last slab to finish for a column block (counted with an
// atomic) adds the partials in slab order, so the result does not depend on the arrival order.
// The scratch is shared by all calls of a process: calls must not overlap on the device (they are
// issued on one stream by the engines).
constexpr int CS_MAX_PART = 1 << 21;    // floats
constexpr int CS_MAX_COLBLOCKS = 1024;
__device__ __align__(16) float g_cs_part[CS_MAX_PART];
__device__ unsigned int g_cs_count[ONO_MAX_JOBS * CS_MAX_COLBLOCKS];

template <typename T>
__device__ __forceinline__ float cs_load(const T* p) {
  if constexpr (sizeof(T) == 4) return *p;
  else return __bfloat162float(*p);
}
// 16 bytes of a row: four f32 or eight bf16 values
template <typename T>
__device__ __forceinline__ void cs_unpack(uint4 w, float* f) {
  if constexpr (sizeof(T) == 4) {
    f[0] = __uint_as_float(w.x); f[1] = __uint_as_float(w.y); f[2] = __uint_as_float(w.z); f[3] = __uint_as_float(w.w);
  } else {
    const float4 lo = unpack16x4(make_uint2(w.x, w.y), 0), hi = unpack16x4(make_uint2(w.z, w.w), 0);
    f[0] = lo.x; f[1] = lo.y; f[2] = lo.z; f[3] = lo.w; f[4] = hi.x; f[5] = hi.y; f[6] = hi.z; f[7] = hi.w;
  }
}

// A thread takes 16 bytes of a row (VEC columns), CW neighbouring threads one run of CW * 16 bytes, the rest of the block's
// 256 threads further rows; eight loads per thread are in flight. Bound by the latency of those loads (a bias gradient is read
// right after it was written, out of L2): with single values per lane 512 x 8192 bf16 took 7.0 us (now 4.6), 401408 x 64 bf16 40.0 us
// (now 11.5), 67032 x 64 f32 14.0 us (now 6.6).
// VECTOR = false (rows that are not 16-byte aligned): the same walk with one column per thread.
struct ColsumSlabs {       // where a matrix is split over several row slabs
  float* part;
  unsigned int* count;     // one counter per column block
  int rows_per, nchunks;
};
template <typename T, int CW, bool VECTOR>
__device__ __forceinline__ void colsum_block(const T* d, int M, int N, int ld, float* out, float beta, const ColsumSlabs sl, int bx,
                                             int by, int gx) {
  constexpr int VEC = VECTOR ? 16 / (int)sizeof(T) : 1, COLS = CW * VEC, RPI = 256 / CW, U = 8;
  static_assert(COLS <= 64, "one block's columns");
  __shared__ float red[8][64];
  __shared__ float fin[256];
  __shared__ int s_last;
  const int nchunks = sl.nchunks, cx = threadIdx.x % CW, ry = threadIdx.x / CW, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col0 = bx * COLS, col = col0 + cx * VEC;
  const int m0 = by * sl.rows_per, m1 = min(M, m0 + sl.rows_per);
  float acc[VEC];
#pragma unroll
  for (int k = 0; k < VEC; ++k) acc[k] = 0.0f;
  if (col + VEC <= N) {
    for (int m = m0 + ry; m < m1; m += U * RPI) {
      if constexpr (VECTOR) {
        uint4 w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          w[u] = make_uint4(0u, 0u, 0u, 0u);
          if (m + u * RPI < m1) w[u] = *reinterpret_cast<const uint4*>(d + (size_t)(m + u * RPI) * ld + col);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          float f[VEC];
          cs_unpack<T>(w[u], f);
#pragma unroll
          for (int k = 0; k < VEC; ++k) acc[k] += f[k];
        }
      } else {
        float w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = m + u * RPI < m1 ? cs_load(d + (size_t)(m + u * RPI) * ld + col) : 0.0f;
#pragma unroll
        for (int u = 0; u < U; ++u) acc[0] += w[u];
      }
    }
  } else if (col < N) {      // the last, partial run of a row: value by value
    for (int m = m0 + ry; m < m1; m += RPI)
#pragma unroll
      for (int k = 0; k < VEC; ++k) if (col + k < N) acc[k] += cs_load(d + (size_t)m * ld + col + k);
  }
#pragma unroll
  for (int k = 0; k < VEC; ++k) {
#pragma unroll
    for (int o = 16; o >= CW; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    if (lane < CW) red[warp][lane * VEC + k] = acc[k];
  }
  __syncthreads();
  float t = 0.0f;
  if (threadIdx.x < COLS) {
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i][threadIdx.x];
  }
  if (nchunks == 1) {
    if (threadIdx.x < COLS && col0 + threadIdx.x < N) {
      float* o = out + col0 + threadIdx.x;
      *o = beta != 0.0f ? beta * (*o) + t : t;
    }
    return;
  }
  const size_t pitch = (size_t)gx * COLS;
  if (threadIdx.x < COLS) sl.part[by * pitch + col0 + threadIdx.x] = t;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&sl.count[bx], 1u) == (unsigned)nchunks - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // 256 / COLS threads per column, each a contiguous run of slabs; the runs are then added in order
  constexpr int PER = 256 / COLS;
  const int c = threadIdx.x % COLS, part = threadIdx.x / COLS, run = (nchunks + PER - 1) / PER;
  float sum = 0.0f;
  for (int k = part * run; k < min(nchunks, (part + 1) * run); k += U) {
    float w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) w[u] = k + u < min(nchunks, (part + 1) * run) ? __ldcg(&sl.part[(size_t)(k + u) * pitch + col0 + c]) : 0.0f;
#pragma unroll
    for (int u = 0; u < U; ++u) sum += w[u];
  }
  fin[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x < COLS && col0 + c < N) {
#pragma unroll
    for (int k = 1; k < PER; ++k) sum += fin[k * COLS + c];
    out[col0 + c] = beta != 0.0f ? beta * out[col0 + c] + sum : sum;
  }
  if (threadIdx.x == 0) sl.count[bx] = 0u;
}
template <typename T, int CW, bool VECTOR>
__global__ void __launch_bounds__(256) colsum_kernel(const T* d, int M, int N, int ld, float* out, float beta, int rows_per, int nchunks) {
  colsum_block<T, CW, VECTOR>(d, M, N, ld, out, beta, ColsumSlabs{g_cs_part, g_cs_count, rows_per, nchunks}, blockIdx.x, blockIdx.y, gridDim.x);
}

// bf16 matrices with 16-byte aligned rows, in one fixed order of additions whatever else changes (a network with bf16 tiles keeps
// its sums from version to version, see fixed_order in the engine). A slab of rows_per rows of 32 columns: row lane t = 0..7 adds
// the rows t, t + 8, t + 16, t + 24 of every 32 into four sums, the last few rows into the first, and adds the four up pairwise; the
// eight lanes are added in order, then the slabs. A warp takes a slab: four threads a row, 16 bytes each, sixteen loads in flight.
// Bound by the latency of those loads and, for the last block, of the partials: 401408 x 64 38.9 us, 100352 x 64 18.7, 512 x 8192
// 13.3 (events around a cold call, which adds about 8; the f32 form, free in its order, 36.9, 16.4 and 11.1 for its twice as many bytes).
constexpr int CS16_WARPS = 4, CS16_FOLD = 256;      // slabs a block, partials folded at a time
struct Cs16Shape { int gx, rows_per, nchunks; };
static Cs16Shape cs16_shape(int M, int N) {
  Cs16Shape q;
  q.gx = (N + 31) / 32;
  q.nchunks = q.gx <= CS_MAX_COLBLOCKS ? std::max(1, std::min({(M + 127) / 128, (4 * 148 + q.gx - 1) / q.gx, CS_MAX_PART / (q.gx * 32)})) : 1;
  q.rows_per = ((M + q.nchunks - 1) / q.nchunks + 7) / 8 * 8;
  q.nchunks = (M + q.rows_per - 1) / q.rows_per;
  return q;
}
__device__ __forceinline__ void colsum16_block(const __nv_bfloat16* d, int M, int N, int ld, float* out, float beta, const ColsumSlabs sl,
                                               int bx, int by, int gx, float (*sm)[32]) {
  constexpr int U = 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cx = lane & 3, ty = lane >> 2;
  const int nchunks = sl.nchunks, chunk = by * CS16_WARPS + warp, col = bx * 32 + 8 * cx, left = N - col;
  const int m0 = min(M, chunk * sl.rows_per), m1 = chunk < nchunks ? min(M, m0 + sl.rows_per) : m0;
  // A whole 16-byte piece may be read of every row that another row follows (the rows' pitch is a multiple of the piece), also where
  // only a part of it are columns; of the last row such a part is read value by value, at the end.
  const int mlim = left >= 8 ? m1 : left > 0 ? min(m1, M - 1) : 0;
  float acc[4][8];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[q][k] = 0.0f;
  auto add = [&](int q, uint4 w) {
    float f[8];
    cs_unpack<__nv_bfloat16>(w, f);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[q][k] += f[k];
  };
  const __nv_bfloat16* p = d + col;
  const int total = m1 > m0 + ty ? (m1 - m0 - ty + 7) / 8 : 0, grouped = total / 4 * 4;      // rows of this lane; those in groups of four
  for (int i = 0; i < grouped; i += 4 * U) {
    uint4 w[4 * U];
#pragma unroll
    for (int u = 0; u < 4 * U; ++u) {
      const int m = m0 + ty + 8 * (i + u);
      w[u] = make_uint4(0u, 0u, 0u, 0u);                                   // adding a zero changes no sum
      if (i + u < grouped && m < mlim) w[u] = *reinterpret_cast<const uint4*>(p + (size_t)m * ld);
    }
#pragma unroll
    for (int u = 0; u < 4 * U; ++u) add(u & 3, w[u]);
  }
  uint4 tail[3];
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    const int m = m0 + ty + 8 * (grouped + u);
    tail[u] = make_uint4(0u, 0u, 0u, 0u);
    if (grouped + u < total && m < mlim) tail[u] = *reinterpret_cast<const uint4*>(p + (size_t)m * ld);
  }
#pragma unroll
  for (int u = 0; u < 3; ++u) add(0, tail[u]);
  if (left > 0 && left < 8 && total > 0 && m0 + ty + 8 * (total - 1) == M - 1) {
    // the matrix' last row is this lane's last: the fourth of a group, or one of those behind the groups
    const int q = total == grouped ? 3 : 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < left) {
        const float f = cs_load(p + (size_t)(M - 1) * ld + k);
        acc[0][k] += q == 0 ? f : 0.0f;
        acc[3][k] += q == 3 ? f : 0.0f;
      }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) sm[warp * 8 + ty][8 * cx + k] = (acc[0][k] + acc[1][k]) + (acc[2][k] + acc[3][k]);
  __syncwarp();
  float t = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += sm[warp * 8 + i][lane];
  const int c = bx * 32 + lane;
  if (nchunks == 1) {
    if (warp == 0 && c < N) out[c] = beta != 0.0f ? beta * out[c] + t : t;
    return;
  }
  const size_t pitch = (size_t)gx * 32;
  if (chunk < nchunks) sl.part[(size_t)chunk * pitch + c] = t;
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&sl.count[bx], 1u) == (unsigned)((nchunks + CS16_WARPS - 1) / CS16_WARPS) - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  float sum = 0.0f;
  for (int k0 = 0; k0 < nchunks; k0 += CS16_FOLD) {
    const int nk = min(CS16_FOLD, nchunks - k0);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < CS16_FOLD * 8 / (32 * CS16_WARPS); ++u) {
      const int i = threadIdx.x + 32 * CS16_WARPS * u, k = i >> 3, q = i & 7;
      if (k < nk) *reinterpret_cast<float4*>(&sm[k][4 * q]) = __ldcg(reinterpret_cast<const float4*>(sl.part + (size_t)(k0 + k) * pitch + bx * 32 + 4 * q));
    }
    __syncthreads();
    if (warp == 0) {
      int k = 0;
      for (; k + 16 <= nk; k += 16) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = sm[k + u][lane];
#pragma unroll
        for (int u = 0; u < 16; ++u) sum += v[u];
      }
      for (; k < nk; ++k) sum += sm[k][lane];
    }
  }
  if (warp == 0 && c < N) out[c] = beta != 0.0f ? beta * out[c] + sum : sum;
  if (threadIdx.x == 0) sl.count[bx] = 0u;
}
__global__ void __launch_bounds__(32 * CS16_WARPS) colsum16_kernel(const __nv_bfloat16* d, int M, int N, int ld, float* out, float beta,
                                                                   int rows_per, int nchunks) {
  __shared__ __align__(16) float sm[CS16_FOLD][32];
  colsum16_block(d, M, N, ld, out, beta, ColsumSlabs{g_cs_part, g_cs_count, rows_per, nchunks}, blockIdx.x, blockIdx.y, gridDim.x, sm);
}

// The bias gradients of several layers in one launch, after the last of them is complete: each is a few microseconds of latency.
// One block shape for all of them, eight threads a row (f32), the one that wide matrices take.
struct ColsumJobs {
  OnoColsum job[ONO_MAX_JOBS];
  int block_end[ONO_MAX_JOBS], gx[ONO_MAX_JOBS], rows_per[ONO_MAX_JOBS], nchunks[ONO_MAX_JOBS];
  int part_at[ONO_MAX_JOBS], count_at[ONO_MAX_JOBS];
};
__global__ void __launch_bounds__(256) colsum_jobs_kernel(const __grid_constant__ ColsumJobs m) {
  int j = 0;
  while ((int)blockIdx.x >= m.block_end[j]) ++j;
  const int b = (int)blockIdx.x - (j ? m.block_end[j - 1] : 0);
  const OnoColsum& q = m.job[j];
  colsum_block<float, 8, true>((const float*)q.d, q.M, q.N, q.ld, q.out, q.beta, ColsumSlabs{g_cs_part + m.part_at[j], g_cs_count + m.count_at[j],
                               m.rows_per[j], m.nchunks[j]}, b % m.gx[j], b / m.gx[j], m.gx[j]);
}
__global__ void __launch_bounds__(32 * CS16_WARPS) colsum16_jobs_kernel(const __grid_constant__ ColsumJobs m) {
  __shared__ __align__(16) float sm[CS16_FOLD][32];
  int j = 0;
  while ((int)blockIdx.x >= m.block_end[j]) ++j;
  const int b = (int)blockIdx.x - (j ? m.block_end[j - 1] : 0);
  const OnoColsum& q = m.job[j];
  colsum16_block((const __nv_bfloat16*)q.d, q.M, q.N, q.ld, q.out, q.beta, ColsumSlabs{g_cs_part + m.part_at[j], g_cs_count + m.count_at[j],
                 m.rows_per[j], m.nchunks[j]}, b % m.gx[j], b / m.gx[j], m.gx[j], sm);
}

template <typename T, int CW, bool VECTOR>
static void launch_colsum(const T* d, int M, int N, int ld, float* out, float beta, cudaStream_t st) {
  constexpr int COLS = CW * (VECTOR ? 16 / (int)sizeof(T) : 1), RPI = 256 / CW;
  const int gx = (N + COLS - 1) / COLS;
  // two blocks per SM; a slab of fewer than eight loads per thread is not worth the second pass over the partials
  int nchunks = 1;
  if (gx <= CS_MAX_COLBLOCKS) nchunks = std::max(1, std::min({(M + 8 * RPI - 1) / (8 * RPI), 2 * 148 / gx, CS_MAX_PART / (gx * COLS)}));
  const int rows_per = (M + nchunks - 1) / nchunks;
  nchunks = (M + rows_per - 1) / rows_per;
  colsum_kernel<T, CW, VECTOR><<<dim3(gx, nchunks), 256, 0, st>>>(d, M, N, ld, out, beta, rows_per, nchunks);
}
template <typename T>
static void colsum_any(const T* d, int M, int N, int ld, float* out, float beta, cudaStream_t st) {
  constexpr int VEC = 16 / (int)sizeof(T);
  if (ld % VEC == 0 && ((uintptr_t)d & 15) == 0) {
    // the fewest of 8, 4 and 2 threads a row that cover it in one run: a narrow matrix leaves no lanes without columns
    const int runs = (N + VEC - 1) / VEC;
    if constexpr (sizeof(T) == 2) {
      const Cs16Shape q = cs16_shape(M, N);
      colsum16_kernel<<<dim3(q.gx, (q.nchunks + CS16_WARPS - 1) / CS16_WARPS), 32 * CS16_WARPS, 0, st>>>(d, M, N, ld, out, beta, q.rows_per, q.nchunks);
    } else if (runs >= 5) launch_colsum<T, 8, true>(d, M, N, ld, out, beta, st);
    else if (runs >= 3) launch_colsum<T, 4, true>(d, M, N, ld, out, beta, st);
    else launch_colsum<T, 2, true>(d, M, N, ld, out, beta, st);
  } else {
    launch_colsum<T, 32, false>(d, M, N, ld, out, beta, st);
  }
}

// ------------------------------------------------------------------------------------------------
// Optimizers (128-bit vectorised main body, scalar tail).
// ------------------------------------------------------------------------------------------------
struct OptimScalars {
  float lr, mu, b1, b2, eps, gs, adam_step;
};

__device__ __forceinline__ float optim_one(int kind, const OptimScalars& s, float p, float g, float* m, float* v) {
  g *= s.gs;
  if (kind == 0) return p - s.lr * g;  // gradient_descent.rs:45-47
  if (kind == 1) {                     // gradient_descent_with_momentum.rs:55-62
    const float vel = s.mu * (*m) + g;
    *m = vel;
    return p - s.lr * vel;
  }
  // adam.rs:75-91: step = lr*sqrt(1-b2^t)/(1-b1^t); p -= step * m / (sqrt(v) + eps)
  const float mm = s.b1 * (*m) + (1.0f - s.b1) * g;
  const float vv = s.b2 * (*v) + (1.0f - s.b2) * g * g;
  *m = mm;
  *v = vv;
  return p - s.adam_step * mm / (sqrtf(vv) + s.eps);
}

__global__ void optim_kernel(const OnoOptim o) {
  OptimScalars s{o.lr, o.mu, o.b1, o.b2, o.eps, o.grad_scale, 0.0f};
  if (o.kind == 2) {
    const float b1t = o.adam_pows[0], b2t = o.adam_pows[1];
    s.adam_step = o.lr * sqrtf(1.0f - b2t) / (1.0f - b1t);
  }
  const long long n4 = o.n >> 2;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float4* p4 = reinterpret_cast<float4*>(o.p);
  const float4* g4 = reinterpret_cast<const float4*>(o.g);
  float4* m4 = reinterpret_cast<float4*>(o.m);
  float4* v4 = reinterpret_cast<float4*>(o.v);
  __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(o.p_bf16);
  for (long long i = tid; i < n4; i += stride) {
    float4 p = p4[i];
    const float4 g = g4[i];
    float4 m = o.kind >= 1 ? m4[i] : make_float4(0, 0, 0, 0);
    float4 v = o.kind == 2 ? v4[i] : make_float4(0, 0, 0, 0);
    p.x = optim_one(o.kind, s, p.x, g.x, &m.x, &v.x);
    p.y = optim_one(o.kind, s, p.y, g.y, &m.y, &v.y);
    p.z = optim_one(o.kind, s, p.z, g.z, &m.z, &v.z);
    p.w = optim_one(o.kind, s, p.w, g.w, &m.w, &v.w);
    p4[i] = p;
    if (o.kind >= 1) m4[i] = m;
    if (o.kind == 2) v4[i] = v;
    if (pb) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y), hi = __floats2bfloat162_rn(p.z, p.w);
      uint2 pk;
      pk.x = *reinterpret_cast<uint32_t*>(&lo);
      pk.y = *reinterpret_cast<uint32_t*>(&hi);
      *reinterpret_cast<uint2*>(pb + 4 * i) = pk;
    }
    if (o.zero_grad) reinterpret_cast<float4*>(const_cast<float*>(o.g))[i] = make_float4(0, 0, 0, 0);
  }
  for (long long i = (n4 << 2) + tid; i < o.n; i += stride) {
    float m = o.kind >= 1 ? o.m[i] : 0.0f, v = o.kind == 2 ? o.v[i] : 0.0f;
    const float p = optim_one(o.kind, s, o.p[i], o.g[i], &m, &v);
    o.p[i] = p;
    if (o.kind >= 1) o.m[i] = m;
    if (o.kind == 2) o.v[i] = v;
    if (pb) pb[i] = __float2bfloat16_rn(p);
    if (o.zero_grad) const_cast<float*>(o.g)[i] = 0.0f;
  }
}

__global__ void adam_tick_kernel(float* pows, float b1, float b2) {
  pows[0] *= b1;
  pows[1] *= b2;
}

__global__ void local_sgd_kernel(float* p, const float* g, float* r, long long n, float lr, __nv_bfloat16* pb) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float gi = g[i];
    const float pi = p[i] - lr * gi;
    p[i] = pi;
    r[i] += gi;
    if (pb) pb[i] = __float2bfloat16_rn(pi);
  }
}

__global__ void sumsq_kernel(const float* x, long long n, double* out) {
  double acc = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float v = x[i];
    acc += (double)v * (double)v;
  }
  __shared__ double s[32];
  float dummy = 0.0f; (void)dummy;
  // warp reduce in double
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += s[w];
    atomicAdd(out, t);
  }
}

__global__ void init_kernel(float* out, long long n, unsigned long long off, unsigned long long seed, int kind,
                            float a, float b) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = philox_sample(off + (unsigned long long)i, seed, kind, a, b);
}

// ------------------------------------------------------------------------------------------------
// Row gather + cast + transpose through a 32x33 shared tile.
// ------------------------------------------------------------------------------------------------
// 32 x 32 tile (bx, by) by a block of 256 threads.
__device__ __forceinline__ void rows_tile32(const OnoRows& r, int bx, int by, float (*tile)[33]) {
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r0 = by * 32, c0 = bx * 32;
  __nv_bfloat16* db = reinterpret_cast<__nv_bfloat16*>(r.dst_bf16);
  __nv_bfloat16* dtb = reinterpret_cast<__nv_bfloat16*>(r.dstT_bf16);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = ty + 8 * j, row = r0 + i, col = c0 + tx;
    float v = 0.0f;
    if (row < r.R && col < r.W) {
      const int srow = r.idx ? r.idx[row] : row;
      v = r.src[(size_t)srow * r.ld_src + col];
      if (r.dst_f32) r.dst_f32[(size_t)row * r.ld_dst + col] = v;
      if (db) db[(size_t)row * r.ld_dst + col] = __float2bfloat16_rn(v);
    }
    tile[i][tx] = v;
  }
  if (!r.dstT_f32 && !dtb) return;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = ty + 8 * j, col = c0 + i, row = r0 + tx;  // output row = source column
    if (col < r.W && row < r.R) {
      const float v = tile[tx][i];
      if (r.dstT_f32) r.dstT_f32[(size_t)col * r.ld_dstT + row] = v;
      if (dtb) dtb[(size_t)col * r.ld_dstT + row] = __float2bfloat16_rn(v);
    }
  }
}
__global__ void __launch_bounds__(256) rows_kernel(const OnoRows r) {
  __shared__ float tile[32][33];
  rows_tile32(r, blockIdx.x, blockIdx.y, tile);
}

static int grid_for(long long n, int block, int per_thread = 4) {
  long long g = (n + (long long)block * per_thread - 1) / ((long long)block * per_thread);
  if (g < 1) g = 1;
  if (g > 148 * 16) g = 148 * 16;
  return (int)g;
}

}  // namespace ono

using namespace ono;

extern "C" int ono_loss(const OnoLoss* l, ono_stream_t st) {
  if (!l || !l->a || !l->y || l->B <= 0 || l->C <= 0) { set_error("bad loss args%s", "", 0, 0); return -1; }
  const int wpb = 4;
  int grid = (l->B + wpb - 1) / wpb;
  if (grid > 148 * 16) grid = 148 * 16;
  const cudaStream_t s = (cudaStream_t)st;
  if (l->C <= 32) loss_kernel<1><<<grid, wpb * 32, 0, s>>>(*l);
  else if (l->C <= 128) loss_kernel<4><<<grid, wpb * 32, 0, s>>>(*l);
  else if (l->C <= LOSS_ROW) loss_kernel<-1><<<grid, wpb * 32, 0, s>>>(*l);
  else loss_kernel<0><<<grid, wpb * 32, 0, s>>>(*l);
  return launch_ok("loss");
}

namespace ono {
__global__ void push_add_kernel(const float* src, float* dst, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    atomicAdd(dst + i, src[i]);   // result unused: compiled to a reduction that needs no reply
}
}  // namespace ono

extern "C" int ono_softmax(const OnoSoftmax* a, ono_stream_t st) {
  if (!a || !a->x || a->B <= 0 || a->C <= 0 || (a->backward && !a->p_f32 && !a->p_bf16)) {
    set_error("bad softmax args%s", "", 0, 0);
    return -1;
  }
  const int wpb = 8;
  int grid = (a->B + wpb - 1) / wpb;
  if (grid > 148 * 8) grid = 148 * 8;
  softmax_kernel<<<grid, wpb * 32, 0, (cudaStream_t)st>>>(*a);
  return launch_ok("softmax");
}

namespace ono {
__global__ void cast16_kernel(const float* src, uint16_t* dst, long long n, int f16, int vec) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n4 = vec ? n >> 2 : 0;
  for (long long i = tid; i < n4; i += stride) {
    const float4 x = __ldcs(reinterpret_cast<const float4*>(src) + i);
    *(reinterpret_cast<uint2*>(dst) + i) = make_uint2(pack16x2(x.x, x.y, f16), pack16x2(x.z, x.w, f16));
  }
  for (long long i = (n4 << 2) + tid; i < n; i += stride) {
    const uint32_t w = pack16x2(src[i], 0.0f, f16);
    dst[i] = (uint16_t)(w & 0xffffu);
  }
}
}  // namespace ono

extern "C" int ono_copy_async(void* dst, const void* src, long long bytes, ono_stream_t st) {
  if (!dst || !src || bytes < 0) { set_error("bad copy args%s", "", 0, 0); return -1; }
  if (bytes == 0) return 0;
  const cudaError_t e = cudaMemcpyAsync(dst, src, (size_t)bytes, cudaMemcpyDefault, (cudaStream_t)st);
  if (e != cudaSuccess) { set_error("cudaMemcpyAsync failed: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}

extern "C" int ono_cast16(const float* src, void* dst, long long n, int f16, ono_stream_t st) {
  if (!src || !dst || n < 0) { set_error("bad cast16 args%s", "", 0, 0); return -1; }
  if (((uintptr_t)dst & 1) != 0) { set_error("cast16 destination must be 2-byte aligned%s", "", 0, 0); return -1; }
  if (n == 0) return 0;
  const int vec = (((uintptr_t)src & 15) == 0 && ((uintptr_t)dst & 7) == 0) ? 1 : 0;
  ono::cast16_kernel<<<grid_for(n, 256, 8), 256, 0, (cudaStream_t)st>>>(src, (uint16_t*)dst, n, f16 ? 1 : 0, vec);
  return launch_ok("cast16");
}

extern "C" int ono_push_add(const float* src, float* dst, long long n, ono_stream_t st) {
  if (!src || !dst || n < 0) { set_error("bad push_add args%s", "", 0, 0); return -1; }
  if (n == 0) return 0;
  ono::push_add_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)st>>>(src, dst, n);
  return launch_ok("push_add");
}

extern "C" int ono_colsum(const void* d, int dtype, int M, int N, int ld, float* out, float beta, ono_stream_t st) {
  if (!d || !out || M <= 0 || N <= 0) { set_error("bad colsum args%s", "", 0, 0); return -1; }
  if (dtype == 0) colsum_any((const float*)d, M, N, ld, out, beta, (cudaStream_t)st);
  else colsum_any((const __nv_bfloat16*)d, M, N, ld, out, beta, (cudaStream_t)st);
  return launch_ok("colsum");
}

extern "C" int ono_colsum_jobs(const OnoColsum* jobs, int n, int dtype, ono_stream_t st) {
  if (!jobs || n <= 0 || n > ONO_MAX_JOBS) { set_error("colsum_jobs: 1 to %s%lld jobs", "", ONO_MAX_JOBS, 0); return -1; }
  const int esz = dtype == 0 ? 4 : 2, cols = 8 * 16 / esz;
  ColsumJobs m;
  int end = 0, part = 0, count = 0;
  for (int j = 0; j < n; ++j) {
    const OnoColsum& q = jobs[j];
    if (!q.d || !q.out || q.M <= 0 || q.N <= 0 || q.ld * esz % 16 != 0 || ((uintptr_t)q.d & 15) != 0) {
      set_error("colsum_jobs: rows must be 16-byte aligned%s", "", 0, 0);
      return -1;
    }
    m.job[j] = q;
    if (dtype != 0) {      // twelve such matrices always fit the scratch
      const Cs16Shape h = cs16_shape(q.M, q.N);
      m.rows_per[j] = h.rows_per; m.gx[j] = h.gx; m.nchunks[j] = h.nchunks; m.part_at[j] = part; m.count_at[j] = count;
      if (h.nchunks > 1) { part += h.nchunks * h.gx * 32; count += h.gx; }
      end += h.gx * ((h.nchunks + CS16_WARPS - 1) / CS16_WARPS);
      m.block_end[j] = end;
      continue;
    }
    const int gx = (q.N + cols - 1) / cols;
    // f32: slabs of at least 256 rows, about two blocks per SM, as far as the scratch reaches (ono_colsum cuts narrow matrices into
    // longer ones: the two agree to rounding)
    int nc = std::max(1, std::min((q.M + 255) / 256, 2 * 148 / gx));
    if (nc > 1 && (count + gx > CS_MAX_COLBLOCKS || part + (long long)nc * gx * cols > CS_MAX_PART)) nc = 1;
    m.rows_per[j] = (q.M + nc - 1) / nc;
    nc = (q.M + m.rows_per[j] - 1) / m.rows_per[j];
    m.gx[j] = gx; m.nchunks[j] = nc; m.part_at[j] = part; m.count_at[j] = count;
    if (nc > 1) { part += nc * gx * cols; count += gx; }
    end += gx * nc;
    m.block_end[j] = end;
  }
  if (dtype == 0) colsum_jobs_kernel<<<end, 256, 0, (cudaStream_t)st>>>(m);
  else colsum16_jobs_kernel<<<end, 32 * CS16_WARPS, 0, (cudaStream_t)st>>>(m);
  return launch_ok("colsum_jobs");
}

extern "C" int ono_optim(const OnoOptim* o, ono_stream_t st) {
  if (!o || !o->p || !o->g || o->n < 0) { set_error("bad optim args%s", "", 0, 0); return -1; }
  if (o->kind >= 1 && !o->m) { set_error("optimizer state m missing%s", "", 0, 0); return -1; }
  if (o->kind == 2 && (!o->v || !o->adam_pows)) { set_error("adam state missing%s", "", 0, 0); return -1; }
  if (((uintptr_t)o->p | (uintptr_t)o->g | (uintptr_t)o->m | (uintptr_t)o->v) & 15) {
    set_error("optimizer buffers must be 16-byte aligned%s", "", 0, 0);
    return -1;
  }
  if (o->p_bf16 && ((uintptr_t)o->p_bf16 & 7)) { set_error("bf16 shadow must be 8-byte aligned%s", "", 0, 0); return -1; }
  if (o->n == 0) return 0;
  optim_kernel<<<grid_for(o->n, 256, 8), 256, 0, (cudaStream_t)st>>>(*o);
  return launch_ok("optim");
}

extern "C" int ono_adam_tick(float* pows, float b1, float b2, ono_stream_t st) {
  adam_tick_kernel<<<1, 1, 0, (cudaStream_t)st>>>(pows, b1, b2);
  return launch_ok("adam_tick");
}

extern "C" int ono_local_sgd(float* p, const float* g, float* r, long long n, float lr, void* pb, ono_stream_t st) {
  if (n <= 0) return 0;
  local_sgd_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)st>>>(p, g, r, n, lr, (__nv_bfloat16*)pb);
  return launch_ok("local_sgd");
}

extern "C" int ono_sumsq(const float* x, long long n, double* out, ono_stream_t st) {
  if (n <= 0) return 0;
  sumsq_kernel<<<grid_for(n, 256, 8), 256, 0, (cudaStream_t)st>>>(x, n, out);
  return launch_ok("sumsq");
}

extern "C" int ono_init(float* out, long long n, unsigned long long off, unsigned long long seed, int kind, float a,
                        float b, ono_stream_t st) {
  if (n <= 0) return 0;
  init_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)st>>>(out, n, off, seed, kind, a, b);
  return launch_ok("init");
}

// f32 copy and/or transpose of an aligned matrix with 16-byte accesses on both sides: 64 x 64 tiles, rows read as
// float4, the transpose written as float4 along the source's rows (R % 4 == 0, W % 4 == 0, 16-byte aligned rows).
__device__ __forceinline__ void rows_tile64(const OnoRows& r, int bx, int by, float (*tile)[65]) {
  const int r0 = by * 64, c0 = bx * 64;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int row = r0 + ty + 16 * p, col = c0 + 4 * tx;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < r.R && col < r.W) {
      v = *reinterpret_cast<const float4*>(r.src + (size_t)row * r.ld_src + col);
      if (r.dst_f32) *reinterpret_cast<float4*>(r.dst_f32 + (size_t)row * r.ld_dst + col) = v;
    }
    float* t = &tile[ty + 16 * p][4 * tx];
    t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w;
  }
  if (!r.dstT_f32) return;
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int col = c0 + ty + 16 * p, row = r0 + 4 * tx;   // output row = source column
    if (col < r.W && row < r.R) {
      const int cl = ty + 16 * p;
      *reinterpret_cast<float4*>(r.dstT_f32 + (size_t)col * r.ld_dstT + row) =
          make_float4(tile[4 * tx][cl], tile[4 * tx + 1][cl], tile[4 * tx + 2][cl], tile[4 * tx + 3][cl]);
    }
  }
}
__global__ void __launch_bounds__(256) rows_vec_kernel(const OnoRows r) {
  __shared__ float tile[64][65];
  rows_tile64(r, blockIdx.x, blockIdx.y, tile);
}
static bool rows_vectorised(const OnoRows* r) {
  return !r->idx && !r->dst_bf16 && !r->dstT_bf16 && (r->dst_f32 || r->dstT_f32) && r->R % 4 == 0 && r->W % 4 == 0 &&
         r->ld_src % 4 == 0 && (!r->dst_f32 || r->ld_dst % 4 == 0) && (!r->dstT_f32 || r->ld_dstT % 4 == 0) &&
         (((uintptr_t)r->src | (uintptr_t)r->dst_f32 | (uintptr_t)r->dstT_f32) & 15) == 0 && (long long)r->R * r->W >= (1 << 16);
}

// Several such jobs in one launch (the two matrices of a batch; the operand copies of every layer after an update): most of them
// move a few hundred kilobytes and cost a launch each, 2 to 3 us in a captured step. `zero`: a double set to zero on the way
// (the loss of the step that the batch belongs to).
struct RowsJobs {
  OnoRows job[ONO_MAX_JOBS];
  int block_end[ONO_MAX_JOBS], vec[ONO_MAX_JOBS], gx[ONO_MAX_JOBS];
  double* zero;
};
__global__ void __launch_bounds__(256) rows_jobs_kernel(const __grid_constant__ RowsJobs m) {
  __shared__ float tile[64 * 65];
  if (blockIdx.x == 0 && threadIdx.x == 0 && m.zero) *m.zero = 0.0;
  int j = 0;
  while ((int)blockIdx.x >= m.block_end[j]) ++j;
  const int b = (int)blockIdx.x - (j ? m.block_end[j - 1] : 0), bx = b % m.gx[j], by = b / m.gx[j];
  if (m.vec[j]) rows_tile64(m.job[j], bx, by, reinterpret_cast<float (*)[65]>(tile));
  else rows_tile32(m.job[j], bx, by, reinterpret_cast<float (*)[33]>(tile));
}

extern "C" int ono_rows_jobs(const OnoRows* jobs, int n, double* zero, ono_stream_t st) {
  if (!jobs || n <= 0 || n > ONO_MAX_JOBS) { set_error("rows_jobs: 1 to %s%lld jobs", "", ONO_MAX_JOBS, 0); return -1; }
  RowsJobs m;
  m.zero = zero;
  long long end = 0;
  for (int j = 0; j < n; ++j) {
    const OnoRows& r = jobs[j];
    if (!r.src || r.R <= 0 || r.W <= 0) { set_error("bad rows args%s", "", 0, 0); return -1; }
    m.job[j] = r;
    m.vec[j] = rows_vectorised(&r) ? 1 : 0;
    const int t = m.vec[j] ? 64 : 32;
    m.gx[j] = (r.W + t - 1) / t;
    end += (long long)m.gx[j] * ((r.R + t - 1) / t);
    if (end >= (1ll << 31)) { set_error("rows_jobs: too many tiles%s", "", 0, 0); return -1; }
    m.block_end[j] = (int)end;
  }
  rows_jobs_kernel<<<(unsigned)end, 256, 0, (cudaStream_t)st>>>(m);
  return launch_ok("rows_jobs");
}

// Row gather out of pinned host memory. The loads cross PCIe, so what counts is bytes in flight, not threads: a few blocks, each thread
// with four independent 16-byte loads outstanding (24 blocks x 256 threads x 64 bytes = 384 KB in flight, several times the
// bandwidth-delay product of a Gen5 x16 link), which leaves the SMs to the kernels of other streams.
constexpr int ROWS_HOST_BLOCKS = 24;
__global__ void __launch_bounds__(256) rows_host_kernel(const OnoRows r) {
  constexpr int U = 4;
  const int w = r.W / 4;
  const long long total = (long long)r.R * w, stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x + threadIdx.x; base < total; base += stride * U) {
    float4 v[U];
    long long at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long e = base + u * stride;
      at[u] = -1;
      if (e < total) {
        const int row = (int)(e / w), c = (int)(e - (long long)row * w) * 4;
        v[u] = *reinterpret_cast<const float4*>(r.src + (size_t)r.idx[row] * r.ld_src + c);
        at[u] = (long long)row * r.ld_dst + c;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) *reinterpret_cast<float4*>(r.dst_f32 + at[u]) = v[u];
  }
}

// A value of device memory to pinned host memory by a store over PCIe. A copy node of a captured step costs about 10 us at the end of
// its chain (8 before the copy engine starts, 2 for eight bytes); this launch, on a branch beside backward, nothing.
namespace ono {
__global__ void report_kernel(const double* value, double* host) { *host = *value; }
// Whether `p` lies in pinned host memory, which kernels may read and write.
bool is_host_memory(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
  return a.type == cudaMemoryTypeHost;
}
}  // namespace ono

extern "C" int ono_report(const double* value, double* host, ono_stream_t st) {
  if (!value || !host || !is_host_memory(host)) { set_error("bad report args%s", "", 0, 0); return -1; }
  report_kernel<<<1, 1, 0, (cudaStream_t)st>>>(value, host);
  return launch_ok("report");
}

// One replayed step: wait for the batch, launch the graph, record that the batch has been consumed and that the loss is on the host.
extern "C" int ono_replay_step(const OnoReplay* r) {
  if (!r || !r->graph_exec) { set_error("bad replay args%s", "", 0, 0); return -1; }
  cudaStream_t s = (cudaStream_t)r->stream;
  cudaError_t e = cudaStreamWaitEvent(s, (cudaEvent_t)r->ready, 0);
  if (e == cudaSuccess) e = cudaGraphLaunch((cudaGraphExec_t)r->graph_exec, s);
  if (e == cudaSuccess) e = cudaEventRecord((cudaEvent_t)r->consumed, s);
  if (e == cudaSuccess) e = cudaEventRecord((cudaEvent_t)r->loss_there, s);
  if (e != cudaSuccess) { set_error("replay_step: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}

extern "C" int ono_rows(const OnoRows* r, ono_stream_t st) {
  if (!r || !r->src || r->R <= 0 || r->W <= 0) { set_error("bad rows args%s", "", 0, 0); return -1; }
  if (r->idx && r->dst_f32 && !r->dst_bf16 && !r->dstT_f32 && !r->dstT_bf16 && r->W % 4 == 0 && r->ld_src % 4 == 0 &&
      r->ld_dst % 4 == 0 && (((uintptr_t)r->src | (uintptr_t)r->dst_f32) & 15) == 0 && is_host_memory(r->src)) {
    rows_host_kernel<<<ROWS_HOST_BLOCKS, 256, 0, (cudaStream_t)st>>>(*r);
    return launch_ok("rows");
  }
  if (rows_vectorised(r)) {
    dim3 grid((r->W + 63) / 64, (r->R + 63) / 64);
    rows_vec_kernel<<<grid, 256, 0, (cudaStream_t)st>>>(*r);
    return launch_ok("rows");
  }
  dim3 grid((r->W + 31) / 32, (r->R + 31) / 32);
  rows_kernel<<<grid, 256, 0, (cudaStream_t)st>>>(*r);
  return launch_ok("rows");
}
