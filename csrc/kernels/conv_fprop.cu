// Forward convolution as one kernel (the reference: arch/layers/conv/conv2d.rs:84-104,119-125, im2col and a product per sample).
//
// As two kernels the column matrix is written by im2col and read back by the product before the weight gradient reads it again. Here it is
// gathered once, into the shared-memory tiles the tensor cores read, and leaves for memory from there:
//
//   warps 0-7    gather a 128-row x 128-byte tile of columns with 16-byte cp.async, zeros where a window hangs over the image, at the
//                places the 128-byte swizzle gives them; a thread's columns of a tile never change, its rows move on with the tile
//   warp 12      issues the tcgen05 products into TMEM (two accumulators), K^T resident in shared memory for the whole launch
//   warp 13      sends every gathered tile to the column matrix by TMA (whole lines, off the load / store unit)
//   warps 8-11   bias, activation, rounding, TMA stores of the result
//
// Columns and products are those of the two kernels to the bit: the same tiles, reduced in the same order. Two kernels and this one, us:
// bf16 3 x 3 stride 2 on 2048 images: 28 x 28 x 32 -> 64 116.0 -> 70.0, 14 x 14 x 64 56.5 -> 41.0; 1024 of 16 x 16 x 48 -> 80 96.1 -> 62.6;
// f32 on 342 images: 28 x 28 x 32 42.1 -> 30.4, 14 x 14 x 64 22.5 -> 16.9; 512 of 14 x 14 x 20 -> 40, 5 x 5, 49.3 -> 40.2; 20 of 28 x 28 x 16
// 10.4 -> 8.2. What bounds it is the column matrix's way to memory (without it the second case takes 32.8); the first case moves its
// bytes at 0.86 of the copy rate.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "act.cuh"
#include "ono_kernels.h"
#include "opt.cuh"
#include "ptx.cuh"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);
int encode_map_2d(CUtensorMap* map, const void* base, int esize, long long rows, long long cols, long long ld, int box_cols, int box_rows,
                  bool swizzle_32b_units);
int encode_out_map(CUtensorMap* map, const void* base, int esize, long long rows, long long cols, long long ld);

constexpr int FP_MAX_STAGES = 8, FP_GATHER = 256;
struct FpropDev {
  OnoConvFprop d;
  int rows, tiles, kb, N, NS;      // output pixels, 128-row tiles, 128-byte blocks of a row, columns of the product (F up to a multiple of 16)
                                   // and of its accumulator
  int stages, out_bufs;
  uint32_t idesc, tmem_cols;
  uint32_t w_at, out_at, tab_at;   // offsets in shared memory (the ring of column tiles is at 0)
};

__device__ __forceinline__ void fprop_fail(const FpropDev& p, volatile int* abort_flag, int code) {
  if (p.d.status) atomicCAS(p.d.status, 0, code);
  *abort_flag = 1;
}

// AHEAD: tiles of a thread's copies in flight behind the newest one. The gather waits for memory, so as many as the ring has room for
// (2048 images of 28 x 28 x 32, bf16: 80.2 us with two, 70.0 with five; without the column matrix to send 66.9 and 68.4).
template <int ESIZE, int AHEAD>
__global__ void __launch_bounds__(576, 1)      // 448 are launched: bounded to 112 registers, for a block of the batch feed beside the CTA
conv_fprop_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmY,
                  const __grid_constant__ FpropDev p) {
  constexpr int BK = 128 / ESIZE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full[FP_MAX_STAGES], empty[FP_MAX_STAGES], acc_full[2], acc_empty[2], w_full, drain_bar;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  volatile int* abortp = &abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const OnoConvGeom& g = p.d.g;
  const uint64_t budget = p.d.timeout_ns;
  const bool with_cols = p.d.cols != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], FP_GATHER); mbar_init(&empty[s], with_cols ? 2 : 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 128); }
    mbar_init(&w_full, 1);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 12) { tmem_alloc(&tmem_base_smem, p.tmem_cols); tmem_relinquish(); }
  if (warp == 13 && lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmY); if (with_cols) tma_prefetch_desc(&tmC); }
  // where a 16-byte piece of a column row comes from: tap (row, column) and offset from the window's origin; row -1: past the last one
  int2* const tab = reinterpret_cast<int2*>(smem + p.tab_at);
  if (warp < 8) {
    constexpr int V = 16 / ESIZE;
    for (int i = threadIdx.x; i < p.kb * 8; i += FP_GATHER) {
      const int q = i * V, tap = q / g.C, c = q - tap * g.C, ky = tap / g.K, kx = tap - ky * g.K;
      tab[i] = tap < g.K * g.K ? make_int2((ky << 16) | kx, (ky * g.W + kx) * p.d.ldx + c) : make_int2(-1, 0);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  if (warp < 8) {
    // ---------------- gather ----------------
    const int u = threadIdx.x & 7, r0 = threadIdx.x >> 3;      // this thread's piece of a tile's rows r0, r0 + 32, ...
    const uint8_t* const x = reinterpret_cast<const uint8_t*>(p.d.x);
    const uint32_t ring = smem_u32(smem);
    bool ok = true;
    int n = 0;                                                  // tiles gathered so far
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
      int iy0[4], ix0[4];
      const uint8_t* at[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = tile * 128 + r0 + 32 * i, rest = m / g.OW, ox = m - rest * g.OW, img = rest / g.OH, oy = rest - img * g.OH;
        iy0[i] = m < p.rows ? oy * g.S - g.P : -(1 << 20);      // (rows past the last pixel: outside every image)
        ix0[i] = ox * g.S - g.P;
        at[i] = x + ((long long)(img * g.H + oy * g.S - g.P) * g.W + ix0[i]) * p.d.ldx * ESIZE;
      }
      for (int k = 0; k < p.kb; ++k, ++n) {
        const int s = n % p.stages;
        const bool free = mbar_wait_bounded(&empty[s], ((n / p.stages) & 1) ^ 1u, abortp, budget);
        if (!__all_sync(0xffffffffu, free)) {
          if (lane == 0) fprop_fail(p, abortp, ONO_ERR_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        const int2 t = tab[k * 8 + u];
        const int ky = t.x >> 16, kx = t.x & 0xffff;
        const uint32_t to = ring + (uint32_t)s * 16384u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = r0 + 32 * i;
          const bool in = t.x >= 0 && (unsigned)(iy0[i] + ky) < (unsigned)g.H && (unsigned)(ix0[i] + kx) < (unsigned)g.W;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)(r * 128 + ((u ^ (r & 7)) << 4))),
                       "l"(in ? at[i] + (long long)t.y * ESIZE : x), "r"(in ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (n >= AHEAD) {      // the copies of the tile AHEAD before this one have landed: the tensor cores and TMA may read it
          asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
          fence_proxy_async_smem();
          mbar_arrive(&full[(n - AHEAD) % p.stages]);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async_smem();
    for (int j = max(0, n - AHEAD); j < n && ok; ++j) mbar_arrive(&full[j % p.stages]);
  } else if (warp < 12) {
    // ---------------- results ----------------
    const int quad = warp & 3;
    uint8_t* const stage0 = smem + p.out_at + (uint32_t)((warp - 8) * p.out_bufs) * 4096u;
    int t = 0, sent = 0;
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, ++t) {
      const int buf = t & 1;
      const bool got = mbar_wait_bounded(&acc_full[buf], (t >> 1) & 1, abortp, budget);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) fprop_fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_FULL);
        break;
      }
      tc_fence_after();
      for (int c = 0; c * 32 < p.d.F; ++c, ++sent) {
        uint32_t r[32];
        tmem_ld_x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * p.NS + c * 32), r);
        float v[32];
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int f = c * 32 + j;
          v[j] = __uint_as_float(r[j]) + (p.d.bias && f < p.d.F ? __ldg(p.d.bias + f) : 0.f);
        }
        act_fwd_n<32>(p.d.act, p.d.act_param, v);
        uint8_t* const stage = stage0 + (uint32_t)(sent & (p.out_bufs - 1)) * 4096u;
        if (lane == 0) {                              // the store that read this tile last is done with it
          if (p.out_bufs == 2) tma_store_wait_read<1>();
          else tma_store_wait_read<0>();
        }
        __syncwarp();
        if (ESIZE == 4) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(pack16x2(v[8 * j], v[8 * j + 1], 0), pack16x2(v[8 * j + 2], v[8 * j + 3], 0), pack16x2(v[8 * j + 4], v[8 * j + 5], 0),
                           pack16x2(v[8 * j + 6], v[8 * j + 7], 0));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmY, stage, c * 32, tile * 128 + quad * 32);
          tma_store_commit();
        }
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[buf]);
    }
    if (lane == 0) tma_store_wait_all<0>();
  } else if (warp == 12) {
    // ---------------- MMA issuer ----------------
    const uint32_t base = smem_u32(smem);
    bool ok = mbar_wait_bounded(&w_full, 0, abortp, budget);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) fprop_fail(p, abortp, ONO_ERR_TIMEOUT_FULL);
    int n = 0, t = 0;
    for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, ++t) {
      const int buf = t & 1;
      const bool drained = mbar_wait_bounded(&acc_empty[buf], ((t >> 1) & 1) ^ 1u, abortp, budget);
      if (!__all_sync(0xffffffffu, drained)) { fprop_fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_EMPTY); ok = false; break; }
      tc_fence_after();
      for (int k = 0; k < p.kb; ++k, ++n) {
        const int s = n % p.stages;
        const bool landed = mbar_wait_bounded(&full[s], (n / p.stages) & 1, abortp, budget);
        if (!__all_sync(0xffffffffu, landed)) { fprop_fail(p, abortp, ONO_ERR_TIMEOUT_FULL); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t ad = make_smem_desc_sw128(base + (uint32_t)s * 16384u, 16, 1024);
          const uint64_t bd = make_smem_desc_sw128(base + p.w_at + (uint32_t)(k * p.N) * 128u, 16, 1024);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (ESIZE == 4) umma_tf32(tmem_base + (uint32_t)(buf * p.NS), ad + 2 * j, bd + 2 * j, p.idesc, (k | j) != 0);
            else umma_f16(tmem_base + (uint32_t)(buf * p.NS), ad + 2 * j, bd + 2 * j, p.idesc, (k | j) != 0);
          }
          umma_commit(&empty[s]);
          if (k == p.kb - 1) umma_commit(&acc_full[buf]);
        }
        __syncwarp();
      }
    }
    if (elect_one()) umma_commit(&drain_bar);      // no MMA may still run when TMEM is released
    __syncwarp();
    mbar_wait_bounded(&drain_bar, 0, abortp, ok ? budget : 1000000ull);
  } else {
    // ---------------- K^T in, columns out ----------------
    if (elect_one()) {
      mbar_expect_tx(&w_full, (uint32_t)(p.kb * p.N) * 128u);
      for (int k = 0; k < p.kb; ++k) tma_load_2d(smem + p.w_at + (uint32_t)(k * p.N) * 128u, &tmW, &w_full, k * BK, 0);
    }
    __syncwarp();
    bool ok = true;
    int n = 0;
    for (int tile = blockIdx.x; tile < p.tiles && ok && with_cols; tile += gridDim.x)
      for (int k = 0; k < p.kb; ++k, ++n) {
        const int s = n % p.stages;
        const bool landed = mbar_wait_bounded(&full[s], (n / p.stages) & 1, abortp, budget);
        if (!__all_sync(0xffffffffu, landed)) { fprop_fail(p, abortp, ONO_ERR_TIMEOUT_FULL); ok = false; break; }
        if (lane == 0) {
          tma_store_2d(&tmC, smem + (uint32_t)s * 16384u, k * BK, tile * 128);
          tma_store_commit();
          if (n > 0) {                                // the previous tile has been read
            tma_store_wait_read<1>();
            mbar_arrive(&empty[(n - 1) % p.stages]);
          }
        }
        __syncwarp();
      }
    if (lane == 0 && with_cols) {
      tma_store_wait_read<0>();
      if (n > 0 && ok) mbar_arrive(&empty[(n - 1) % p.stages]);
      tma_store_wait_all<0>();
    }
    // K^T has landed before the CTA may retire its shared memory, also when everyone else has given up
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&w_full, 0, abortp, budget))) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 12) { tc_fence_after(); tmem_dealloc(tmem_base, p.tmem_cols); }
}

constexpr uint32_t FPROP_SMEM = 225u * 1024u;      // the rest is a block's of the batch feed
static bool fprop_plan(const OnoConvFprop* d, FpropDev* p) {
  const OnoConvGeom& g = d->g;
  const int esz = d->dtype == 0 ? 4 : 2, V = 16 / esz;
  if (g.B <= 0 || g.C <= 0 || g.C % V || d->F <= 0 || d->F % V || d->F > 256 || g.K < 1 || g.S < 1 || g.P < 0 || g.OH <= 0 || g.OW <= 0) return false;
  const long long rows = (long long)g.B * g.OH * g.OW, ckk = (long long)g.C * g.K * g.K;
  // (32-bit indices of pixels and of the offsets inside a window)
  if (rows + 128 >= (1ll << 30) || (long long)g.B * g.H * g.W >= (1ll << 30) || g.K >= (1 << 14) || ckk * esz > 128 * 256 ||
      (long long)(g.K + 1) * g.W * d->ldx >= (1ll << 30)) return false;
  memset(p, 0, sizeof(*p));
  p->rows = (int)rows;
  p->tiles = (int)((rows + 127) / 128);
  p->kb = (int)((ckk * esz + 127) / 128);
  p->N = (d->F + 15) / 16 * 16;
  p->tmem_cols = 32;
  p->NS = (p->N + 31) / 32 * 32;
  while (p->tmem_cols < 2u * (uint32_t)p->NS) p->tmem_cols *= 2;
  const uint32_t fixed = (uint32_t)(p->kb * p->N) * 128u + (uint32_t)p->kb * 64u + 1024u;
  for (p->out_bufs = 2; p->out_bufs >= 1; --p->out_bufs) {
    const uint32_t taken = fixed + 4u * 4096u * (uint32_t)p->out_bufs;
    p->stages = taken >= FPROP_SMEM ? 0 : (int)std::min<uint32_t>(FP_MAX_STAGES, (FPROP_SMEM - taken) / 16384u);
    if (p->stages >= 4) break;
  }
  if (p->out_bufs == 0) p->out_bufs = 1;
  if (p->stages < 3) return false;
  p->w_at = (uint32_t)p->stages * 16384u;
  p->out_at = p->w_at + (uint32_t)(p->kb * p->N) * 128u;
  p->tab_at = p->out_at + 4u * 4096u * (uint32_t)p->out_bufs;
  const uint32_t fmt = esz == 4 ? 2u : 1u;
  p->idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p->N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  return true;
}
static bool fprop_aligned(const OnoConvFprop* d) {
  const int esz = d->dtype == 0 ? 4 : 2, ckk = d->g.C * d->g.K * d->g.K;
  if ((d->ldx * esz | d->ld_kop * esz | d->ld_y * esz | (d->cols ? d->ld_cols * esz : 0)) & 15) return false;
  if (((uintptr_t)d->x | (uintptr_t)d->kop | (uintptr_t)d->y | (uintptr_t)d->cols) & 15) return false;
  return d->ldx >= d->g.C && d->ld_kop >= ckk && d->ld_y >= d->F && (!d->cols || d->ld_cols >= ckk);
}
}  // namespace ono

using namespace ono;

extern "C" int ono_conv_fprop_fits(const OnoConvFprop* d) {
  FpropDev p;
  return d && fprop_aligned(d) && fprop_plan(d, &p) ? 1 : 0;
}

// Whether this kernel is the faster form for sizes that it takes. A CTA goes through a tile's blocks of 128 bytes one after the other, and a product of
// few tiles may split them over a cluster: up to 32 tiles of f32 this kernel takes 3.7 us + 0.56 a block + 0.026 a filter, im2col and the product 6.7 +
// 0.36 a block, whatever the tiles (409 drawn layers, within 0.9 and 1.2 us). The line below is a little beyond the one where they meet, where as
// much is lost on either side: 12 x 12 x 20 -> 40, 5 x 5, of 4 to 32 images 16.2 us here and 14.1 as two, 14 x 14 x 64 -> 64, stride 2, of 8 15.7 and 14.9,
// 28 x 28 x 16 -> 32, of 8 8.0 and 9.3. bf16 has half the blocks and a product that keeps its order of sums, i.e. does not split them there
// (where it does, the caller takes the two kernels): never slower here by more than 1.02 times.
extern "C" int ono_conv_fprop_pays(const OnoConvGeom* g, int F, int dtype) {
  if (!g) return 0;
  const long long tiles = ((long long)g->B * g->OH * g->OW + 127) / 128, blocks = ((long long)g->C * g->K * g->K * 4 + 127) / 128;
  return dtype != 0 || tiles > 32 || 8 * blocks + F <= 8 * 18;
}

template <int ESIZE, int AHEAD>
static int fprop_launch(const CUtensorMap& tw, const CUtensorMap& tc, const CUtensorMap& ty, const FpropDev& p, cudaStream_t st) {
  auto kern = conv_fprop_kernel<ESIZE, AHEAD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FPROP_SMEM);
  if (e == cudaSuccess) {
    kern<<<std::min(p.tiles, ono_num_sms()), 448, p.tab_at + (size_t)p.kb * 64 + 1024, st>>>(tw, tc, ty, p);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) { set_error("conv_fprop: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}

extern "C" int ono_conv_fprop(const OnoConvFprop* d, ono_stream_t st) {
  FpropDev p;
  if (!d || !d->x || !d->kop || !d->y || !fprop_aligned(d) || !fprop_plan(d, &p)) { set_error("bad conv_fprop args%s", "", 0, 0); return -1; }
  p.d = *d;
  if (!p.d.timeout_ns) p.d.timeout_ns = 2000000000ull;
  const int esz = d->dtype == 0 ? 4 : 2, BK = 128 / esz, ckk = d->g.C * d->g.K * d->g.K;
  CUtensorMap tw, tc, ty;
  int rc = encode_map_2d(&tw, d->kop, esz, d->F, ckk, d->ld_kop, BK, p.N, false);
  if (!rc) rc = encode_out_map(&ty, d->y, esz, p.rows, d->F, d->ld_y);
  tc = tw;
  if (!rc && d->cols) rc = encode_map_2d(&tc, d->cols, esz, p.rows, ckk, d->ld_cols, BK, 128, false);
  if (rc) return rc;
  const cudaStream_t s = (cudaStream_t)st;
  if (p.stages >= 7) return esz == 4 ? fprop_launch<4, 5>(tw, tc, ty, p, s) : fprop_launch<2, 5>(tw, tc, ty, p, s);
  if (p.stages >= 5) return esz == 4 ? fprop_launch<4, 3>(tw, tc, ty, p, s) : fprop_launch<2, 3>(tw, tc, ty, p, s);
  return esz == 4 ? fprop_launch<4, 1>(tw, tc, ty, p, s) : fprop_launch<2, 1>(tw, tc, ty, p, s);
}
