// Input gradient of a convolution as one kernel (the reference: arch/layers/conv/conv2d.rs:84-104,202-266, K^T x dy per sample, then col2im).
//
// As two kernels the column gradient [pixels, k * k * C] goes to memory and comes back: of 32 channels under a 3 x 3 kernel with stride 2 it
// is 2.25 times the input gradient that remains of it. Here it stays in shared memory. A CTA takes the output pixels of one or a few
// images (at most 256, one or two 128-row tiles) and walks the input channels in chunks of 16 to 64 bytes; for a chunk
//
//   warp 16  brings dy (once) and the chunk's rows of K^T, for all taps one 3-D box, by TMA;
//   warp 17  issues the tcgen05 products into TMEM: [256 pixels][taps x chunk], f32;
//   warps 0-15 move the tiles to shared memory, rounded to the tile type as the column matrix was, then gather: an input pixel adds
//              the taps of the windows over it, in f32 and in tap order, applies act' and stores 16 bytes. Meanwhile the products of the
//              next chunk run, and the stored activations it needs first are under way.
//
// Which windows lie over a pixel is the same in every image: a table in shared memory, made once per CTA, holds the place of a pixel's
// first tap and a mask of those that exist; the others follow at fixed steps. Every value is that of the two kernels to the bit: the same products,
// reduced in the same order, the same rounding, the same sums. Product and fold as two kernels -> here, us: 2048 images of 28 x 28 x 32 under 64
// filters, 3 x 3, stride 2, bf16 155.2 -> 107.6; of 14 x 14 x 64 72.5 -> 58.9; 342 of the former, f32, 53.7 -> 40.4; 512 of 14 x 14 x 20 under 40 filters,
// 5 x 5, bf16 79.4 -> 23.2; 700 x 11 under 30, f32, 85.3 -> 24.7; 64 x 6 under 16 11.8 -> 7.0. What bounds it is the gather's instructions (48 and 44 %
// of the issue slots over all phases of the first two); bf16 values are added as they are (unpacked first 123 us of the 107.6), taps that a pixel does not have
// cost nothing. Room for the columns of two chunks, so that one is moved while the other is gathered, gave nothing (106.7, and registers: f32 60).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "act.cuh"
#include "ono_kernels.h"
#include "opt.cuh"
#include "piece.cuh"
#include "ptx.cuh"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);
int encode_map_2d(CUtensorMap* map, const void* base, int esize, long long rows, long long cols, long long ld, int box_cols, int box_rows,
                  bool swizzle_32b_units);
int encode_map_3d(CUtensorMap* map, const void* base, int esize, long long nz, long long rows, long long cols, long long ld, int box_cols,
                  int box_rows, int box_z);

struct DgradDev {
  OnoConvDgrad d;
  int G, units, tiles;        // images of a work unit, units, 128-row tiles of a unit
  int taps, pc, cc;           // k * k, 16-byte pieces and channels of a chunk
  int passes, split, per;     // chunks of C; a unit's chunks are dealt to `split` work items of `per`
  int kb;                     // 128-byte blocks of F
  int N, parts, NS, Q;        // columns of a tile's product and the instructions they take (at most 256 each), TMEM columns of a tile, pieces of a
                              // row in shared memory (odd: rows start in all banks)
  int a_bufs, b_bufs;
  uint32_t tmem_cols, idesc, b_bytes, b_block;      // bytes a chunk's K^T brings per block of F, and the room it takes
  uint32_t a_at, b_at, col_at, tab_at;              // offsets in shared memory
  uint32_t inv_hw;            // 2^32 / (H * W) rounded up: exact for the pixels of a unit (at most 256 images of 4096)
  int step_i, step_j;         // pieces from a tap to the next one of a pixel, downwards and to the right
};

__device__ __forceinline__ void dgrad_fail(const DgradDev& p, volatile int* abort_flag, int code) {
  if (p.d.status) atomicCAS(p.d.status, 0, code);
  *abort_flag = 1;
}

constexpr int DG_WARPS = 16, DG_THREADS = 32 * DG_WARPS;      // of the gather

template <int ESIZE, int KT>
__global__ void __maxnreg__(88)      // of 576 threads; room for a block of the batch feed beside the CTA
conv_dgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ DgradDev p) {
  using T = std::conditional_t<ESIZE == 4, float, __nv_bfloat16>;
  constexpr int BK = 128 / ESIZE, V = 16 / ESIZE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t a_full[2], a_empty[2], b_full[2], b_empty[2], acc_full, acc_empty, drain_bar;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  volatile int* abortp = &abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const OnoConvGeom& g = p.d.g;
  const int OHW = g.OH * g.OW, HW = g.H * g.W;
  const uint64_t budget = p.d.timeout_ns;

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) { mbar_init(&a_full[b], 1); mbar_init(&a_empty[b], 1); mbar_init(&b_full[b], 1); mbar_init(&b_empty[b], 1); }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, DG_THREADS);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == DG_WARPS && lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); }
  if (warp == DG_WARPS + 1) { tmem_alloc(&tmem_base_smem, p.tmem_cols); tmem_relinquish(); }
  // the windows over each pixel of an image
  int2* const tab = reinterpret_cast<int2*>(smem + p.tab_at);
  if (warp < DG_WARPS)
    for (int i = threadIdx.x; i < HW; i += DG_THREADS) {
      const int iyp = i / g.W + g.P, ixp = i % g.W + g.P, ky0 = iyp % g.S, kx0 = ixp % g.S, oy0 = iyp / g.S, ox0 = ixp / g.S;
      uint32_t mask = 0;
      for (int a = 0; a < KT; ++a)
        for (int b = 0; b < KT; ++b) {
          const int ky = ky0 + g.S * a, kx = kx0 + g.S * b, oy = oy0 - a, ox = ox0 - b;
          if (ky < g.K && kx < g.K && oy >= 0 && ox >= 0 && oy < g.OH && ox < g.OW) mask |= 1u << (a * KT + b);
        }
      tab[i] = make_int2((oy0 * g.OW + ox0) * p.Q + (ky0 * g.K + kx0) * p.pc, (int)mask);
    }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  const int items = p.units * p.split;

  if (warp == DG_WARPS) {
    // ---------------- TMA producer ----------------
    bool ok = true;
    int na = 0, nb = 0;
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++na) {
      const int unit = it / p.split, c0 = (it - unit * p.split) * p.per, c1 = min(p.passes, c0 + p.per);
      const int ab = na % p.a_bufs;
      const bool free = mbar_wait_bounded(&a_empty[ab], ((na / p.a_bufs) & 1) ^ 1u, abortp, budget);
      if (!__all_sync(0xffffffffu, free)) { dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_EMPTY); ok = false; break; }
      if (elect_one()) {
        mbar_expect_tx(&a_full[ab], (uint32_t)(p.tiles * p.kb) * 16384u);
        for (int t = 0; t < p.tiles; ++t)
          for (int k = 0; k < p.kb; ++k)
            tma_load_2d(smem + p.a_at + (uint32_t)((ab * p.tiles + t) * p.kb + k) * 16384u, &tmA, &a_full[ab], k * BK, unit * p.G * OHW + t * 128);
      }
      __syncwarp();
      for (int c = c0; c < c1; ++c, ++nb) {
        const int bb = nb % p.b_bufs;
        const bool room = mbar_wait_bounded(&b_empty[bb], ((nb / p.b_bufs) & 1) ^ 1u, abortp, budget);
        if (!__all_sync(0xffffffffu, room)) { dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_EMPTY); ok = false; break; }
        if (elect_one()) {
          mbar_expect_tx(&b_full[bb], p.b_bytes * (uint32_t)p.kb);
          for (int k = 0; k < p.kb; ++k) tma_load_3d(smem + p.b_at + (uint32_t)(bb * p.kb + k) * p.b_block, &tmB, &b_full[bb], k * BK, c * p.cc, 0);
        }
        __syncwarp();
      }
    }
    if (!ok) {      // copies already in flight land before the CTA retires its shared memory
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
    }
  } else if (warp == DG_WARPS + 1) {
    // ---------------- MMA issuer ----------------
    bool ok = true;
    int na = 0, nb = 0;
    const uint32_t base = smem_u32(smem);
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++na) {
      const int unit = it / p.split, c0 = (it - unit * p.split) * p.per, c1 = min(p.passes, c0 + p.per);
      const int ab = na % p.a_bufs;
      const bool here = mbar_wait_bounded(&a_full[ab], (na / p.a_bufs) & 1, abortp, budget);
      if (!__all_sync(0xffffffffu, here)) { dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_FULL); ok = false; break; }
      for (int c = c0; c < c1; ++c, ++nb) {
        const int bb = nb % p.b_bufs;
        bool go = mbar_wait_bounded(&b_full[bb], (nb / p.b_bufs) & 1, abortp, budget);
        if (!__all_sync(0xffffffffu, go)) { dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_FULL); ok = false; break; }
        go = mbar_wait_bounded(&acc_empty, (nb & 1) ^ 1u, abortp, budget);
        if (!__all_sync(0xffffffffu, go)) { dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_EMPTY); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          for (int t = 0; t < p.tiles; ++t)
            for (int k = 0; k < p.kb; ++k) {
              const uint64_t ad = make_smem_desc_sw128(base + p.a_at + (uint32_t)((ab * p.tiles + t) * p.kb + k) * 16384u, 16, 1024);
              const uint64_t bd = make_smem_desc_sw128(base + p.b_at + (uint32_t)(bb * p.kb + k) * p.b_block, 16, 1024);
              const int n1 = p.N / p.parts;
              for (int h = 0; h < p.parts; ++h) {
                const uint32_t to = tmem_base + (uint32_t)(t * p.NS + h * n1);
                const uint64_t bh = bd + (uint32_t)(h * n1 * 128 >> 4);
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                  if (ESIZE == 4) umma_tf32(to, ad + 2 * s, bh + 2 * s, p.idesc, (k | s) != 0);
                  else umma_f16(to, ad + 2 * s, bh + 2 * s, p.idesc, (k | s) != 0);
                }
              }
            }
          umma_commit(&b_empty[bb]);
          if (c == c1 - 1) umma_commit(&a_empty[ab]);
          umma_commit(&acc_full);
        }
        __syncwarp();
      }
    }
    if (elect_one()) umma_commit(&drain_bar);      // no MMA may still run when TMEM is released
    __syncwarp();
    mbar_wait_bounded(&drain_bar, 0, abortp, ok ? budget : 1000000ull);
  } else {
    // ---------------- tiles to shared memory, gather ----------------
    bool ok = true;
    uint4* const col = reinterpret_cast<uint4*>(smem + p.col_at);
    const int tile = (warp >> 2) & 1, quad = warp & 3, half = warp >> 3, row = tile * 128 + quad * 32 + lane, live = p.taps * p.pc;
    const T* const aux = reinterpret_cast<const T*>(p.d.aux);
    T* const dx = reinterpret_cast<T*>(p.d.dx);
    const int lg = p.pc >> 1, pm = p.pc - 1;       // pieces of a chunk: 1, 2 or 4
    // Pixels of a thread in one round, and their stored values: those of the next round (of the next chunk or unit at the end of one)
    // are fetched as this round's are used up, so that they come while the products are waited for and moved. More pixels a round only
    // make the code longer (bf16, 2 x 2 taps: four 114.7 us, two 107.6, one 127.4; 3 x 3 taps: two 55.1, one 52.3).
    constexpr int U = KT <= 2 ? 2 : 1;
    uint4 av[U];
    struct Place { long long pix0; int total, ch0; };      // a chunk: its first pixel, pieces of all its pixels, first channel
    auto place = [&](int it, int c) {
      Place w{0, 0, 0};
      if (it < items) {
        const int unit = it / p.split;
        if (c < 0) c = (it - unit * p.split) * p.per;
        w.pix0 = (long long)unit * p.G * HW;
        w.total = (min(p.G, g.B - unit * p.G) * HW) << lg;
        w.ch0 = c * p.cc;
      }
      return w;
    };
    auto fetch = [&](const Place& w, int e) {
      const int ch = w.ch0 + (e & pm) * V;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (p.d.dact != ACT_NONE && e < w.total && ch < g.C) v = *reinterpret_cast<const uint4*>(aux + (w.pix0 + (e >> lg)) * p.d.ld_aux + ch);
      return v;
    };
    {
      const Place w = place(blockIdx.x, -1);
#pragma unroll
      for (int u = 0; u < U; ++u) av[u] = fetch(w, threadIdx.x + u * DG_THREADS);
    }
    int n = 0;
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
      const int unit = it / p.split, c0 = (it - unit * p.split) * p.per, c1 = min(p.passes, c0 + p.per);
      for (int c = c0; c < c1; ++c, ++n) {
        const bool got = mbar_wait_bounded(&acc_full, n & 1, abortp, budget);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) dgrad_fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_FULL);
          ok = false;
        }
        tc_fence_after();
        if (ok && tile < p.tiles) {
          for (int q0 = half; q0 < p.NS / 32; q0 += 2) {
            uint32_t r[32];
            tmem_ld_x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(tile * p.NS + q0 * 32), r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32 / V; ++j) {
              const int q = q0 * (32 / V) + j;
              if (q >= live) continue;
              uint4 w;
              if (ESIZE == 4) w = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
              else {
                const float* f = reinterpret_cast<const float*>(r) + 8 * (ESIZE == 2 ? j : 0);
                w = make_uint4(pack16x2(f[0], f[1], 0), pack16x2(f[2], f[3], 0), pack16x2(f[4], f[5], 0), pack16x2(f[6], f[7], 0));
              }
              col[row * p.Q + q] = w;
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&acc_empty);
        // the tile is there; all warps go on, or none does (a warp that left alone would be waited for below)
        uint32_t stop;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                     : "=r"(stop) : "r"((uint32_t)(!ok || *abortp)), "n"(DG_THREADS) : "memory");
        ok = !stop;
        if (!ok) break;
        const Place here = place(it, c);
#pragma unroll 1
        for (int eb = threadIdx.x; eb - (int)threadIdx.x < here.total; eb += U * DG_THREADS) {
          const bool more = eb - (int)threadIdx.x + U * DG_THREADS < here.total;
          const Place next = more ? here : c + 1 < c1 ? place(it, c + 1) : place(it + gridDim.x, -1);
          const int en = more ? eb + U * DG_THREADS : threadIdx.x;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int e = eb + u * DG_THREADS, px = e >> lg, piece = e & pm, ch = here.ch0 + piece * V;
            if (e < here.total && ch < g.C) {
              const int im = HW > 1 ? (int)__umulhi((uint32_t)px, p.inv_hw) : px;
              const int2 tb = tab[px - im * HW];
              const uint4* at = col + im * OHW * p.Q + tb.x + piece;
              float acc[V];
#pragma unroll
              for (int k = 0; k < V; ++k) acc[k] = 0.f;
              constexpr int R = KT <= 2 ? KT : 1;      // rows of taps fetched together
#pragma unroll
              for (int i0 = 0; i0 < KT; i0 += R) {
                uint4 w[R * KT];
#pragma unroll
                for (int i = 0; i < R * KT; ++i)
                  if ((tb.y >> (i0 * KT + i)) & 1) w[i] = at[(i0 + i / KT) * p.step_i + i % KT * p.step_j];
#pragma unroll
                for (int i = 0; i < R * KT; ++i)
                  if ((tb.y >> (i0 * KT + i)) & 1) add_piece<T, V>(acc, w[i]);
              }
              if (p.d.dact != ACT_NONE) {
                float a[V];
                unpack_piece<T, uint4>(av[u], a);
                act_bwd_n<V>(p.d.dact, p.d.dact_param, p.d.relu_quirk, a, acc);
              }
              *reinterpret_cast<uint4*>(dx + (here.pix0 + px) * p.d.ld_dx + ch) = pack_piece<T, uint4>(acc);
            }
            av[u] = fetch(next, en + u * DG_THREADS);
          }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(DG_THREADS) : "memory");      // the column tile has been read
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == DG_WARPS + 1) { tc_fence_after(); tmem_dealloc(tmem_base, p.tmem_cols); }
}

constexpr uint32_t DGRAD_SMEM = 225u * 1024u;      // the rest is a block's of the batch feed
// The plan with chunks of `pc` pieces and up to `G` images a unit; false: it does not fit.
static bool dgrad_plan_as(const OnoConvDgrad* d, DgradDev* p, int sms, int pc, int G, int split) {
  const OnoConvGeom& g = d->g;
  const int esz = d->dtype == 0 ? 4 : 2, V = 16 / esz;
  memset(p, 0, sizeof(*p));
  p->taps = g.K * g.K;
  p->pc = pc;
  p->cc = pc * V;
  p->parts = p->taps * p->cc > 256 ? 2 : 1;
  p->N = (p->taps * p->cc + 16 * p->parts - 1) / (16 * p->parts) * (16 * p->parts);
  p->NS = (p->N + 31) / 32 * 32;
  p->Q = (p->taps * p->pc) | 1;
  p->kb = (d->F * esz + 127) / 128;
  p->passes = (g.C + p->cc - 1) / p->cc;
  p->inv_hw = (uint32_t)(((1ull << 32) + (unsigned)(g.H * g.W) - 1) / (unsigned)(g.H * g.W));
  p->step_i = g.S * g.K * p->pc - g.OW * p->Q;
  p->step_j = g.S * p->pc - p->Q;
  // no fewer units than SMs
  p->G = std::max(1, std::min(G, (g.B + sms - 1) / sms));
  p->tiles = (p->G * g.OH * g.OW + 127) / 128;
  p->units = (g.B + p->G - 1) / p->G;
  p->per = (p->passes + split - 1) / split;
  p->split = (p->passes + p->per - 1) / p->per;
  p->b_bytes = (uint32_t)(p->taps * p->cc * 128);
  p->b_block = ((uint32_t)(p->N * 128) + 1023u) & ~1023u;
  p->tmem_cols = 32;
  while (p->tmem_cols < (uint32_t)(p->tiles * p->NS)) p->tmem_cols *= 2;
  if (p->tiles > 2 || p->tmem_cols > 512 || p->N / p->parts > 256) return false;
  const uint32_t colb = (uint32_t)(p->tiles * 128 * p->Q) * 16u, tabb = (uint32_t)(g.H * g.W) * 8u;
  for (int v = 0; v < 3; ++v) {                  // two buffers each, one of dy, one each
    p->a_bufs = v == 0 ? 2 : 1;
    p->b_bufs = v <= 1 ? 2 : 1;
    p->a_at = 0;
    p->b_at = (uint32_t)(p->a_bufs * p->tiles * p->kb) * 16384u;
    p->col_at = p->b_at + (uint32_t)(p->b_bufs * p->kb) * p->b_block;
    p->tab_at = p->col_at + colb;
    if (p->tab_at + tabb + 1024u <= DGRAD_SMEM) break;
    if (v == 2) return false;
  }
  const uint32_t fmt = esz == 4 ? 2u : 1u;
  p->idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)((p->N / p->parts) >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  return true;
}
// Everything that follows from the sizes; false: not a problem for this kernel. A warp's 16-byte
// accesses to pixels touch 32 / pc lines, each of its tap loads takes eight cycles; beside it a chunk costs about 1500 cycles in
// waits, barriers and the tile's way to shared memory. One tile of fewer images with wider chunks often beats two with narrow ones
// (2048 images, 14 x 14, 64 channels, bf16: 78.6 us with two tiles of 32-byte chunks, 64.0 with one of 64-byte chunks). A unit's chunks go to
// several CTAs where that fills the last round better (342 images of 28 x 28 x 32, f32: three rounds of 148 units 44.7 us, five of half a unit 40.4).
static bool dgrad_plan(const OnoConvDgrad* d, DgradDev* p, int sms) {
  const OnoConvGeom& g = d->g;
  if (g.B <= 0 || g.C <= 0 || d->F <= 0 || g.K < 1 || g.K > 5 || g.S < 1 || g.P < 0 || g.OH <= 0 || g.OW <= 0 || g.OH * g.OW > 256) return false;
  if ((long long)g.H * g.W > 4096 || (long long)g.B * g.H * g.W >= (1ll << 30)) return false;
  const int OHW = g.OH * g.OW, KT = (g.K + g.S - 1) / g.S;
  double best = 0.0;
  DgradDev q;
  for (int pc = 4; pc >= 1; pc /= 2)
    for (int tiles = 1; tiles <= 2; ++tiles)
      for (int split = 1; split == 1 || split <= q.passes; ++split) {
        if (128 * tiles < OHW || !dgrad_plan_as(d, &q, sms, pc, 128 * tiles / OHW, split)) break;
        const double chunk = 1500.0 + 1.4 * q.G * g.H * g.W * pc / 32.0 * (64.0 / pc + 8.0 * KT * KT);
        const double cost = (chunk * q.per + 500.0) * ((q.units * q.split + sms - 1) / sms);
        if (best == 0.0 || cost < best) { best = cost; *p = q; }
      }
  return best > 0.0;
}
static bool dgrad_aligned(const OnoConvDgrad* d) {
  const int esz = d->dtype == 0 ? 4 : 2, V = 16 / esz, up = (d->g.C + V - 1) / V * V;
  const bool aux = d->dact != ACT_NONE;
  if ((d->ld_dy * esz | d->ld_kt * esz | d->ld_dx * esz | (aux ? d->ld_aux * esz : 0)) & 15) return false;
  if (((uintptr_t)d->dy | (uintptr_t)d->kt | (uintptr_t)d->dx | (aux ? (uintptr_t)d->aux : 0)) & 15) return false;
  return d->ld_dy >= d->F && d->ld_kt >= d->F && d->ld_dx >= up && (!aux || d->ld_aux >= up);
}
}  // namespace ono

using namespace ono;

extern "C" int ono_conv_dgrad_fits(const OnoConvDgrad* d) {
  DgradDev p;
  return d && dgrad_aligned(d) && dgrad_plan(d, &p, ono_num_sms()) ? 1 : 0;
}

// Whether this kernel is the faster form for sizes that it takes. A unit brings all of K^T to its SM and moves whole 128-row tiles, however few
// output pixels an image has; a plain product shares both among images. So with few output pixels and many filters or channels the product and the
// fold win: 128 images of 4 x 4 x 64 under 256 filters, f32, 32.0 us here and 10.7 as two, 7 x 7 x 96 under 96, 5 x 5, 37.0 and 22.3, bf16 24.9
// and 17.0. Both times were fitted to 1589 drawn layers (4 to 32 pixels wide, 1 to 128 channels, 4 to 256 filters, 1 to 2048 images; this kernel's
// within 8 %, the other within 10), us: the line lets 5 % pass, which is what they scatter by. Of the drawn layers 67 were slower here by
// more than 3 % (at most 2.2 times), 55 take two kernels now, and of the others none is slower by more than 1.14 times where the fold has its vector form;
// of 1320 more, up to four times the size, 41 were slower by more than 5 %, and 13 still are.
// That form is for kernels of 3 and 5, strides of 1 and 2 and channels in whole pieces; other layers take this kernel (4 x 4: 0.3 of the time).
extern "C" int ono_conv_dgrad_pays(const OnoConvGeom* g, int F, int dtype) {
  OnoConvDgrad d = {};
  DgradDev p;
  if (!g) return 0;
  d.g = *g;
  d.F = F;
  d.dtype = dtype;
  const int sms = ono_num_sms(), esz = dtype == 0 ? 4 : 2;
  if (!dgrad_plan(&d, &p, sms)) return 0;
  if ((g->K != 3 && g->K != 5) || g->S > 2 || g->C % (16 / esz)) return 1;
  const double MB = 1e-6 * esz, rows = (double)g->B * g->OH * g->OW, ckk = (double)g->C * p.taps;
  const int KT = (g->K + g->S - 1) / g->S, rounds = (p.units * p.split + sms - 1) / sms;
  const double pieces = (double)p.G * g->H * g->W * p.pc;
  const double chunk = 0.674 + 0.00345 * p.N + (0.000886 + 0.000079 * KT * KT) * pieces + 0.000615 * p.tiles * p.N * p.kb;
  const double one = 4.07 + rounds * (p.per * chunk + 0.194 + 0.131 * p.tiles * p.kb);
  const double tiles = std::ceil(rows / 128) * std::ceil(ckk / 128), waves = std::ceil(tiles / sms);
  const double two = 6.49 + 0.184 * MB * rows * ckk + 0.461 * MB * g->B * g->H * g->W * g->C + waves * (0.829 + 0.141 * p.kb) + 0.051 * p.kb;
  return one <= 1.05 * two;
}

template <int ESIZE, int KT>
static int dgrad_launch(const CUtensorMap& ta, const CUtensorMap& tb, const DgradDev& p, int grid, size_t smem, cudaStream_t st) {
  auto kern = conv_dgrad_kernel<ESIZE, KT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DGRAD_SMEM);
  if (e == cudaSuccess) {
    kern<<<grid, DG_THREADS + 64, smem, st>>>(ta, tb, p);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) { set_error("conv_dgrad: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}

extern "C" int ono_conv_dgrad(const OnoConvDgrad* d, ono_stream_t st) {
  DgradDev p;
  if (!d || !d->dy || !d->kt || !d->dx || (d->dact != ACT_NONE && !d->aux) || !dgrad_aligned(d) || !dgrad_plan(d, &p, ono_num_sms())) {
    set_error("bad conv_dgrad args%s", "", 0, 0);
    return -1;
  }
  p.d = *d;
  if (!p.d.timeout_ns) p.d.timeout_ns = 2000000000ull;
  const OnoConvGeom& g = d->g;
  const int esz = d->dtype == 0 ? 4 : 2, BK = 128 / esz;
  CUtensorMap ta, tb;
  int rc = encode_map_2d(&ta, d->dy, esz, (long long)g.B * g.OH * g.OW, d->F, d->ld_dy, BK, 128, false);
  if (!rc) rc = encode_map_3d(&tb, d->kt, esz, p.taps, g.C, d->F, d->ld_kt, BK, p.cc, p.taps);
  if (rc) return rc;
  const int grid = std::min(p.units * p.split, ono_num_sms()), KT = (g.K + g.S - 1) / g.S;
  const size_t smem = p.tab_at + (size_t)g.H * g.W * 8 + 1024;
  const cudaStream_t s = (cudaStream_t)st;
#define ONO_DGRAD(KK) case KK: return esz == 4 ? dgrad_launch<4, KK>(ta, tb, p, grid, smem, s) : dgrad_launch<2, KK>(ta, tb, p, grid, smem, s)
  switch (KT) {
    ONO_DGRAD(1);
    ONO_DGRAD(2);
    ONO_DGRAD(3);
    ONO_DGRAD(4);
    default: return esz == 4 ? dgrad_launch<4, 5>(ta, tb, p, grid, smem, s) : dgrad_launch<2, 5>(ta, tb, p, grid, smem, s);
  }
#undef ONO_DGRAD
}
