// Persistent, warp-specialised tcgen05 GEMM for sm_100a: the dense forward / dgrad / wgrad work of
// the reference's Dense layer (machine_learning/src/arch/layers/dense.rs:36-64) and the GEMM half
// of its im2col convolution (arch/layers/conv/conv2d.rs:119-125), rebuilt for Blackwell.
//
//   warp 4 (one elected lane)  TMA producer: cp.async.bulk.tensor tiles -> 128B-swizzled smem ring
//   warp 5 (one elected lane)  MMA issuer:   tcgen05.mma (kind::tf32 | kind::f16/bf16), f32
//                                            accumulators in TMEM, double buffered (2 x BN columns)
//   warps 0-3 and 6-9          epilogue:     two groups taking alternate 32-column chunks: tcgen05.ld
//                                            TMEM -> registers, bias / activation / activation-
//                                            derivative / accumulate, stores (row-major through a
//                                            swizzled staging tile + TMA store, transposed, f32, bf16)
//
// Operands may be K-major or MN-major (bf16 and tf32); the difference is confined to the TMA box
// pattern and three descriptor fields computed on the host (see make_operand()).
// All mbarrier waits are bounded; on a timeout the kernel records a code in *status, every role
// leaves its loop, TMEM is freed and the kernel returns normally.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "act.cuh"
#include "ono_kernels.h"
#include "opt.cuh"
#include "ptx.cuh"

namespace ono {

struct OperandDev {
  int mn_major;       // 0: K contiguous in global memory, 1: MN contiguous
  int n_box;          // TMA boxes per stage
  int box_mn;         // MN extent covered by one box
  uint32_t box_stride_bytes;
  uint32_t lbo_bytes, sbo_bytes, kstep_bytes;
  uint32_t layout_type;  // shared-memory descriptor layout: 2 = 128B swizzle, 1 = 128B swizzle on 32B units
};

struct GemmDev {
  int M, N, K;
  OperandDev a, b;
  uint32_t idesc;
  OnoEpilogue epi;
  int* status;
  unsigned long long timeout_ns;
  int split_k;  // > 1: K is split over that many work items per tile; split s writes its partial product to slab s of `slabs`
  int tma_out;  // plain result through TMA: 1: out_f32 store; 2: out_bf16 store; 3: out_f32 += reduce-add. 0: everything else
  int staged;   // 1: epilogue_rows on the staged tile (no split, no optimizer, no TMA store)
  int vec;      // row-major outputs and aux are aligned for accesses of four columns
  int vec_t;    // transposed outputs are aligned for accesses of four rows
  float* slabs;            // split-K partial products: [split_k][M][slab_ld] f32
  long long slab_elems;    // M * slab_ld
  int slab_ld;
  OnoApply apply;          // optimizer applied to the result tile in the epilogue (apply.p != nullptr)
  const unsigned int* gate;          // flags that must reach *gate_target before the first operand load (nullptr: none)
  const unsigned int* gate_target;
  int gate_stride;
  unsigned int gate_mask;
};

template <int BN>
struct TileCfg {
  static constexpr int STAGES = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
  static constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
};

__device__ __forceinline__ void fail(const GemmDev& p, volatile int* abort_flag, int code) {
  if (p.status) atomicCAS(p.status, 0, code);
  *abort_flag = 1;
}

// ---------------- epilogue arithmetic on groups of four columns ----------------
// The activation is chosen once for a whole group of values, and the code of one group is a few hundred instructions: the
// choice made per element, unrolled over 32 columns, cost small launches their time in instruction fetches (a 32 x 128 x 10
// product with a ReLU derivative and a transposed copy: 19.7 us before, 18.3 after).
template <int G>
__device__ __forceinline__ void act_fwd_group(int kind, float prm, float4 (&v)[G]) {
  float* f = reinterpret_cast<float*>(v);
  switch (kind) {
    case ACT_RELU:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_fwd(ACT_RELU, prm, f[j]);
      break;
    case ACT_SIGMOID:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_fwd(ACT_SIGMOID, prm, f[j]);
      break;
    case ACT_TANH:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_fwd(ACT_TANH, prm, f[j]);
      break;
    case ACT_GELU:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_fwd(ACT_GELU, prm, f[j]);
      break;
    default: break;
  }
}
template <int G>
__device__ __forceinline__ void act_bwd_group(int kind, float prm, int quirk, const float4 (&s)[G], float4 (&v)[G]) {
  float* f = reinterpret_cast<float*>(v);
  const float* a = reinterpret_cast<const float*>(s);
  switch (kind) {
    case ACT_RELU:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_bwd(ACT_RELU, prm, quirk, a[j], f[j]);
      break;
    case ACT_SIGMOID:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_bwd(ACT_SIGMOID, prm, quirk, a[j], f[j]);
      break;
    case ACT_TANH:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_bwd(ACT_TANH, prm, quirk, a[j], f[j]);
      break;
    case ACT_GELU:
#pragma unroll
      for (int j = 0; j < 4 * G; ++j) f[j] = act_bwd(ACT_GELU, prm, quirk, a[j], f[j]);
      break;
    default: break;
  }
}

// Four consecutive values of which `left` (>= 1) are inside the matrix; `vec`: the address is aligned for one access.
__device__ __forceinline__ float4 load_f32x4(const float* p, int left, int vec) {
  if (left >= 4 && vec) return *reinterpret_cast<const float4*>(p);
  return make_float4(p[0], left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ void store_f32x4(float* p, float4 v, int left, int vec) {
  if (left >= 4 && vec) { *reinterpret_cast<float4*>(p) = v; return; }
  p[0] = v.x;
  if (left > 1) p[1] = v.y;
  if (left > 2) p[2] = v.z;
  if (left > 3) p[3] = v.w;
}
__device__ __forceinline__ float4 load_b16x4(const void* base, size_t off, int left, int vec) {
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(base) + off;
  if (left >= 4 && vec) return unpack16x4(*reinterpret_cast<const uint2*>(p), 0);
  return make_float4(__bfloat162float(p[0]), left > 1 ? __bfloat162float(p[1]) : 0.f, left > 2 ? __bfloat162float(p[2]) : 0.f,
                     left > 3 ? __bfloat162float(p[3]) : 0.f);
}
__device__ __forceinline__ void store_b16x4(void* base, size_t off, float4 v, int left, int vec, int f16) {
  uint16_t* p = reinterpret_cast<uint16_t*>(base) + off;
  const uint2 w = make_uint2(pack16x2(v.x, v.y, f16), pack16x2(v.z, v.w, f16));
  if (left >= 4 && vec) { *reinterpret_cast<uint2*>(p) = w; return; }
  p[0] = (uint16_t)(w.x & 0xffffu);
  if (left > 1) p[1] = (uint16_t)(w.x >> 16);
  if (left > 2) p[2] = (uint16_t)(w.y & 0xffffu);
  if (left > 3) p[3] = (uint16_t)(w.y >> 16);
}
__device__ __forceinline__ float4 load_bias4(const OnoEpilogue& e, int n, int left) {
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (left <= 0) return b;
  float* f = reinterpret_cast<float*>(&b);
  if (e.bias) {
#pragma unroll
    for (int j = 0; j < 4; ++j) if (j < left) f[j] = __ldg(e.bias + n + j);
  } else if (e.bias_bf16) {
    const __nv_bfloat16* bb = reinterpret_cast<const __nv_bfloat16*>(e.bias_bf16) + n;
#pragma unroll
    for (int j = 0; j < 4; ++j) if (j < left) f[j] = __bfloat162float(bb[j]);
  }
  return b;
}
__device__ __forceinline__ float4 load_aux4(const OnoEpilogue& e, int m, int n, int left, int vec) {
  const size_t off = (size_t)m * e.ld_aux + n;
  return e.aux_f32 ? load_f32x4(e.aux_f32 + off, left, vec) : load_b16x4(e.aux_bf16, off, left, vec);
}
// The same in two steps, for values fetched ahead of their use: four f32, or four bf16 in the first two words. (Unpacked where they are
// loaded, they would be waited for there.)
__device__ __forceinline__ uint4 load_aux4_raw(const OnoEpilogue& e, int m, int n, int left, int vec) {
  const size_t off = (size_t)m * e.ld_aux + n;
  uint4 w = make_uint4(0u, 0u, 0u, 0u);
  if (e.aux_f32) {
    const float4 v = load_f32x4(e.aux_f32 + off, left, vec);
    return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
  }
  const uint16_t* p = reinterpret_cast<const uint16_t*>(e.aux_bf16) + off;
  if (left >= 4 && vec) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    w.x = u.x; w.y = u.y;
  } else {
    w.x = p[0];
    if (left > 1) w.x |= (uint32_t)p[1] << 16;
    if (left > 2) w.y = p[2];
    if (left > 3) w.y |= (uint32_t)p[3] << 16;
  }
  return w;
}
__device__ __forceinline__ float4 aux4(const OnoEpilogue& e, uint4 w) {
  if (e.aux_f32) return make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
  return unpack16x4(make_uint2(w.x, w.y), 0);
}

// Rows m[0..G) of four columns starting at n (`left` of them inside the matrix): everything between the accumulator and
// the row-major outputs. Rows >= M are computed and not stored.
template <int G>
__device__ __forceinline__ void epilogue_rows(const OnoEpilogue& e, float4 (&v)[G], const int (&m)[G], int n, int left, int vec,
                                              int M, float4 bias, const float4 (&aux)[G]) {
#pragma unroll
  for (int i = 0; i < G; ++i) {
    v[i].x = fmaf(v[i].x, e.alpha, bias.x); v[i].y = fmaf(v[i].y, e.alpha, bias.y);
    v[i].z = fmaf(v[i].z, e.alpha, bias.z); v[i].w = fmaf(v[i].w, e.alpha, bias.w);
  }
  if (e.pre_f32) {
#pragma unroll
    for (int i = 0; i < G; ++i) if (m[i] < M) store_f32x4(e.pre_f32 + (size_t)m[i] * e.ld_out + n, v[i], left, vec);
  } else if (e.pre_bf16) {
#pragma unroll
    for (int i = 0; i < G; ++i) if (m[i] < M) store_b16x4(e.pre_bf16, (size_t)m[i] * e.ld_out + n, v[i], left, vec, 0);
  }
  act_fwd_group<G>(e.act, e.act_param, v);
  if (e.dact != ACT_NONE) act_bwd_group<G>(e.dact, e.dact_param, e.relu_quirk, aux, v);
  if (e.out_f32) {
#pragma unroll
    for (int i = 0; i < G; ++i)
      if (m[i] < M) {
        float* o = e.out_f32 + (size_t)m[i] * e.ld_out + n;
        if (e.beta != 0.0f) {
          const float4 old = load_f32x4(o, left, vec);
          v[i].x += e.beta * old.x; v[i].y += e.beta * old.y; v[i].z += e.beta * old.z; v[i].w += e.beta * old.w;
        }
        store_f32x4(o, v[i], left, vec);
      }
  }
  if (e.out_bf16) {
#pragma unroll
    for (int i = 0; i < G; ++i) if (m[i] < M) store_b16x4(e.out_bf16, (size_t)m[i] * e.ld_out + n, v[i], left, vec, e.out16_f16);
  }
}

// PAIR = true: two CTAs of a cluster work on one 256 x BN tile (tcgen05 cta_group::2). Each CTA stages its own
// 128 rows of A and its own BN/2 rows of B, so every byte of B crosses L2 -> SM once per pair instead of
// once per CTA; the leader CTA (cluster rank 0) issues the MMAs for both, each CTA drains its own TMEM.
// APPLY = true: the instantiation whose epilogue applies the optimizer through TMA: the operand ring shrinks to two
// stages and every epilogue warp gets APPLY_WARP_BYTES of shared memory for the tiles of the master, the optimizer state
// and the bf16 shadow that belong to the 32 x 32 accumulator chunk it is working on (see the epilogue below).
struct ApplyMaps { CUtensorMap p, m, v, s; };
constexpr uint32_t APPLY_WARP_BYTES = 20480;

// Registers: an SM's file has to hold blocks of other streams' kernels (the batch feed, the optimizer) beside the CTA; 168 registers left
// room for none. 152 leave a warp of the feed its place in each quarter of the file: steps back to back with 168 and so, three dense layers of 4096
// on 1024 rows 631 -> 597 us, eight of 8192 on 512 3396 -> 3261, four of 2048 and the convolutions level. Pairs with 128 597 -> 598. Without
// pairs 128 cost nothing and leave room for two.
template <int ESIZE, int BN, bool PAIR, bool APPLY>
__global__ void __maxnreg__(PAIR ? 152 : 128)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, const __grid_constant__ ApplyMaps am, const GemmDev p) {
  constexpr int BM = 128;              // rows per CTA
  constexpr int TILE_M = PAIR ? 256 : 128;
  constexpr int BK = 128 / ESIZE;      // one 128-byte swizzle row of K per stage
  constexpr int UMMA_K = 32 / ESIZE;   // 8 for tf32, 16 for bf16
  constexpr int KSTEPS = BK / UMMA_K;  // 4
  constexpr int BN_CTA = PAIR ? BN / 2 : BN;   // rows of B staged by one CTA
  constexpr uint32_t A_BYTES = BM * 128, B_BYTES = BN_CTA * 128, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int STAGES = APPLY ? 2 : TileCfg<BN_CTA>::STAGES;
  constexpr uint32_t TMEM_COLS = TileCfg<BN>::TMEM_COLS;
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u;
  const bool leader = crank == 0u;
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;      // CTA or CTA pair
  const int units = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  // eight 4 KB output staging tiles (one per epilogue warp: 32 rows x 128 B) behind the operand ring, for TMA stores
  uint8_t* cstage = smem + (size_t)STAGES * STAGE_BYTES;

  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tmem_full_bar[2];
  __shared__ __align__(8) uint64_t tmem_empty_bar[2];
  __shared__ __align__(8) uint64_t drain_bar;
  __shared__ __align__(8) uint64_t apply_bar[APPLY ? 16 : 1];   // [epilogue warp][buffer]: tiles of a chunk have landed
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // the same for the whole warp, also for the compiler
  const int lane = threadIdx.x & 31;
  volatile int* abortp = &abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full_bar[b], 1);
      mbar_init(&tmem_empty_bar[b], PAIR ? 512 : 256);   // 8 epilogue warps; a pair's leader counts both CTAs'
    }
    mbar_init(&drain_bar, 1);
    if (APPLY)
      for (int b = 0; b < 16; ++b) mbar_init(&apply_bar[b], 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (p.tma_out) tma_prefetch_desc(&tmC);
    if (APPLY) { tma_prefetch_desc(&am.p); tma_prefetch_desc(&am.m); tma_prefetch_desc(&am.v); tma_prefetch_desc(&am.s); }
  }
  if (warp == 5) {
    if (PAIR) { tmem_alloc_pair(&tmem_base_smem, TMEM_COLS); tmem_relinquish_pair(); }
    else { tmem_alloc(&tmem_base_smem, TMEM_COLS); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();   // the peer's barriers exist before anything is signalled across CTAs
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  const int num_m = (p.M + TILE_M - 1) / TILE_M;
  const int num_n = (p.N + BN - 1) / BN;
  const int total_tiles = num_m * num_n;
  const int KB = (p.K + BK - 1) / BK;
  const uint64_t budget = p.timeout_ns;
  // with a gate the producer may legitimately spend its whole budget before the first load: the roles behind it wait longer,
  // so that a gate that never opens is reported as such and not as a stalled pipeline
  const uint64_t cbudget = p.gate ? 2 * budget + 1000000ull : budget;
  // split-K: a work item is (tile, split); split s reduces k-blocks [s*KB_PER, min(KB, (s+1)*KB_PER))
  // and stores its partial product in slab s of the workspace (the host guarantees no split is empty).
  const int SPLITS = p.split_k > 1 ? p.split_k : 1;
  const int KB_PER = (KB + SPLITS - 1) / SPLITS;
  const int total_work = total_tiles * SPLITS;

  // The producer and the MMA issuer run their loops with the whole warp and elect a lane for each group of asynchronous
  // instructions: addresses, coordinates and descriptors are then the warp's (uniform registers), which is the form these
  // instructions take them in. Issued from a loop under `if (lane == 0)`, every operand of every instruction was moved over one
  // at a time, and a stage cost 0.41 us whatever its tile (with the loads or the MMAs taken out just as well). 512 x 8192 x 8192
  // bf16, plain result: 60.8 -> 53.8 us (1.28 PFLOP/s), with GELU 71.4 -> 62.0; 1024 x 4096 x 4096 tf32 60.1 -> 56.3.
  if (warp == 4) {
    // ---------------- TMA producer ----------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    if (p.gate) {
      // the operands are still being delivered (e.g. fresh weights arriving from their owners): wait, bounded, for every
      // selected flag, then order the TMA (async proxy) reads behind the acquire
      if (lane == 0) {
        const uint32_t want = *p.gate_target;
        for (int i = 0; i < 32 && ok; ++i)
          if (((p.gate_mask >> i) & 1u) && !wait_flag_ge(p.gate + (size_t)i * p.gate_stride, want, budget)) {
            fail(p, abortp, ONO_ERR_TIMEOUT_PEER_FLAG);
            ok = false;
          }
      }
      ok = __all_sync(0xffffffffu, ok);
      asm volatile("fence.proxy.async;" ::: "memory");
    }
    // pair: both CTAs' copies complete on the leader's barriers
    const uint32_t full_remote0 = PAIR ? mapa_shared(smem_u32(&full_bar[0]), 0u) : 0u;
    const int a_mn = p.a.mn_major, b_mn = p.b.mn_major;
    for (int work = unit; work < total_work && ok; work += units) {
      const int tile = work / SPLITS, split = work % SPLITS;
      const int m0 = (APPLY ? tile / num_n : tile % num_m) * TILE_M + (int)crank * BM;
      const int n0 = (APPLY ? tile % num_n : tile / num_m) * BN + (int)crank * (PAIR ? BN_CTA : 0);
      const int kb0 = split * KB_PER, kb1 = min(KB, kb0 + KB_PER);
      for (int kb = kb0; kb < kb1; ++kb) {
        const bool free = mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, abortp, budget);
        if (!__all_sync(0xffffffffu, free)) {
          fail(p, abortp, ONO_ERR_TIMEOUT_EMPTY);
          ok = false;
          break;
        }
        uint8_t* sa = smem + (size_t)stage * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        const int k0 = kb * BK;
        const uint32_t full_remote = full_remote0 + 8u * stage;
        if (elect_one()) {
          // the leader's barrier expects the bytes of both CTAs
          if (!PAIR) mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
          else if (leader) mbar_expect_tx(&full_bar[stage], 2u * STAGE_BYTES);
          for (int i = 0; i < p.a.n_box; ++i) {
            const int mn = m0 + i * p.a.box_mn;
            if (PAIR) tma_load_2d_pair(sa + i * p.a.box_stride_bytes, &tmA, full_remote, a_mn ? mn : k0, a_mn ? k0 : mn);
            else tma_load_2d(sa + i * p.a.box_stride_bytes, &tmA, &full_bar[stage], a_mn ? mn : k0, a_mn ? k0 : mn);
          }
          for (int i = 0; i < p.b.n_box; ++i) {
            const int mn = n0 + i * p.b.box_mn;
            if (PAIR) tma_load_2d_pair(sb + i * p.b.box_stride_bytes, &tmB, full_remote, b_mn ? mn : k0, b_mn ? k0 : mn);
            else tma_load_2d(sb + i * p.b.box_stride_bytes, &tmB, &full_bar[stage], b_mn ? mn : k0, b_mn ? k0 : mn);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
    if (!ok) {
      // Give copies already in flight time to land before the CTA retires its shared memory.
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
    }
  } else if (warp == 5) {
    if (leader) {
      // ---------------- MMA issuer (the pair's leader issues for both CTAs) ----------------
      int stage = 0;
      uint32_t phase = 0;
      int t = 0;
      bool ok = true;
      const uint32_t ring = smem_u32(smem);
      const uint64_t adesc0 = make_smem_desc_sw128(ring, p.a.lbo_bytes, p.a.sbo_bytes, p.a.layout_type);
      const uint64_t bdesc0 = make_smem_desc_sw128(ring + A_BYTES, p.b.lbo_bytes, p.b.sbo_bytes, p.b.layout_type);
      const uint32_t akstep = p.a.kstep_bytes >> 4, bkstep = p.b.kstep_bytes >> 4;   // descriptors address 16-byte units
      const uint32_t idesc = p.idesc;
      for (int work = unit; work < total_work && ok; work += units, ++t) {
        const int split = work % SPLITS;
        const int kb0 = split * KB_PER, kb1 = min(KB, kb0 + KB_PER);
        const int buf = t & 1;
        const uint32_t acc_phase = (t >> 1) & 1;
        const bool drained = mbar_wait_bounded(&tmem_empty_bar[buf], acc_phase ^ 1u, abortp, cbudget);
        if (!__all_sync(0xffffffffu, drained)) {
          fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_EMPTY);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          const bool landed = mbar_wait_bounded(&full_bar[stage], phase, abortp, cbudget);
          if (!__all_sync(0xffffffffu, landed)) {
            fail(p, abortp, ONO_ERR_TIMEOUT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t adesc = adesc0 + (uint32_t)stage * (STAGE_BYTES >> 4), bdesc = bdesc0 + (uint32_t)stage * (STAGE_BYTES >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < KSTEPS; ++k) {
              const uint32_t acc = (kb != kb0) || (k != 0);
              if (PAIR) {
                if (ESIZE == 4) umma_tf32_pair(d_tmem, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
                else umma_f16_pair(d_tmem, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
              } else {
                if (ESIZE == 4) umma_tf32(d_tmem, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
                else umma_f16(d_tmem, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
              }
            }
            // the stage is free (in both CTAs of a pair) once these MMAs have read it
            if (PAIR) umma_commit_pair_mc(&empty_bar[stage], 3);
            else umma_commit(&empty_bar[stage]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok && elect_one()) {
          if (PAIR) umma_commit_pair_mc(&tmem_full_bar[buf], 3);
          else umma_commit(&tmem_full_bar[buf]);
        }
        __syncwarp();
      }
      // Make sure no MMA is still running before TMEM is released.
      if (elect_one()) {
        if (PAIR) umma_commit_pair(&drain_bar);
        else umma_commit(&drain_bar);
      }
      __syncwarp();
      mbar_wait_bounded(&drain_bar, 0, abortp, ok ? cbudget : 1000000ull);
    }
  } else {
    // ---------------- epilogue warps 0..3 (TMEM lanes 32*warp .. 32*warp+31) ----------------
    int t = 0;
    bool ok = true;
    // Two groups of four warps (warps 0-3 and 6-9) take alternate 32-column chunks of the
    // accumulator. Every warp owns a 4 KB staging tile (its 32 rows x 32 columns) and its own TMA-store queue, so eight
    // stores are in flight per CTA and no warp waits for another.
    const int grp = warp >= 6 ? 1 : 0;
    const int quad = warp & 3;                 // TMEM lane quadrant this warp may read
    uint8_t* const wstage = cstage + (size_t)(grp * 4 + quad) * 4096u;
    const uint32_t tmem_empty_remote[2] = {PAIR ? mapa_shared(smem_u32(&tmem_empty_bar[0]), 0u) : 0u,
                                           PAIR ? mapa_shared(smem_u32(&tmem_empty_bar[1]), 0u) : 0u};
    if constexpr (APPLY) {
      // ---------------- optimizer in the epilogue, tiles moved by TMA ----------------
      // For every 32 x 32 chunk of dW the warp brings the matching tiles of the f32 master and of the optimizer state
      // into shared memory with TMA loads (issued one chunk ahead when two buffers fit, also across output tiles, since
      // they do not depend on the MMAs), updates them in place with the gradient values it reads from TMEM (a lane
      // holds one row in both), writes the bf16 shadow tile next to them and sends everything back with TMA stores.
      // Out-of-range rows and columns are zero-filled by the loads and clipped by the stores.
      const OnoApply& ap = p.apply;
      const int narr = 1 + (ap.kind >= 1 ? 1 : 0) + (ap.kind == 2 ? 1 : 0);
      const uint32_t slot_bytes = (uint32_t)narr * 4096u + 2048u;
      const int nbuf = APPLY_WARP_BYTES / slot_bytes >= 2 ? 2 : 1;
      const int ew = grp * 4 + quad;                                   // epilogue warp index 0..7
      uint8_t* const wbase = cstage + (size_t)ew * APPLY_WARP_BYTES;
      uint64_t* const bars = &apply_bar[ew * 2];
      OptScal os{ap.kind, ap.lr, ap.mu, ap.b1, ap.b2, ap.eps, ap.grad_scale, 0.0f};
      if (ap.kind == 2) os.adam_step = ap.lr * sqrtf(1.0f - __ldg(ap.adam_pows + 1)) / (1.0f - __ldg(ap.adam_pows));
      // chunk iterator over this warp's (work item, column chunk) sequence
      // (the two groups of four warps take alternate chunks of 32 columns, and the tiles are numbered along the rows of the
      // matrix, so that at any time the CTAs read and write long runs of a few rows. With tiles numbered down the columns and
      // each group on its own half of the columns 8192 x 8192 x 512 with momentum took 249 us (now 229: 5.3 TB/s of state),
      // with SGD 165 (152))
      constexpr int CPG = BN / 64;                 // chunks per group and tile
      auto first_chunk = [&](int& w, int& c) {
        c = grp;
        while (w < total_work && (w % num_n) * BN + c * 32 >= p.N) w += units;
      };
      auto next_chunk = [&](int& w, int& c) {
        c += 2;
        if (c >= 2 * CPG || (w % num_n) * BN + c * 32 >= p.N) { w += units; first_chunk(w, c); }
      };
      auto issue = [&](int w, int c, int b) {      // lane 0: loads of chunk (w, c) into buffer b
        const int y = (w / num_n) * TILE_M + (int)crank * BM + quad * 32;
        const int x = (w % num_n) * BN + c * 32;
        uint8_t* dst = wbase + (size_t)b * slot_bytes;
        mbar_expect_tx(&bars[b], (uint32_t)narr * 4096u);
        tma_load_2d(dst, &am.p, &bars[b], x, y);
        if (ap.kind >= 1) tma_load_2d(dst + 4096, &am.m, &bars[b], x, y);
        if (ap.kind == 2) tma_load_2d(dst + 8192, &am.v, &bars[b], x, y);
      };
      int pw = unit, pc = 0;                       // next chunk to prefetch
      first_chunk(pw, pc);
      long long issued = 0, done = 0;
      if (lane == 0)
        for (; issued < nbuf && pw < total_work; ++issued) { issue(pw, pc, (int)issued); next_chunk(pw, pc); }
      for (int work = unit; work < total_work && ok; work += units, ++t) {
        const int m0 = (work / num_n) * TILE_M + (int)crank * BM;
        const int n0 = (work % num_n) * BN;
        const int buf = t & 1;
        const uint32_t acc_phase = (t >> 1) & 1;
        const bool got = mbar_wait_bounded(&tmem_full_bar[buf], acc_phase, abortp, cbudget);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_FULL);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
#pragma unroll 1
        for (int c = grp; c < 2 * CPG; c += 2) {
          const int nc = n0 + c * 32;
          if (nc >= p.N) break;
          const int b = (int)(done % nbuf);
          const bool landed = mbar_wait_bounded(&bars[b], (uint32_t)((done / nbuf) & 1), abortp, cbudget);
          if (!__all_sync(0xffffffffu, landed)) {
            if (lane == 0) fail(p, abortp, ONO_ERR_TIMEOUT_FULL);
            ok = false;
            break;
          }
          uint32_t r[32];
          tmem_ld_x32(t_row + (uint32_t)(c * 32), r);
          tmem_ld_wait();
          uint8_t* const tp = wbase + (size_t)b * slot_bytes + lane * 128;      // this lane's row of the master tile
          uint8_t* const ts = wbase + (size_t)b * slot_bytes + (size_t)narr * 4096u + lane * 64;   // and of the shadow tile
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) {
            float4 out[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int j = 2 * jj + h;
              const uint32_t o = (uint32_t)((j ^ (lane & 7)) << 4);
              const float4 g = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                           __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
              float4 P = *reinterpret_cast<const float4*>(tp + o);
              float4 Mo = make_float4(0.f, 0.f, 0.f, 0.f), Vo = Mo;
              if (ap.kind >= 1) Mo = *reinterpret_cast<const float4*>(tp + 4096 + o);
              if (ap.kind == 2) Vo = *reinterpret_cast<const float4*>(tp + 8192 + o);
              P = opt_apply4(os, P, g, Mo, Vo);
              *reinterpret_cast<float4*>(tp + o) = P;
              if (ap.kind >= 1) *reinterpret_cast<float4*>(tp + 4096 + o) = Mo;
              if (ap.kind == 2) *reinterpret_cast<float4*>(tp + 8192 + o) = Vo;
              out[h] = P;
            }
            if (ap.p_bf16) {
              const uint2 lo = pack_bf16x4(out[0]), hi = pack_bf16x4(out[1]);
              *reinterpret_cast<uint4*>(ts + ((jj ^ ((lane >> 1) & 3)) << 4)) = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int y = m0 + quad * 32;
            uint8_t* src = wbase + (size_t)b * slot_bytes;
            tma_store_2d(&am.p, src, nc, y);
            if (ap.kind >= 1) tma_store_2d(&am.m, src + 4096, nc, y);
            if (ap.kind == 2) tma_store_2d(&am.v, src + 8192, nc, y);
            if (ap.p_bf16) tma_store_2d(&am.s, src + (size_t)narr * 4096u, nc, y);
            tma_store_commit();
            if (pw < total_work) {                  // refill this buffer once its stores have read it
              tma_store_wait_read<0>();
              issue(pw, pc, b);
              next_chunk(pw, pc);
              ++issued;
            }
          }
          __syncwarp();
          ++done;
        }
        tc_fence_before();
        if (PAIR) mbar_arrive_cluster(tmem_empty_remote[buf]);
        else mbar_arrive(&tmem_empty_bar[buf]);
      }
      if (lane == 0) {
        tma_store_wait_all<0>();
        if (!ok) {      // loads already issued into this warp's buffers must land before the CTA retires its shared memory
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
        }
      }
    } else {
    // The stored activations (aux) of this lane's eight row segments of a chunk do not depend on the product: they are loaded one
    // chunk ahead, the first chunk's while the MMAs of its tile still run, and unpacked in the chunk that uses them: 512 x 8192 x 8192
    // bf16 with GELU's derivative 78.3 us with the unpacking (and so the wait) where they are loaded, 66.4 so.
    uint4 aux_now[8];
    auto load_aux = [&](int w, int c) {
      const int n = ((w / SPLITS) / num_m) * BN + c * 32 + 4 * (lane & 7), left = p.N - n;
      const int mb = ((w / SPLITS) % num_m) * TILE_M + (int)crank * BM + quad * 32 + (lane >> 3);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        aux_now[i] = make_uint4(0u, 0u, 0u, 0u);
        if (left > 0 && mb + 4 * i < p.M) aux_now[i] = load_aux4_raw(p.epi, mb + 4 * i, n, left, p.vec);
      }
    };
    const bool with_aux = p.staged && p.epi.dact != ACT_NONE;
    if (with_aux && unit < total_work) load_aux(unit, grp);
    for (int work = unit; work < total_work && ok; work += units, ++t) {
      const int tile = work / SPLITS;
      const int m0 = (tile % num_m) * TILE_M + (int)crank * BM;
      const int n0 = (tile / num_m) * BN;
      const int buf = t & 1;
      const uint32_t acc_phase = (t >> 1) & 1;
      const bool got = mbar_wait_bounded(&tmem_full_bar[buf], acc_phase, abortp, cbudget);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_FULL);
        ok = false;
        break;
      }
      tc_fence_after();
      const int row = quad * 32 + lane;
      const int m = m0 + row;
      const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
#pragma unroll 1
      for (int c = grp; c < BN / 32; c += 2) {
        const int nc = n0 + c * 32;
        if (nc >= p.N) break;  // uniform across the CTA
        uint32_t r[32];
        tmem_ld_x32(t_row + (uint32_t)(c * 32), r);
        float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.staged) bias4 = load_bias4(p.epi, nc + 4 * (lane & 7), p.N - nc - 4 * (lane & 7));
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        if (SPLITS > 1) {
          // partial product of one K range: plain stores into this split's own slab; the finishing pass adds the
          // slabs in split order, so the sum does not depend on which CTA finished first
          if (m < p.M) {
            float* o = p.slabs + (size_t)(work % SPLITS) * p.slab_elems + (size_t)m * p.slab_ld + nc;
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              if (nc + j < p.slab_ld) *reinterpret_cast<float4*>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          }
          continue;
        }
        if (p.apply.p) {
          // Optimizer in the epilogue. The warp stages its 32 x 32 tile of dW, then walks the tile so that eight
          // lanes cover one 128-byte row segment: every access to the master, the state and the shadow is a full line.
          __syncwarp();                       // the previous chunk's reads of the staging tile are done
          {
            uint8_t* rp = wstage + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(rp + ((j ^ (lane & 7)) << 4)) =
                  make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
          __syncwarp();
          const OnoApply& ap = p.apply;
          OptScal os{ap.kind, ap.lr, ap.mu, ap.b1, ap.b2, ap.eps, ap.grad_scale, 0.0f};
          if (ap.kind == 2) os.adam_step = ap.lr * sqrtf(1.0f - __ldg(ap.adam_pows + 1)) / (1.0f - __ldg(ap.adam_pows));
          const int c4 = lane & 7, rsub = lane >> 3;
          const int col = nc + c4 * 4;
          const int mbase = m0 + quad * 32 + rsub;
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            float4 P[4], Mo[4], Vo[4];
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int mr = mbase + h * 16 + it * 4;
              P[it] = Mo[it] = Vo[it] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (col < p.N && mr < p.M) {
                const size_t off = (size_t)mr * ap.ld + col;
                P[it] = __ldcs(reinterpret_cast<const float4*>(ap.p + off));
                if (ap.kind >= 1) Mo[it] = __ldcs(reinterpret_cast<const float4*>(ap.m + off));
                if (ap.kind == 2) Vo[it] = __ldcs(reinterpret_cast<const float4*>(ap.v + off));
              }
            }
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int r = h * 16 + it * 4 + rsub;
              const int mr = mbase + h * 16 + it * 4;
              if (col < p.N && mr < p.M) {
                const size_t off = (size_t)mr * ap.ld + col;
                const float4 g = *reinterpret_cast<const float4*>(wstage + r * 128 + ((c4 ^ (r & 7)) << 4));
                const float4 pp = opt_apply4(os, P[it], g, Mo[it], Vo[it]);
                __stcs(reinterpret_cast<float4*>(ap.p + off), pp);
                if (ap.kind >= 1) __stcs(reinterpret_cast<float4*>(ap.m + off), Mo[it]);
                if (ap.kind == 2) __stcs(reinterpret_cast<float4*>(ap.v + off), Vo[it]);
                if (ap.p_bf16) *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ap.p_bf16) + off) = pack_bf16x4(pp);
              }
            }
          }
          continue;
        }
        if (p.tma_out) {
          // plain result (the host allows nothing but alpha here): registers -> swizzled staging tile -> one TMA store per
          // warp and 32 x 32 chunk; the TMA unit clips rows >= M and columns >= N
          if (p.epi.alpha != 1.0f) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= p.epi.alpha;
          }
          if (lane == 0) tma_store_wait_read<0>();  // this warp's previous store has read the tile
          __syncwarp();
          if (p.tma_out != 2) {
            uint8_t* rp = wstage + lane * 128;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(rp + ((j ^ (row & 7)) << 4)) =
                  make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          } else {
            uint8_t* rp = wstage + lane * 64;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 pk;
              pk.x = pack16x2(v[8 * j], v[8 * j + 1], p.epi.out16_f16);
              pk.y = pack16x2(v[8 * j + 2], v[8 * j + 3], p.epi.out16_f16);
              pk.z = pack16x2(v[8 * j + 4], v[8 * j + 5], p.epi.out16_f16);
              pk.w = pack16x2(v[8 * j + 6], v[8 * j + 7], p.epi.out16_f16);
              *reinterpret_cast<uint4*>(rp + ((j ^ ((row >> 1) & 3)) << 4)) = pk;
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (p.tma_out == 3) tma_reduce_add_2d(&tmC, wstage, nc, m0 + quad * 32);
            else tma_store_2d(&tmC, wstage, nc, m0 + quad * 32);
            tma_store_commit();
          }
          continue;
        }
        // Any other epilogue: the chunk goes through the warp's staging tile so that eight lanes cover one row's 32 columns.
        // Operand loads (aux) and stores are then whole 64- or 128-byte row segments, four rows an instruction; with a row
        // per lane they were 32 separate 16-byte pieces. The tile's swizzle, unit ^ (row ^ row >> 2), is free of bank
        // conflicts for the writes (a row per lane), the row reads and the transposed reads alike.
        const OnoEpilogue& e = p.epi;
        const int c4 = lane & 7, rsub = lane >> 3, n = nc + 4 * c4, left = p.N - n;
        const int mb = m0 + quad * 32 + rsub;
        __syncwarp();                                   // the previous chunk's reads of the staging tile are done
        {
          uint8_t* rp = wstage + lane * 128;
          const int sw = (lane ^ (lane >> 2)) & 7;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(rp + ((j ^ sw) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        __syncwarp();
        const bool keep = e.outT_f32 || e.outT_bf16;
        float4 aux_h[4], aux_l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { aux_h[i] = aux4(e, aux_now[i]); aux_l[i] = aux4(e, aux_now[i + 4]); }
        if (with_aux) {
          if (c + 2 < BN / 32 && nc + 64 < p.N) load_aux(work, c + 2);
          else if (work + units < total_work) load_aux(work + units, grp);
        }
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          float4 q[4];
          int mr[4];
          uint8_t* at[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = h * 16 + 4 * i + rsub;
            mr[i] = mb + h * 16 + 4 * i;
            at[i] = wstage + r * 128 + ((c4 ^ ((r ^ (r >> 2)) & 7)) << 4);
            q[i] = *reinterpret_cast<const float4*>(at[i]);
          }
          if (left > 0) epilogue_rows<4>(e, q, mr, n, left, p.vec, p.M, bias4, aux_h);
          if (keep) {
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(at[i]) = q[i];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) aux_h[i] = aux_l[i];
        }
        if (keep) {
          // transposed copy: a lane takes four rows of one column, eight lanes one 128-byte run of the copy
          __syncwarp();
          const int mt = m0 + quad * 32 + 4 * c4;
#pragma unroll 2
          for (int it = 0; it < 8; ++it) {
            const int c = 4 * it + rsub;
            float4 q;
            float* qf = reinterpret_cast<float*>(&q);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int r = 4 * c4 + k;
              qf[k] = *reinterpret_cast<const float*>(wstage + r * 128 + ((it ^ ((r ^ (r >> 2)) & 7)) << 4) + 4 * rsub);
            }
            if (nc + c < p.N && mt < p.M) {
              const size_t off = (size_t)(nc + c) * e.ld_outT + mt;
              if (e.outT_f32) store_f32x4(e.outT_f32 + off, q, p.M - mt, p.vec_t);
              if (e.outT_bf16) store_b16x4(e.outT_bf16, off, q, p.M - mt, p.vec_t, 0);
            }
          }
        }
      }
      tc_fence_before();
      if (PAIR) mbar_arrive_cluster(tmem_empty_remote[buf]);
      else mbar_arrive(&tmem_empty_bar[buf]);
    }
    }
    if (!APPLY && p.tma_out && lane == 0) tma_store_wait_all<0>();  // global writes done before exit
  }

  tc_fence_before();
  __syncthreads();
  // pair: neither CTA retires its shared memory, barriers or TMEM while the other may still touch them
  if (PAIR) cluster_sync_all();
  if (warp == 5) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------
// Small problems: one 128 x BN tile per cluster, K split over the cluster's CTAs
// ------------------------------------------------------------------------------------------------
// A problem with few output tiles is bound by latency: one CTA walks the whole reduction at the rate one SM can draw from
// L2, and its eight epilogue warps then walk 128 x 128 values, both while most of the chip idles. Here a cluster of S CTAs
// splits K; CTA s multiplies its share into its own TMEM and hands every 32 x 32 block of the partial tile to the CTA that
// owns the block, in that CTA's shared memory (st.shared::cluster). The owner adds the S partial blocks in split order, so
// the result is the same to the bit from run to run, and runs the epilogue on its 1/S of the tile: reduction and epilogue
// are both S times shorter, with no slabs in memory and no finishing pass. Operands of the epilogue (bias, aux) are loaded
// while the MMAs run. See pick_cluster() for the choice of BN and S.
template <int BN>
struct ClusterCfg {
  static constexpr int STAGES = BN == 128 ? 5 : (BN == 64 ? 6 : 8);
  static constexpr uint32_t RECV_BYTES = BN * 128 * 4;      // S partial blocks of each of the (4 * BN / 32) / S owned blocks
};

template <int ESIZE, int BN>
__global__ void __launch_bounds__(320, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmDev p) {
  constexpr int BM = 128, BK = 128 / ESIZE, UMMA_K = 32 / ESIZE, KSTEPS = BK / UMMA_K;
  constexpr uint32_t A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int STAGES = ClusterCfg<BN>::STAGES;
  constexpr uint32_t TMEM_COLS = BN;
  constexpr int UNITS = 4 * (BN / 32);                      // 32 x 32 blocks of the tile: unit u = 4 * (column chunk) + row quadrant
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* recv = smem + (size_t)STAGES * STAGE_BYTES;      // [source CTA][owned unit][32 rows][128 bytes, swizzled]
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_bar;
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  volatile int* abortp = &abort_flag;
  const int S = p.split_k;                                  // cluster size, a power of two <= UNITS
  const int rank = (int)cluster_ctarank();
  const int upc = UNITS / S;                                // units owned by a CTA

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&acc_bar, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4 && lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); }
  if (warp == 5) { tmem_alloc(&tmem_base_smem, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_arrive();                                         // "this CTA runs": nobody writes to its shared memory before
  const uint32_t tmem_base = tmem_base_smem;
  const int tile = (int)blockIdx.x / S;
  const int num_m = (p.M + BM - 1) / BM;
  const int m0 = (tile % num_m) * BM, n0 = (tile / num_m) * BN;
  const int KB = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)KB * rank / S), kb1 = (int)((long long)KB * (rank + 1) / S);   // S <= KB: never empty
  const uint64_t budget = p.timeout_ns;
  const OnoEpilogue& e = p.epi;

  // this warp's share of the epilogue: rows [4 * rg, 4 * rg + 4 * upc) of the owned units, numbered unit after unit
  const int grp = warp >= 6 ? 1 : 0, quad = warp & 3, ew = grp * 4 + quad;
  const int c4 = lane & 7, rsub = lane >> 3;

  if (warp == 4) {               // TMA producer (see gemm_tcgen05_kernel for the form of the two loops)
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const int a_mn = p.a.mn_major, b_mn = p.b.mn_major;
    for (int kb = kb0; kb < kb1; ++kb) {
      const bool free = mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, abortp, budget);
      if (!__all_sync(0xffffffffu, free)) { fail(p, abortp, ONO_ERR_TIMEOUT_EMPTY); ok = false; break; }
      uint8_t* sa = smem + (size_t)stage * STAGE_BYTES;
      uint8_t* sb = sa + A_BYTES;
      const int k0 = kb * BK;
      if (elect_one()) {
        mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
        for (int i = 0; i < p.a.n_box; ++i) {
          const int mn = m0 + i * p.a.box_mn;
          tma_load_2d(sa + i * p.a.box_stride_bytes, &tmA, &full_bar[stage], a_mn ? mn : k0, a_mn ? k0 : mn);
        }
        for (int i = 0; i < p.b.n_box; ++i) {
          const int mn = n0 + i * p.b.box_mn;
          tma_load_2d(sb + i * p.b.box_stride_bytes, &tmB, &full_bar[stage], b_mn ? mn : k0, b_mn ? k0 : mn);
        }
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    if (!ok) {      // copies already in flight land before the CTA retires its shared memory
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) { __nanosleep(1000); }
    }
  } else if (warp == 5) {        // MMA issuer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t ring = smem_u32(smem);
    const uint64_t adesc0 = make_smem_desc_sw128(ring, p.a.lbo_bytes, p.a.sbo_bytes, p.a.layout_type);
    const uint64_t bdesc0 = make_smem_desc_sw128(ring + A_BYTES, p.b.lbo_bytes, p.b.sbo_bytes, p.b.layout_type);
    const uint32_t akstep = p.a.kstep_bytes >> 4, bkstep = p.b.kstep_bytes >> 4, idesc = p.idesc;
    for (int kb = kb0; kb < kb1; ++kb) {
      const bool landed = mbar_wait_bounded(&full_bar[stage], phase, abortp, budget);
      if (!__all_sync(0xffffffffu, landed)) { fail(p, abortp, ONO_ERR_TIMEOUT_FULL); ok = false; break; }
      tc_fence_after();
      const uint64_t adesc = adesc0 + (uint32_t)stage * (STAGE_BYTES >> 4), bdesc = bdesc0 + (uint32_t)stage * (STAGE_BYTES >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < KSTEPS; ++k) {
          const uint32_t acc = (kb != kb0) || (k != 0);
          if (ESIZE == 4) umma_tf32(tmem_base, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
          else umma_f16(tmem_base, adesc + k * akstep, bdesc + k * bkstep, idesc, acc);
        }
        umma_commit(&empty_bar[stage]);
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    if (elect_one()) umma_commit(&acc_bar);       // also after a failure: no MMA may still run when TMEM is released
    __syncwarp();
    mbar_wait_bounded(&acc_bar, 0, abortp, ok ? budget : 1000000ull);
  }
  __syncwarp();

  // Bias and aux of the first batch of rows: in flight while the MMAs run.
  const int G = upc < 4 ? upc : 4;
  const int flat0 = ew * upc;                                // first row group (of four rows) of this warp
  float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f), aux[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) aux[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  auto unit_of = [&](int flat) { return rank * upc + (flat >> 3); };
  auto load_operands = [&](int flat) {
    const int u = unit_of(flat), n = n0 + (u >> 2) * 32 + 4 * c4, left = p.N - n;
    const int mb = m0 + (u & 3) * 32 + 4 * (flat & 7) + rsub;
    bias4 = load_bias4(e, n, left);
    if (e.dact != ACT_NONE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) if (i < G && left > 0 && mb + 4 * i < p.M) aux[i] = load_aux4(e, mb + 4 * i, n, left, p.vec);
    }
  };
  const bool epi_warp = warp < 4 || warp >= 6;
  if (epi_warp) {
    load_operands(flat0);
    const bool got = mbar_wait_bounded(&acc_bar, 0, abortp, budget);
    if (!__all_sync(0xffffffffu, got) && lane == 0) fail(p, abortp, ONO_ERR_TIMEOUT_TMEM_FULL);
  }
  tc_fence_after();
  cluster_wait();                                            // every CTA of the cluster runs
  if (epi_warp) {
    const int sw = (lane ^ (lane >> 2)) & 7;
#pragma unroll 1
    for (int c = grp; c < BN / 32; c += 2) {
      if (n0 + c * 32 >= p.N || m0 + quad * 32 >= p.M) continue;        // nothing of this block is inside the matrix
      uint32_t r[32];
      tmem_ld_x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * 32), r);
      tmem_ld_wait();
      const int u = 4 * c + quad, owner = u / upc;
      const uint32_t dst = mapa_shared(smem_u32(recv + ((size_t)rank * upc + (u - owner * upc)) * 4096u + lane * 128), (uint32_t)owner);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        st_cluster_v4(dst + ((j ^ sw) << 4), make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                         __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
    }
    tc_fence_before();
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();                                            // all partial blocks have arrived; nothing remote is touched after this
  if (warp == 5) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
  if (!epi_warp) return;
  const bool keep = e.outT_f32 || e.outT_bf16;
#pragma unroll 1
  for (int b = 0; b < upc; b += G) {
    const int flat = flat0 + b, u = unit_of(flat);
    if (b) load_operands(flat);
    const int nc = n0 + (u >> 2) * 32, mq = m0 + (u & 3) * 32;
    if (nc >= p.N || mq >= p.M) continue;
    const int n = nc + 4 * c4, left = p.N - n;
    uint8_t* const blk = recv + (size_t)(u - rank * upc) * 4096u;
    float4 q[4];
    int mr[4];
    uint8_t* at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = (4 * (flat & 7) + 4 * i + rsub) & 31;
      mr[i] = i < G ? mq + r : p.M;                          // rows past the batch are computed and not stored
      at[i] = blk + r * 128 + ((c4 ^ ((r ^ (r >> 2)) & 7)) << 4);
      q[i] = *reinterpret_cast<const float4*>(at[i]);
    }
#pragma unroll 1
    for (int s = 1; s < S; ++s) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 t = *reinterpret_cast<const float4*>(at[i] + (size_t)s * upc * 4096u);
        q[i].x += t.x; q[i].y += t.y; q[i].z += t.z; q[i].w += t.w;
      }
    }
    if (left > 0) epilogue_rows<4>(e, q, mr, n, left, p.vec, p.M, bias4, aux);
    if (keep) {
#pragma unroll
      for (int i = 0; i < 4; ++i) if (i < G) *reinterpret_cast<float4*>(at[i]) = q[i];
    }
  }
  if (!keep) return;
  asm volatile("bar.sync 1, 256;" ::: "memory");             // the eight epilogue warps: a unit's rows come from several of them
#pragma unroll 1
  for (int b = 0; b < upc; ++b) {
    // transposed copy: a lane takes four rows of one column, eight lanes one run of 32 rows
    const int flat = flat0 + b, u = unit_of(flat), it = flat & 7;
    const int nc = n0 + (u >> 2) * 32, mt = m0 + (u & 3) * 32 + 4 * c4, c = 4 * it + rsub;
    const uint8_t* const blk = recv + (size_t)(u - rank * upc) * 4096u;
    if (nc + c < p.N && mt < p.M) {
      float4 q;
      float* qf = reinterpret_cast<float*>(&q);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = 4 * c4 + k;
        qf[k] = *reinterpret_cast<const float*>(blk + r * 128 + ((it ^ ((r ^ (r >> 2)) & 7)) << 4) + 4 * rsub);
      }
      const size_t off = (size_t)(nc + c) * e.ld_outT + mt;
      if (e.outT_f32) store_f32x4(e.outT_f32 + off, q, p.M - mt, p.vec_t);
      if (e.outT_bf16) store_b16x4(e.outT_bf16, off, q, p.M - mt, p.vec_t, 0);
    }
  }
}

// Two-pass form (split-K). Used for problems with a handful of output tiles and a long reduction (e.g. 342 x 128 x 3136:
// three tiles, i.e. three SMs streaming 98 k-blocks each) and whenever the caller asks for a split: the reduction is
// split over the SMs, split s stores its partial product into slab s of a workspace, and this pass adds the slabs in
// split order and runs the regular epilogue (bias, activation, derivative, every output form) on the sums. The result
// is the same to the bit from run to run. The workspace comes from the caller (OnoGemm::workspace, e.g. one per
// stream); without one a static buffer is used, and such GEMMs must then not overlap on the device.
constexpr long long SPLIT_SCRATCH_ELEMS = 4ll << 20;
__device__ float g_split_scratch[SPLIT_SCRATCH_ELEMS];

// A block owns 32 groups of four columns (consecutive in row-major order), eight warps: warp w adds the slabs w, w + 8,
// w + 16, ... of its lane's group with four 16-byte loads in flight, the eight partial sums are then added in warp order
// through shared memory, and warp 0 runs the epilogue. The order of every addition is fixed, so the result does not depend on
// timing. What bounds it is the latency of a warp's slab loads. (One block per 32 x 32 tile with a row per lane read
// 32 separate rows per load: 342 x 128 out of 49 slabs took 16.4 us.) 32 registers, of which the epilogue spills two words: two warps then fit
// a quarter of an SM's register file beside a convolution's input gradient, and the chain behind it does not wait for that one's end. With the 38 it
// would take, and so: convolutional step of 342 images 260 -> 254 us, of 2048 in bf16 624 -> 630; product and pass, 342 x 128 x 3136 in 49
// splits 10.7 either way, 1024 x 256 x 4096 in 8 17.4 -> 16.7 (tf32) and 14.5 -> 13.9 (bf16), 2048 x 512 x 4096 in 4 42.1 -> 39.5 and 31.5 ->
// 29.4, none of 56 forms more than 1.4 % longer.
__global__ void __maxnreg__(32) gemm_finish_kernel(const float* slabs, long long slab_elems, int nslabs, int ld, int M,
                                                          int N, int vec, const OnoEpilogue e) {
  __shared__ float4 part[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ng = (N + 3) >> 2;
  const int g = blockIdx.x * 32 + lane;
  const int m = g / ng, n = (g - m * ng) * 4;
  const bool in = m < M;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in) {
    const float* src = slabs + (size_t)m * ld + n;
    int sidx = warp;
    for (; sidx + 24 < nslabs; sidx += 32) {
      float4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = __ldcs(reinterpret_cast<const float4*>(src + (size_t)(sidx + 8 * u) * slab_elems));
#pragma unroll
      for (int u = 0; u < 4; ++u) { v.x += q[u].x; v.y += q[u].y; v.z += q[u].z; v.w += q[u].w; }
    }
    for (; sidx < nslabs; sidx += 8) {
      const float4 q = __ldcs(reinterpret_cast<const float4*>(src + (size_t)sidx * slab_elems));
      v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
    }
  }
  part[warp][lane] = v;
  __syncthreads();
  if (warp != 0 || !in) return;
#pragma unroll
  for (int w = 1; w < 8; ++w) {
    const float4 q = part[w][lane];
    v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
  }
  const int left = N - n;
  float4 vv[1] = {v}, aux[1] = {make_float4(0.f, 0.f, 0.f, 0.f)};
  const int mm[1] = {m};
  if (e.dact != ACT_NONE) aux[0] = load_aux4(e, m, n, left, vec);
  epilogue_rows<1>(e, vv, mm, n, left, vec, M, load_bias4(e, n, left), aux);
  const float* f = reinterpret_cast<const float*>(vv);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < left) {
      const size_t off = (size_t)(n + j) * e.ld_outT + m;
      if (e.outT_f32) e.outT_f32[off] = f[j];
      if (e.outT_bf16) reinterpret_cast<__nv_bfloat16*>(e.outT_bf16)[off] = __float2bfloat16_rn(f[j]);
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
static thread_local char g_err[512] = "";
void set_error(const char* fmt, const char* a = "", long long b = 0, long long c = 0) {
  snprintf(g_err, sizeof(g_err), fmt, a, b, c);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  });
  return fn;
}

// 2-D row-major global matrix [rows, cols] with leading dimension ld (elements); box = {box_cols
// (innermost, 128 bytes), box_rows}; 128-byte swizzle.
int encode_map_2d(CUtensorMap* map, const void* base, int esize, long long rows, long long cols,
                  long long ld, int box_cols, int box_rows, bool swizzle_32b_units = false) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) { set_error("cuTensorMapEncodeTiled unavailable%s", ""); return -2; }
  if (((uintptr_t)base & 15) != 0) { set_error("TMA base not 16-byte aligned%s", ""); return -3; }
  if ((ld * esize) % 16 != 0) { set_error("TMA row stride %s%lld bytes not a multiple of 16", "", ld * esize); return -3; }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * esize)};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUresult r = fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle_32b_units ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%s%lld)", "", (long long)r); return -4; }
  return 0;
}

// The same for a box of `box_rows` x `box_z` rows of a matrix whose rows are numbered (z, row): [nz][rows][cols], rows ld apart.
int encode_map_3d(CUtensorMap* map, const void* base, int esize, long long nz, long long rows, long long cols, long long ld, int box_cols,
                  int box_rows, int box_z) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) { set_error("cuTensorMapEncodeTiled unavailable%s", ""); return -2; }
  if (((uintptr_t)base & 15) != 0 || (ld * esize) % 16 != 0) { set_error("TMA base or rows not 16-byte aligned%s", ""); return -3; }
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)nz};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * esize), (cuuint64_t)(ld * esize * rows)};
  cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, (cuuint32_t)box_z};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (3d) failed (%s%lld)", "", (long long)r); return -4; }
  return 0;
}

// Output tile map for the TMA-store epilogue: box = {32 columns, 32 rows}; the 128-byte (f32) or
// 64-byte (bf16) rows use the matching swizzle so that the staging writes are bank-conflict free.
int encode_out_map(CUtensorMap* map, const void* base, int esize, long long rows, long long cols, long long ld) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) { set_error("cuTensorMapEncodeTiled unavailable%s", ""); return -2; }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * esize)};
  cuuint32_t box[2] = {32u, 32u};   // one epilogue warp's rows
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, esize == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  esize == 4 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (output) failed (%s%lld)", "", (long long)r); return -4; }
  return 0;
}

// Fills the device-side operand description and encodes the operand's tensor map.
static int make_operand(OperandDev* od, CUtensorMap* map, const void* ptr, int esize, int major,
                        int MN, int K, int ld, int tile_mn) {
  const int BK = 128 / esize;
  if (major == ONO_K_MAJOR) {
    od->mn_major = 0;
    od->n_box = 1;
    od->box_mn = tile_mn;
    od->box_stride_bytes = 0;
    od->lbo_bytes = 16;      // unused for a single swizzle atom along K
    od->sbo_bytes = 1024;    // 8 rows x 128 bytes
    od->kstep_bytes = 32;    // one UMMA_K slice inside the 128-byte row
    od->layout_type = 2;
    return encode_map_2d(map, ptr, esize, MN, K, ld, BK, tile_mn);
  }
  if (esize == 4) {
    // 32-bit MN-major operands: rows of 32 elements (128 bytes) of MN, swizzled on 32-byte units in atoms of 4 K-rows
    // (the layout tcgen05 defines for tf32 operands whose MN dimension is contiguous); one MMA (UMMA_K = 8) reads two atoms.
    const int chunk4 = 32;
    od->mn_major = 1;
    od->n_box = tile_mn / chunk4;
    if (od->n_box < 1) { set_error("MN-major tile too narrow%s", ""); return -5; }
    od->box_mn = chunk4;
    od->box_stride_bytes = (uint32_t)BK * 128u;
    od->lbo_bytes = od->box_stride_bytes;   // between 32-wide MN atoms
    od->sbo_bytes = 512;                    // between groups of 4 K-rows
    od->kstep_bytes = 8u * 128u;            // UMMA_K rows of K
    od->layout_type = 1;
    return encode_map_2d(map, ptr, esize, K, MN, ld, chunk4, BK, true);
  }
  const int chunk = 128 / esize;  // 64 elements of MN per 128-byte row
  od->mn_major = 1;
  od->n_box = tile_mn / chunk;
  if (od->n_box < 1) { set_error("MN-major tile too narrow%s", ""); return -5; }
  od->box_mn = chunk;
  od->box_stride_bytes = (uint32_t)BK * 128u;  // BK rows of K, 128 bytes each
  od->lbo_bytes = od->box_stride_bytes;        // between 64-wide MN atoms
  od->sbo_bytes = 1024;                        // between groups of 8 K-rows
  od->kstep_bytes = (32 / esize) * 128u;       // UMMA_K rows of K
  od->layout_type = 2;
  return encode_map_2d(map, ptr, esize, K, MN, ld, chunk, BK);
}

// cudaFuncSetAttribute, symbol addresses and SM counts belong to a device: caches are kept per device.
constexpr int kMaxDevices = 64;
static int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  return dev;
}
static int num_sms() {
  static int sms[kMaxDevices] = {0};
  const int dev = current_device();
  if (sms[dev] == 0) {
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    if (sms[dev] <= 0) sms[dev] = 148;
  }
  return sms[dev];
}

static ApplyMaps g_no_apply_maps;   // zero-filled: instantiations without the TMA optimizer epilogue never touch it

template <int ESIZE, int BN, bool PAIR, bool APPLY = false>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmDev& p, int max_ctas,
                  cudaStream_t stream, const ApplyMaps& am = g_no_apply_maps) {
  constexpr int BN_CTA = PAIR ? BN / 2 : BN;
  constexpr int STAGES = APPLY ? 2 : TileCfg<BN_CTA>::STAGES;
  constexpr size_t smem = (size_t)STAGES * (128 * 128 + BN_CTA * 128) + (APPLY ? 8 * APPLY_WARP_BYTES : 2 * 16384) + 1024;
  static bool attr_done[kMaxDevices] = {false};
  static int max_pairs_dev[kMaxDevices] = {0};
  const int dev = current_device();
  bool& attr_set = attr_done[dev];
  int& max_pairs = max_pairs_dev[dev];
  auto kern = gemm_tcgen05_kernel<ESIZE, BN, PAIR, APPLY>;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return -6; }
    if (PAIR) {
      // how many 2-CTA clusters the device can hold at once (an SM count that is odd inside a GPC loses one)
      cudaLaunchConfig_t q = {};
      q.gridDim = dim3(2 * num_sms());
      q.blockDim = dim3(320);
      q.dynamicSmemBytes = smem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
      q.attrs = at;
      q.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &q) != cudaSuccess || n <= 0) { cudaGetLastError(); n = num_sms() / 2; }
      max_pairs = n;
    }
    attr_set = true;
  }
  const int tile_m = PAIR ? 256 : 128;
  const int tiles = ((p.M + tile_m - 1) / tile_m) * ((p.N + BN - 1) / BN) * (p.split_k > 1 ? p.split_k : 1);
  if (!PAIR) {
    int grid = max_ctas > 0 ? max_ctas : num_sms();
    if (grid > tiles) grid = tiles;
    kern<<<grid, 320, smem, stream>>>(ta, tb, tc, am, p);
  } else {
    int pairs = max_ctas > 0 ? std::max(1, max_ctas / 2) : max_pairs;
    if (pairs > max_pairs) pairs = max_pairs;
    if (pairs > tiles) pairs = tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t le = cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, am, p);
    if (le != cudaSuccess) { set_error("gemm pair launch: %s", cudaGetErrorString(le)); return -7; }
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("gemm launch: %s", cudaGetErrorString(e)); return -7; }
  return 0;
}

template <int ESIZE, int BN>
static int launch_cluster(const CUtensorMap& ta, const CUtensorMap& tb, const GemmDev& p, cudaStream_t stream) {
  constexpr size_t smem = (size_t)ClusterCfg<BN>::STAGES * (128 * 128 + BN * 128) + ClusterCfg<BN>::RECV_BYTES + 1024;
  static bool attr_done[kMaxDevices] = {false};
  auto kern = gemm_cluster_kernel<ESIZE, BN>;
  bool& attr_set = attr_done[current_device()];
  if (!attr_set) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return -6; }
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((p.M + 127) / 128) * ((p.N + BN - 1) / BN) * p.split_k);
  cfg.blockDim = dim3(320);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.split_k; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tb, p);
  if (e != cudaSuccess) { set_error("gemm cluster launch: %s", cudaGetErrorString(e)); return -7; }
  return 0;
}

// Tile width and cluster size of gemm_cluster_kernel for a problem, or {0, 0} when the persistent kernel is the better one. Returns
// whether that is because the two-pass form takes the problem (a preference for CTA pairs yields to it then).
// The cost of a form is a straight line in the k-blocks of one CTA, fitted to a sweep of 32 shapes on a B200 (us; every form,
// M 32 .. 2048, N 10 .. 8192, K 10 .. 8192, both types, run back to back): 0.33 per k-block whatever the tile, and a constant
// that grows with the share of the epilogue that one CTA is left with. All CTAs have to be resident at once: 148 SMs hold 37
// clusters of four but only 12 of eight (16 of them took twice as long: 23.5 against 10.9 us for 256 x 1024 x 1024 tf32).
// A 128-column tile without a split is left out: there the persistent kernel draws level (512 x 4096 x 2048: 23.8 to 24.4 us,
// 1024 x 2048 x 256, plain output: 9.4 to 7.5 us). Examples, persistent -> cluster: 32 x 128 x 10 with a derivative (and a
// transposed copy, which no step asks for any more) 18.3 -> 6.3 us, 64 x 120 x 400 tf32 14.2 -> 6.9, 256 x 2048 x 2048 bf16 20.3 -> 11.6, 512 x 1000 x 8192
// bf16 47.9 -> 21.3, 342 x 3136 x 128 tf32 19.8 -> 10.9.
static bool pick_cluster(int M, int N, int K, int esize, int b_major, int ctas_max, int* bn_out, int* s_out) {
  static const float fixed[3][4] = {{5.6f, 5.6f, 6.0f, 0.f}, {8.0f, 6.3f, 6.3f, 6.6f}, {0.f, 8.6f, 9.3f, 7.5f}};   // [bn][S], 0: no such form
  constexpr float PER_KBLOCK = 0.33f, TWO_PASS = 11.3f;
  *bn_out = *s_out = 0;
  const int KB = (int)(((long long)K * esize + 127) / 128);
  const long long tm = (M + 127) / 128;
  float best = 1e30f;
  for (int b = 0; b < 3; ++b) {
    const int bn = 32 << b;
    if (b_major == ONO_MN_MAJOR && esize == 2 && bn < 64) continue;     // one MN-major box of bf16 is 64 wide
    for (int l = 0; l < 4; ++l) {
      const int S = 1 << l;
      const long long ctas = tm * ((N + bn - 1) / bn) * S;
      if (fixed[b][l] == 0.f || S > KB || ctas > (S == 8 ? std::min(ctas_max, 96) : ctas_max)) continue;
      const float cost = fixed[b][l] + PER_KBLOCK * (float)((KB + S - 1) / S);
      if (cost < best) { best = cost; *bn_out = bn; *s_out = S; }
    }
  }
  // a reduction so long that eight CTAs a tile are few: the two-pass form spreads it over all SMs (1024 x 10 x 4096 tf32: 9.3
  // against 11.4 us; 342 x 128 x 3136, just below the line: 11.7 against 10.9 us)
  if (!(best > TWO_PASS && KB >= 64 && tm * ((N + 127) / 128) * 8 <= ctas_max)) return false;
  *bn_out = *s_out = 0;
  return true;
}
}  // namespace ono

extern "C" const char* ono_last_error(void) { return ono::g_err; }
extern "C" int ono_num_sms(void) { return ono::num_sms(); }

extern "C" int ono_gemm(const OnoGemm* g, ono_stream_t stream_) {
  using namespace ono;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (!g || !g->A || !g->B || g->M <= 0 || g->N <= 0 || g->K <= 0) { set_error("bad gemm args%s", ""); return -1; }
  const int esize = g->dtype == ONO_TF32 ? 4 : 2;
  const OnoEpilogue& e = g->epi;
  // A plain result: one row-major output, nothing applied but alpha (the weight gradients).
  const bool plain = !e.bias && !e.bias_bf16 && e.act == ACT_NONE && e.dact == ACT_NONE && e.beta == 0.0f && !e.pre_f32 &&
                     !e.pre_bf16 && !e.outT_f32 && !e.outT_bf16;
  int bn = g->bn;
  if (bn == 0) {
    // The narrowest tile that holds the row (401408 x 64 x 288 bf16: 79.4 us with 128 columns, 56.5 with 64; 100352 x 60 x 300:
    // 24.6, 20.0). Wider rows: 256 columns unless that leaves most SMs idle, or unless the reduction is so short that the
    // epilogue is all there is (2048 x 3136 x 128 bf16 with a derivative: 54.9 us with 256, 44.0 with 128; 512 x 4096 x 2048: 38.4, 26.9).
    const int KB = (int)(((long long)g->K * esize + 127) / 128);
    if (g->N <= 32) bn = 32;
    else if (g->N <= 64) bn = 64;
    else if (g->N <= 128) bn = 128;
    else {
      const long long t256 = (long long)((g->M + 127) / 128) * ((g->N + 255) / 256);
      bn = t256 >= (long long)num_sms() * 3 / 4 && (plain || KB > 4) ? 256 : 128;
    }
  } else if (bn != 32 && bn != 128 && bn != 256 && !(bn == 64 && g->cluster > 0)) {
    set_error("bn must be 32, 128 or 256%s", "");
    return -1;
  }
  if (g->b_major == ONO_MN_MAJOR && bn < 64) bn = g->bn ? 128 : 64;
  if ((e.out_f32 || e.out_bf16 || e.pre_f32 || e.pre_bf16) && e.ld_out < g->N) { set_error("ld_out < N%s", ""); return -1; }
  if ((e.outT_f32 || e.outT_bf16) && e.ld_outT < g->M) { set_error("ld_outT < M%s", ""); return -1; }
  // The vectorised epilogue paths need 16-byte aligned rows.
  if ((e.out_f32 || e.pre_f32) && e.ld_out % 4 != 0 && !(e.any_ld && !e.reduce_out)) { set_error("ld_out must be a multiple of 4 for f32 outputs%s", ""); return -1; }
  if ((e.out_bf16 || e.pre_bf16) && (e.ld_out % 8 != 0)) { set_error("ld_out must be a multiple of 8 for bf16 outputs%s", ""); return -1; }
  if (e.dact != ACT_NONE) {
    if (!e.aux_f32 && !e.aux_bf16) { set_error("dact needs aux%s", ""); return -1; }
    if (e.aux_f32 && e.ld_aux % 4 != 0) { set_error("ld_aux must be a multiple of 4%s", ""); return -1; }
    if (e.aux_bf16 && e.ld_aux % 8 != 0) { set_error("ld_aux must be a multiple of 8%s", ""); return -1; }
  }

  GemmDev p;
  memset(&p, 0, sizeof(p));
  p.M = g->M; p.N = g->N; p.K = g->K;
  p.epi = g->epi;
  p.status = g->status;
  p.timeout_ns = g->timeout_ns ? g->timeout_ns : 2000000000ull;
  if (g->gate) {
    if (!g->gate_target || !g->gate_mask || g->gate_stride < 0) { set_error("gate needs a target word and a flag mask%s", ""); return -1; }
    p.gate = g->gate; p.gate_target = g->gate_target; p.gate_stride = g->gate_stride; p.gate_mask = g->gate_mask;
  }
  // One cluster per tile (see gemm_cluster_kernel) where pick_cluster() finds room for it; `cluster` < 0 keeps the persistent
  // kernel, > 0 asks for that cluster size (and `bn` for the tile width).
  int cl_bn = 0, cl_s = 0;
  bool split_over_pair = false;
  if (g->cluster >= 0 && !g->gate && !g->apply.p && !e.reduce_out && g->pair != 1 && (g->cluster > 0 || (g->bn == 0 && g->split_k == 0))) {
    const int limit = g->max_ctas > 0 ? std::min(g->max_ctas, num_sms()) : num_sms();
    if (g->cluster > 0) {
      const int kb = (int)(((long long)g->K * esize + 127) / 128);
      const bool pow2 = g->cluster == 1 || g->cluster == 2 || g->cluster == 4 || g->cluster == 8;
      if (!pow2 || (g->bn != 32 && g->bn != 64 && g->bn != 128) || g->cluster > kb || g->cluster > g->bn / 8 ||
          (g->b_major == ONO_MN_MAJOR && esize == 2 && g->bn < 64)) {
        set_error("cluster: needs a size of 1, 2, 4 or 8 within the k-blocks and a tile of 32, 64 or 128 columns%s", "");
        return -1;
      }
      cl_bn = g->bn; cl_s = g->cluster;
    } else {
      split_over_pair = pick_cluster(g->M, g->N, g->K, esize, g->b_major, limit, &cl_bn, &cl_s);
    }
  }
  CUtensorMap ta, tb;
  if (cl_s > 0) {
    int rc = make_operand(&p.a, &ta, g->A, esize, g->a_major, g->M, g->K, g->lda, 128);
    if (rc) return rc;
    if ((rc = make_operand(&p.b, &tb, g->B, esize, g->b_major, g->N, g->K, g->ldb, cl_bn))) return rc;
    p.split_k = cl_s;
    p.vec = e.ld_out % 4 == 0 && (((uintptr_t)e.out_f32 | (uintptr_t)e.pre_f32 | (uintptr_t)e.aux_f32) & 15) == 0 &&
            (((uintptr_t)e.out_bf16 | (uintptr_t)e.pre_bf16 | (uintptr_t)e.aux_bf16) & 7) == 0;
    p.vec_t = (((uintptr_t)e.outT_f32 & 15) | ((uintptr_t)e.outT_bf16 & 7)) == 0 && e.ld_outT % 4 == 0;
    p.idesc = (1u << 4) | ((esize == 4 ? 2u : 1u) << 7) | ((esize == 4 ? 2u : 1u) << 10) | ((uint32_t)p.a.mn_major << 15) |
              ((uint32_t)p.b.mn_major << 16) | ((uint32_t)(cl_bn >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    if (esize == 4) {
      if (cl_bn == 32) return launch_cluster<4, 32>(ta, tb, p, stream);
      if (cl_bn == 64) return launch_cluster<4, 64>(ta, tb, p, stream);
      return launch_cluster<4, 128>(ta, tb, p, stream);
    }
    if (cl_bn == 32) return launch_cluster<2, 32>(ta, tb, p, stream);
    if (cl_bn == 64) return launch_cluster<2, 64>(ta, tb, p, stream);
    return launch_cluster<2, 128>(ta, tb, p, stream);
  }
  int rc = make_operand(&p.a, &ta, g->A, esize, g->a_major, g->M, g->K, g->lda, 128);
  if (rc) return rc;
  // CTA pairs: on request (ops/gemm.py asks for them from a few k-blocks on), where M spans more than one 128-row block. A request
  // that is a preference yields to the two-pass form, on which pick_cluster() has counted: run as pairs on a handful of SMs instead,
  // 384 x 512 x 3136 tf32 took 43 us (two passes 21.5), 256 x 256 x 8192 bf16 51 (18), 256 x 1152 x 100352 bf16 491 (91; events
  // around a cold call, which adds about 8 to each).
  const bool pair = g->pair > 0 && bn >= 128 && g->M > 128 && !(g->pair == 2 && split_over_pair);
  rc = make_operand(&p.b, &tb, g->B, esize, g->b_major, g->N, g->K, g->ldb, pair ? bn / 2 : bn);
  if (rc) return rc;
  // Optimizer in the epilogue: the result tile updates the master / state tiles and is not stored.
  const OnoApply& ap = g->apply;
  if (ap.p) {
    if (e.out_f32 || e.out_bf16 || e.outT_f32 || e.outT_bf16 || e.pre_f32 || e.pre_bf16 || e.bias || e.bias_bf16 ||
        e.act != ACT_NONE || e.dact != ACT_NONE || e.reduce_out) {
      set_error("apply: the epilogue optimizer excludes every other output%s", "");
      return -1;
    }
    if (ap.kind < 0 || ap.kind > 2 || (ap.kind >= 1 && !ap.m) || (ap.kind == 2 && (!ap.v || !ap.adam_pows))) {
      set_error("apply: optimizer kind or state missing%s", "");
      return -1;
    }
    if (g->N % 4 != 0 || ap.ld % 4 != 0 || ap.ld < g->N || (((uintptr_t)ap.p | (uintptr_t)ap.m | (uintptr_t)ap.v) & 15) ||
        ((uintptr_t)ap.p_bf16 & 7)) {
      set_error("apply: N and ld must be multiples of 4 and the matrices 16-byte aligned%s", "");
      return -1;
    }
    if (g->split_k > 1) { set_error("apply: split-K is not supported%s", ""); return -1; }
    p.apply = ap;
  }
  // split-K (g->split_k > 1, or 0 = automatic for long-K problems with few output tiles): see gemm_finish_kernel.
  bool two_pass = false;
  {
    const int BKe = 128 / esize;
    const int KBh = (g->K + BKe - 1) / BKe;
    const long long tiles0 = (long long)((g->M + (pair ? 255 : 127)) / (pair ? 256 : 128)) * ((g->N + bn - 1) / bn);
    const long long ldn = ((long long)g->N + 3) / 4 * 4;
    int want = g->split_k > 1 ? g->split_k : 0;
    if (g->split_k == 0 && !ap.p && !e.reduce_out && !pair && tiles0 * 8 <= num_sms() && KBh >= 16)
      want = (int)std::min<long long>(KBh / 4, num_sms() / tiles0);
    if (want > KBh) want = KBh;
    if (want >= 2) {
      if (e.reduce_out) { set_error("split-K cannot be combined with reduce_out%s", ""); return -1; }
      float* ws = g->workspace;
      long long ws_elems = g->workspace_elems;
      if (!ws) {
        static float* scratch_dev[kMaxDevices] = {nullptr};
        float*& sp = scratch_dev[current_device()];
        if (!sp && cudaGetSymbolAddress((void**)&sp, g_split_scratch) != cudaSuccess) {
          set_error("split scratch address unavailable%s", "");
          return -6;
        }
        ws = sp;
        ws_elems = SPLIT_SCRATCH_ELEMS;
      } else if (((uintptr_t)ws & 15) != 0) {
        set_error("split-K workspace must be 16-byte aligned%s", "");
        return -1;
      }
      const long long slab = (long long)g->M * ldn;
      if (want > ws_elems / slab) want = (int)(ws_elems / slab);   // as many slabs as the workspace holds
      if (want >= 2) {
        const int per = (KBh + want - 1) / want;
        p.split_k = (KBh + per - 1) / per;                         // no empty split
        p.slabs = ws;
        p.slab_elems = slab;
        p.slab_ld = (int)ldn;
        two_pass = p.split_k > 1;
      } else if (g->split_k > 1 && slab > ws_elems) {
        set_error("split-K workspace too small for one slab (%s%lld elements needed)", "", slab);
        return -1;
      }
    }
    if (!two_pass) p.split_k = 1;
  }
  // A plain result (one row-major output, nothing applied but alpha: the weight gradients) leaves through TMA stores, off the
  // LSU path; every other epilogue stores from the staged tile.
  CUtensorMap tc;
  memset(&tc, 0, sizeof(tc));
  p.tma_out = 0;
  if (two_pass || ap.p) {
    // plain stores into the slabs / updates in place, no TMA store
  } else if (e.reduce_out) {
    if (!e.out_f32 || e.out_bf16 || e.outT_f32 || e.outT_bf16 || e.pre_f32 || e.pre_bf16 || ((uintptr_t)e.out_f32 & 15)) {
      set_error("reduce_out supports a plain, 16-byte aligned f32 output only%s", "");
      return -1;
    }
    rc = encode_out_map(&tc, e.out_f32, 4, g->M, g->N, e.ld_out);
    if (rc) return rc;
    p.tma_out = 3;
  } else if (plain && e.out_f32 && !e.out_bf16 && ((uintptr_t)e.out_f32 & 15) == 0 && g->N % 4 == 0 && e.ld_out % 4 == 0) {
    if (encode_out_map(&tc, e.out_f32, 4, g->M, g->N, e.ld_out) == 0) p.tma_out = 1;
  } else if (plain && e.out_bf16 && !e.out_f32 && ((uintptr_t)e.out_bf16 & 15) == 0 && g->N % 8 == 0) {
    if (encode_out_map(&tc, e.out_bf16, 2, g->M, g->N, e.ld_out) == 0) p.tma_out = 2;
  }
  p.staged = !two_pass && !ap.p && !p.tma_out;
  p.vec = e.ld_out % 4 == 0 && (((uintptr_t)e.out_f32 | (uintptr_t)e.pre_f32 | (uintptr_t)e.aux_f32) & 15) == 0 &&
          (((uintptr_t)e.out_bf16 | (uintptr_t)e.pre_bf16 | (uintptr_t)e.aux_bf16) & 7) == 0;
  p.vec_t = (((uintptr_t)e.outT_f32 & 15) | ((uintptr_t)e.outT_bf16 & 7)) == 0 && e.ld_outT % 4 == 0;
  // (A TMA store writes whole 16-byte units: with a row of N elements that ends inside a unit it would put the
  // zero-filled rest of the unit into the columns after N, which belong to the caller when the output is a view of a
  // wider matrix. Such shapes leave through thread stores. The reduce-add form adds those zeros, which changes nothing.)
  const uint32_t fmt = g->dtype == ONO_TF32 ? 2u : 1u;  // TF32 / BF16
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)p.a.mn_major << 15) |
            ((uint32_t)p.b.mn_major << 16) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)((pair ? 256 : 128) >> 4) << 24);

  // The TMA form of the optimizer epilogue: bf16 CTA pairs with 256-column tiles (the weight gradients of wide layers),
  // a reduction short enough for the two-stage operand ring, shadow rows that a bf16 tensor map can address.
  ApplyMaps am;
  // Momentum and SGD fit two chunk buffers per warp (loads run one chunk ahead); Adam's three state tiles fit only one,
  // which measured slower than reading them from registers (8192 x 8192 x 512: 0.48 ms against 0.44 ms), so Adam stays
  // on the register form. A TMA store writes whole 16-byte units, hence the shadow needs N % 8 == 0 here.
  const bool apply_tma = ap.p && pair && esize == 2 && bn == 256 && g->K <= 2048 && ap.kind <= 1 &&
                         (!ap.p_bf16 || (g->N % 8 == 0 && ap.ld % 8 == 0 && ((uintptr_t)ap.p_bf16 & 15) == 0));
  if (apply_tma) {
    memset(&am, 0, sizeof(am));
    if ((rc = encode_out_map(&am.p, ap.p, 4, g->M, g->N, ap.ld))) return rc;
    if (ap.kind >= 1 && (rc = encode_out_map(&am.m, ap.m, 4, g->M, g->N, ap.ld))) return rc;
    if (ap.kind == 2 && (rc = encode_out_map(&am.v, ap.v, 4, g->M, g->N, ap.ld))) return rc;
    if (ap.p_bf16 && (rc = encode_out_map(&am.s, ap.p_bf16, 2, g->M, g->N, ap.ld))) return rc;
    // unused maps still get prefetched by the kernel: point them at the master's map
    if (ap.kind < 1) am.m = am.p;
    if (ap.kind < 2) am.v = am.p;
    if (!ap.p_bf16) am.s = am.p;
  }
  auto run = [&]() -> int {
    if (apply_tma) return launch<2, 256, true, true>(ta, tb, tc, p, g->max_ctas, stream, am);
    if (pair) {
      if (esize == 4) return bn == 128 ? launch<4, 128, true>(ta, tb, tc, p, g->max_ctas, stream)
                                       : launch<4, 256, true>(ta, tb, tc, p, g->max_ctas, stream);
      return bn == 128 ? launch<2, 128, true>(ta, tb, tc, p, g->max_ctas, stream)
                       : launch<2, 256, true>(ta, tb, tc, p, g->max_ctas, stream);
    }
    if (esize == 4) {
      if (bn == 32) return launch<4, 32, false>(ta, tb, tc, p, g->max_ctas, stream);
      if (bn == 64) return launch<4, 64, false>(ta, tb, tc, p, g->max_ctas, stream);
      if (bn == 128) return launch<4, 128, false>(ta, tb, tc, p, g->max_ctas, stream);
      return launch<4, 256, false>(ta, tb, tc, p, g->max_ctas, stream);
    }
    if (bn == 32) return launch<2, 32, false>(ta, tb, tc, p, g->max_ctas, stream);
    if (bn == 64) return launch<2, 64, false>(ta, tb, tc, p, g->max_ctas, stream);
    if (bn == 128) return launch<2, 128, false>(ta, tb, tc, p, g->max_ctas, stream);
    return launch<2, 256, false>(ta, tb, tc, p, g->max_ctas, stream);
  };
  rc = run();
  if (rc || !two_pass) return rc;
  const int groups = g->M * ((g->N + 3) / 4);
  gemm_finish_kernel<<<(groups + 31) / 32, 256, 0, stream>>>(p.slabs, p.slab_elems, p.split_k, p.slab_ld, g->M, g->N, p.vec, g->epi);
  if (cudaGetLastError() != cudaSuccess) { set_error("gemm_finish launch failed%s", ""); return -7; }
  return 0;
}
