// Forward, loss and backward of a small dense network in two launches (f32 parameters, tf32 products).
//
// A product of such a network occupies a few SMs for less time than its launch, set-up and drain take: as launches of the tcgen05
// kernels (csrc/kernels/gemm_tcgen05.cu) the steps of 784-128-10 at batch 32 were eight kernels of 3 to 7 us in a row. Only the weight
// gradients sum over samples, everything before them works row by row. So here a cluster of CTAs takes 16 or 32 samples from the first
// layer to the loss and back: its CTAs share out the columns of every layer and hand each other their results in shared memory
// (st.shared::cluster), a cluster barrier between layers, no trip through memory. A second launch computes all weight and bias
// gradients. What bounds either is latency (L2 loads, barriers), not any unit's rate, so the products run on mma.sync, whose
// operands are registers: no descriptors, no TMEM, and 16-row tiles where tcgen05 has 128.
//
// All that does not depend on the samples before it, i.e. the CTA's columns of every weight matrix and, for the way back, its rows of them,
// comes into shared memory by asynchronous copies at the start, so that no layer waits for L2. The code is kept short (one loop for either
// direction, activations out of line): every part of it runs once or twice per launch, and with the loads of the weights unrolled into
// the products in aligned and unaligned forms, instruction fetch alone cost each layer about 3000 cycles of 8000.
//
// Fragments are read 16 bytes at a time: the index of the reduction, and the columns of a group of 32, are dealt to the lanes in runs
// of four (the same permutation on both operands), so that one load serves four products.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "act.cuh"
#include "loss.cuh"
#include "ono_kernels.h"
#include "ptx.cuh"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);
bool is_host_memory(const void* p);

constexpr int DS_THREADS = 256;
constexpr int DS_MAX_CTAS = 148;      // see ds_shape
__host__ __device__ inline int ds_pitch(int n) { return (n + 31) / 32 * 32 + 16; }   // rows of a tile start 16 banks apart

__device__ __forceinline__ void mma_tf32(float (&d)[4], const float (&a)[4], float b0, float b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
// Four consecutive values of a row, of which `left` exist (the rest are zero). V: rows are 16-byte aligned and multiples of four long, so
// that there are four or none. (Chosen at run time, the choice is a branch around every load, and the loads go one after the other.)
template <bool V>
__device__ __forceinline__ float4 ds_load4(const float* p, int left) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (V) {
    if (left > 0) v = *reinterpret_cast<const float4*>(p);
    return v;
  }
  if (left > 0) v.x = p[0];
  if (left > 1) v.y = p[1];
  if (left > 2) v.z = p[2];
  if (left > 3) v.w = p[3];
  return v;
}
__device__ __forceinline__ void ds_store4(float* p, float4 v, int left, bool vec) {
  if (left >= 4 && vec) { *reinterpret_cast<float4*>(p) = v; return; }
  if (left > 0) p[0] = v.x;
  if (left > 1) p[1] = v.y;
  if (left > 2) p[2] = v.z;
  if (left > 3) p[3] = v.w;
}
__device__ __forceinline__ float4 ds_cut(float4 v, int left) {      // the first `left` values, zeros behind them
  return make_float4(left > 0 ? v.x : 0.f, left > 1 ? v.y : 0.f, left > 2 ? v.z : 0.f, left > 3 ? v.w : 0.f);
}
__device__ __noinline__ float4 ds_act_fwd(int kind, float prm, float4 v) {
  float* f = reinterpret_cast<float*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = act_fwd(kind, prm, f[j]);
  return v;
}
__device__ __noinline__ float4 ds_act_bwd(int kind, float prm, int quirk, float4 a, float4 v) {
  const float* q = reinterpret_cast<const float*>(&a);
  float* f = reinterpret_cast<float*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = act_bwd(kind, prm, quirk, q[j], f[j]);
  return v;
}

// Four values of a row into shared memory, asynchronously; those past the matrix (`left` <= 0: all) become zero, which the copy itself does, so
// that nothing branches. V as for ds_load4; `base`: any address of the matrix.
template <bool V>
__device__ __forceinline__ void ds_copy4(float* dst, const float* base, const float* p, int left) {
  const uint32_t to = smem_u32(dst);
  if (V) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(left > 0 ? p : base), "r"(left > 0 ? 16 : 0) : "memory");
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4 * j), "l"(left > j ? p + j : base), "r"(left > j ? 4 : 0) : "memory");
}
// rows x cols values, zero up to pr rows and pc columns (a multiple of four), to rows `pitch` apart: a row a warp.
template <bool V>
__device__ __forceinline__ void ds_stage(const float* src, int ld, int rows, int cols, int pr, int pc, float* dst, int pitch) {
#pragma unroll 1
  for (int r = threadIdx.x >> 5; r < pr; r += DS_THREADS / 32)
#pragma unroll 4
    for (int c = 4 * (threadIdx.x & 31); c < pc; c += 128) ds_copy4<V>(dst + r * pitch + c, src, src + (size_t)r * ld + c, r < rows ? cols - c : 0);
}

// A group of 32 columns of W[K][N]: row k at 32 k, its four-column units swizzled so that the fragment reads below are free of conflicts.
__device__ __forceinline__ int ds_wf(int k, int c) { return k * 32 + ((((c >> 2) ^ ((k >> 1) & 6)) << 2) | (c & 3)); }
__host__ __device__ inline int ds_wb_pitch(int out) { return (out + 15) / 16 * 16 + 4; }

// Such a group: W's rows k < K (zero up to kp), `cols` of its columns.
template <bool V>
__device__ __forceinline__ void ds_stage_cols(const float* src, int ld, int K, int cols, int kp, float* dst) {
  const int c = 4 * (threadIdx.x & 7);
#pragma unroll 4
  for (int k = threadIdx.x >> 3; k < kp; k += DS_THREADS / 8) ds_copy4<V>(dst + ds_wf(k, c), src, src + (size_t)k * ld + c, k < K ? cols - c : 0);
}

// One product of a cluster's rows, out[R, N] = A[R, K] x B, the columns dealt to its CTAs in groups of 32. A and B in shared memory, zero up to
// a multiple of 16 of the reduction; B: this CTA's groups one after the other, W's columns (ds_wf) or, TRANS, W's rows (`ldb` apart).
// `done(row, col, v)` gets four columns of a row at a time. The eight warps are dealt out over the groups of this CTA and, where these are
// few, over K; partial sums meet in `red` and are added in order.
template <int RT, int S, bool TRANS, class Done>
__device__ __forceinline__ void ds_product(const float* A, int lda, const float* B, int ldb, int K, int N, int rank, float* red, Done done) {
  constexpr int R = 16 * RT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int groups = (N + 31) >> 5, mine = (groups - rank + S - 1) / S, most = (groups + S - 1) / S;
  const int lg = most > 4 ? 3 : most > 2 ? 2 : most > 1 ? 1 : 0, gw = 1 << lg;      // groups worked on at a time; the same in every CTA
  const int kw = 8 >> lg, slot = warp >> (3 - lg), ks = warp & (kw - 1);
  const int KG = (K + 15) >> 4, k0 = (KG * ks) >> (3 - lg), k1 = (KG * (ks + 1)) >> (3 - lg);
  const int per_group = 32 * (TRANS ? ldb : KG * 16);
#pragma unroll 1
  for (int p0 = 0; p0 < mine; p0 += gw) {
    const int grp = p0 + slot;
    float acc[RT][4][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[r][t][i] = 0.f;
    if (grp < mine) {
      const float* w0 = B + (size_t)grp * per_group;
#pragma unroll 2
      for (int kg = k0; kg < k1; ++kg) {
        float4 w[4], av[RT][2];
#pragma unroll
        for (int t = 0; t < 4; ++t)      // value t of column 4 g + t, or row 4 c + t of the reduction
          w[t] = *reinterpret_cast<const float4*>(TRANS ? w0 + (4 * g + t) * ldb + kg * 16 + 4 * c : w0 + ds_wf(kg * 16 + 4 * c + t, 4 * g));
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int h = 0; h < 2; ++h) av[r][h] = *reinterpret_cast<const float4*>(A + (16 * r + 8 * h + g) * lda + kg * 16 + 4 * c);
        // two steps of eight: lane c holds reduction indices 4 c, 4 c + 1, then 4 c + 2, 4 c + 3
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int r = 0; r < RT; ++r) {
            const float a[4] = {s ? av[r][0].z : av[r][0].x, s ? av[r][1].z : av[r][1].x, s ? av[r][0].w : av[r][0].y, s ? av[r][1].w : av[r][1].y};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if (TRANS) mma_tf32(acc[r][t], a, s ? w[t].z : w[t].x, s ? w[t].w : w[t].y);
              else {
                const float4 lo = w[2 * s], hi = w[2 * s + 1];
                mma_tf32(acc[r][t], a, t == 0 ? lo.x : t == 1 ? lo.y : t == 2 ? lo.z : lo.w, t == 0 ? hi.x : t == 1 ? hi.y : t == 2 ? hi.z : hi.w);
              }
            }
          }
      }
    }
    // column 4 j + t of the group is column j of product t: a lane holds columns 8 c .. 8 c + 7 of rows g and g + 8
    __syncthreads();                           // the sums of the previous groups have been read
    float* mr = red + (size_t)warp * R * 32;
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = 16 * r + 8 * h + g;
        float4* q = reinterpret_cast<float4*>(mr + row * 32);
        q[(2 * c) ^ (row & 7)] = make_float4(acc[r][0][2 * h], acc[r][1][2 * h], acc[r][2][2 * h], acc[r][3][2 * h]);
        q[(2 * c + 1) ^ (row & 7)] = make_float4(acc[r][0][2 * h + 1], acc[r][1][2 * h + 1], acc[r][2][2 * h + 1], acc[r][3][2 * h + 1]);
      }
    __syncthreads();
#pragma unroll 1
    for (int i = threadIdx.x; i < gw * R * 8; i += DS_THREADS) {
      const int sl = i / (R * 8), rest = i - sl * (R * 8), row = rest >> 3, c8 = rest & 7;
      if (p0 + sl >= mine) break;
      const float* src = red + ((size_t)(sl * kw) * R + row) * 32 + ((c8 ^ (row & 7)) << 2);
      float4 v = *reinterpret_cast<const float4*>(src);
      for (int k = 1; k < kw; ++k) {
        const float4 o = *reinterpret_cast<const float4*>(src + (size_t)k * R * 32);
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      done(row, (rank + (p0 + sl) * S) * 32 + 4 * c8, v);
    }
  }
}

// This CTA's columns of a tile in shared memory to memory (behind the barrier that shared them, which would wait for the stores).
template <int R, int S>
__device__ __forceinline__ void ds_put(const float* h, int pitch, int rows, int N, int rank, float* out, int ld) {
  const int groups = (N + 31) >> 5, mine = (groups - rank + S - 1) / S;
  const bool vec = ld % 4 == 0 && ((uintptr_t)out & 15) == 0;
#pragma unroll 1
  for (int i = threadIdx.x; i < mine * R * 8; i += DS_THREADS) {
    const int sl = i / (R * 8), rest = i - sl * (R * 8), row = rest >> 3, col = (rank + sl * S) * 32 + 4 * (rest & 7);
    if (row < rows) ds_store4(out + (size_t)row * ld + col, *reinterpret_cast<const float4*>(h + row * pitch + col), N - col, vec);
  }
}

// What the CTAs of a step hand the last one of them (OnoDenseStep::scratch).
struct DenseScratch {
  double loss[DS_MAX_CTAS];
  int correct[DS_MAX_CTAS];
  unsigned int ticket;
};
static_assert(sizeof(DenseScratch) <= ONO_DENSE_SCRATCH, "scratch of a dense step");

// Where everything lies in shared memory (in floats).
struct DenseDev {
  OnoDenseStep s;
  int x_at, y_at, red_at;
  int h_at[ONO_DENSE_MAX], z_at[ONO_DENSE_MAX], b_at[ONO_DENSE_MAX];      // a layer's output (GELU: and its pre-activation), its bias
  int wf_at[ONO_DENSE_MAX], wb_at[ONO_DENSE_MAX];                         // this CTA's columns of its weights, and rows for the way back
};

template <int RT, int S>
__global__ void __launch_bounds__(DS_THREADS, 1) dense_rows_kernel(const __grid_constant__ DenseDev p) {
  constexpr int R = 16 * RT;
  extern __shared__ __align__(16) float ds_smem[];
  __shared__ double s_loss[8];
  __shared__ int s_correct[8];
  const OnoDenseStep& s = p.s;
  const int rank = (int)cluster_ctarank();
  const int cl = (int)blockIdx.x / S, row0 = cl * R, rows = min(R, s.rows - row0), L = s.n_layers, first = s.dx ? 0 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const red = ds_smem + p.red_at;
  cluster_arrive();                             // "this CTA runs": nobody writes to its shared memory before
  auto to_all = [&](float* local, float4 v) {   // the same place in every CTA of the cluster
    *reinterpret_cast<float4*>(local) = v;
    const uint32_t at = smem_u32(local);
#pragma unroll
    for (int q = 1; q < S; ++q) st_cluster_v4(mapa_shared(at, (uint32_t)((rank + q) & (S - 1))), v);
  };

  // the samples and the first layer's weights, then everything else there is
  {
    const int in = s.layer[0].in, pitch = ds_pitch(in);
    float* const x = ds_smem + p.x_at;
    const float* from = s.x + (size_t)row0 * s.ldx;
    if (in % 4 == 0 && s.ldx % 4 == 0 && ((uintptr_t)s.x & 15) == 0) ds_stage<true>(from, s.ldx, rows, in, R, (in + 15) & ~15, x, pitch);
    else ds_stage<false>(from, s.ldx, rows, in, R, (in + 15) & ~15, x, pitch);
  }
#pragma unroll 1
  for (int l = 0; l < L; ++l) {
    const OnoDenseLayer& d = s.layer[l];
    const bool vec = d.out % 4 == 0 && ((uintptr_t)d.w & 15) == 0;
    const int kp = (d.in + 15) & ~15, groups = (d.out + 31) / 32;
    float* w = ds_smem + p.wf_at[l];
#pragma unroll 1
    for (int q = rank; q < groups; q += S, w += kp * 32) {
      if (vec) ds_stage_cols<true>(d.w + q * 32, d.out, d.in, min(32, d.out - q * 32), kp, w);
      else ds_stage_cols<false>(d.w + q * 32, d.out, d.in, min(32, d.out - q * 32), kp, w);
    }
    for (int i = threadIdx.x; i < groups * 32; i += DS_THREADS) ds_smem[p.b_at[l] + i] = d.b && i < d.out ? __ldg(d.b + i) : 0.f;
    if (l == 0) asm volatile("cp.async.commit_group;" ::: "memory");
  }
#pragma unroll 1
  for (int l = first; l < L; ++l) {
    const OnoDenseLayer& d = s.layer[l];
    const bool vec = d.out % 4 == 0 && ((uintptr_t)d.w & 15) == 0;
    const int ldb = ds_wb_pitch(d.out), groups = (d.in + 31) / 32;
    float* w = ds_smem + p.wb_at[l];
#pragma unroll 1
    for (int q = rank; q < groups; q += S, w += 32 * ldb) {
      const float* from = d.w + (size_t)q * 32 * d.out;
      if (vec) ds_stage<true>(from, d.out, min(32, d.in - q * 32), d.out, 32, (d.out + 15) & ~15, w, ldb);
      else ds_stage<false>(from, d.out, min(32, d.in - q * 32), d.out, 32, (d.out + 15) & ~15, w, ldb);
    }
  }
  for (int i = threadIdx.x; i < rows * s.loss.C; i += DS_THREADS) {
    const int r = i / s.loss.C, c = i - r * s.loss.C;
    ds_smem[p.y_at + i] = s.loss.y[(size_t)(row0 + r) * s.loss.ldy + c];
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  cluster_wait();

  // forward
#pragma unroll 1
  for (int l = 0; l < L; ++l) {
    const OnoDenseLayer& d = s.layer[l];
    float* const h = ds_smem + p.h_at[l];
    float* const z = p.z_at[l] >= 0 ? ds_smem + p.z_at[l] : nullptr;
    const float* const bias = ds_smem + p.b_at[l];
    const int pitch = ds_pitch(d.out);
    auto done = [&](int row, int col, float4 v) {
      const float4 b = *reinterpret_cast<const float4*>(bias + col);      // (zero past the last column, as the product is)
      v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
      if (z) *reinterpret_cast<float4*>(z + row * pitch + col) = v;
      if (d.act != ACT_NONE) v = ds_act_fwd(d.act, d.act_param, v);
      to_all(h + row * pitch + col, ds_cut(v, d.out - col));      // an activation of zero need not be zero
    };
    ds_product<RT, S, false>(ds_smem + (l ? p.h_at[l - 1] : p.x_at), ds_pitch(d.in), ds_smem + p.wf_at[l], 0, d.in, d.out, rank, red, done);
    if (l == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");      // seen by the others behind the barrier
    __syncwarp();
    cluster_sync_all();
    if (l < L - 1) ds_put<R, S>(h, pitch, rows, d.out, rank, d.a + (size_t)row0 * d.ld_a, d.ld_a);
  }

  // loss and the gradient of the last pre-activation, in place: a row a warp, at most one each, dealt to the CTAs, who hand each other the result
  {
    float* const h = ds_smem + p.h_at[L - 1];
    const int C = s.loss.C, row = rank + S * warp, pitch = ds_pitch(C);
    // Whether a product reads the gradient here. Where none does (one layer, no gradient for what is below it) no barrier follows, and a CTA with
    // fewer rows may have ended: nothing may be stored in its shared memory.
    const bool shared = L > first;
    static_assert(R <= 8 * S, "rows of the loss");
    LossRow r{0.f, 0};
    if (row < rows) {
      float* hr = h + row * pitch;
      float* out = s.loss.d_f32 + (size_t)(row0 + row) * s.loss.ld_d;
      auto put = [&](int j, float prob, float dv) {
        if (shared) {
          const uint32_t at = smem_u32(hr + j);
#pragma unroll
          for (int q = 0; q < S; ++q) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_shared(at, (uint32_t)q)), "f"(dv) : "memory");
        }
        out[j] = dv;
      };
      r = loss_row<1>(s.loss, hr, ds_smem + p.y_at + row * C, nullptr, nullptr, lane, put);
    }
    if (lane == 0) { s_loss[warp] = (double)r.loss; s_correct[warp] = r.correct; }
    if (shared) {
      __syncwarp();
      cluster_sync_all();
    }
  }

  // backward: d(l) = d(l + 1) W^T, through the activation below (below the first layer only if the caller has one); a layer's gradient
  // takes the place of its activation
#pragma unroll 1
  for (int l = L - 1; l >= first; --l) {
    const OnoDenseLayer& d = s.layer[l];
    const OnoDenseLayer& e = s.layer[l ? l - 1 : 0];
    const bool more = l > first;
    float* const h = ds_smem + p.h_at[l ? l - 1 : 0];
    const float* const st = l && p.z_at[l - 1] >= 0 ? ds_smem + p.z_at[l - 1] : h;
    const int pitch = ds_pitch(d.in), ldg = l ? e.ld_d : s.ld_dx;
    float* const out = (l ? e.d : s.dx) + (size_t)row0 * ldg;
    const bool g_vec = ldg % 4 == 0 && ((uintptr_t)out & 15) == 0;
    auto done = [&](int row, int col, float4 v) {
      if (l && e.act != ACT_NONE) v = ds_act_bwd(e.act, e.act_param, s.relu_quirk, *reinterpret_cast<const float4*>(st + row * pitch + col), v);
      if (!l && s.dx_act != ACT_NONE && row < rows)
        v = ds_act_bwd(s.dx_act, s.dx_param, s.relu_quirk, ds_load4<false>(s.dx_aux + (size_t)(row0 + row) * s.ld_dx_aux + col, d.in - col), v);
      if (more) to_all(h + row * pitch + col, ds_cut(v, d.in - col));
      else if (row < rows) ds_store4(out + (size_t)row * ldg + col, v, d.in - col, g_vec);
    };
    ds_product<RT, S, true>(ds_smem + p.h_at[l], ds_pitch(d.out), ds_smem + p.wb_at[l], ds_wb_pitch(d.out), d.out, d.in, rank, red, done);
    if (more) {
      __syncwarp();
      cluster_sync_all();
      ds_put<R, S>(h, pitch, rows, d.in, rank, out, ldg);
    }
  }

  // the loss, behind everything the step waits for (its fence and counter took one warp, and so all, 5000 cycles where the rows were done)
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    int n = 0;
    for (int w = 0; w < 8; ++w) { t += s_loss[w]; n += s_correct[w]; }
    DenseScratch* const sc = reinterpret_cast<DenseScratch*>(s.scratch);
    sc->loss[blockIdx.x] = t;
    sc->correct[blockIdx.x] = n;
    __threadfence();
    if (atomicAdd(&sc->ticket, 1u) == gridDim.x - 1u) {      // the last CTA adds up, in order
      __threadfence();
      t = 0.0;
      n = 0;
      for (unsigned q = 0; q < gridDim.x; ++q) { t += __ldcg(sc->loss + q); n += __ldcg(sc->correct + q); }
      t *= (double)(1.0f / ((float)s.loss.B * (float)s.loss.C));
      if (!s.zero_loss) t += *s.loss.loss_sum;
      *s.loss.loss_sum = t;
      if (s.loss.correct) *s.loss.correct += n;
      if (s.host_loss) *s.host_loss = t;
      sc->ticket = 0u;
    }
  }
}

// All weight and bias gradients: dW[i][o] = sum over samples a[b][i] d[b][o], a 32 x 32 tile a block. The eight warps take interleaved groups of
// eight samples, their sums meet in shared memory and are added in order; blocks of the first tile row also sum the deltas (bias).
struct DenseGrads {
  int n, rows;
  struct { const float* a; const float* d; float* gw; float* gb; int lda, ldd, in, out, end, av, dv; } job[ONO_DENSE_MAX];
  float beta;
};

template <bool AV, bool DV>
__device__ __forceinline__ void dense_grads_tile(const DenseGrads& p, int j, float (*red)[32 * 32], float (*bred)[32]) {
  const auto& q = p.job[j];
  const int tile = (int)blockIdx.x - (j ? p.job[j - 1].end : 0), ot = (q.out + 31) / 32;
  const int i0 = tile / ot * 32, o0 = tile % ot * 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  float acc[2][4][4], bs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][t][i] = 0.f;
  constexpr int U = 4;
  const int il = q.in - (i0 + 4 * g), ol = q.out - (o0 + 4 * g);
  for (int b0 = warp * 8; b0 < p.rows; b0 += 64 * U) {
    float4 a[U][2], d[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int b = b0 + 64 * u + 4 * h + c;
        a[u][h] = d[u][h] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (b < p.rows) {
          a[u][h] = ds_load4<AV>(q.a + (size_t)b * q.lda + i0 + 4 * g, il);
          d[u][h] = ds_load4<DV>(q.d + (size_t)b * q.ldd + o0 + 4 * g, ol);
        }
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float* al = reinterpret_cast<const float*>(&a[u][0]);
      const float* ah = reinterpret_cast<const float*>(&a[u][1]);
      const float* dl = reinterpret_cast<const float*>(&d[u][0]);
      const float* dh = reinterpret_cast<const float*>(&d[u][1]);
#pragma unroll
      for (int t = 0; t < 4; ++t) bs[t] += dl[t] + dh[t];
#pragma unroll
      for (int m = 0; m < 2; ++m) {      // rows g and g + 8 of product m are rows 4 g + 2 m and 4 g + 2 m + 1 of the tile
        const float av[4] = {al[2 * m], al[2 * m + 1], ah[2 * m], ah[2 * m + 1]};
#pragma unroll
        for (int t = 0; t < 4; ++t) mma_tf32(acc[m][t], av, dl[t], dh[t]);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = 4 * g + 2 * m + h;
      float4* r4 = reinterpret_cast<float4*>(red[warp] + row * 32);
      r4[(2 * c) ^ (row & 7)] = make_float4(acc[m][0][2 * h], acc[m][1][2 * h], acc[m][2][2 * h], acc[m][3][2 * h]);
      r4[(2 * c + 1) ^ (row & 7)] = make_float4(acc[m][0][2 * h + 1], acc[m][1][2 * h + 1], acc[m][2][2 * h + 1], acc[m][3][2 * h + 1]);
    }
  if (i0 == 0) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      bs[t] += __shfl_xor_sync(0xffffffffu, bs[t], 1);
      bs[t] += __shfl_xor_sync(0xffffffffu, bs[t], 2);
      if (c == 0) bred[warp][4 * g + t] = bs[t];
    }
  }
  __syncthreads();
  const int row = threadIdx.x >> 3, c8 = threadIdx.x & 7, i = i0 + row, o = o0 + 4 * c8;
  const int at = row * 32 + ((c8 ^ (row & 7)) << 2);
  float4 v = *reinterpret_cast<const float4*>(red[0] + at);
#pragma unroll
  for (int w = 1; w < 8; ++w) {
    const float4 x = *reinterpret_cast<const float4*>(red[w] + at);
    v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
  }
  if (i < q.in && o < q.out) {
    float* dst = q.gw + (size_t)i * q.out + o;
    const bool vec = q.out % 4 == 0 && ((uintptr_t)q.gw & 15) == 0;
    const int left = q.out - o;
    if (p.beta != 0.f) {
      const float4 x = ds_load4<false>(dst, left);
      v.x += p.beta * x.x; v.y += p.beta * x.y; v.z += p.beta * x.z; v.w += p.beta * x.w;
    }
    ds_store4(dst, v, left, vec);
  }
  if (i0 == 0 && threadIdx.x < 32 && o0 + (int)threadIdx.x < q.out) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += bred[w][threadIdx.x];
    float* dst = q.gb + o0 + threadIdx.x;
    *dst = p.beta != 0.f ? p.beta * *dst + t : t;
  }
}

__global__ void __launch_bounds__(DS_THREADS) dense_grads_kernel(const __grid_constant__ DenseGrads p) {
  __shared__ __align__(16) float red[8][32 * 32];
  __shared__ float bred[8][32];
  int j = 0;
  while (j < p.n - 1 && (int)blockIdx.x >= p.job[j].end) ++j;
  if (p.job[j].av && p.job[j].dv) dense_grads_tile<true, true>(p, j, red, bred);
  else dense_grads_tile<false, false>(p, j, red, bred);
}

// Shared memory of a CTA with R rows and S CTAs to a cluster (bytes), and where everything lies in it.
static size_t ds_layout(const OnoDenseStep* s, int R, int S, DenseDev* p) {
  long long at = 0;
  auto take = [&](long long n) { const long long a = at; at += (n + 3) / 4 * 4; return (int)std::min<long long>(a, 1 << 30); };
  p->x_at = take((long long)R * ds_pitch(s->layer[0].in));
  for (int l = 0; l < s->n_layers; ++l) {
    const long long in = s->layer[l].in, out = s->layer[l].out, n = (long long)R * ds_pitch((int)out);
    const long long go = ((out + 31) / 32 + S - 1) / S, gi = ((in + 31) / 32 + S - 1) / S;
    p->h_at[l] = take(n);
    p->z_at[l] = s->layer[l].act == ACT_GELU && l + 1 < s->n_layers ? take(n) : -1;
    p->b_at[l] = take((out + 31) / 32 * 32);
    p->wf_at[l] = take(go * ((in + 15) / 16 * 16) * 32);
    p->wb_at[l] = l > 0 || s->dx ? take(gi * 32 * ds_wb_pitch((int)out)) : 0;
  }
  p->y_at = take((long long)R * s->layer[s->n_layers - 1].out);
  p->red_at = take(8ll * R * 32);
  return (size_t)at * 4;
}
}  // namespace ono

using namespace ono;

// Rows of a cluster and its CTAs: as many small clusters as can be resident at once (148 SMs hold 12 of eight CTAs, 37 of four; more would
// run one after the other). DS_MAX_CTAS bounds the scratch; ono_dense_step_fits and the launch both come here.
constexpr int DS_OF_8 = 12, DS_OF_4 = 32;
static_assert(8 * DS_OF_8 <= DS_MAX_CTAS && 4 * DS_OF_4 <= DS_MAX_CTAS, "clusters of a dense step");
static bool ds_shape(int rows, int* rt, int* cs) {
  if (rows <= DS_OF_8 * 16) { *rt = 1; *cs = 8; }
  else if (rows <= DS_OF_8 * 32) { *rt = 2; *cs = 8; }
  else if (rows <= DS_OF_4 * 32) { *rt = 2; *cs = 4; }
  else return false;
  return true;
}

extern "C" int ono_dense_step_fits(const OnoDenseStep* s) {
  int rt, cs;
  if (!s || s->n_layers < 1 || s->n_layers > ONO_DENSE_MAX || !ds_shape(s->rows, &rt, &cs)) return 0;
  DenseDev p;
  for (int l = 0; l < s->n_layers; ++l)
    if (s->layer[l].out <= 0 || s->layer[l].in <= 0 || s->layer[l].out > 8192 || s->layer[l].in > 8192) return 0;
  return s->layer[s->n_layers - 1].out <= 32 && ds_layout(s, 16 * rt, cs, &p) <= 225u * 1024u;
}

extern "C" int ono_dense_step(const OnoDenseStep* s, ono_stream_t st) {
  if (!s || !s->x || !s->scratch || !s->loss.y || !s->loss.d_f32 || !s->loss.loss_sum || s->rows <= 0 || s->loss.B != s->rows ||
      !ono_dense_step_fits(s) || s->loss.C != s->layer[s->n_layers - 1].out) {
    set_error("bad dense_step args%s", "", 0, 0);
    return -1;
  }
  for (int l = 0; l < s->n_layers; ++l) {
    const OnoDenseLayer& d = s->layer[l];
    const bool last = l == s->n_layers - 1;
    if (!d.w || (!last && (!d.a || !d.d || ((uintptr_t)d.a & 15) || ((uintptr_t)d.d & 15) || d.ld_a < d.out || d.ld_d < d.out)) ||
        (l && d.in != s->layer[l - 1].out) || (last && d.act == ACT_GELU)) {
      set_error("bad dense_step layer %s%lld", "", l, 0);
      return -1;
    }
  }
  if (s->dx_act != ACT_NONE && (!s->dx || !s->dx_aux || s->ld_dx_aux < s->layer[0].in)) { set_error("dense_step: dx_act needs dx and dx_aux%s", "", 0, 0); return -1; }
  if (s->host_loss && !is_host_memory(s->host_loss)) { set_error("dense_step: host_loss must be pinned%s", "", 0, 0); return -1; }
  int rt, cs;
  ds_shape(s->rows, &rt, &cs);
  DenseDev p;
  p.s = *s;
  const size_t smem = ds_layout(s, 16 * rt, cs, &p);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((s->rows + 16 * rt - 1) / (16 * rt) * cs));
  cfg.blockDim = dim3(DS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  auto go = [&](auto kern) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return e != cudaSuccess ? e : cudaLaunchKernelEx(&cfg, kern, p);
  };
  const cudaError_t e = rt == 1 ? go(dense_rows_kernel<1, 8>) : cs == 8 ? go(dense_rows_kernel<2, 8>) : go(dense_rows_kernel<2, 4>);
  if (e != cudaSuccess) { set_error("dense_step: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}

extern "C" int ono_dense_grads(const OnoDenseStep* s, float beta, ono_stream_t st) {
  if (!s || !s->x || s->n_layers < 1 || s->n_layers > ONO_DENSE_MAX || s->rows <= 0 || !s->loss.d_f32) { set_error("bad dense_grads args%s", "", 0, 0); return -1; }
  DenseGrads p;
  p.n = s->n_layers;
  p.rows = s->rows;
  p.beta = beta;
  long long end = 0;
  for (int l = 0; l < s->n_layers; ++l) {
    const OnoDenseLayer& d = s->layer[l];
    auto& q = p.job[l];
    q.a = l ? s->layer[l - 1].a : s->x;
    q.lda = l ? s->layer[l - 1].ld_a : s->ldx;
    const bool last = l == s->n_layers - 1;
    q.d = last ? s->loss.d_f32 : d.d;
    q.ldd = last ? s->loss.ld_d : d.ld_d;
    q.gw = d.gw; q.gb = d.gb; q.in = d.in; q.out = d.out;
    if (!q.a || !q.d || !q.gw || !q.gb || d.in <= 0 || d.out <= 0) { set_error("bad dense_grads layer %s%lld", "", l, 0); return -1; }
    q.av = q.lda % 4 == 0 && q.in % 4 == 0 && ((uintptr_t)q.a & 15) == 0;
    q.dv = q.ldd % 4 == 0 && q.out % 4 == 0 && ((uintptr_t)q.d & 15) == 0;
    end += (long long)((d.in + 31) / 32) * ((d.out + 31) / 32);
    if (end >= (1ll << 31)) { set_error("dense_grads: too many tiles%s", "", 0, 0); return -1; }
    q.end = (int)end;
  }
  dense_grads_kernel<<<(unsigned)end, DS_THREADS, 0, (cudaStream_t)st>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("dense_grads: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}
