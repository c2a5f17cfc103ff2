// Mini-batches out of pinned host memory.
//
// One launch gathers samples and labels, a row a warp; the row numbers come out of pinned memory as well, 32 of a warp at a time. PCIe bounds
// it (2048 rows of 784 and 10 floats: 139 us, 47 GB/s), so what the shape below is for is the step that runs beside it. The products of the
// step are persistent, one CTA an SM with a fixed share of the tiles: a CTA that finds no room beside a block of the feed starts when that block
// ends, and its kernel ends late. For the room
//   - the feed keeps its rows in registers: a CTA of the products takes 225 KB of the 228 KB of shared memory, and a block costs 1 KB as it is;
//   - it asks for the largest cut of shared memory: an SM that it reached first could not be recut for such a CTA while it runs;
//   - it takes at most 56 registers (46, none spilled) and blocks of two warps: a quarter of an SM's registers (16384) serves every fourth warp
//     of a CTA and has 1792 left beside three warps of 152 (products in clusters; 144, 128, 112 of the other products leave more).
// Steps back to back with 24 blocks of 256 threads, 64 registers and 8 KB, and so: convolution of 2048 images 688 -> 630 us, of 342 258 -> 254,
// three dense layers of 4096 on 1024 rows 624 -> 597, four of 2048 on 256 218 -> 211, eight of 8192 on 512 3350 -> 3261, 1001 and 333 on 200
// 84.3 -> 78.3. With other work between the steps less of it shows: the dense layers of 4096 take 643 then, and took 644 with neither this feed nor
// the bound on the products' registers.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "ono_kernels.h"

namespace ono {
void set_error(const char* fmt, const char* a, long long b, long long c);
bool is_host_memory(const void* p);

// 48 x 64 threads x 64 bytes in flight: 32 blocks take 152 us for the rows above and 72 no less than 48 (beside a step: 0.5 % slower).
constexpr int FEED_THREADS = 64, FEED_BLOCKS = 48;
template <typename V>
__device__ __forceinline__ void feed_row(const float* src, float* dst, int width, int lane) {
  constexpr int U = sizeof(V) == 16 ? 4 : 8;      // 512 rows of 517 single floats: 34.5 us with eight, 42.5 with four, 35.9 with sixteen
  const int w = width / (int)(sizeof(V) / sizeof(float));
  const V* s = reinterpret_cast<const V*>(src) + lane;
  V* d = reinterpret_cast<V*>(dst) + lane;
#pragma unroll 1
  for (int left = w - lane; left > 0; left -= 32 * U, s += 32 * U, d += 32 * U) {
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (left > 32 * u) v[u] = s[32 * u];
#pragma unroll
    for (int u = 0; u < U; ++u) if (left > 32 * u) d[32 * u] = v[u];
  }
}
__global__ void __maxnreg__(56) feed_kernel(const OnoFeed f, int x_vec, int y_vec) {
  const int lane = threadIdx.x & 31, first = blockIdx.x * (FEED_THREADS / 32) + (threadIdx.x >> 5), warps = gridDim.x * (FEED_THREADS / 32);
  for (int r0 = first; r0 < f.n; r0 += 32 * warps) {
    const int mine = r0 + lane * warps < f.n ? f.idx[r0 + lane * warps] : 0;
    for (int i = 0, r = r0; i < 32 && r < f.n; ++i, r += warps) {
      const int from = __shfl_sync(0xffffffffu, mine, i);
      const float y0 = lane < f.y_size ? f.y[(size_t)from * f.y_size + lane] : 0.f;      // under way with the samples; most labels are no longer
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {      // the samples, then what is left of the labels; one copy of the code below
        const int size = part ? f.y_size : f.x_size, skip = part ? 32 : 0;
        const float* s = (part ? f.y : f.x) + (size_t)from * size + skip;
        float* d = (part ? f.y_dst : f.x_dst) + (size_t)r * size + skip;
        if (part ? y_vec : x_vec) feed_row<float4>(s, d, size - skip, lane);
        else feed_row<float>(s, d, size - skip, lane);
      }
      if (lane < f.y_size) f.y_dst[(size_t)r * f.y_size + lane] = y0;
    }
  }
}
}  // namespace ono

using namespace ono;

extern "C" int ono_feed(const OnoFeed* f, ono_stream_t st, void* free_event, void* ready_event) {
  if (!f || !f->idx || !f->x || !f->y || !f->x_dst || !f->y_dst || f->n <= 0 || f->x_size <= 0 || f->y_size <= 0) {
    set_error("bad feed args%s", "", 0, 0);
    return -1;
  }
  if (!is_host_memory(f->idx)) { set_error("feed: the row numbers must be pinned%s", "", 0, 0); return -1; }
  cudaError_t e = cudaStreamWaitEvent((cudaStream_t)st, (cudaEvent_t)free_event, 0);
  if (e != cudaSuccess) { set_error("feed: cudaStreamWaitEvent: %s", cudaGetErrorString(e), 0, 0); return -7; }
  const int x_vec = f->x_size % 4 == 0 && (((uintptr_t)f->x | (uintptr_t)f->x_dst) & 15) == 0;
  const int y_vec = f->y_size % 4 == 0 && (((uintptr_t)f->y | (uintptr_t)f->y_dst) & 15) == 0;
  e = cudaFuncSetAttribute(feed_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) { set_error("feed: cudaFuncSetAttribute: %s", cudaGetErrorString(e), 0, 0); return -7; }
  feed_kernel<<<FEED_BLOCKS, FEED_THREADS, 0, (cudaStream_t)st>>>(*f, x_vec, y_vec);
  e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("feed launch: %s", cudaGetErrorString(e), 0, 0); return -5; }
  e = cudaEventRecord((cudaEvent_t)ready_event, (cudaStream_t)st);
  if (e != cudaSuccess) { set_error("feed: cudaEventRecord: %s", cudaGetErrorString(e), 0, 0); return -7; }
  return 0;
}
