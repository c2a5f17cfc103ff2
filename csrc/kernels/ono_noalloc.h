// Allocation-free entry point of the fused optimizer/synchronisation step.
//
// This has no counterpart in the reference (which has no GPU code at all); it exists for callers of
// this library that must not allocate device memory: a plug-in inside a serving or training process
// whose framework has already handed the whole HBM to its own caching allocator, code that runs
// between another component's captured CUDA graphs, or a recovery path that must not take the
// allocator's lock. There cudaMalloc can fail, stall the whole device, or wait on a lock the caller's
// own thread already holds.
//
// ono_sync_step (ono_kernels.h) takes a flag pad and per-block epoch words from its caller besides the tensors it works on.
// ono_sync_step_noalloc is the single-GPU form of the step, one rank that owns the whole vector, i.e. the fused
// "scale the gradient, apply SGD / momentum / Adam, refresh the bf16 shadow, accumulate the gradient norm" pass. It needs
// no scratch: the kernel waits for nobody.
//
// Rules of use:
//   * The caller passes every input and output (p, g, m, v, p_bf16, adam_pows, sumsq, status); the
//     call launches one kernel on `stream` and calls no allocating routine.
//   * nblocks is at most ONO_NOALLOC_MAX_BLOCKS (a larger request is rejected and nothing is launched); within that the
//     library picks the grid.
#pragma once
#include "ono_kernels.h"

#ifdef __cplusplus
extern "C" {
#endif

#define ONO_NOALLOC_MAX_BLOCKS 512

typedef struct OnoNoAllocStep {
  float* p;                // [n] parameters, updated in place
  const float* g;          // [n] gradient
  float* m;                // [n] first-moment / velocity state (momentum, Adam), else null
  float* v;                // [n] second-moment state (Adam), else null
  void* p_bf16;            // optional [n] bf16 copy of the updated parameters, 8-byte aligned
  long long n;             // element count, a multiple of 4 (pad the buffers); p, g, m, v 16-byte aligned
  int kind;                // 0 SGD, 1 momentum, 2 Adam
  float lr, mu, b1, b2, eps;
  int n_workers;           // the gradient is divided by this first (values below 1 mean 1)
  const float* adam_pows;  // device float[2] = {b1^t, b2^t} for this step (Adam only)
  double* sumsq;           // optional device double (8-byte aligned), += sum of squares of the scaled gradient
  int* status;             // optional device int, left alone: nothing in this form waits
  int nblocks;             // at most ONO_NOALLOC_MAX_BLOCKS; 0 = no wish
} OnoNoAllocStep;

// Returns 0 on success, a negative value if the arguments are rejected or the launch failed
// (ono_last_error() has the text).
int ono_sync_step_noalloc(const OnoNoAllocStep* s, ono_stream_t stream);

#ifdef __cplusplus
}
#endif
