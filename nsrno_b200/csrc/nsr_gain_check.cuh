// Gain-index validation shared by every entry point that reads gains (host code).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "nsrno_b200.h"

namespace {
// Pinned index buffer of one host thread, given back when the thread ends.
struct PinnedIndices {
  int32_t* words = nullptr;
  int capacity = 0;
  ~PinnedIndices() { if (words) cudaFreeHost(words); }

  cudaError_t reserve(int count) {
    if (count <= capacity) return cudaSuccess;
    if (words) cudaFreeHost(words);
    words = nullptr;
    capacity = 0;
    const int want = count < 1024 ? 1024 : count;
    const cudaError_t ce = cudaHostAlloc((void**)&words, sizeof(int32_t) * (size_t)want, cudaHostAllocDefault);
    if (ce != cudaSuccess) words = nullptr;
    else capacity = want;
    return ce;
  }
};

// The check in two parts: start() refuses what the host can see and copies the
// indices to pinned memory behind the stream's earlier work, finish() waits for
// that copy alone and looks at them.  What a caller launches in between runs
// while the host waits (four 256 x 384 fields through nsr_learned_precondition:
// 71 us a call with the stream drained first, 59 us this way).  The copy never
// outlives the check: calls of one thread use its buffer one after the other,
// whatever their streams.
struct GainCheck {
  const int32_t* host = nullptr;   // indices under way, nullptr when none are
  int count = 0, n_gain = 0;
  cudaEvent_t copied = nullptr;
  ~GainCheck() {
    if (host) cudaEventSynchronize(copied);   // the caller gave up between the two parts
    if (copied) cudaEventDestroy(copied);
  }

  int start(const NsrLearned* L, int n_systems, cudaStream_t st) {
    if (!L) return 0;
    if (!L->params) return NSR_ERR_ARGUMENT;
    if (!L->gains) return 0;
    if (L->n_gain <= 0) return NSR_ERR_ARGUMENT;
    if (!L->gain_index) return n_systems <= L->n_gain ? 0 : NSR_ERR_ARGUMENT;
    if (n_systems <= 0) return 0;
    static thread_local PinnedIndices pinned;
    cudaError_t ce = pinned.reserve(n_systems);
    if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&copied, cudaEventDisableTiming);
    if (ce != cudaSuccess) return (int)ce;
    ce = cudaMemcpyAsync(pinned.words, L->gain_index, sizeof(int32_t) * (size_t)n_systems, cudaMemcpyDeviceToHost, st);
    if (ce != cudaSuccess) return (int)ce;
    ce = cudaEventRecord(copied, st);
    if (ce != cudaSuccess) {
      cudaStreamSynchronize(st);
      return (int)ce;
    }
    host = pinned.words;
    count = n_systems;
    n_gain = L->n_gain;
    return 0;
  }

  int finish() {
    if (!host) return 0;
    const int32_t* index = host;
    host = nullptr;
    const cudaError_t ce = cudaEventSynchronize(copied);
    if (ce != cudaSuccess) return (int)ce;
    for (int s = 0; s < count; ++s)
      if (index[s] < 0 || index[s] >= n_gain) return NSR_ERR_ARGUMENT;
    return 0;
  }
};
}  // namespace
