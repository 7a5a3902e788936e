// ragged_fft.h -- pairs of a ragged batch through the fused FFT kernels
// (ragged_fft.cu; kernels in fft_engine.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "xc_internal.h"

namespace xc {
namespace fe {

// One FP32 pair on the caller's buffers.
struct FftPair {
  const float* left;
  const float* right;
  float* out;
  Geometry g;
};

// The launches of a set of pairs: per chunk of pairs (whose spectra fit the
// workspace together) the row transforms, the column products and the inverse
// rows, one launch per transform length each.
struct RaggedFft {
  struct Launch {
    const void* fn;
    unsigned blocks;
    int threads, smem;
    std::vector<char> args;
  };
  std::vector<std::vector<Launch>> phases;  // launches of a phase are independent of each other
  void* tables = nullptr;                   // device: records, CTA lists, twiddles
};

// The kernels have lengths for the pair's output.
bool ragged_fft_takes(const Geometry& g);
// Workspace bytes of a set of pairs (at most about `cap`, or one pair's).
size_t ragged_fft_workspace(const std::vector<FftPair>& pairs, size_t cap);
xc_status ragged_fft_build(RaggedFft* f, const std::vector<FftPair>& pairs, void* workspace, size_t cap);
// Enqueues (or captures) the launches, phase after phase, over the streams;
// starts after work queued on streams[0] and ends joined to it.
xc_status ragged_fft_enqueue(const RaggedFft& f, const cudaStream_t* streams, int n_streams, cudaEvent_t fork,
                             const cudaEvent_t* joins);
void ragged_fft_release(RaggedFft* f);

}  // namespace fe
}  // namespace xc
