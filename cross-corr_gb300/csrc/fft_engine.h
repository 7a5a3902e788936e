// fft_engine.h -- host side of the fused FFT correlation (fft_engine.cu):
// what a plan keeps, and how it is made and run.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "fft_engine.cuh"
#include "xc_internal.h"

namespace xc {
namespace fe {

// One uniform problem: transform lengths, kernels, twiddle tables and the
// workspace layout (byte offsets).
struct Engine {
  bool ready = false;
  xc_dtype dtype = XC_F32;
  Geometry g{};
  PairMap pm{};
  long long n_right = 0;
  int nx = 0, ny = 0, nblk = 0;
  RowKernels rk{};
  ColKernels ck{};
  void* tw = nullptr;      // device: row table, column table, a row of zeros
  size_t tw_col = 0, zeros = 0;  // byte offsets of the last two
  bool shared = false;     // every right serves several lefts: all spectra are made first
  bool lpre = false;       // left spectra are made first
  int l_chunk = 1, k_chunk = 1, kc = 1;
  int sms = 0;
  size_t off_al = 0, off_ar = 0, off_fl = 0, off_fr = 0, off_b = 0, bytes = 0;
};

// 1 / (nx ny), the scale of an unnormalised pair of transforms, as powers of
// two on the left and right spectra and the rest at the end.  `early` puts all
// of the power on the spectra, half each, as unitary transforms have it:
// nothing leaves the type's range above before the result does (ragged
// batches, whose pairs would else run on the split path, which has no scale).
// Otherwise half of it stays for the end: the product of the spectra then lies
// sqrt(nx ny) above its unitary size, so that what it loses below the smallest
// normal number is below the result's own last place, as with transforms that
// are scaled at the end.  (FP32, 256x256 by 256x256, both of 2^-66: error
// 2.4e-5 of the result with all of the power on the spectra.)  Above, results
// up to 2^127 / sqrt(nx ny) are finite, 2^127 / (nx ny) with all of it at the end.
struct Scales {
  double left, right, rest;
};
Scales spectrum_scales(int nx, int ny, bool early);
// Smallest length >= n that the kernels have; 0 when n is beyond the largest.
int length_for(int n);
// Twiddle tables of a length's row or column passes: a complex value of the
// problem's type per entry (FP32 tables of pairs, ready for the packed
// products, were twice as large: 511x511 x 64 took 80.0 us against 74.6).
size_t twiddle_bytes(int n, bool rows, xc_dtype dtype);
void fill_twiddles(int n, bool rows, xc_dtype dtype, void* out);

// Plans a problem within `ws_bytes` of workspace.  *e stays not ready (and
// XC_OK is returned) when the sizes are beyond the kernels' lengths or the
// workspace is too small; an error only when the device calls fail.
xc_status engine_plan(Engine* e, xc_dtype dtype, const Geometry& g, const PairMap& pm, long long n_right,
                      size_t ws_bytes);
xc_status engine_run(const Engine& e, const void* left, const void* right, void* out, char* ws, cudaStream_t stream);
void engine_release(Engine* e);

}  // namespace fe
}  // namespace xc
