// fft_cols_f64.cu -- the column kernels of the fused FFT correlation, FP64, every
// length (a translation unit of its own, so that the four build in parallel).
#include "fft_engine.cuh"

namespace xc {
namespace fe {

#define XC_FFT_S double
bool col_kernels_f64(int n, ColKernels* k) {
  switch (n) {
    XC_FFT_COLS(XC_COL_CASE)
    default: return false;
  }
}

}  // namespace fe
}  // namespace xc
