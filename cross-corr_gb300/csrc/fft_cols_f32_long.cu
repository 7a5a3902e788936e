// fft_cols_f32_long.cu -- the column kernels of the fused FFT correlation, FP32, the longer
// lengths (translation units of their own, so that they build in parallel).
#include "fft_engine.cuh"

namespace xc {
namespace fe {

#define XC_FFT_S f2
bool col_kernels_f32_long(int n, ColKernels* k) {
  switch (n) {
    XC_FFT_COLS_LONG(XC_COL_CASE)
    default: return false;
  }
}

}  // namespace fe
}  // namespace xc
