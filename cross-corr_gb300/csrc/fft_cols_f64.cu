// fft_cols_f64.cu -- the column kernels of the fused FFT correlation, FP64, the shorter
// lengths (translation units of their own, so that they build in parallel).
#include "fft_engine.cuh"

namespace xc {
namespace fe {

#define XC_FFT_S double
bool col_kernels_f64(int n, ColKernels* k) {
  switch (n) {
    XC_FFT_COLS_SHORT(XC_COL_CASE)
    default: return col_kernels_f64_long(n, k);
  }
}

}  // namespace fe
}  // namespace xc
