// fft_rows_f64.cu -- the row kernels of the fused FFT correlation, FP64, every
// length (a translation unit of its own, so that the four build in parallel).
#include "fft_engine.cuh"

namespace xc {
namespace fe {

#define XC_FFT_S double
bool row_kernels_f64(int n, RowKernels* k) {
  switch (n) {
    XC_FFT_ROWS(XC_ROW_CASE)
    default: return false;
  }
}

}  // namespace fe
}  // namespace xc
