// fft_rows_f32.cu -- the row kernels of the fused FFT correlation, FP32, every
// length (a translation unit of its own, so that the four build in parallel).
#include "fft_engine.cuh"

namespace xc {
namespace fe {

#define XC_FFT_S f2
bool row_kernels_f32(int n, RowKernels* k) {
  switch (n) {
    XC_FFT_ROWS(XC_ROW_CASE)
    default: return false;
  }
}

}  // namespace fe
}  // namespace xc
