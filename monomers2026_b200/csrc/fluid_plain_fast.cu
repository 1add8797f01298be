// fluid_plain_fast.cu - the compile-time spectral kernels of the
// reference-structured FP64 form
#include "fluid_fast.h"
#define SELM_EVEN_SIZES(X) SELM_EVEN_SIZES_64(X)
#include "fluid_fast_impl.cuh"
#include "fluid_plain_fast.cuh"

namespace selm {

#define SELM_ALL_SIZES(X) SELM_TUNED_SIZES(X) SELM_EVEN_SIZES_64(X)

cudaError_t plain_fast_attrs(int n) {
  switch (n) {
#define SELM_CASE(N) \
  case N:            \
    return PlainKernels<N>::attrs();
    SELM_ALL_SIZES(SELM_CASE)
#undef SELM_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t plain_fast_stage(int stage, int n, const PlainBufs& b, const FftTables<double>& tb, cudaStream_t st) {
  switch (n) {
#define SELM_CASE(N) \
  case N:            \
    return PlainKernels<N>::run(stage, b, tb, st);
    SELM_ALL_SIZES(SELM_CASE)
#undef SELM_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace selm
