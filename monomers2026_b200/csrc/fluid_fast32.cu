// fluid_fast32.cu - the compile-time spectral kernels in FP32
#include "fluid_fast.h"
#define SELM_EVEN_SIZES(X) SELM_EVEN_SIZES_32(X)
#include "fluid_fast_impl.cuh"

namespace selm {

bool fast_tuned_size(int n) {
  switch (n) {
#define SELM_CASE(N) case N:
    SELM_TUNED_SIZES(SELM_CASE)
#undef SELM_CASE
    return true;
    default:
      return false;
  }
}
bool fast_size(int n, int precision) {
  if (fast_tuned_size(n)) return true;
  switch (n) {
#define SELM_CASE(N) case N:
    SELM_EVEN_SIZES_64(SELM_CASE)
    return true;
    SELM_EVEN_SIZES_ABOVE_64(SELM_CASE)
    return precision == 32;
#undef SELM_CASE
    default:
      return false;
  }
}

template cudaError_t fast_attrs_for<float>(int);
template cudaError_t fast_stage<float>(int, int, int, int, const FastBufs<float>&, const ZGeom&, const FftTables<float>&,
                                       const double*, const double*, const double*, int, long, const CUtensorMap*,
                                       cudaStream_t);

}  // namespace selm
