// fluid_fast64.cu - the compile-time spectral kernels in FP64
#include "fluid_fast.h"
#define SELM_EVEN_SIZES(X) SELM_EVEN_SIZES_64(X)
#include "fluid_fast_impl.cuh"

namespace selm {

template cudaError_t fast_attrs_for<double>(int);
template cudaError_t fast_stage<double>(int, int, int, int, const FastBufs<double>&, const ZGeom&,
                                        const FftTables<double>&, const double*, const double*, const double*, int, long,
                                        const CUtensorMap*, cudaStream_t);

}  // namespace selm
