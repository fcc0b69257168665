// Instantiation of the pointwise pass: arithmetic and stage storage double, BSSN.
#include "pointwise.cuh"

namespace amss {
template cudaError_t launch_pointwise<double, double, false>(const void*, const int2*, int, int, RKConst, int, unsigned*,
                                                  cudaStream_t, const void*);
}  // namespace amss
