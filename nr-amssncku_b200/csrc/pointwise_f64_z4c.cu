// Instantiation of the pointwise pass: arithmetic and stage storage double, Z4c.
#include "pointwise.cuh"

namespace amss {
template cudaError_t launch_pointwise<double, double, true>(const void*, const int2*, int, int, RKConst, int, unsigned*,
                                                  cudaStream_t, const void*);
}  // namespace amss
