// Instantiation of the stencil pass: arithmetic and stage storage double.
#include "deriv.cuh"

namespace amss {
template cudaError_t launch_deriv<double, double>(const void*, const DerivItem*, int, int, void*, int, int, int, int,
                                             cudaStream_t);
}  // namespace amss
