// Instantiation of the stencil pass: arithmetic and stage storage float.
#include "deriv.cuh"

namespace amss {
template cudaError_t launch_deriv<float, float>(const void*, const DerivItem*, int, int, void*, int, int, int, int,
                                             cudaStream_t);
}  // namespace amss
