// substep_common.cuh -- point indexing and the global-memory point accessor
// shared by the RK4 substep kernels.
#pragma once
#include "deriv.cuh"

namespace amss {

__device__ __forceinline__ void point_ijk(long long p, const int* ex, int& i, int& j, int& k) {
  const long long s1 = (long long)ex[0] * ex[1];
  k = (int)(p / s1);
  const long long r = p - (long long)k * s1;
  j = (int)(r / ex[0]);
  i = (int)(r - (long long)j * ex[0]);
}

template <typename SI, bool SYMM>
__device__ __forceinline__ Pt<SI, SYMM> make_pt(const SI* base, const BlockView& b, long long p,
                                               const double* side = nullptr) {
  Pt<SI, SYMM> q;
  q.base = base;
  q.side = side;
  q.fs = b.fs;
  q.p = p;
  q.sy = b.ex[0];
  q.sz = (long long)b.ex[0] * b.ex[1];
  point_ijk(p, b.ex, q.i, q.j, q.k);
  q.ex0 = b.ex[0];
  q.ex1 = b.ex[1];
  q.ex2 = b.ex[2];
  return q;
}

}  // namespace amss
