// substep_common.cuh -- point indexing, the tile lists and the global-memory
// point accessor shared by the RK4 substep kernels.
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

// Region of a tile: -1 the whole array, else the index into StepBlock::rlo/rn.
__device__ __forceinline__ int tile_region(int x) {
  return (x & kRegionTile) ? ((x & kOwnRegion) ? 1 : 0) : -1;
}

// Points of a tile list's range in a block: its array, or one of its regions.
template <typename T>
__device__ __forceinline__ long long tile_count(const StepBlock<T>& B, int rg) {
  return rg >= 0 ? (long long)B.rn[rg][0] * B.rn[rg][1] * B.rn[rg][2] : B.npts;
}

// Array point of entry q of a tile's point range, or -1 past its end.
template <typename T>
__device__ __forceinline__ long long tile_point(const StepBlock<T>& B, int rg, long long q) {
  if (q >= tile_count(B, rg)) return -1;
  if (rg < 0) return q;
  const int* lo = B.rlo[rg];
  const int* n = B.rn[rg];
  const long long n01 = (long long)n[0] * n[1];
  const int k = (int)(q / n01);
  const long long r = q - (long long)k * n01;
  const int j = (int)(r / n[0]), i = (int)(r - (long long)j * n[0]);
  return (long long)(i + lo[0]) + (long long)B.b.ex[0] * ((long long)(j + lo[1]) + (long long)B.b.ex[1] * (k + lo[2]));
}

}  // namespace amss
