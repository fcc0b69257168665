// substep_impl.cuh -- the fused RK4 substep kernel template and its launcher,
// and the drop-in right-hand sides.  Instantiated in one translation unit per
// (precision, symmetry) pair so the large kernels compile in parallel.
#pragma once
#include "substep_common.cuh"

#ifndef AMSS_SUBSTEP_MINB   // resident CTAs of 128 threads the kernel is compiled for
#define AMSS_SUBSTEP_MINB 2
#endif
#ifndef AMSS_SUBSTEP_MINB_F32   // the same for FP32 arithmetic (fits 168 registers without spills)
#define AMSS_SUBSTEP_MINB_F32 3
#endif

namespace amss {

// Fused RK4 substep over a tile list of one level, every stencil evaluated
// from global memory.  Substep `sub` reads (sub0: u0, sub1: A, sub2: B,
// sub3: A) and writes (A, B, A, unew).
template <typename T, typename SI, typename SO, bool SYMM>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? AMSS_SUBSTEP_MINB_F32 : AMSS_SUBSTEP_MINB) k_substep(
    const StepBlock<T>* __restrict__ blocks, const int2* __restrict__ tiles, int ntiles, int sub, RKConst rk,
    int enforce, unsigned* status) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const int region = tile_region(tile.x);
    const StepBlock<T>& B = blocks[tile.x & kTileIndex];
    const long long p = tile_point(B, region, (long long)tile.y + threadIdx.x);
    if (p < 0) continue;
    const int cur = B.lvl[0];
    double* u0 = B.tl[cur];
    const SI* in = sub == 0 ? (const SI*)u0 : (const SI*)B.stage[sub == 2 ? 1 : 0];
    SO* out = sub == 3 ? (SO*)B.tl[(cur + 1) % 3] : (SO*)B.stage[sub == 1 ? 1 : 0];
    const double* in_side = sub == 0 ? nullptr : B.side[sub == 2 ? 1 : 0];
    auto q = make_pt<SI, SYMM>(in, B.b, p, in_side);
    EpiRK<T, SO> epi;
    epi.out_side = sub == 3 ? nullptr : B.side[sub == 1 ? 1 : 0];
    epi.u0 = u0;
    epi.K = B.K;
    epi.out = out;
    epi.fs = B.b.fs;
    epi.p = p;
    epi.sub = sub;
    epi.enforce = enforce != 0;
    epi.c = rk;
    const int fm = B.b.face_mask;
    const bool on_face = ((fm & 1) && q.i == q.ex0 - 1) || ((fm & 2) && q.j == q.ex1 - 1) ||
                         ((fm & 4) && q.k == q.ex2 - 1) || ((fm & 8) && q.i == 0) || ((fm & 16) && q.j == 0) ||
                         ((fm & 32) && q.k == 0);
    // outer-face points are updated by k_face (a separate list), so no warp
    // here carries the Sommerfeld path for a few of its lanes
    if (on_face) continue;
    unsigned st;
    const PointGates G = point_gates(B.b, q.i, q.j, q.k);
    RhsAux aux{};
    st = bssn_rhs_point<T, SI, SYMM, false>(q, B.C, G, aux, epi);
    if (st) atomicOr(status, st);
  }
}

template <typename T, typename SS, bool SYMM>
cudaError_t launch_substep(const void* blocks, const int2* tiles, int ntiles, int sub, RKConst rk, int enforce,
                           unsigned* status, int grid, cudaStream_t s) {
  const StepBlock<T>* bl = (const StepBlock<T>*)blocks;
  if (sub == 0)
    k_substep<T, double, SS, SYMM><<<grid, 128, 0, s>>>(bl, tiles, ntiles, sub, rk, enforce, status);
  else if (sub == 3)
    k_substep<T, SS, double, SYMM><<<grid, 128, 0, s>>>(bl, tiles, ntiles, sub, rk, enforce, status);
  else
    k_substep<T, SS, SS, SYMM><<<grid, 128, 0, s>>>(bl, tiles, ntiles, sub, rk, enforce, status);
  return cudaGetLastError();
}

// Drop-in RHS: all points of one block, RHS plus the diagnostic outputs.
template <bool SYMM>
__global__ void __launch_bounds__(128) k_rhs_dropin(BlockView b, Coefs<double> C, const double* __restrict__ u,
                                                    double* __restrict__ rhs, RhsAux aux, unsigned* status) {
  const long long n = (long long)b.ex[0] * b.ex[1] * b.ex[2];
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    auto q = make_pt<double, SYMM>(u, b, p);
    const PointGates G = point_gates(b, q.i, q.j, q.k);
    EpiStore<double> epi{rhs, b.fs, p};
    const unsigned st = bssn_rhs_point<double, double, SYMM, true>(q, C, G, aux, epi);
    if (st) atomicOr(status, st);
  }
}

template <bool SYMM>
cudaError_t launch_rhs_dropin(int grid, cudaStream_t s, BlockView b, Coefs<double> C, const double* u, double* rhs,
                              RhsAux aux, unsigned* status) {
  k_rhs_dropin<SYMM><<<grid, 128, 0, s>>>(b, C, u, rhs, aux, status);
  return cudaGetLastError();
}

// Drop-in Z4c RHS: all points of one block, the 25 right-hand sides (the
// diagnostic outputs come from k_rhs_dropin, as ricci_gamma + constraint_bssn
// evaluate the BSSN formulas).
template <bool SYMM>
__global__ void __launch_bounds__(128) k_rhs_dropin_z4c(BlockView b, Coefs<double> C, const double* __restrict__ u,
                                                        double* __restrict__ rhs, const double* matter,
                                                        unsigned* status) {
  const long long n = (long long)b.ex[0] * b.ex[1] * b.ex[2];
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x) {
    auto q = make_pt<double, SYMM>(u, b, p);
    const PointGates G = point_gates(b, q.i, q.j, q.k);
    EpiStore<double> epi{rhs, b.fs, p};
    RhsAux aux{};
    aux.matter = matter;
    aux.fs = b.fs;
    const unsigned st = bssn_rhs_point<double, double, SYMM, false, true>(q, C, G, aux, epi);
    if (st) atomicOr(status, st);
  }
}

template <bool SYMM>
cudaError_t launch_rhs_dropin_z4c(int grid, cudaStream_t s, BlockView b, Coefs<double> C, const double* u,
                                  double* rhs, const double* matter, unsigned* status) {
  k_rhs_dropin_z4c<SYMM><<<grid, 128, 0, s>>>(b, C, u, rhs, matter, status);
  return cudaGetLastError();
}

}  // namespace amss
