// amr_types.cuh -- host/device descriptors of the AMR data movement (amr.cuh).
#pragma once
#include "bssn_step.cuh"

namespace amss {

// Per-block buffers as the AMR kernels see them (one table for all levels).
struct AmrBlock {
  int org[3];          // global level index of array element 0
  int ex[3];
  long long fs;
  double* tl[3];       // three time levels of the FP64 state; tl[cur] is current
  void* st[2];         // stage buffers (FP64, or FP32 in the mixed form)
  double* side[2];     // FP64 chi, alpha, beta^i of the stages (mixed form, kSideFields each)
  double* K;           // RK accumulator, reused as the time-interpolated parent state
  const int* lvl;      // level state {cur, steps taken}
  int nf;              // evolved fields: 24 (BSSN) or 25 (Z4c)
};

// A box of work: [lo, lo + n) in global level indices of the destination.
struct AmrBox {
  int dst, src;        // block ids
  int lo[3];
  int n[3];
};

// Work units of the prolongation over a box of fine cells (k_amr_prolong):
// coarse cells c0 .. with a child in the box, pieces of seg - 6 of them along
// x on segments of seg lanes, per_warp segments a warp; `count` units a field.
struct ProlongUnits {
  int c0[3], nc, seg, per_warp, nx, ny, count;
  __host__ __device__ explicit ProlongUnits(const AmrBox& b) {
    int n[3];
    for (int d = 0; d < 3; ++d) {
      c0[d] = b.lo[d] >> 1;
      n[d] = ((b.lo[d] + b.n[d] - 1) >> 1) - c0[d] + 1;
    }
    nc = n[0];
    seg = nc <= 4 ? 10 : (nc <= 10 ? 16 : 32);
    per_warp = 32 / seg;
    nx = (nc + seg - 7) / (seg - 6);
    ny = n[1];
    count = nx * ny * n[2];
  }
};

// Work units of the restriction over a box of coarse cells (k_amr_restrict):
// pieces of 14 cells along x, kRestrictRows rows along y; `count` units a field.
constexpr int kRestrictRows = 4;
struct RestrictUnits {
  int nx, ny, count;
  __host__ __device__ explicit RestrictUnits(const AmrBox& b) {
    nx = (b.n[0] + 13) / 14;
    ny = (b.n[1] + kRestrictRows - 1) / kRestrictRows;
    count = nx * ny * b.n[2];
  }
};

enum AmrBuf : int { BUF_STATE = 0, BUF_STAGE_A = 1, BUF_STAGE_B = 2, BUF_TEMP = 3 };

}  // namespace amss
