// amr.cuh -- device side of the AMR data movement (ghost sync, restriction,
// prolongation, time interpolation) between blocks resident in HBM.
//
// Every operation is a list of boxes in global level indices; a box names a
// destination block and a source block.  Threads are mapped to box points
// through a tile list (128 points per tile), so one launch serves all boxes
// of a level, whatever their sizes.  Each thread moves all nf fields of one
// point.  Nothing here applies enforce_ga: as in the reference, restricted and
// prolonged values are enforced by the pass at the start of the next step.
#pragma once
#include "amr_types.cuh"

namespace amss {

__device__ __forceinline__ long long amr_idx(const AmrBlock& b, int gi, int gj, int gk) {
  return (long long)(gi - b.org[0]) + (long long)b.ex[0] * ((long long)(gj - b.org[1]) + (long long)b.ex[1] * (gk - b.org[2]));
}
__device__ __forceinline__ bool amr_inside(const AmrBlock& b, int gi, int gj, int gk) {
  return gi >= b.org[0] && gi < b.org[0] + b.ex[0] && gj >= b.org[1] && gj < b.org[1] + b.ex[1] &&
         gk >= b.org[2] && gk < b.org[2] + b.ex[2];
}
__device__ __forceinline__ double* amr_state(const AmrBlock& b) { return b.tl[b.lvl[0]]; }

// Copies the n fields of one point: eight loads in flight before their stores
// (the compiler may not move a load past a store it cannot tell apart).  With
// the time interpolation's batches below, the 7-level binary's coarse step
// 276.7 -> 275.5 ms, mixed 206.7 -> 205.7 ms.
template <typename V>
__device__ __forceinline__ void copy_point(V* d, const V* s, long long dfs, long long sfs, int n) {
  for (int f0 = 0; f0 < n; f0 += 8) {
    V v[8];
#pragma unroll
    for (int f = 0; f < 8; ++f)
      if (f0 + f < n) v[f] = s[(f0 + f) * sfs];
#pragma unroll
    for (int f = 0; f < 8; ++f)
      if (f0 + f < n) d[(f0 + f) * dfs] = v[f];
  }
}

// Same-level ghost fill: copy the nf fields of each box point from src to dst.
template <typename SS>
__global__ void k_amr_sync(const AmrBlock* __restrict__ blocks, const AmrBox* __restrict__ boxes,
                           const int2* __restrict__ tiles, int ntiles, int which, unsigned* status) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBox& bx = boxes[tile.x];
    const int p = tile.y + threadIdx.x;
    const int np = bx.n[0] * bx.n[1] * bx.n[2];
    if (p >= np) continue;
    const int gi = bx.lo[0] + p % bx.n[0], gj = bx.lo[1] + (p / bx.n[0]) % bx.n[1], gk = bx.lo[2] + p / (bx.n[0] * bx.n[1]);
    const AmrBlock& D = blocks[bx.dst];
    const AmrBlock& S = blocks[bx.src];
    if (!amr_inside(D, gi, gj, gk) || !amr_inside(S, gi, gj, gk)) { atomicOr(status, ST_BAD_ARG); continue; }
    const long long od = amr_idx(D, gi, gj, gk), os = amr_idx(S, gi, gj, gk);
    if (which == BUF_STATE || which == BUF_TEMP) {
      const double* s = which == BUF_STATE ? amr_state(S) : S.K;
      double* d = which == BUF_STATE ? amr_state(D) : D.K;
      copy_point(d + od, s + os, D.fs, S.fs, D.nf);
    } else {
      const int sl = which == BUF_STAGE_A ? 0 : 1;
      const SS* s = (const SS*)S.st[sl];
      SS* d = (SS*)D.st[sl];
      copy_point(d + od, s + os, D.fs, S.fs, D.nf);
      if constexpr (sizeof(SS) == 4) copy_point(D.side[sl] + od, (const double*)S.side[sl] + os, D.fs, S.fs, kSideFields);
    }
  }
}

// prolongrestrict_cell.f90:1937-1942 and :2350
__device__ __constant__ double kProlongW[6] = {7.7e1 / 8.192e3, -6.93e2 / 8.192e3, 3.465e3 / 4.096e3,
                                               1.155e3 / 4.096e3, -4.95e2 / 8.192e3, 6.3e1 / 8.192e3};

// Fine buffer cells of dst (fine) from the parent level's src block:
// prolong3 (prolongrestrict_cell.f90:1915-2164), z then y then x; g odd is
// the right child of k = g >> 1 (coarse k-2..k+3, weights C1..C6), g even
// the left child (coarse k-3..k+2, weights C6..C1).
//
// The pass is bound by its loads: one thread a run of fine cells read 31
// values a cell from lines of its own (208 us a call of the 48^3 boxes).  A
// lane takes one coarse x column instead, so that a warp's loads are
// consecutive, and the four (y, z) rows of fine cells over one coarse cell
// share the column's 7 x 7 values: it reduces them over z and y for each row;
// the x sums of its coarse cell's children then read the columns of the
// neighbouring lanes by shuffle, in the reference's order of operations.
// 79 us now.  A unit is (field, z pair, y pair, x piece): a segment of
// `seg` lanes, whose inner seg - 6 have children to write.  Boxes a few cells
// wide pack three segments of 10 lanes, or two of 16, into a warp.
__global__ void __launch_bounds__(128) k_amr_prolong(const AmrBlock* __restrict__ blocks,
                                                     const AmrBox* __restrict__ boxes, const int2* __restrict__ tiles,
                                                     int ntiles, int from_temp, unsigned* status) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBox& bx = boxes[tile.x];
    const ProlongUnits U(bx);
    const AmrBlock& D = blocks[bx.dst];
    const AmrBlock& S = blocks[bx.src];
    const int s = lane / U.seg, l = lane - s * U.seg;   // segment of the warp, lane in it
    const int uu = tile.y + warp * U.per_warp + s;
    const bool on = s < U.per_warp && uu < U.count * D.nf;
    const int f = on ? uu / U.count : 0, u = on ? uu - f * U.count : 0;
    const int m0 = U.c0[0] + (u % U.nx) * (U.seg - 6);       // first coarse cell of the piece
    const int cy = U.c0[1] + (u / U.nx) % U.ny, cz = U.c0[2] + u / (U.nx * U.ny);
    const int cx = m0 - 3 + l;                               // this lane's column
    int lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) { lo[d] = bx.lo[d]; hi[d] = bx.lo[d] + bx.n[d]; }
    // which rows and cells exist, and the coarse values they read
    const int mine = m0 + U.seg - 6 < U.c0[0] + U.nc ? m0 + U.seg - 6 : U.c0[0] + U.nc;   // end of the piece
    const int fx0 = 2 * m0 < lo[0] ? lo[0] : 2 * m0, fx1 = 2 * mine < hi[0] ? 2 * mine : hi[0];   // its fine cells
    const bool ye = 2 * cy >= lo[1], yo = 2 * cy + 1 < hi[1], ze = 2 * cz >= lo[2], zo = 2 * cz + 1 < hi[2];
    const int xa = (fx0 & 1) ? (fx0 >> 1) - 2 : (fx0 >> 1) - 3, xb = (fx1 >> 1) + 2;
    const int ra = ye ? 0 : 1, rb = yo ? 6 : 5, qa = ze ? 0 : 1, qb = zo ? 6 : 5;
    bool ok = on;
    if (on && (!amr_inside(D, fx0, ye ? 2 * cy : 2 * cy + 1, ze ? 2 * cz : 2 * cz + 1) ||
               !amr_inside(D, fx1 - 1, yo ? 2 * cy + 1 : 2 * cy, zo ? 2 * cz + 1 : 2 * cz) ||
               !amr_inside(S, xa, cy - 3 + ra, cz - 3 + qa) || !amr_inside(S, xb, cy - 3 + rb, cz - 3 + qb))) {
      atomicOr(status, ST_BAD_ARG);
      ok = false;
    }
    // T[2 zr + yr]: the column reduced over z and y for the row of fine parity (yr, zr)
    double T[4] = {0.0, 0.0, 0.0, 0.0};
    if (ok && cx >= xa && cx <= xb) {
      const double* q = (from_temp ? S.K : amr_state(S)) + f * S.fs + amr_idx(S, cx, cy - 3, cz - 3);
      const long long sy = S.ex[0], sz = (long long)S.ex[0] * S.ex[1];
#pragma unroll
      for (int r = 0; r < 7; ++r) {
        if (r < ra || r > rb) continue;
        double v[7];
#pragma unroll
        for (int m = 0; m < 7; ++m) v[m] = m >= qa && m <= qb ? q[r * sy + m * sz] : 0.0;
        double te = __dmul_rn(kProlongW[5], v[0]), to = __dmul_rn(kProlongW[0], v[1]);
#pragma unroll
        for (int m = 1; m < 6; ++m) {
          te = __dadd_rn(te, __dmul_rn(kProlongW[5 - m], v[m]));
          to = __dadd_rn(to, __dmul_rn(kProlongW[m], v[m + 1]));
        }
        if (r < 6) {   // left child in y: rows 0 .. 5, weights C6 .. C1
          T[0] = r == 0 ? __dmul_rn(kProlongW[5], te) : __dadd_rn(T[0], __dmul_rn(kProlongW[5 - r], te));
          T[2] = r == 0 ? __dmul_rn(kProlongW[5], to) : __dadd_rn(T[2], __dmul_rn(kProlongW[5 - r], to));
        }
        if (r > 0) {   // right child: rows 1 .. 6, weights C1 .. C6
          T[1] = r == 1 ? __dmul_rn(kProlongW[0], te) : __dadd_rn(T[1], __dmul_rn(kProlongW[r - 1], te));
          T[3] = r == 1 ? __dmul_rn(kProlongW[0], to) : __dadd_rn(T[3], __dmul_rn(kProlongW[r - 1], to));
        }
      }
    }
    // x sums of the lane's coarse cell: its children 2 cx and 2 cx + 1
    double* dst = amr_state(D) + f * D.fs;
    const bool wl = ok && l >= 3 && l < U.seg - 3 && 2 * cx >= fx0 && 2 * cx < fx1;
    const bool wr = ok && l >= 3 && l < U.seg - 3 && 2 * cx + 1 >= fx0 && 2 * cx + 1 < fx1;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double vl = 0.0, vr = 0.0;
#pragma unroll
      for (int a = 0; a < 7; ++a) {
        const double c = __shfl_sync(0xffffffffu, T[m], lane - 3 + a);
        if (a < 6) vl = a == 0 ? __dmul_rn(kProlongW[5], c) : __dadd_rn(vl, __dmul_rn(kProlongW[5 - a], c));
        if (a > 0) vr = a == 1 ? __dmul_rn(kProlongW[0], c) : __dadd_rn(vr, __dmul_rn(kProlongW[a - 1], c));
      }
      const bool row = ((m & 1) ? yo : ye) && ((m & 2) ? zo : ze);
      if (row && (wl || wr)) {
        double* o = dst + amr_idx(D, 2 * cx, 2 * cy + (m & 1), 2 * cz + (m >> 1));
        if (wl) o[0] = vl;
        if (wr) o[1] = vr;
      }
    }
  }
}

// Coarse cells of dst (coarse) from fine src: restrict3
// (prolongrestrict_cell.f90:2330-2468): fine 2k-2..2k+3 with weights
// C1 C2 C3 C3 C2 C1, z then y then x.  Writes the current state or the
// time-interpolated temp.
//
// A lane takes one fine x column and kRestrictRows coarse rows along y: it
// reduces the column over z once a fine y row (rows of neighbouring coarse
// cells share four of their six) and over y; every second lane then forms a
// coarse cell's x sum from its own and five neighbouring columns by shuffle,
// in the reference's order.  A thread a cell read 216 values of it, every
// second one of a line (94 us a call of the 48^3 boxes, 33 us now).  A
// unit is (field, z row, group of y rows, piece of 14 coarse cells): one warp.
constexpr int kRestrictCells = 14;   // (32 - 4) / 2 coarse cells a warp
__global__ void __launch_bounds__(128) k_amr_restrict(const AmrBlock* __restrict__ blocks,
                                                      const AmrBox* __restrict__ boxes, const int2* __restrict__ tiles,
                                                      int ntiles, int to_temp, unsigned* status) {
  const double C1 = 3.0 / 2.56e2, C2 = -2.5e1 / 2.56e2, C3 = 7.5e1 / 1.28e2;
  auto sum6 = [&](double a, double b, double c, double d, double e, double g) {
    return __dadd_rn(__dadd_rn(__dmul_rn(C1, __dadd_rn(a, g)), __dmul_rn(C2, __dadd_rn(b, e))),
                     __dmul_rn(C3, __dadd_rn(c, d)));
  };
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBox& bx = boxes[tile.x];
    const AmrBlock& D = blocks[bx.dst];
    const AmrBlock& S = blocks[bx.src];
    const RestrictUnits U(bx);
    const int uu = tile.y + warp;
    if (uu >= U.count * D.nf) continue;   // a whole warp
    const int f = uu / U.count, u = uu - f * U.count;
    const int c0 = bx.lo[0] + (u % U.nx) * kRestrictCells;             // first coarse cell of the piece
    const int y0 = bx.lo[1] + ((u / U.nx) % U.ny) * kRestrictRows, z = bx.lo[2] + u / (U.nx * U.ny);
    const int nc = c0 + kRestrictCells < bx.lo[0] + bx.n[0] ? kRestrictCells : bx.lo[0] + bx.n[0] - c0;
    const int nr = y0 + kRestrictRows < bx.lo[1] + bx.n[1] ? kRestrictRows : bx.lo[1] + bx.n[1] - y0;
    if (!amr_inside(D, c0, y0, z) || !amr_inside(D, c0 + nc - 1, y0 + nr - 1, z) ||
        !amr_inside(S, 2 * c0 - 2, 2 * y0 - 2, 2 * z - 2) ||
        !amr_inside(S, 2 * (c0 + nc - 1) + 3, 2 * (y0 + nr - 1) + 3, 2 * z + 3)) {
      if (lane == 0) atomicOr(status, ST_BAD_ARG);
      continue;
    }
    const long long sy = S.ex[0], sz = (long long)S.ex[0] * S.ex[1];
    const bool col = lane < 2 * nc + 4;   // this lane's fine column 2 c0 - 2 + lane is read
    const double* q = amr_state(S) + f * S.fs + amr_idx(S, 2 * c0 - 2 + (col ? lane : 0), 2 * y0 - 2, 2 * z - 2);
    double w[6];   // z sums of fine y rows 2 y - 2 .. 2 y + 3 of the current coarse row
    auto zsum = [&](int r) {
      const double* p = q + r * sy;
      return sum6(p[0], p[sz], p[2 * sz], p[3 * sz], p[4 * sz], p[5 * sz]);
    };
#pragma unroll
    for (int r = 0; r < 4; ++r) w[r + 2] = zsum(r);
    double* dst = (to_temp ? D.K : amr_state(D)) + f * D.fs;
#pragma unroll
    for (int y = 0; y < kRestrictRows; ++y) {
      if (y >= nr) break;   // the same in the whole warp
#pragma unroll
      for (int r = 0; r < 4; ++r) w[r] = w[r + 2];
      w[4] = zsum(2 * y + 4);
      w[5] = zsum(2 * y + 5);
      const double T = sum6(w[0], w[1], w[2], w[3], w[4], w[5]);
      double x[6];
#pragma unroll
      for (int a = 0; a < 6; ++a) x[a] = __shfl_sync(0xffffffffu, T, lane + a);
      if ((lane & 1) == 0 && lane / 2 < nc) dst[amr_idx(D, c0 + lane / 2, y0 + y, z)] = sum6(x[0], x[1], x[2], x[3], x[4], x[5]);
    }
  }
}

// Parent state at the child's intermediate time into K (prepare_inter_time_level,
// Parallel.C:4329-4441): average2 (fmisc.f90:1569-1592, 3/8 new + 3/4 old
// - 1/8 older) once the level has two steps behind it, else average
// (fmisc.f90:1532, (new + old)/2), at array point p of block B.
__device__ __forceinline__ void timeinterp_point(const AmrBlock& B, long long p) {
  const int cur = B.lvl[0];
  const double* f1 = B.tl[cur];
  const double* f2 = B.tl[(cur + 2) % 3];
  const double* f3 = B.tl[(cur + 1) % 3];
  const bool second = B.lvl[1] >= 2;
  const double C1 = 3.0 / 8.0, C2 = 3.0 / 4.0, C3 = -1.0 / 8.0;
  // four fields' loads in flight before their stores
  for (int f0 = 0; f0 < B.nf; f0 += 4) {
    double v1[4], v2[4], v3[4];
#pragma unroll
    for (int f = 0; f < 4; ++f)
      if (f0 + f < B.nf) {
        const long long o = (f0 + f) * B.fs + p;
        v1[f] = f1[o];
        v2[f] = f2[o];
        v3[f] = second ? f3[o] : 0.0;
      }
#pragma unroll
    for (int f = 0; f < 4; ++f)
      if (f0 + f < B.nf)
        B.K[(f0 + f) * B.fs + p] =
            second ? __dadd_rn(__dadd_rn(__dmul_rn(C1, v1[f]), __dmul_rn(C2, v2[f])), __dmul_rn(C3, v3[f]))
                   : __dmul_rn(0.5, __dadd_rn(v1[f], v2[f]));
  }
}

// Over every point of a level's blocks: one thread per block point.
__global__ void k_amr_timeinterp(const AmrBlock* __restrict__ blocks, const int2* __restrict__ tiles, int ntiles) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBlock& B = blocks[tile.x];
    const long long p = (long long)tile.y + threadIdx.x;
    const long long np = (long long)B.ex[0] * B.ex[1] * B.ex[2];
    if (p >= np) continue;
    timeinterp_point(B, p);
  }
}

// Over boxes of cells (dst = the block; the cells a finer level's
// prolongation reads from it): one thread per box cell.
__global__ void k_amr_timeinterp_boxes(const AmrBlock* __restrict__ blocks, const AmrBox* __restrict__ boxes,
                                       const int2* __restrict__ tiles, int ntiles, unsigned* status) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBox& bx = boxes[tile.x];
    const int q = tile.y + threadIdx.x;
    if (q >= bx.n[0] * bx.n[1] * bx.n[2]) continue;
    const AmrBlock& B = blocks[bx.dst];
    const int x = bx.lo[0] + q % bx.n[0], y = bx.lo[1] + (q / bx.n[0]) % bx.n[1], z = bx.lo[2] + q / (bx.n[0] * bx.n[1]);
    if (!amr_inside(B, x, y, z)) {
      atomicOr(status, ST_BAD_ARG);
      continue;
    }
    timeinterp_point(B, amr_idx(B, x, y, z));
  }
}

// enforce_ga in place on the current state of every block of a level, as the
// reference does on StateList at the start of each level step
// (bssn_class.C:3052).  One thread per block point.
__global__ void k_amr_enforce(const AmrBlock* __restrict__ blocks, const int2* __restrict__ tiles, int ntiles) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int2 tile = tiles[t];
    const AmrBlock& B = blocks[tile.x];
    const long long p = (long long)tile.y + threadIdx.x;
    const long long np = (long long)B.ex[0] * B.ex[1] * B.ex[2];
    if (p >= np) continue;
    double* u = B.tl[B.lvl[0]];
    double g[6], a[6];
    for (int m = 0; m < 6; ++m) { g[m] = u[(F_GXX + m) * B.fs + p]; a[m] = u[(F_AXX + m) * B.fs + p]; }
    enforce_ga_point(g, a);
    for (int m = 0; m < 6; ++m) { u[(F_GXX + m) * B.fs + p] = g[m]; u[(F_AXX + m) * B.fs + p] = a[m]; }
  }
}

// Advance a level's time-level ring and step counter.
__global__ void k_amr_rotate(int* lvl) {
  lvl[0] = (lvl[0] + 1) % 3;
  lvl[1] = lvl[1] + 1;
}

}  // namespace amss
