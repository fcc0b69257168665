// pointwise.cuh -- the pointwise pass of the split RK4 substep: the
// right-hand side of every point from its centre values and the stencil terms
// D that the stencil pass (deriv.cuh) stored, and the RK4 update.
//
// The pass streams 1.7 KB a point (FP64) through about 3,600 instructions
// that hold 250 registers, so only eight warps fit an SM and a load that a
// warp waits for costs it hundreds of cycles: with one load per use the pass
// spent 60,000 cycles on a 128-point tile, 12 % of them issuing (282 us on
// 70^3 points, 28 % of DRAM bandwidth).  Each warp therefore copies the rows
// of its 32 points into a shared-memory region of its own, with cp.async and
// several groups ahead of their use (25 KB a warp, 200 KB of an SM), and the
// point function reads shared memory: 160-173 us on 70^3 points, 3.4-3.9 TB/s; Z4c on
// 134^3 points 2,103 -> 1,110 us; the mixed form on 70^3 points 205 -> 120 us.
// No CTA barrier: a warp waits for its own copies only.  What remains is the
// latency of dependent FP64 operations at two warps a scheduler.
//
// The point function uses its inputs in nine phases (phase<N> in
// bssn_rhs.cuh).  A phase's rows are copied as one group into a fixed slot of
// the region; four of the phases reuse a slot once its first phase is done:
//
//   slot 0: phase 0 (centre values), then 4, then 8
//   slot 1: phase 1, then 5         slot 2: phases 2 and 3, then 6
//   slot 3: phase 7
//
// D's rows are in the order the phases use them (dl::g, dl::h, dl::a), so
// that a phase's terms are one run of rows: 16 bytes a lane, two (FP64) or
// four (FP32) rows an instruction.
#pragma once
#include "substep_common.cuh"

namespace amss {

template <typename T, typename SI, bool Z4C>
struct PwStage {
  static constexpr int kNf = Z4C ? NFIELDS_Z4C : NFIELDS_BSSN;
  // The centre values are staged where they need no conversion; the mixed
  // form's FP64 state (substep 0) is read directly, which keeps the region
  // small enough for three CTAs an SM.
  static constexpr bool kCentre = sizeof(SI) == sizeof(T);
  static constexpr int kRow = 32 * sizeof(T);   // bytes of a D row of a warp
  static constexpr int kRow8 = 256;             // of a row of FP64 values

  // fields each phase finishes: their state (u0) and accumulator (K) rows
  static constexpr int nput(int ph) { return ph == 1 ? 5 : ph == 3 ? 6 : ph == 5 ? 6 : ph == 8 ? (Z4C ? 8 : 7) : 0; }
  static constexpr int put_field(int ph, int i) {
    constexpr int p1[5] = {F_CHI, F_LAP, F_BETAX, F_BETAY, F_BETAZ};
    constexpr int p5[6] = {F_GAMX, F_GAMY, F_GAMZ, F_DTSFX, F_DTSFY, F_DTSFZ};
    constexpr int p8[8] = {F_AXX, F_AXY, F_AXZ, F_AYY, F_AYZ, F_AZZ, F_TRK, F_TZ};
    return ph == 1 ? p1[i] : ph == 3 ? F_GXX + i : ph == 5 ? p5[i] : p8[i];
  }
  static constexpr int put_phase(int F) {
    for (int ph = 1; ph <= 8; ++ph)
      for (int i = 0; i < nput(ph); ++i)
        if (put_field(ph, i) == F) return ph;
    return -1;
  }
  static constexpr int put_index(int F) {
    const int ph = put_phase(F);
    for (int i = 0; i < nput(ph); ++i)
      if (put_field(ph, i) == F) return i;
    return -1;
  }
  // D rows of a phase: [d0, d0 + nd), and Theta's (Z4c: rows 135 .. 138)
  static constexpr int d0(int ph) { return dl::first(ph); }
  static constexpr int nd(int ph) { return dl::first(ph + 1) - dl::first(ph); }
  static constexpr int dz0(int ph) { return ph == 4 ? dl::kTheta : dl::kTheta + 3; }
  static constexpr int ndz(int ph) { return !Z4C ? 0 : ph == 4 ? 3 : ph == 8 ? 1 : 0; }

  static constexpr int centre_bytes() {
    if (!kCentre) return 0;
    int n = 0;
    for (int F = 0; F < kNf; ++F) n += sizeof(SI) == 4 && !is_wide(F) ? 128 : kRow8;
    return n;
  }
  static constexpr int bytes(int ph) { return ph == 0 ? centre_bytes() : (nd(ph) + ndz(ph)) * kRow + 2 * nput(ph) * kRow8; }
  static constexpr int max3(int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }
  static constexpr int kSlot1 = max3(bytes(0), bytes(4), bytes(8));
  static constexpr int kSlot2 = kSlot1 + max3(bytes(1), bytes(5), 0);
  static constexpr int kSlot3 = kSlot2 + max3(bytes(2) + bytes(3), bytes(6), 0);
  static constexpr int kWarp = kSlot3 + bytes(7);   // bytes of a warp's region
  static constexpr int start(int ph) {
    return ph == 1 || ph == 5 ? kSlot1
                              : ph == 2 || ph == 6 ? kSlot2 : ph == 3 ? kSlot2 + bytes(2) : ph == 7 ? kSlot3 : 0;
  }
  static_assert(kWarp % 16 == 0, "rows are copied 16 bytes at a time");

  // byte offsets in the region (of lane 0)
  static constexpr int off_c(int F) {
    int o = start(0);
    for (int f = 0; f < F; ++f) o += sizeof(SI) == 4 && !is_wide(f) ? 128 : kRow8;
    return o;
  }
  static constexpr int off_d(int row) {
    if (row >= dl::kTheta) {
      const int ph = row < dl::kTheta + 3 ? 4 : 8;
      return start(ph) + (nd(ph) + row - dz0(ph)) * kRow;
    }
    int ph = 1;
    while (dl::first(ph + 1) <= row) ++ph;
    return start(ph) + (row - d0(ph)) * kRow;
  }
  static constexpr int off_u(int F) {
    const int ph = put_phase(F);
    return start(ph) + (nd(ph) + ndz(ph)) * kRow + put_index(F) * kRow8;
  }
  static constexpr int off_k(int F) { return off_u(F) + nput(put_phase(F)) * kRow8; }
};

__device__ __forceinline__ void cp_async16(unsigned sdst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sdst), "l"(gsrc) : "memory");
}

// Accessor of the pointwise pass over a warp's staged rows.
template <typename T, typename SI, bool Z4C>
struct StagedPt {
  static constexpr bool kPre = true;
  using S = PwStage<T, SI, Z4C>;
  const unsigned char* reg;     // the warp's region
  unsigned sreg;                // its shared-memory address
  int lane;
  const T* drow0;               // D of the tile, at this warp's 32 points: row r at + r * kDTile
  const SI* in;                 // stage input, at the point
  const double* in_side;        // FP64 side slots of an FP32 stage input, at the point
  const double* u0;             // state at t_n, at the point
  const double* K;              // accumulator, at the point
  long long fs, p;
  int sub;

  // copies the rows of phase PH into its slot, as one group
  template <int PH>
  __device__ __forceinline__ void issue() const {
    if constexpr (PH == 0) {
      if constexpr (S::kCentre) {
#pragma unroll
        for (int F = 0; F < S::kNf; ++F) {
          if constexpr (sizeof(SI) == 8) cp_async8(sreg + S::off_c(F) + lane * 8, in + F * fs);
          else if (is_wide(F)) cp_async8(sreg + S::off_c(F) + lane * 8, in_side + side_slot(F) * fs);
          else cp_async4(sreg + S::off_c(F) + lane * 4, in + F * fs);
        }
      }
    } else {
      copy_rows<S::nd(PH)>(S::d0(PH), S::start(PH));
      if constexpr (S::ndz(PH) > 0) copy_rows<S::ndz(PH)>(S::dz0(PH), S::start(PH) + S::nd(PH) * S::kRow);
#pragma unroll
      for (int i = 0; i < S::nput(PH); ++i) {
        const int F = S::put_field(PH, i);
        cp_async8(sreg + S::start(PH) + (S::nd(PH) + S::ndz(PH)) * S::kRow + i * S::kRow8 + lane * 8, u0 + F * fs);
      }
      if (S::nput(PH) > 0 && sub != 0) {
#pragma unroll
        for (int i = 0; i < S::nput(PH); ++i) {
          const int F = S::put_field(PH, i);
          cp_async8(sreg + S::start(PH) + (S::nd(PH) + S::ndz(PH)) * S::kRow + (S::nput(PH) + i) * S::kRow8 + lane * 8,
                       K + F * fs);
        }
      }
    }
    cp_async_commit();
  }
  template <int N>
  __device__ __forceinline__ void copy_rows(int row0, int off) const {
    constexpr int kLpr = S::kRow / 16, kPer = 32 / kLpr;   // lanes a row, rows an instruction
    const int h = lane / kLpr, c = lane % kLpr;
    const unsigned char* g = (const unsigned char*)(drow0 + (long long)(row0 + h) * kDTile) + c * 16;
    const unsigned s = sreg + off + h * S::kRow + c * 16;
#pragma unroll
    for (int r = 0; r < N; r += kPer)
      if (r + kPer <= N || r + h < N) cp_async16(s + r * S::kRow, g + r * kDTile * sizeof(T));
  }
  // the region's phases in order: what may be issued once phase PH - 1 is
  // done (every lane has read its rows: the warp syncs first), then the wait
  // for PH's own group, counted in groups issued after it
  template <int PH>
  __device__ __forceinline__ void phase() const {
    __syncwarp();
    if constexpr (PH == 0) {
      issue<0>(); issue<1>(); issue<2>(); issue<3>(); issue<7>();
      cp_async_wait<4>();
    }
    if constexpr (PH == 1) { issue<4>(); cp_async_wait<4>(); }
    if constexpr (PH == 2) { issue<5>(); cp_async_wait<4>(); }
    if constexpr (PH == 3) cp_async_wait<3>();
    if constexpr (PH == 4) { issue<6>(); cp_async_wait<2>(); }
    if constexpr (PH == 5) { issue<8>(); cp_async_wait<2>(); }
    if constexpr (PH == 6) cp_async_wait<1>();   // and with it phase 7's rows
    if constexpr (PH == 8) cp_async_wait<0>();
    __syncwarp();   // the copies of every lane are seen by every lane
  }

  template <typename U, int F>
  __device__ __forceinline__ U v(int, int, int) const {   // centre values only
    if constexpr (!S::kCentre) return (U)__ldg(in + F * fs);
    else if constexpr (sizeof(SI) == 4 && !is_wide(F)) return (U)*(const float*)(reg + S::off_c(F) + lane * 4);
    else return (U)*(const double*)(reg + S::off_c(F) + lane * 8);
  }
  template <typename U, int SLOT>
  __device__ __forceinline__ U dv() const {
    constexpr int o = S::off_d(dl::row(SLOT));
    return (U)*(const T*)(reg + o + lane * (int)sizeof(T));
  }
};

// RK4 epilogue over a warp's staged rows: EpiRK with u0 and K from the region.
// An inactive lane (past the tile's points, or an outer face) stores nothing.
template <typename T, typename SI, typename SO, bool Z4C>
struct StagedRK {
  using S = PwStage<T, SI, Z4C>;
  const unsigned char* reg;
  int lane;
  double* K;          // at the point
  SO* out;
  double* out_side;
  long long fs;
  int sub;
  bool enforce, act;
  RKConst c;
  double g[6], a[6];

  template <int F>
  __device__ __forceinline__ void put(T kv) {
    const double k = (double)kv;
    const double u = *(const double*)(reg + S::off_u(F) + lane * 8);
    double r;
    if (sub == 0) {
      r = u + c.half_dt * k;
      if (act) K[F * fs] = k;
    } else {
      const double kk = *(const double*)(reg + S::off_k(F) + lane * 8);
      if (sub == 3) {
        r = u + c.sixth_dt * (k + kk);
      } else {
        if (act) K[F * fs] = kk + 2.0 * k;
        r = sub == 1 ? u + c.half_dt * k : u + c.dt * k;
      }
    }
    if constexpr (F == F_CHI) {
      if (r < c.chitiny) r = c.chitiny;
    }
    if constexpr (F >= F_GXX && F <= F_GZZ) g[F - F_GXX] = r;
    else if constexpr (F >= F_AXX && F <= F_AZZ) a[F - F_AXX] = r;
    else if (act) {
      if constexpr (sizeof(SO) == 4 && is_wide(F)) out_side[side_slot(F) * fs] = r;
      else out[F * fs] = (SO)r;
    }
  }
  __device__ __forceinline__ void finish() {
    if (enforce) enforce_ga_point(g, a);
    if (!act) return;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      out[(F_GXX + m) * fs] = (SO)g[m];
      out[(F_AXX + m) * fs] = (SO)a[m];
    }
  }
};

// CTAs of 128 threads an SM: FP64 takes 250 registers, FP32 fits 168
template <typename T>
constexpr int kPwResident = sizeof(T) == 4 ? 3 : 2;

// Substep `sub` over a tile list of one level: reads (sub0: u0, sub1: A,
// sub2: B, sub3: A), writes (A, B, A, unew).
template <typename T, typename SI, typename SO, bool Z4C>
__global__ void __launch_bounds__(kPointwiseTile, kPwResident<T>)
k_pointwise(const StepBlock<T>* __restrict__ blocks, const int2* __restrict__ tiles, int sub, RKConst rk, int enforce,
            unsigned* status, const T* __restrict__ D) {
  using S = PwStage<T, SI, Z4C>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  constexpr int kSlots = Z4C ? D_SLOTS_Z4C : D_SLOTS;
  // a CTA a tile, its four warps on their own: a grid of eight CTAs an SM that
  // loops over the tiles took 342 us longer on 134^3 points (Z4c), two resident
  // CTAs looping with the next tile prefetched into L2 261 us longer, and CTAs
  // of one or two warps 430 and 330 us longer
  const int2 tile = tiles[blockIdx.x];
  const int region = tile_region(tile.x);
  const StepBlock<T>& B = blocks[tile.x & kTileIndex];
  const long long q0 = (long long)tile.y + warp * 32;
  if (q0 >= tile_count(B, region)) return;   // no point of this warp
  const long long pt = tile_point(B, region, q0 + lane);
  const long long p = pt >= 0 ? pt : tile_point(B, region, q0);
  int i, j, k;
  point_ijk(p, B.b.ex, i, j, k);
  const int fm = B.b.face_mask;
  // outer-face points are updated by k_face (a separate list)
  const bool on_face = ((fm & 1) && i == B.b.ex[0] - 1) || ((fm & 2) && j == B.b.ex[1] - 1) ||
                       ((fm & 4) && k == B.b.ex[2] - 1) || ((fm & 8) && i == 0) || ((fm & 16) && j == 0) ||
                       ((fm & 32) && k == 0);
  const int cur = B.lvl[0];
  const long long fs = B.b.fs;
  StagedPt<T, SI, Z4C> q;
  q.reg = smem + warp * S::kWarp;
  q.sreg = (unsigned)__cvta_generic_to_shared(q.reg);
  q.lane = lane;
  q.drow0 = D + (long long)(B.dtile + tile.y / kDTile) * (kSlots * kDTile) + warp * 32;
  q.u0 = B.tl[cur] + p;
  q.in = sub == 0 ? (const SI*)B.tl[cur] + p : (const SI*)B.stage[sub == 2 ? 1 : 0] + p;
  q.in_side = sub == 0 ? nullptr : B.side[sub == 2 ? 1 : 0] + p;
  q.K = B.K + p;
  q.fs = fs;
  q.p = p;
  q.sub = sub;
  StagedRK<T, SI, SO, Z4C> epi;
  epi.reg = q.reg;
  epi.lane = lane;
  epi.K = B.K + p;
  epi.out = sub == 3 ? (SO*)B.tl[(cur + 1) % 3] + p : (SO*)B.stage[sub == 1 ? 1 : 0] + p;
  epi.out_side = sub == 3 ? nullptr : B.side[sub == 1 ? 1 : 0] + p;
  epi.fs = fs;
  epi.sub = sub;
  epi.enforce = enforce != 0;
  epi.act = pt >= 0 && !on_face;
  epi.c = rk;
  const PointGates G{};   // the stencil terms are formed already
  const RhsAux aux{};
  const unsigned st = bssn_rhs_point<T, SI, false, false, Z4C>(q, B.C, G, aux, epi);
  if (st && epi.act) atomicOr(status, st);
}

template <typename T, typename SI, typename SO, bool Z4C>
cudaError_t launch_pointwise_as(const void* blocks, const int2* tiles, int ntiles, int sub, RKConst rk, int enforce,
                                unsigned* status, cudaStream_t s, const void* D) {
  constexpr int smem = PwStage<T, SI, Z4C>::kWarp * (kPointwiseTile / 32);
  const cudaError_t e =
      cudaFuncSetAttribute(k_pointwise<T, SI, SO, Z4C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  k_pointwise<T, SI, SO, Z4C><<<ntiles, kPointwiseTile, smem, s>>>((const StepBlock<T>*)blocks, tiles, sub, rk,
                                                                   enforce, status, (const T*)D);
  return cudaGetLastError();
}

template <typename T, typename SS, bool Z4C>
cudaError_t launch_pointwise(const void* blocks, const int2* tiles, int ntiles, int sub, RKConst rk, int enforce,
                             unsigned* status, cudaStream_t s, const void* D) {
  if (sub == 0)
    return launch_pointwise_as<T, double, SS, Z4C>(blocks, tiles, ntiles, sub, rk, enforce, status, s, D);
  if (sub == 3)
    return launch_pointwise_as<T, SS, double, Z4C>(blocks, tiles, ntiles, sub, rk, enforce, status, s, D);
  return launch_pointwise_as<T, SS, SS, Z4C>(blocks, tiles, ntiles, sub, rk, enforce, status, s, D);
}

}  // namespace amss
