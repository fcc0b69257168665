// deriv.cuh -- the stencil pass of the split RK4 substep.
//
// One CTA takes one field of one (x, y) tile of a block and marches through z,
// over the planes [k0, k1) of a z-slab.  A thread owns two columns, adjacent
// in y.  Planes of the tile lie in a shared-memory ring with a 3-cell halo,
// filled as the reference's padded copy fh of symmetry_bd (fmisc.f90:877-901):
// cells at negative indices hold the mirrored value times the field's parity,
// cells past the block end are never read by the gated stencils and hold 0.
// x-, y- and z-lines and the xy cross stencil read the ring.  The mixed
// derivatives with z are Dz(Dx f) and Dz(Dy f) -- the reference's 16-point
// cross stencils of fdderivs are exactly these tensor products of its 1-D
// stencils, so only the rounding of the coefficient product differs -- over
// register windows of Dx f and Dy f at planes k-4 .. k, and are stored two
// planes late, so that each is formed once.
//
// The pass is bound by instruction issue (43 % of the cycles) and latency, not
// by memory (417 MB in 268 us on 70^3 points), and most of what it issues is
// not arithmetic (2,100 of 10,200 thread instructions a point were FP64 in the
// 291 us form below), so the layout serves those: two columns a thread share the row differences of the
// cross stencil, the y-line, and a step's barrier, gates and addresses; the
// row stride is a constant, so that a stencil's reads differ by immediates;
// the shift comes through shared memory two planes ahead, the coefficients
// from shared memory; stencils that do not fit are chosen by selects or, for
// the 2nd-order ones next to an edge, stored over the 4th-order ones; points
// that are not the thread's to store go to a spare tile, so that the step is
// straight-line code; what the march needs of the block is in registers, as
// its waits would have it read again.  One column a thread with a register
// column and per-stencil branches, 35 x 7 tiles and whole-block marches took
// 359 us (mixed 293 us, 196 us now), two columns with branches for the points'
// stores and the block read again 291 us (mixed 226 us).  A second, full-width
// path beside the gated one took 22 % fewer instructions and was slower where
// tiles hold many edge points (134^3 Z4c +9 %): its warps wait for the others
// at the plane's barrier.
//
// The planes are copied by cp.async into a ring of nine (k-3 .. k+3 in use, k+4
// landing, k+5 issued), one barrier a plane.  A source that needs conversion
// (the mixed form's FP64 state at substep 0) lands in a buffer of its own and
// is converted by the thread that copied it.
//
// Per point the pass stores, for the field's kind (stencil.cuh: dslots):
// gradient, Hessian, and one "adv" value = upwinded advection
// (lopsidediff.f90:321-481) + eps/64 * KO line sums (kodiss.f90:190-207).
// The formulas and gates are those of diff_new.f90:946-1528.
#pragma once
#include <vector>

#include "bssn_step.cuh"

namespace amss {

constexpr int DTHREADS = 256;
constexpr int DWMAX = 38;                   // widest tile
constexpr int DHMAX = 18;                   // highest tile
constexpr int DS = DWMAX + 6;               // row stride of a plane in shared memory
constexpr int DPLANE = DS * (DHMAX + 6);    // a plane's slot in the ring
constexpr int DRING = 9;                    // planes k-3 .. k+3 in use, k+4 landing, k+5 issued
constexpr int DBETA = 3;                    // planes of the shift: k in use, k+1 landing, k+2 issued
constexpr int DPER = 4;                     // plane cells a thread copies (deriv_cells_fit)
// Shared memory: the ring in the widest arithmetic type, which also covers the
// FP32 ring and its landing planes, then the shift, then the block's stencil
// coefficients (in registers they spill, from global memory they are waited
// for).  Two CTAs an SM.
constexpr size_t kDerivRing = (size_t)DRING * DPLANE * sizeof(double);
constexpr size_t kDerivCoef = kDerivRing + (size_t)DBETA * 6 * DTHREADS * sizeof(double);
constexpr size_t kDerivSmem = kDerivCoef + sizeof(Coef<double>);
static_assert((size_t)DRING * DPLANE * 4 + 2 * DPER * DTHREADS * sizeof(double) <= kDerivRing, "landing planes");
static_assert(2 * (kDerivSmem + 1024) <= 228 * 1024, "two CTAs an SM");
constexpr int kDerivMinEx = 8;              // the split form needs blocks at least this wide in x
constexpr int kPointwiseTile = kDTile;      // points of a tile of the pointwise pass
constexpr int kMinSlab = 8;                 // fewest planes of a z-slab that is asked for
constexpr int kAutoSlab = 4;                // and of one that deriv_slabs chooses
constexpr int kMaxTileW = 64;               // widest tile amss_engine_set_level_tiling takes (used up to DWMAX)

// Tile of a region n0 x n1 columns wide: width w (at most wmax) and height h
// (even, two rows a thread), cutting the region into near-equal tiles of at
// most DTHREADS column pairs.
struct DerivTile { int w, h; };
__host__ __device__ constexpr DerivTile deriv_tile(int n0, int n1, int wmax) {
  const int wm = wmax < DWMAX ? wmax : DWMAX;
  const int nx = (n0 + wm - 1) / wm, w = (n0 + nx - 1) / nx;
  const int hm = 2 * (DTHREADS / w) < DHMAX ? 2 * (DTHREADS / w) : DHMAX;
  const int ny = (n1 + hm - 1) / hm;
  return DerivTile{w, 2 * ((n1 + 2 * ny - 1) / (2 * ny))};
}
constexpr bool deriv_cells_fit() {
  for (int w = 1; w <= DWMAX; ++w) {
    const int hm = 2 * (DTHREADS / w) < DHMAX ? 2 * (DTHREADS / w) : DHMAX;
    if ((w + 6) * (hm + 6) > DPER * DTHREADS || w * (hm / 2) > DTHREADS) return false;
  }
  return true;
}
static_assert(deriv_cells_fit(), "a tile has more cells or columns than its threads take");

struct DerivItem {
  int block;           // index into the level's StepBlock table
  int x0, y0;          // tile origin (array indices)
  int field;
  int k0, k1;          // planes [k0, k1)
  int x1, y1;          // columns x < x1, y < y1 only
  int w, h;            // tile
};

// Appends the work items (of field 0) of a block's region [lo, lo + n): tiles
// at most wmax wide, `slabs` z-slabs of near-equal height (at least `least`).
inline void deriv_push(std::vector<DerivItem>& v, int block, const int lo[3], const int n[3], int wmax, int slabs,
                       int least) {
  const DerivTile t = deriv_tile(n[0], n[1], wmax);
  const int most = n[2] / least, ns = slabs < 1 || most < 1 ? 1 : slabs < most ? slabs : most;
  for (int z = 0; z < ns; ++z) {
    const int k0 = lo[2] + (int)((long long)n[2] * z / ns), k1 = lo[2] + (int)((long long)n[2] * (z + 1) / ns);
    for (int y0 = lo[1]; y0 < lo[1] + n[1]; y0 += t.h)
      for (int x0 = lo[0]; x0 < lo[0] + n[0]; x0 += t.w)
        v.push_back(DerivItem{block, x0, y0, 0, k0, k1, lo[0] + n[0], lo[1] + n[1], t.w, t.h});
  }
}
// z-slabs of a level whose tiling nobody set, from its items at one slab a
// block: the number with the least expected time on `ctas` resident CTAs.  An
// item of p planes takes p + 6 steps (four of warm-up, the prologue about two)
// of relative cost 1, 0.65 or 0.5 by its field's kind; the launch takes the
// longest item, or all items shared out plus part of a last one.  A 24^3 block
// is 48 items of 30 steps uncut and 288 of 10 in six slabs (a step 459 and
// 216 us); 70^3 points go in two (1.92 ms a step; 2.17 uncut, 1.94 in three,
// 1.90 in four), 134^3 of Z4c in one or two alike (12.4 ms).
inline int deriv_slabs(const std::vector<DerivItem>& one, bool z4c, int ctas) {
  const double per_tile = 11.0 + (z4c ? 5 : 4) * 0.65 + 9 * 0.5;
  int best = 1;
  double least = 0.0;
  for (int ns = 1; ns <= 16; ++ns) {
    double sum = 0.0, longest = 0.0;
    for (const DerivItem& it : one) {
      const int p = it.k1 - it.k0, most = p / kAutoSlab, n = most < 1 ? 1 : ns < most ? ns : most;
      const double steps = (p + n - 1) / n + 6;
      sum += n * steps;
      if (steps > longest) longest = steps;
    }
    const double shared = sum * per_tile / ctas + 0.25 * longest, t = shared > longest ? shared : longest;
    if (ns == 1 || t < least) { least = t; best = ns; }
  }
  return best;
}

// kind of a field's stencil record: 0 gradient + Hessian + adv, 1 gradient + adv, 2 adv
__host__ __device__ constexpr int dkind(int F) { return dslots(F) == 10 ? 0 : (dslots(F) == 4 ? 1 : 2); }

// Asynchronous copies global -> shared of one 8- or 4-byte cell; zero-filled
// when !valid (the source address is then not read).
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gsrc), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned sdst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sdst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned sdst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sdst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// A stencil term into D: written once here and read once by the pointwise
// pass: the store is marked evict-first (st.global.cs) and leaves L2 to the
// fields the stencil pass re-reads.
template <typename T>
__device__ __forceinline__ void dstore(T* a, T v) { __stcs(a, v); }

// The plane cells one thread copies, fixed for the whole march.  A: type in
// the ring, S: type of the source.
template <typename A, typename S>
struct PlaneCells {
  const S* src;
  long long sz;
  int ex2;
  int off[DPER];     // i + j * ex0 of the (mirrored) cell; -1: past the block's end, -2: no cell
  int pos[DPER];     // its place in a ring slot
  unsigned neg;      // bit e: x/y mirroring flips the sign of cell e
  int odd;           // bit d: the field's parity in direction d is odd

  __device__ __forceinline__ void init(const S* s, int F, const int* ex, int x0, int y0, int w, int h) {
    src = s;
    sz = (long long)ex[0] * ex[1];
    ex2 = ex[2];
    odd = (soa_sign(F, 0) < 0 ? 1 : 0) | (soa_sign(F, 1) < 0 ? 2 : 0) | (soa_sign(F, 2) < 0 ? 4 : 0);
    neg = 0;
    const int sx = w + 6, np = sx * (h + 6);
#pragma unroll
    for (int e = 0; e < DPER; ++e) {
      const int t = threadIdx.x + e * DTHREADS;
      const int cj = t / sx, ci = t - cj * sx;
      off[e] = -2;
      pos[e] = 0;
      if (t < np) {
        int i = x0 - 3 + ci, j = y0 - 3 + cj;
        bool m = false;
        if (i < 0) { i = -i - 1; m ^= (odd & 1) != 0; }
        if (j < 0) { j = -j - 1; m ^= (odd & 2) != 0; }
        off[e] = i < ex[0] && j < ex[1] ? i + j * ex[0] : -1;
        pos[e] = cj * DS + ci;
        if (m) neg |= 1u << e;
      }
    }
  }
  // whether cell e of plane kk takes the opposite sign of its source
  __device__ __forceinline__ bool flips(int e, int kk) const { return (((neg >> e) & 1u) != 0) != (kk < 0 && (odd & 4)); }
  // issues the copies of plane kk (negative: mirrored): into the ring slot (no
  // conversion), or into buf, one cell per thread and e.  Cells past the
  // block's end are set to 0 at once.
  __device__ __forceinline__ void issue(int kk, A* slot, S* buf) const {
    const int k = kk < 0 ? -kk - 1 : kk;
    const S* pl = src + k * sz;
    const bool kin = k < ex2;
#pragma unroll
    for (int e = 0; e < DPER; ++e) {
      S* d = sizeof(A) == sizeof(S) ? reinterpret_cast<S*>(slot) + pos[e] : buf + threadIdx.x + e * DTHREADS;
      if (kin && off[e] >= 0) {
        const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
        if constexpr (sizeof(S) == 8) cp_async8(sa, pl + off[e]);
        else cp_async4(sa, pl + off[e]);
      } else if (off[e] >= -1) {
        *d = S(0);
      }
    }
  }
  // once this thread's copies of plane kk landed: their signs, and the conversion
  __device__ __forceinline__ void land(int kk, A* slot, const S* buf) const {
    if constexpr (sizeof(A) == sizeof(S)) {
      if (!neg && !(kk < 0 && (odd & 4))) return;
#pragma unroll
      for (int e = 0; e < DPER; ++e)
        if (off[e] >= 0 && flips(e, kk)) slot[pos[e]] = -slot[pos[e]];
    } else {
#pragma unroll
      for (int e = 0; e < DPER; ++e)
        if (off[e] >= -1) {
          const A v = (A)buf[threadIdx.x + e * DTHREADS];
          slot[pos[e]] = flips(e, kk) ? -v : v;
        }
    }
  }
};

// Upwinded term of one direction (lopsidediff.f90:321-481) over a line f(o),
// o = -3 .. 3 relative to the point; f already includes the +1 of the
// diagonal metric.  bd = beta * d12.  Which stencil a point takes depends on
// the sign of beta and on the room towards the ends of the line: 0 forward, 1
// centred, 2 backward -- the forward arithmetic on the mirrored line --, 3
// none; lop_codes packs the form for beta > 0 (bits 0, 1) and < 0 (bits 2, 3).
__device__ __forceinline__ int lop_codes(int idx, int lo, int hi) {
  const int p = idx + 3 <= hi ? 0 : (idx + 2 <= hi ? 1 : (idx + 1 <= hi ? 2 : 3));
  const int n = idx - 3 >= lo ? 2 : (idx - 2 >= lo ? 1 : (idx - 1 >= lo ? 0 : 3));
  return p | (n << 2);
}
template <typename A, typename FN>
__device__ __forceinline__ A lop_term(const FN& f, A b, A bd, int codes) {
  const int form = b > A(0) ? (codes & 3) : (b < A(0) ? codes >> 2 : 3);
  const bool fwd = form == 0;
  const A F3 = A(3), F10 = A(10), F18 = A(18), F6 = A(6);
  const A fa = fwd ? f(-1) : f(1), fb = f(0), fc = fwd ? f(1) : f(-1);
  const A fd = fwd ? f(2) : f(-2), fe = fwd ? f(3) : f(-3);
  const A s = -F3 * fa - F10 * fb + F18 * fc - F6 * fd + fe;
  A r = (fwd ? bd : -bd) * s;
  if (form & 1) r = form == 1 ? bd * (f(-2) - A(8) * f(-1) + A(8) * f(1) - f(2)) : A(0);
  return r;
}

// a / dx of a KO line sum.  FP64: the product with the rounded reciprocal,
// corrected by its remainder (Markstein 1990, "Computation of elementary
// functions on the IBM RISC System/6000 processor"): the rounded quotient in
// four operations instead of a division (below 1e-305, where the remainder is
// subnormal, one unit in the last place off); an infinite quotient, whose
// remainder is no number, stays as it is.
template <typename T>
__device__ __forceinline__ T ko_quotient(T a, const Coef<T>& c, int d) {
  if constexpr (sizeof(T) == 8) {
    const T q = a * c.hinv[d];
    const T r = fma(fma(-q, c.h[d], a), c.hinv[d], q);
    return fabs(q) < T(1.7976931348623157e308) ? r : q;
  } else {
    return a * c.hinv[d];
  }
}

// KO dissipation of a point from its three lines.
template <typename A, typename FX, typename FY, typename FZ>
__device__ __forceinline__ A ko_term(const FX& X, const FY& Y, const FZ& Z, const Coef<A>& C) {
  return ko_quotient(ko_sum_rn<A, false>(X), C, 0) + ko_quotient(ko_sum_rn<A, false>(Y), C, 1) +
         ko_quotient(ko_sum_rn<A, false>(Z), C, 2);
}

// March one field of one tile.  A: stencil arithmetic type, S: type of the
// field's source array, SI: type of the stage input (for the shift), T: type
// of the D array.
template <typename A, int KIND, bool Z4C, typename T, typename S, typename SI>
__device__ __forceinline__ void deriv_march(const StepBlock<T>& B, const S* src, const SI* in, const double* bsh,
                                            int F, const DerivItem& it, T* D, int slots, int region, int spare,
                                            unsigned char* smem) {
  const Coef<A>& C = *reinterpret_cast<const Coef<A>*>(smem + kDerivCoef);
  if (threadIdx.x < sizeof(Coef<A>) / 4)
    reinterpret_cast<unsigned*>(smem + kDerivCoef)[threadIdx.x] = reinterpret_cast<const unsigned*>(&pick<A>(B.C))[threadIdx.x];
  A* ring = reinterpret_cast<A*>(smem);
  S* land = reinterpret_cast<S*>(smem + (size_t)DRING * DPLANE * sizeof(A));   // two planes, where A != S
  // the thread's shift values, component c of point a in slot s at
  // (6 s + 2 c + a) * DTHREADS
  const double* bet = reinterpret_cast<double*>(smem + kDerivRing) + threadIdx.x;
  const unsigned bet_s = (unsigned)__cvta_generic_to_shared(bet);
  const int ex0 = B.b.ex[0], ex1 = B.b.ex[1], ex2 = B.b.ex[2];
  const int x0 = it.x0, y0 = it.y0, k0 = it.k0, k1 = it.k1, W = it.w, NP = it.h / 2;
  const long long fs = B.b.fs;
  const int fm = B.b.face_mask, ls = B.b.lowsym_mask;
  const int lox = (ls & 1) ? -3 : 0, loy = (ls & 2) ? -3 : 0, loz = (ls & 4) ? -3 : 0;

  // The thread's column pair (li, 2 pj), (li, 2 pj + 1) of the tile, row by row.
  const int pj = threadIdx.x / W, li = threadIdx.x - pj * W;
  const bool any = pj < NP;
  const int i = x0 + li, j = y0 + 2 * pj;
  const bool xin = any && i < it.x1 && !((fm & 1) && i == ex0 - 1) && !((fm & 8) && i == 0);
  const bool m0 = xin && j < it.y1 && !((fm & 2) && j == ex1 - 1) && !((fm & 16) && j == 0);
  const bool m1 = xin && j + 1 < it.y1 && !((fm & 2) && j + 1 == ex1 - 1);
  const int own = any ? (2 * pj + 3) * DS + li + 3 : 0;   // in a ring slot
  // which stencils fit in x and y at the two points (the z part is the plane's):
  // bit 0 4th order, 1 2nd order, 2 KO, 3 advection (point_gates)
  auto fits_xy = [&](int jj) -> int {
    const int lx = (ls & 1) ? -2 : 0, ly = (ls & 2) ? -2 : 0;
    const int nx = i - lx < ex0 - 1 - i ? i - lx : ex0 - 1 - i, ny = jj - ly < ex1 - 1 - jj ? jj - ly : ex1 - 1 - jj;
    const int n = nx < ny ? nx : ny;   // cells to the nearest end, mirrored ones (two of them) included
    const int mx = i - lox < ex0 - 1 - i ? i - lox : ex0 - 1 - i, my = jj - loy < ex1 - 1 - jj ? jj - loy : ex1 - 1 - jj;
    return (n >= 2 ? 1 : 0) | (n >= 1 ? 2 : 0) | ((mx < my ? mx : my) >= 3 ? 4 : 0) |
           (i <= ex0 - 2 && jj <= ex1 - 2 ? 8 : 0);
  };
  const int fit0 = fits_xy(j), fit1 = fits_xy(j + 1);
  auto fits_z = [&](int k) -> int {
    const int lz = (ls & 4) ? -2 : 0, n = k - lz < ex2 - 1 - k ? k - lz : ex2 - 1 - k;
    return (n >= 2 ? 1 : 0) | (n >= 1 ? 2 : 0) | (k - 3 >= loz && k + 3 < ex2 ? 4 : 0) | (k <= ex2 - 2 ? 8 : 0);
  };

  // entries of the points in their tiles' order, and the D rows of the field
  const int rn0 = region < 0 ? ex0 : B.rn[region][0], rn1 = region < 0 ? ex1 : B.rn[region][1];
  const int rx = region < 0 ? 0 : B.rlo[region][0], ry = region < 0 ? 0 : B.rlo[region][1];
  const int rz = region < 0 ? 0 : B.rlo[region][2];
  const int og = dl::g(F) * kDTile, oh = dl::h(F) * kDTile, oa = dl::a(F) * kDTile;
  const int rn01 = rn0 * rn1, dt0 = B.dtile;   // locals: the march's waits would have B read again each time
  int dq = (i - rx) + rn0 * ((j - ry) + rn1 * (k0 - 2 - rz));   // entry of the first point at plane k
  // a thread without a point of its own stores into the tile past the last
  // (spare): straight-line code instead of a branch per point
  T* const sp = D + (long long)spare * (slots * kDTile) + (threadIdx.x & 127);
  auto dptr = [&](bool m, int q) -> T* {
    T* d = D + ((long long)(dt0 + (q >> 7)) * (slots * kDTile) + (q & 127));
    return m ? d : sp;
  };
  static_assert(kDTile == 128, "dptr");

  // the diagonal metric is advected as g = d + 1 (bssn_rhs.f90:948-953) in FP64,
  // bit-faithful to the reference; FP32 advects d (the constant drops out)
  const A add1 = (sizeof(A) == 8 && (F == F_GXX || F == F_GYY || F == F_GZZ)) ? A(1) : A(0);

  PlaneCells<A, S> P;
  P.init(src, F, B.b.ex, x0, y0, W, it.h);

  A wx0[5], wy0[5];        // Dx f, Dy f at planes k-4 .. k (KIND 0)
  A wx1[5], wy1[5];
#pragma unroll
  for (int t = 0; t < 5; ++t) wx0[t] = wy0[t] = wx1[t] = wy1[t] = A(0);

  // the shift at the points of plane k + 2, from the stage input (bsh: its FP64
  // side slots in the mixed form), copied two planes ahead into slot sw
  const double* gb = (sizeof(SI) == 4 ? bsh : (const double*)in + F_BETAX * fs) + i + (long long)j * ex0 +
                     (long long)k0 * P.sz;
  auto shift = [&](int sw) {
    const unsigned s = bet_s + sw * (6 * DTHREADS * 8);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (m0) cp_async8(s + 2 * c * DTHREADS * 8, gb + c * fs);
      if (m1) cp_async8(s + (2 * c + 1) * DTHREADS * 8, gb + c * fs + ex0);
    }
  };

  // Planes kA-1 .. kA+4, kA = k0 - 2, fill six slots of the ring: plane m in
  // slot (m - kA) mod DRING.  (Planes kA-3, kA-2 are read by no point.)
  const int kA = k0 - 2;
  auto first = [&](int m) { return ring + (m < 0 ? DRING - 1 : m) * DPLANE; };
  if constexpr (sizeof(A) == sizeof(S)) {
#pragma unroll 1
    for (int m = -1; m <= 4; ++m) {
      P.issue(kA + m, first(m), land);
      if (m >= 3) cp_async_commit();
    }
    cp_async_wait<1>();
#pragma unroll 1
    for (int m = -1; m <= 3; ++m) P.land(kA + m, first(m), land);
  } else {
    // one plane after another through the landing buffer
#pragma unroll 1
    for (int m = -1; m <= 3; ++m) {
      P.issue(kA + m, nullptr, land + (m & 1) * (DPER * DTHREADS));
      cp_async_commit();
      if (m >= 0) {
        cp_async_wait<1>();
        P.land(kA + m - 1, first(m - 1), land + ((m - 1) & 1) * (DPER * DTHREADS));
      }
    }
    cp_async_wait<0>();
    P.land(kA + 3, first(3), land + DPER * DTHREADS);
    P.issue(kA + 4, nullptr, land);
    cp_async_commit();
  }
  __syncthreads();

  const A F8 = A(8);
  const int kE = KIND == 0 ? k1 + 2 : k1;
  const int cx = lop_codes(i, lox, ex0 - 1), cy0 = lop_codes(j, loy, ex1 - 1), cy1 = lop_codes(j + 1, loy, ex1 - 1);
  // element offsets of the slots of planes k-3 .. k+5 (k-3, k-2 of the first plane: any)
  int so[DRING];
#pragma unroll
  for (int m = 0; m < DRING; ++m) so[m] = ((m + DRING - 3) % DRING) * DPLANE;
#pragma unroll 1
  for (int k = kA, br = 0; k < kE; ++k) {
    const int bw = br == 0 ? 2 : br - 1;         // the shift's slots of planes k (br) and k + 2
    const int par = (k - kA + 5) & 1;            // landing buffer of k+5
    P.issue(k + 5, ring + so[8], land + par * (DPER * DTHREADS));
    if (k + 2 >= k0 && k + 2 < k1) {
      shift(bw);
      gb += P.sz;
    }
    cp_async_commit();
    const A* q = ring + so[3] + own;
    const bool outp = k >= k0 && k < k1 && !((fm & 4) && k == ex2 - 1) && !((fm & 32) && k == 0);
    if (any && outp) {
      const int fz = fits_z(k), cz = lop_codes(k, loz, ex2 - 1);
      const int f0 = fit0 & fz, f1 = fit1 & fz;
      T* d0 = dptr(m0, dq);
      T* d1 = dptr(m1, dq + rn0);
      A X0[7], X1[7], Y[8];   // x-lines of the two points; the y-line from row -3 to row 4
#pragma unroll
      for (int o = -3; o <= 3; ++o)
        { X0[3 + o] = q[o]; X1[3 + o] = q[DS + o]; }
#pragma unroll
      for (int r = -3; r <= 4; ++r) Y[3 + r] = r == 0 ? X0[3] : r == 1 ? X1[3] : q[r * DS];
      A c0[7], c1[7];         // z-lines
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        c0[m] = m == 3 ? X0[3] : ring[so[m] + own];
        c1[m] = m == 3 ? X1[3] : ring[so[m] + own + DS];
      }
      // 4th-order stencils; points where they do not fit are stored over below
      if constexpr (KIND == 0) {
        // row differences f(-2) - 8 f(-1) + 8 f(1) - f(2) of rows -2 .. 3
        A ds[6];
        auto row = [&](int r) {
          const A* u = q + r * DS;
          return u[-2] - F8 * u[-1] + F8 * u[1] - u[2];
        };
        ds[0] = row(-2); ds[1] = row(-1); ds[4] = row(2); ds[5] = row(3);
        ds[2] = X0[1] - F8 * X0[2] + F8 * X0[4] - X0[5];
        ds[3] = X1[1] - F8 * X1[2] + F8 * X1[4] - X1[5];
        wx0[4] = C.d12[0] * ds[2];
        wx1[4] = C.d12[0] * ds[3];
        wy0[4] = C.d12[1] * (Y[1] - F8 * Y[2] + F8 * Y[4] - Y[5]);
        wy1[4] = C.d12[1] * (Y[2] - F8 * Y[3] + F8 * Y[5] - Y[6]);
        auto dd = [&](A fm2, A fm1, A f0, A f1, A f2, A cf) {
          return cf * (-fm2 + A(16) * fm1 - A(30) * f0 - f2 + A(16) * f1);
        };
        dstore(d0 + og, (T)wx0[4]);
        dstore(d0 + og + kDTile, (T)wy0[4]);
        dstore(d0 + oh, (T)dd(X0[1], X0[2], X0[3], X0[4], X0[5], C.Fdd[0]));
        dstore(d0 + oh + 1 * kDTile, (T)(C.Fxy * (ds[0] - F8 * ds[1] + F8 * ds[3] - ds[4])));
        dstore(d0 + oh + 3 * kDTile, (T)dd(Y[1], Y[2], Y[3], Y[4], Y[5], C.Fdd[1]));
        dstore(d0 + oh + 5 * kDTile, (T)dd(c0[1], c0[2], c0[3], c0[4], c0[5], C.Fdd[2]));
        dstore(d1 + og, (T)wx1[4]);
        dstore(d1 + og + kDTile, (T)wy1[4]);
        dstore(d1 + oh, (T)dd(X1[1], X1[2], X1[3], X1[4], X1[5], C.Fdd[0]));
        dstore(d1 + oh + 1 * kDTile, (T)(C.Fxy * (ds[1] - F8 * ds[2] + F8 * ds[4] - ds[5])));
        dstore(d1 + oh + 3 * kDTile, (T)dd(Y[2], Y[3], Y[4], Y[5], Y[6], C.Fdd[1]));
        dstore(d1 + oh + 5 * kDTile, (T)dd(c1[1], c1[2], c1[3], c1[4], c1[5], C.Fdd[2]));
      }
      if constexpr (KIND == 1) {
        dstore(d0 + og, (T)(C.d12[0] * (X0[1] - F8 * X0[2] + F8 * X0[4] - X0[5])));
        dstore(d0 + og + kDTile, (T)(C.d12[1] * (Y[1] - F8 * Y[2] + F8 * Y[4] - Y[5])));
        dstore(d1 + og, (T)(C.d12[0] * (X1[1] - F8 * X1[2] + F8 * X1[4] - X1[5])));
        dstore(d1 + og + kDTile, (T)(C.d12[1] * (Y[2] - F8 * Y[3] + F8 * Y[5] - Y[6])));
      }
      if constexpr (KIND <= 1) {
        dstore(d0 + og + 2 * kDTile, (T)(C.d12[2] * (c0[1] - F8 * c0[2] + F8 * c0[4] - c0[5])));
        dstore(d1 + og + 2 * kDTile, (T)(C.d12[2] * (c1[1] - F8 * c1[2] + F8 * c1[4] - c1[5])));
      }
      // FP64 advects the diagonal metric as g = d + 1; Z4c dissipates it so too
      // (Z4c_rhs.f90:1240-1245), so there the lines are shifted once for both
      constexpr bool kMetric = KIND == 0 && sizeof(A) == 8;
      if constexpr (kMetric && Z4C) {
#pragma unroll
        for (int m = 0; m < 7; ++m) { X0[m] = X0[m] + add1; X1[m] = X1[m] + add1; }
#pragma unroll
        for (int m = 0; m < 8; ++m) Y[m] = Y[m] + add1;
#pragma unroll
        for (int m = 0; m < 7; ++m) { c0[m] = c0[m] + add1; c1[m] = c1[m] + add1; }
      }
      auto adv = [&](const auto& fX, const auto& fY, const auto& fZ, int a, int cy, int fit) -> A {
        const double* sb = bet + (6 * br + a) * DTHREADS;
        auto line = [&](const auto& f, int d, int codes) {
          const A bv = (A)(T)sb[2 * d * DTHREADS];   // rounded as the pointwise pass sees it
          const A bd = bv * C.d12[d];
          if constexpr (kMetric && !Z4C) return lop_term<A>([&](int o) { return f(o) + add1; }, bv, bd, codes);
          else return lop_term<A>(f, bv, bd, codes);
        };
        const A r = line(fX, 0, cx) + line(fY, 1, cy) + line(fZ, 2, cz);
        const A ko = C.ko * ko_term<A>(fX, fY, fZ, C);
        return ((fit & 8) ? r : A(0)) + ((fit & 4) ? ko : A(0));
      };
      const A a0 = adv([&](int o) { return X0[3 + o]; }, [&](int o) { return Y[3 + o]; },
                       [&](int o) { return c0[3 + o]; }, 0, cy0, f0);
      dstore(d0 + oa, (T)a0);
      const A a1 = adv([&](int o) { return X1[3 + o]; }, [&](int o) { return Y[4 + o]; },
                       [&](int o) { return c1[3 + o]; }, 1, cy1, f1);
      dstore(d1 + oa, (T)a1);
      if constexpr (KIND <= 1) {
        // next to an edge the derivatives are of 2nd order, on it zero.  One
        // copy of the code for both points
        if ((m0 && !(f0 & 1)) || (m1 && !(f1 & 1))) {
#pragma unroll 1
          for (int a = 0; a < 2; ++a) {
            const int fit = a ? f1 : f0;
            if (!(a ? m1 : m0) || (fit & 1)) continue;
            const A* u = q + a * DS;
            const A* um = ring + so[2] + own + a * DS;   // planes k-1, k+1
            const A* up = ring + so[4] + own + a * DS;
            T* d = a ? d1 : d0;
            auto put = [&](int o, A v) { dstore(d + o, (fit & 2) ? (T)v : T(0)); };
            put(og, C.d2[0] * (-u[-1] + u[1]));
            put(og + kDTile, C.d2[1] * (-u[-DS] + u[DS]));
            put(og + 2 * kDTile, C.d2[2] * (-um[0] + up[0]));
            if constexpr (KIND == 0) {
              const A TWO = A(2), f = u[0];
              put(oh, C.Sdd[0] * (u[-1] - TWO * f + u[1]));
              put(oh + 1 * kDTile, C.Sxy * (u[-1 - DS] - u[1 - DS] - u[-1 + DS] + u[1 + DS]));
              put(oh + 2 * kDTile, C.d2[2] * (-(C.d2[0] * (-um[-1] + um[1])) + C.d2[0] * (-up[-1] + up[1])));
              put(oh + 3 * kDTile, C.Sdd[1] * (u[-DS] - TWO * f + u[DS]));
              put(oh + 4 * kDTile, C.d2[2] * (-(C.d2[1] * (-um[-DS] + um[DS])) + C.d2[1] * (-up[-DS] + up[DS])));
              put(oh + 5 * kDTile, C.Sdd[2] * (um[0] - TWO * f + up[0]));
            }
          }
        }
      }
    } else if constexpr (KIND == 0) {
      if (any) {   // a plane of the windows only
        auto dx4 = [&](const A* u) { return C.d12[0] * (u[-2] - F8 * u[-1] + F8 * u[1] - u[2]); };
        auto dy4 = [&](const A* u) { return C.d12[1] * (u[-2 * DS] - F8 * u[-DS] + F8 * u[DS] - u[2 * DS]); };
        wx0[4] = dx4(q); wy0[4] = dy4(q);
        wx1[4] = dx4(q + DS); wy1[4] = dy4(q + DS);
      }
    }
    if constexpr (KIND == 0) {
      // the mixed xz, yz derivatives of plane k-2 where they are of 4th order
      const int kl = k - 2;
      if (kl >= k0 && !((fm & 4) && kl == ex2 - 1) && !((fm & 32) && kl == 0)) {
        const int fl = fits_z(kl);
        T* d0 = dptr(m0 && (fit0 & fl & 1), dq - 2 * rn01) + oh;
        T* d1 = dptr(m1 && (fit1 & fl & 1), dq - 2 * rn01 + rn0) + oh;
        dstore(d0 + 2 * kDTile, (T)(C.d12[2] * (wx0[0] - F8 * wx0[1] + F8 * wx0[3] - wx0[4])));
        dstore(d0 + 4 * kDTile, (T)(C.d12[2] * (wy0[0] - F8 * wy0[1] + F8 * wy0[3] - wy0[4])));
        dstore(d1 + 2 * kDTile, (T)(C.d12[2] * (wx1[0] - F8 * wx1[1] + F8 * wx1[3] - wx1[4])));
        dstore(d1 + 4 * kDTile, (T)(C.d12[2] * (wy1[0] - F8 * wy1[1] + F8 * wy1[3] - wy1[4])));
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        wx0[t] = wx0[t + 1]; wy0[t] = wy0[t + 1];
        wx1[t] = wx1[t + 1]; wy1[t] = wy1[t + 1];
      }
    }
    // plane k+4 lands in a slot no thread reads in this step
    cp_async_wait<1>();
    P.land(k + 4, ring + so[7], land + (par ^ 1) * (DPER * DTHREADS));
    __syncthreads();
    const int s0 = so[0];
#pragma unroll
    for (int m = 0; m < DRING - 1; ++m) so[m] = so[m + 1];
    so[DRING - 1] = s0;
    dq += rn01;
    br = br == 2 ? 0 : br + 1;
  }
  cp_async_wait<0>();   // the copies still in flight land before the ring is reused
}

// Stencil pass over a work list of (block, tile, slab, field) items, ordered
// by field so that resident CTAs share one code path.
template <typename T, typename SI, bool Z4C>
__global__ void __launch_bounds__(DTHREADS, 2) k_deriv(const StepBlock<T>* __restrict__ blocks,
                                                       const DerivItem* __restrict__ items, int nitems, int sub,
                                                       T* __restrict__ D, int slots, int region, int spare) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
    const DerivItem it = items[w];
    const StepBlock<T>& B = blocks[it.block];
    const int cur = B.lvl[0];
    const SI* in = sub == 0 ? (const SI*)B.tl[cur] : (const SI*)B.stage[sub == 2 ? 1 : 0];
    const int F = it.field;
    const long long fs = B.b.fs;
    // the mixed form's stages keep the shift in their FP64 side slots
    const double* bsh = sizeof(SI) == 4 ? B.side[sub == 2 ? 1 : 0] + side_slot(F_BETAX) * fs : nullptr;
    if constexpr (sizeof(T) == 4) {
      if (is_wide(F)) {
        // wide fields of the mixed form: FP64 source (state, or the FP64 side stage) and arithmetic
        const double* src = sizeof(SI) == 4 ? B.side[sub == 2 ? 1 : 0] + side_slot(F) * fs
                                            : (const double*)in + F * fs;
        deriv_march<double, 0, Z4C>(B, src, in, bsh, F, it, D, slots, region, spare, smem);
        __syncthreads();
        continue;
      }
    }
    const SI* src = in + F * fs;
    switch (dkind(F)) {
      case 0: deriv_march<T, 0, Z4C>(B, src, in, bsh, F, it, D, slots, region, spare, smem); break;
      case 1: deriv_march<T, 1, Z4C>(B, src, in, bsh, F, it, D, slots, region, spare, smem); break;
      default: deriv_march<T, 2, Z4C>(B, src, in, bsh, F, it, D, slots, region, spare, smem); break;
    }
    __syncthreads();
  }
}

// Stencil pass launcher: substep 0 reads the FP64 state, 1-3 the stages;
// region: the D order of the points (-1: whole arrays, else StepBlock::rlo);
// spare: a tile of D that holds no points (any rubbish may be stored there).
template <typename T, typename SS>
cudaError_t launch_deriv(const void* blocks, const DerivItem* items, int nitems, int sub, void* D, int slots,
                         int region, int spare, int grid, cudaStream_t s) {
  const StepBlock<T>* bl = (const StepBlock<T>*)blocks;
  auto go = [&](auto kernel) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDerivSmem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, DTHREADS, kDerivSmem, s>>>(bl, items, nitems, sub, (T*)D, slots, region, spare);
    return cudaGetLastError();
  };
  if (slots == D_SLOTS_Z4C) return sub == 0 ? go(k_deriv<T, double, true>) : go(k_deriv<T, SS, true>);
  return sub == 0 ? go(k_deriv<T, double, false>) : go(k_deriv<T, SS, false>);
}

}  // namespace amss
