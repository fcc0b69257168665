// face.cu -- the outer-face pass of the RK4 substep.
#include "substep_common.cuh"

namespace amss {

// Outer-face points of a level (Sommerfeld on level 0, sommerfeld_rout.f90:
// 223-449; frozen on refined patch faces, :122-139) from the list faces[] =
// (block, point), with the NaN check, the RK4 update, the chi floor and
// enforce_ga of the pointwise pass.
//
// A CTA takes kFacePts points: lane = point, warp = fields warp, warp + 8, ...
// The pass is latency bound -- a face point reads up to nine scattered values
// a field, and the points of an x face share no line -- so the fields of a
// point go to different warps and their loads are in flight together: 82 us a
// launch on a 70^3 block (28,568 face points) and 93 us on a 24^3 block with
// one thread taking the 24 fields of a point in turn, 30 us and 10 us
// now.  enforce_ga couples 12 fields of a point, which meet in shared memory;
// warp 0 then finishes one point per lane.
constexpr int kFacePts = 32;
constexpr int kFaceWarps = 8;
constexpr int kFaceFields = (NFIELDS_Z4C + kFaceWarps - 1) / kFaceWarps;   // fields a warp takes

template <typename T, typename SI, typename SO>
__global__ void __launch_bounds__(kFacePts * kFaceWarps) k_face(const StepBlock<T>* __restrict__ blocks,
                                                                const int2* __restrict__ faces, int nfaces, int sub,
                                                                RKConst rk, int enforce, unsigned* status) {
  __shared__ double ga[12][kFacePts];   // metric and A~ values of the points, before enforce_ga
  const int lane = threadIdx.x % kFacePts, warp = threadIdx.x / kFacePts;
  for (int t0 = blockIdx.x * kFacePts; t0 < nfaces; t0 += gridDim.x * kFacePts) {
    const bool mine = t0 + lane < nfaces;
    const int2 fc = faces[mine ? t0 + lane : nfaces - 1];
    const StepBlock<T>& B = blocks[fc.x];
    const BlockView& b = B.b;
    const long long p = fc.y, fs = b.fs;
    const int cur = B.lvl[0];
    const double* u0 = B.tl[cur];
    const SI* in = sub == 0 ? (const SI*)u0 : (const SI*)B.stage[sub == 2 ? 1 : 0];
    const double* in_side = sub == 0 ? nullptr : B.side[sub == 2 ? 1 : 0];
    SO* out = sub == 3 ? (SO*)B.tl[(cur + 1) % 3] : (SO*)B.stage[sub == 1 ? 1 : 0];
    double* out_side = sub == 3 ? nullptr : B.side[sub == 1 ? 1 : 0];
    if (mine) {
      int id[3];
      point_ijk(p, b.ex, id[0], id[1], id[2]);
      // The Sommerfeld rule (sommerfeld_rout.f90:378-440, one-sided 2nd order,
      // upwinded by the sign of x_d) in FP64 in both precisions.  Per
      // direction: which stencil (0 backward, 1 centred, 2 forward, 3 none)
      // and its two points besides the centre, mirrored below index 0.
      double pos[3] = {0.0, 0.0, 0.0}, R = 1.0;
      int form[3] = {3, 3, 3};
      long long o1[3] = {0, 0, 0}, o2[3] = {0, 0, 0};
      unsigned neg = 0;
      if (B.lev0) {
        pos[0] = b.X[id[0]]; pos[1] = b.Y[id[1]]; pos[2] = b.Z[id[2]];
        R = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]);
        const long long st[3] = {1, b.ex[0], (long long)b.ex[0] * b.ex[1]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int lo = ((b.lowsym_mask >> d) & 1) ? -1 : 0, hi = b.ex[d] - 1;
          if (pos[d] > 0.0) form[d] = id[d] - 2 >= lo ? 0 : (id[d] - 1 >= lo ? 1 : 2);
          else if (pos[d] < 0.0) form[d] = id[d] + 2 <= hi ? 2 : (id[d] + 1 <= hi ? 1 : 0);
          const int a1 = form[d] == 3 ? 0 : (form[d] == 2 ? 1 : -1);
          const int a2 = form[d] == 3 ? 0 : (form[d] == 0 ? -2 : (form[d] == 1 ? 1 : 2));
          const int m1 = id[d] + a1, m2 = id[d] + a2;
          o1[d] = (long long)((m1 < 0 ? -m1 - 1 : m1) - id[d]) * st[d];
          o2[d] = (long long)((m2 < 0 ? -m2 - 1 : m2) - id[d]) * st[d];
          neg |= (m1 < 0 ? 1u << (2 * d) : 0u) | (m2 < 0 ? 2u << (2 * d) : 0u);
        }
      }
      unsigned bad = 0;
#pragma unroll
      for (int m = 0; m < kFaceFields; ++m) {
        const int F = warp + m * kFaceWarps;
        if (F >= B.nf) break;
        const bool wide = sizeof(SI) == 4 && is_wide(F);
        auto ld = [&](long long o) -> double {
          return wide ? __ldg(in_side + side_slot(F) * fs + p + o) : (double)__ldg(in + F * fs + p + o);
        };
        // every load of the field is issued before the first use
        const double f0 = ld(0), u = u0[F * fs + p];
        double f1[3], f2[3], kk = 0.0;
        double* K = B.K + F * fs + p;
        if (B.lev0) {
#pragma unroll
          for (int d = 0; d < 3; ++d) { f1[d] = ld(o1[d]); f2[d] = ld(o2[d]); }
          if (sub != 0) kk = *K;
        }
        if (F <= F_BETAZ || B.nf == NFIELDS_Z4C) {   // Z4c_rhs.f90:230-262 checks all 25
          const T c = (T)f0;
          bad |= nan_bits(&c, 1);
        }
        double r = u;   // refined patch: frozen at u0; its accumulator is never read
        if (B.lev0) {
          const double v = (F == F_CHI || F == F_TRK || F == F_LAP) ? 1.4142135623730951 : 1.0;
          double fd[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const bool odd = soa_sign(F, d) < 0;
            const double a = odd && (neg & (1u << (2 * d))) ? -f1[d] : f1[d];
            const double c = odd && (neg & (2u << (2 * d))) ? -f2[d] : f2[d];
            const double d2 = B.C.d.d2[d];
            fd[d] = form[d] == 0   ? d2 * (3.0 * f0 - 4.0 * a + c)
                    : form[d] == 1 ? d2 * (-a + c)
                    : form[d] == 2 ? d2 * (-c + 4.0 * a - 3.0 * f0)
                                   : 0.0;
          }
          const double k = -v * (fd[0] * pos[0] + fd[1] * pos[1] + fd[2] * pos[2] + f0) / R;
          if (sub == 0) {
            r = u + rk.half_dt * k;
            *K = k;
          } else if (sub == 3) {
            r = u + rk.sixth_dt * (k + kk);
          } else {
            *K = kk + 2.0 * k;
            r = sub == 1 ? u + rk.half_dt * k : u + rk.dt * k;
          }
        }
        if (F == F_CHI && r < rk.chitiny) r = rk.chitiny;
        if (enforce && F >= F_GXX && F <= F_AZZ) ga[F - F_GXX][lane] = r;
        else if (sizeof(SO) == 4 && is_wide(F)) out_side[side_slot(F) * fs + p] = r;
        else out[F * fs + p] = (SO)r;
      }
      if (bad) atomicOr(status, bad);
    }
    if (enforce) {
      __syncthreads();
      if (warp == 0 && mine) {
        double g[6], a[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) { g[m] = ga[m][lane]; a[m] = ga[6 + m][lane]; }
        enforce_ga_point(g, a);
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          out[(F_GXX + m) * fs + p] = (SO)g[m];
          out[(F_AXX + m) * fs + p] = (SO)a[m];
        }
      }
      __syncthreads();
    }
  }
}

template <typename T, typename SS>
cudaError_t launch_face(const void* blocks, const int2* faces, int nfaces, int sub, RKConst rk, int enforce,
                        unsigned* status, cudaStream_t s) {
  if (nfaces == 0) return cudaSuccess;
  const StepBlock<T>* bl = (const StepBlock<T>*)blocks;
  const int grid = (nfaces + kFacePts - 1) / kFacePts < 148 * 16 ? (nfaces + kFacePts - 1) / kFacePts : 148 * 16;
  if (sub == 0)
    k_face<T, double, SS><<<grid, kFacePts * kFaceWarps, 0, s>>>(bl, faces, nfaces, sub, rk, enforce, status);
  else if (sub == 3)
    k_face<T, SS, double><<<grid, kFacePts * kFaceWarps, 0, s>>>(bl, faces, nfaces, sub, rk, enforce, status);
  else
    k_face<T, SS, SS><<<grid, kFacePts * kFaceWarps, 0, s>>>(bl, faces, nfaces, sub, rk, enforce, status);
  return cudaGetLastError();
}

template cudaError_t launch_face<double, double>(const void*, const int2*, int, int, RKConst, int, unsigned*,
                                                 cudaStream_t);
template cudaError_t launch_face<float, float>(const void*, const int2*, int, int, RKConst, int, unsigned*,
                                               cudaStream_t);

}  // namespace amss
