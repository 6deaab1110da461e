// The flux of one face from its eight-cell stencil, shared by the per-face
// sweep (k_flux, gcs_sweeps.cuh) and the staged one (k_flux_tma,
// gcs_flux_tma.cuh), which differ only in where the stencil cells are read.
#pragma once

#include "gcs_kernel_util.cuh"
#include "gcs_physics.cuh"

namespace gcs {

// A face: its indices, its node in the full arrays and in the Bulk view's.
// Node indices fit 32 bits (a context of 2^32 nodes would need 8 TB), which
// halves the address arithmetic of the sweeps' loads.
struct FaceAt {
  int f, i, j, k;
  unsigned c, cb;
};

// The eight nodes n - 4 (n = 0..7) around a node along one axis; kUnit: the
// contiguous one, where the offsets are immediates of the loads.
template <bool kUnit>
struct LineStencil {
  unsigned at[8];
  __device__ __forceinline__ LineStencil(unsigned c, int stride) {
#pragma unroll
    for (int n = 0; n < 8; ++n) at[n] = c + (unsigned)((n - 4) * stride);
  }
  template <typename T>
  __device__ __forceinline__ void load(const T *p, T q[8]) const {
#pragma unroll
    for (int n = 0; n < 8; ++n) q[n] = kUnit ? (p + at[4])[n - 4] : p[at[n]];
  }
};

// The stencil cells of a face in global memory, `stride` apart.
template <typename T>
struct GlobalStencil {
  const Bulk<T> &B;
  LineStencil<false> at;
  __device__ __forceinline__ GlobalStencil(const Bulk<T> &B_, unsigned cb, int stride)
      : B(B_), at(cb, stride) {}
  __device__ __forceinline__ void load(const T *p, T q[8]) const { at.load(p, q); }
  __device__ __forceinline__ void volume(T q[8]) const { load(B.vol, q); }
  __device__ __forceinline__ void prim(int m, T q[8]) const { load(B.Pr[m], q); }
  __device__ __forceinline__ void field(int m, T q[8]) const { load(B.Bp[m], q); }
};

template <typename T>
__device__ __forceinline__ T inv_gm1(const Opts &O);
template <>
__device__ __forceinline__ double inv_gm1<double>(const Opts &O) { return O.s_igm1; }
template <>
__device__ __forceinline__ float inv_gm1<float>(const Opts &O) { return O.s_igm1_f32; }

// nonorthogonal_sweep.c:408-548 for one face of direction d: only the
// interpolation weights, one variable's stencil and the reconstructed states
// are live at once.  d is a run-time value: the three directions share one
// instruction stream (a body per direction, run side by side, overflows the
// instruction cache: three of the eight cycles between issues waited for it).
template <bool kOrtho, typename T, typename Stencil>
__device__ __forceinline__ void face_flux(int d, const Stencil &cells, const Dims &D,
                                          const DevState &S, const Bulk<T> &B,
                                          const Opts &O, DevStatus *st, const FaceAt &at) {
  const unsigned c = at.c, cb = at.cb;
  // No branch between the loads: every check sets a flag that is tested
  // before the stores, so the loads of the next variables are in flight
  // while one is reconstructed.
  const unsigned long long first = failure_word(st);
  const T iv = B.iv[d][cb];
  bool recon_ok = !isnan(iv);
  const T pdm2 = T(2.0) * (T)O.pdm;
  PrimT<T> st2[2];
  T mag[2][3] = {{T(0.0), T(0.0), T(0.0)}, {T(0.0), T(0.0), T(0.0)}};
  {
    T qa[8], qb[8];
    cells.volume(qa);
    cells.prim(0, qb);
    const Up7Weights<T> w(qa, Num<T>::rcp(iv));
    cells.prim(1, qa);
#pragma unroll
    for (int n = 0; n < 8; ++n) recon_ok = recon_ok && !isnan(qb[n]);
    up7_pdm(w, qb, pdm2, &st2[0].rho, &st2[1].rho);
    cells.prim(2, qb);
    up7_pdm(w, qa, pdm2, &st2[0].vx, &st2[1].vx);
    cells.prim(3, qa);
    up7_pdm(w, qb, pdm2, &st2[0].vy, &st2[1].vy);
    cells.prim(4, qb);
    up7_pdm(w, qa, pdm2, &st2[0].vz, &st2[1].vz);
    if (O.s_mhd) cells.field(0, qa);
    up7_pdm(w, qb, pdm2, &st2[0].p, &st2[1].p);
    if (O.s_mhd) {
      cells.field(1, qb);
      up7_pdm(w, qa, pdm2, &mag[0][0], &mag[1][0]);
      cells.field(2, qa);
      up7_pdm(w, qb, pdm2, &mag[0][1], &mag[1][1]);
      up7_pdm(w, qa, pdm2, &mag[0][2], &mag[1][2]);
    }
  }
  FaceFrame<T> fr;
  fr.nx = B.fn[d][0][cb]; fr.ny = B.fn[d][1][cb]; fr.nz = B.fn[d][2][cb];
  if (!kOrtho) {
    fr.t1x = B.ft1[d][0][cb]; fr.t1y = B.ft1[d][1][cb]; fr.t1z = B.ft1[d][2][cb];
    fr.t2x = B.ft2[d][0][cb]; fr.t2y = B.ft2[d][1][cb]; fr.t2z = B.ft2[d][2][cb];
  }
  T bn = T(0.0), b0n = T(0.0);
  T b0[3] = {T(0.0), T(0.0), T(0.0)};
  if (O.s_mhd) {
    bn = B.BN[d][cb];
    if (O.s_bg) {
      b0[0] = B.fb0[d][0][cb];
      b0[1] = B.fb0[d][1][cb];
      b0[2] = B.fb0[d][2][cb];
      b0n = B.fb0n[d][cb];
    }
  }
  const T area = B.area[d][cb];
  FluidFlux<T> fl;
  const bool fluid_ok = kinetic_fluid_flux<kOrtho>(st2, inv_gm1<T>(O), fr, &fl) == 0;
  MaxwellFlux<T> mx;
  mx.m[0] = mx.m[1] = mx.m[2] = T(0.0);
  bool maxwell_ok = true;
  if (O.s_mhd) {
    maxwell_ok = kinetic_maxwell_flux(mag, bn, fr, O.s_bg, b0, b0n, O.s_boris,
                                      (T)O.s_ic2, fl, &mx) == 0;
    if (O.hogs)
      apply_hogs(&fl, &mx, st2, inv_gm1<T>(O), (T)O.hogs_h, (T)O.hogs_m, O.s_boris,
                 (T)O.s_ic2);
  }
  if (stopped(first, kPassFlux)) return;
  if (!(recon_ok && fluid_ok && maxwell_ok)) {
    fail(st, !recon_ok ? kStageReconstruct : !fluid_ok ? kStageKineticFluid
                                                       : kStageKineticMaxwell,
         d, at.f, at.i, at.j, at.k);
    return;
  }
  if (O.s_mhd && O.hogs && O.s_boris) {
    bool applied;
    T speed;
    if (emergency_diffusion(&fl, st2, S.Up, (long long)c - D.stride(d), c, (T)O.s_c,
                            &applied, &speed)) {
      fail(st, kStageEmergency, d, at.f, at.i, at.j, at.k);
      return;
    }
    if (applied) {
      atomicAdd(&st->emergency_count[at.f], 1ULL);
      atomicMax(&st->emergency_max_bits[at.f],
                (unsigned long long)__double_as_longlong((double)speed));
    }
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) B.F[d][m][c] = (double)(area * fl.f[m]);
#pragma unroll
  for (int m = 0; m < 3; ++m) B.M[d][m][c] = (double)(area * mx.m[m]);
}

}  // namespace gcs
