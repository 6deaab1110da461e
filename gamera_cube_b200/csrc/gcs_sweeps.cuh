// Predictor, flux and EMF sweeps, CT and cell update, generic in the bulk
// type T of the sweeps.
//
// T = double is the plain FP64 path: every array of the Bulk<double> view
// is the FP64 array of DevState/DevGeom/DevBg.  The flux, face-velocity and
// edge-EMF sweeps (gcs_kernels_fp64.cu) are built with FMA contraction and
// take reciprocals, roots and the erfc/exp pair of gcs_physics.cuh: the
// reference's formulas to a few roundings.  The predictor, CT and cell update
// (gcs_kernels.cu) keep the reference's operations, without contraction.
// T = float is the FP32-bulk path (gcs_kernels_bulk.cu, built with FMA):
// the predictor still advances the FP64 state and also writes FP32 copies
// of the cell primitives, cell B, face normal fields and EMF weights; the
// flux, face-velocity and edge-EMF sweeps of the radial layers where the
// background field is weak compute in FP32 from FP32 metric and background,
// the layers near the inner boundary (strong dipole) in FP64; every sweep
// stores FP64 fluxes, face velocities and EMFs, which CT and the cell
// update accumulate into the FP64 face flux and conserved state.  Each
// sweep launch covers one radial range [i0, i1).
#pragma once

#include "gcs_kernel_util.cuh"
#include "gcs_kernels.cuh"
#include "gcs_physics.cuh"
#include "gcs_face_flux.cuh"
#include "gcs_flux_tma.cuh"

namespace gcs {

#ifndef GCS_SWEEPS_TEMPLATES_ONLY
// The non-template kernels below are compiled in gcs_kernels.cu only.

// Predictor over every cell/face (nonorthogonal_step.c:379-419): Phi~, U~,
// B~ in FP64; primitives of U~ with the sweep options (rho NaN where the
// conversion fails), Phi~/area and the EMF weights V m / max(rho, floor)
// for the sweeps, in FP64 and (bulk) FP32.
__global__ void __launch_bounds__(256, 4) k_predict(Dims D, DevState S, DevGeom G, Bulk<float> B32, int bulk,
                          Opts O, const StepParams *prm, DevStatus *st) {
  const unsigned long long first = failure_word(st);
  int f, i, j, k;
  const Box b{0, 0, 0, D.N1, D.N2, D.E0 + 1};
  if (!box_coord(b, &f, &i, &j, &k)) return;
  const double r = prm->ratio;
  const unsigned c = (unsigned)(f * D.Nn + D.node(i, j, k));
  // FP32 copies exist for the layers [B32.lo, N0) only
  const bool wb = bulk && i >= B32.lo;
  const unsigned cb = wb ? (unsigned)B32.at(f, D.node(i, j, k)) : 0;
  const bool cell = i < D.E0 && j < D.E1 && k < D.E2;
  const int coord[3] = {i, j, k};
  double phi[6], bn[3];
  bool in[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    in[d] = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) in[d] = in[d] && coord[a] < D.ext(a) + (a == d ? 1 : 0);
    phi[2 * d] = bn[d] = 0.0;
    if (in[d]) {
      const double p = S.P[d][c];
      phi[2 * d] = p + r * (p - S.Po[d][c]);
      bn[d] = phi[2 * d] / G.area[d][c];
    }
  }
  double up[5], bp[3], prv[5], v = 0.0;
  bool ok = true, recovered = true;
  if (cell) {
    double uo[5], uc[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      uo[m] = S.Uo[m][c];
      uc[m] = S.U[m][c];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const unsigned u = c + (unsigned)D.stride(d);
      const double p = S.P[d][u];
      phi[2 * d + 1] = p + r * (p - S.Po[d][u]);
    }
    v = G.vol[c];
    recovered = recover_cell(G, c, phi, bp);
    ok = predict_cell(uo, uc, r, O.u_gamma, O.u_rho_floor, O.u_p_floor, up) == 0;
    Prim pr;
    if (cons_to_prim(up, O.s_gamma, O.s_rho_floor, O.s_p_floor, &pr)) pr.rho = NAN;
    prv[0] = pr.rho;
    prv[1] = pr.vx;
    prv[2] = pr.vy;
    prv[3] = pr.vz;
    prv[4] = pr.p;
  }
  if (stopped(first, kPassPredict)) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!in[d]) continue;
    S.Pp[d][c] = phi[2 * d];
    S.BN[d][c] = bn[d];
    if (wb) B32.BN[d][cb] = (float)bn[d];
  }
  if (!cell) return;
  if (!ok) {
    fail(st, kStagePredict, 0, f, i, j, k);
    return;
  }
  if (!recovered) fail(st, kStageRecoverPredict, 0, f, i, j, k);
  const double rho = fmax(up[0], O.e_rho_floor);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    S.Up[m][c] = up[m];
    S.Pr[m][c] = prv[m];
    if (wb) B32.Pr[m][cb] = (float)prv[m];
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double w = v * up[1 + m] / rho;
    S.W[m][c] = w;
    S.Bp[m][c] = bp[m];
    if (wb) {
      B32.W[m][cb] = (float)w;
      B32.Bp[m][cb] = (float)bp[m];
    }
  }
}
#endif  // GCS_SWEEPS_TEMPLATES_ONLY

// Minimum resident blocks of 128 threads per SM the sweeps are compiled for
// (register caps 128 and 80 in FP64, 80 and 64 in FP32), from measured full-step
// sweeps at 6 x 96x96x192.
template <typename T>
struct SweepOccupancy {
  static constexpr int flux = 4;
  static constexpr int edge = 6;
};
template <>
struct SweepOccupancy<float> {
  static constexpr int flux = 6;
  static constexpr int edge = 8;
};

// ---------------------------------------------------------------------------
// Face-flux sweep, all three directions (nonorthogonal_sweep.c:408-548).
// Each thread owns one face; the eight-cell stencil of one variable at a
// time is read from the predictor's cell primitives (face_flux,
// gcs_face_flux.cuh).
// Bound: FP64 issue and latency at 16 warps an SM (128 registers; 3 to 5
// blocks of 128 measured within 2 %).  All directions in one launch find a
// layer's cells in L2 (a launch each: 3.81 against 3.67 ms).  6 x 96x96x192:
// 4.46 -> 3.01 ms a step, 2774 -> 1740 instructions a face.
template <bool kOrtho, typename T>
__global__ void __launch_bounds__(128, SweepOccupancy<T>::flux)
    k_flux(Dims D, DevState S, const __grid_constant__ Bulk<T> B, Opts O, DevStatus *st,
           const __grid_constant__ Boxes X) {
  const int group = (int)blockIdx.y / 3, d = (int)blockIdx.y - 3 * group;
  int f, i, j, k;
  if (!box_coord(X.b[d], &f, &i, &j, &k, group)) return;
  const FaceAt at{f, i, j, k, (unsigned)(f * D.Nn + D.node(i, j, k)),
                  (unsigned)B.at(f, D.node(i, j, k))};
  const GlobalStencil<T> cells(B, at.cb, (int)D.stride(d));
  face_flux<kOrtho, T>(d, cells, D, S, B, O, st, at);
}

#ifndef GCS_SWEEPS_TEMPLATES_ONLY
// Seam flux synchronisation (cubedsphere_interface.c:40-81): the fluid and
// Maxwell face fluxes of each seam face pair are set to their oriented mean.
__global__ void k_seam_flux(Dims D, const Seam *seams, DevState S, DevStatus *st) {
  if (failed(st)) return;
  const long long per = (long long)D.nr * D.n;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 12 * per) return;
  const Seam sm = seams[t / per];
  const int rem = (int)(t % per);
  const int i = D.g + rem / D.n;
  const int along = rem % D.n;
  const int dalong = sm.reversed ? D.n - 1 - along : along;
  int src[3] = {i, D.g + along, D.g + along};
  int tgt[3] = {i, D.g + dalong, D.g + dalong};
  src[sm.src_axis] = sm.src_b;
  tgt[sm.dst_axis] = sm.dst_b;
  const long long s = sm.face * D.Nn + D.node(src[0], src[1], src[2]);
  const long long d = sm.nface * D.Nn + D.node(tgt[0], tgt[1], tgt[2]);
  const double o = sm.orient;
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    double *a = S.F[sm.src_axis][m], *b = S.F[sm.dst_axis][m];
    const double common = 0.5 * (a[s] + o * b[d]);
    a[s] = common;
    b[d] = o * common;
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    double *a = S.M[sm.src_axis][m], *b = S.M[sm.dst_axis][m];
    const double common = 0.5 * (a[s] + o * b[d]);
    a[s] = common;
    b[d] = o * common;
  }
}

#endif  // GCS_SWEEPS_TEMPLATES_ONLY

// ---------------------------------------------------------------------------
// Face velocities of face family a (nonorthogonal_sweep.c:223-259):
// central8 of the per-cell weights over central8 of the volumes, for every
// face the edge velocities of edge family (a+2)%3 read.
template <int a, typename T>
__device__ __forceinline__ void velocity_thread(const Dims &D, const Bulk<T> &B,
                                                DevStatus *st, const Box &b, int group) {
  const unsigned long long first = failure_word(st);
  int f, x[3];
  if (!box_coord(b, &f, &x[0], &x[1], &x[2], group)) return;
  const unsigned c = (unsigned)(f * D.Nn + D.node(x[0], x[1], x[2]));
  const unsigned cb = (unsigned)B.at(f, D.node(x[0], x[1], x[2]));
  const LineStencil<a == 2> at(cb, (int)D.stride(a));
  const T iv = B.iv[a][cb];
  T w[3][8];
#pragma unroll
  for (int m = 0; m < 3; ++m) at.load(B.W[m], w[m]);
  const T riv = Num<T>::rcp(iv);
  if (first != 0ULL) return;
#pragma unroll
  for (int m = 0; m < 3; ++m) B.FV[a][m][c] = (double)(central8(w[m]) * riv);
}
template <typename T>
__global__ void k_face_velocity(Dims D, Bulk<T> B, DevStatus *st, Boxes X) {
  const int group = (int)blockIdx.y / 3, a = (int)blockIdx.y - 3 * group;
  if (a == 0)
    velocity_thread<0, T>(D, B, st, X.b[0], group);
  else if (a == 1)
    velocity_thread<1, T>(D, B, st, X.b[1], group);
  else
    velocity_thread<2, T>(D, B, st, X.b[2], group);
}

// ---------------------------------------------------------------------------
// Edge EMF sweep of edge family e (nonorthogonal_sweep.c:624-752).
// Bound: L2 and HBM traffic (225 B an edge from HBM at 4.5 TB/s, 13 TB/s from
// L2).  The three families run in one launch because they read the same face
// velocities, areas and fields: 6 x 96x96x192, with the face velocities, 2.40
// -> 2.11 ms a step, against 3.02 with a launch per family.
template <int e, typename T>
__device__ __forceinline__ void edge_thread(const Dims &D, const DevState &S,
                                            const unsigned char *edge_ok, const Bulk<T> &B,
                                            const Opts &O, const StepParams *prm,
                                            DevStatus *st, const Box &b, int group) {
  constexpr int a = (e + 1) % 3, bb = (e + 2) % 3;
  const unsigned long long first = failure_word(st);
  int f, x[3];
  if (!box_coord(b, &f, &x[0], &x[1], &x[2], group)) return;
  const unsigned c = (unsigned)(f * D.Nn + D.node(x[0], x[1], x[2]));
  const unsigned cb = (unsigned)B.at(f, D.node(x[0], x[1], x[2]));
  const unsigned char geometry = edge_ok[c];
  const int sa = (int)D.stride(a), sb = (int)D.stride(bb);
  const T pdm2 = T(2.0) * (T)O.e_pdm;
  // edge velocity: faces of family a along bb
  T fld[8];
  T v[3];
  T fl, fr, sl, sr;
  {
    const LineStencil<bb == 2> at(cb, sb), full(c, sb);
    T ar[8];
    at.load(B.area[a], ar);
    const T rca = Num<T>::rcp(B.ca[e][cb]);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double fv[8];
      full.load(B.FV[a][m], fv);
      T w[8];
#pragma unroll
      for (int n = 0; n < 8; ++n) w[n] = ar[n] * (T)fv[n];
      v[m] = central8(w) * rca;
    }
    // transverse face fields (nonorthogonal_sweep.c:372-406)
    at.load(B.BN[a], fld);
    up7_pdm(Up7Weights<T>(ar, rca), fld, pdm2, &fl, &fr);
  }
  const T vt1 = dot3(v[0], v[1], v[2], B.et1[e][0][cb], B.et1[e][1][cb], B.et1[e][2][cb]);
  const T vt2 = dot3(v[0], v[1], v[2], B.et2[e][0][cb], B.et2[e][1][cb], B.et2[e][2][cb]);
  {
    const LineStencil<a == 2> at(cb, sa);
    T ar[8];
    at.load(B.area[bb], ar);
    at.load(B.BN[bb], fld);
    up7_pdm(Up7Weights<T>(ar, Num<T>::rcp(B.cb[e][cb])), fld, pdm2, &sl, &sr);
  }
  // 2x2 edge solve (nonorthogonal_operators.c:56-79)
  const T f1 = T(0.5) * (fl + fr);
  const T f2 = T(0.5) * (sl + sr);
  const T inv = B.einv[e][cb];
  const T n10 = B.en1[e][0][cb], n11 = B.en1[e][1][cb];
  const T n20 = B.en2[e][0][cb], n21 = B.en2[e][1][cb];
  T ef0 = inv * (n21 * f1 - n11 * f2);
  T ef1 = inv * (-n20 * f1 + n10 * f2);
  if (O.e_bg) {
    ef0 += B.eb0t1[e][cb];
    ef1 += B.eb0t2[e][cb];
  }
  const T jump = (sr - sl) - (fr - fl);
  // edge density (nonorthogonal_sweep.c:351-370), from the FP64 state
  const double *up0 = S.Up[0];
  double rho = 0.0;
  rho += 0.25 * up0[c];
  rho += 0.25 * up0[c - (unsigned)sb];
  rho += 0.25 * up0[c - (unsigned)sa];
  rho += 0.25 * up0[c - (unsigned)(sa + sb)];
  const bool rho_ok = isfinite(rho) && rho > DBL_MIN;
  T emf;
  const bool emf_ok =
      edge_emf(vt1, vt2, ef0, ef1, jump, (T)rho, B.elen[e][cb], (T)O.e_diff, O.e_boris,
               sizeof(T) == 8 ? (T)O.e_c : (T)O.e_ic2,
               (T)(O.e_cfl * Num<double>::rcp(prm->dt)), &emf) == 0;
  if (stopped(first, kPassEmf)) return;
  if (geometry != 0 || !rho_ok || !emf_ok) {
    fail(st, geometry != 0 ? geometry : !rho_ok ? kStageEdgeDensity : kStageEdgeEmf, e, f,
         x[0], x[1], x[2]);
    return;
  }
  B.E[e][c] = (double)emf;
}
template <typename T>
__global__ void __launch_bounds__(128, SweepOccupancy<T>::edge)
    k_edge_emf(Dims D, DevState S, DevGeom G, Bulk<T> B, Opts O, const StepParams *prm,
               DevStatus *st, Boxes X) {
  const int group = (int)blockIdx.y / 3, e = (int)blockIdx.y - 3 * group;
  if (e == 0)
    edge_thread<0, T>(D, S, G.edge_ok[0], B, O, prm, st, X.b[0], group);
  else if (e == 1)
    edge_thread<1, T>(D, S, G.edge_ok[1], B, O, prm, st, X.b[1], group);
  else
    edge_thread<2, T>(D, S, G.edge_ok[2], B, O, prm, st, X.b[2], group);
}

#ifndef GCS_SWEEPS_TEMPLATES_ONLY
// Signed mean over each group of coincident seam/corner edges
// (cubedsphere_interface.c:217-242); members in the reference's sorted
// order.
__global__ void k_edge_sync(Dims D, const int *offsets, const EdgeMember *mem,
                            int groups, DevState S, DevStatus *st) {
  if (failed(st)) return;
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= groups) return;
  const int b = offsets[gi], e = offsets[gi + 1];
  double common = 0.0;
  for (int t = b; t < e; ++t) {
    const EdgeMember m = mem[t];
    common += (double)m.sign * S.E[m.dir][m.face * D.Nn + m.node];
  }
  common /= (double)(e - b);
  for (int t = b; t < e; ++t) {
    const EdgeMember m = mem[t];
    S.E[m.dir][m.face * D.Nn + m.node] = (double)m.sign * common;
  }
}

// ---------------------------------------------------------------------------
// Save Phi -> Phi_old on every face, then the CT curl on active faces
// (nonorthogonal_step.c:233-298, 361-377): the three faces of a node share
// its edge EMFs, nine reads where a launch per family makes twelve.  families:
// bit per face family of the launch.
__global__ void k_ct(Dims D, DevState S, Opts O, int families, const StepParams *prm,
                     DevStatus *st) {
  const unsigned long long first = failure_word(st);
  int f, x[3];
  const Box b{0, 0, 0, D.E1 + 1, D.E2 + 1, D.E0 + 1};
  if (!box_coord(b, &f, &x[0], &x[1], &x[2])) return;
  const unsigned c = (unsigned)(f * D.Nn + D.node(x[0], x[1], x[2]));
  const unsigned s0 = (unsigned)D.stride(0), s1 = (unsigned)D.stride(1);
  bool in[3], active[3];
  double old[3], curl[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    in[d] = families >> d & 1;
    active[d] = in[d] && O.u_mhd;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      in[d] = in[d] && x[a] < D.ext(a) + (a == d);
      active[d] = active[d] && x[a] >= D.g && x[a] < D.g + D.act(a) + (a == d);
    }
    old[d] = in[d] ? S.P[d][c] : 0.0;
  }
  double *const *E = S.E;
  if (active[0] || active[1] || active[2]) {
    // edge reads of an inactive face of the node stay inside the arrays
    const double e0 = E[0][c], e1 = E[1][c], e2 = E[2][c];
    if (active[0]) curl[0] = E[2][c + s1] - e2 - E[1][c + 1] + e1;
    if (active[1]) curl[1] = E[0][c + 1] - e0 - E[2][c + s0] + e2;
    if (active[2]) curl[2] = E[1][c + s0] - e1 - E[0][c + s1] + e0;
  }
  const double dt = prm->dt;
  if (first != 0ULL) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (in[d]) S.Po[d][c] = old[d];
    if (active[d]) S.P[d][c] = old[d] - dt * curl[d];
  }
}

// Cell update (nonorthogonal_step.c:527-610 with the stress rates of
// nonorthogonal_sweep.c:550-622) and final recovery (cubedsphere_step.c:
// 142-152) of every cell: save U, B as old, on active cells U += dt * rate,
// recover B from the CT-updated Phi, apply the Boris (nonorthogonal_state.c:
// 161-280) or Maxwell momentum update, store B; in driver mode the CFL time
// step of the new state (nonorthogonal_step.c:449-525).
//
// The reference recovers B before the seam sync of Phi for the momentum
// update and again after it on every cell.  The two sides of a seam face
// carry the same synced Phi and edge EMFs, so the sync moves Phi by the
// rounding of the curl only; here it runs before this kernel (after it only
// where a host callback may have set the sides apart) and one recovery serves
// both uses, which saves a second pass over the recovery
// map, Phi, U and B0 (264 B per cell).  Bound: HBM (4.9 TB/s).  Four blocks an
// SM (124 registers): at six, the bound without the recovery, it spills.
// 6 x 96x96x192, CT, update and recovery: 2.72 -> 1.79 ms a step (six blocks
// 2.21, five 1.99).
__global__ void __launch_bounds__(128, 4) k_update(Dims D, DevState S, DevGeom G,
                                                DevBg BG, Opts O, int with_cfl,
                                                const StepParams *prm,
                                                DevStatus *st) {
  const unsigned long long first = failure_word(st);
  int f, i, j, k;
  const Box b{0, 0, 0, D.E1, D.E2, D.E0};
  double cand = DBL_MAX;
  if (box_coord(b, &f, &i, &j, &k)) {
    const unsigned c = (unsigned)(f * D.Nn + D.node(i, j, k));
    const unsigned sdir[3] = {(unsigned)D.stride(0), (unsigned)D.stride(1), 1u};
    const bool active = i >= D.g && i < D.g + D.nr && j >= D.g && j < D.g + D.n &&
                        k >= D.g && k < D.g + D.n;
    double uold[5], bo[3], bn[3] = {0.0, 0.0, 0.0}, b0[3] = {0.0, 0.0, 0.0};
    bool recovered = true;
#pragma unroll
    for (int m = 0; m < 5; ++m) uold[m] = S.U[m][c];
#pragma unroll
    for (int m = 0; m < 3; ++m) bo[m] = S.B[m][c];
    if (O.u_mhd) {
      double phi[6];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        phi[2 * d] = S.P[d][c];
        phi[2 * d + 1] = S.P[d][c + sdir[d]];
      }
      recovered = recover_cell(G, c, phi, bn);
    }
    double u[5];
    int code = recovered ? kStageNone : active ? kStageRecoverUpdate : kStageRecoverFinal;
    if (active) {
      const double dt = prm->dt;
      const double iv = G.ivol[c];
      double rate[5], mrate[3];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        double diff = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) diff += S.F[d][m][c] - S.F[d][m][c + sdir[d]];
        rate[m] = diff * iv;
        u[m] = uold[m] + dt * rate[m];
      }
      if (O.u_mhd) {
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          double diff = 0.0;
#pragma unroll
          for (int d = 0; d < 3; ++d)
            diff += S.M[d][m][c] - S.M[d][m][c + sdir[d]];
          mrate[m] = diff * iv;
          if (O.u_bg) mrate[m] += BG.force[m][c];
          if (O.u_bg || (with_cfl && O.t_bg)) b0[m] = BG.b0[m][c];
        }
        if (O.u_boris) {
          double nb[3], ob[3];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            nb[m] = O.u_bg ? bn[m] + b0[m] : bn[m];
            ob[m] = O.u_bg ? bo[m] + b0[m] : bo[m];
          }
          if (apply_boris(u, uold, nb, ob, rate, mrate, O.u_c, dt, O.u_gamma,
                          O.u_rho_floor, O.u_p_floor) &&
              code == kStageNone)
            code = kStageUpdate;
        } else {
          apply_maxwell(u, mrate, dt, O.u_gamma, O.u_rho_floor, O.u_p_floor);
        }
      }
    }
    if (!stopped(first, kPassUpdate, kPassTimestep)) {
#pragma unroll
      for (int m = 0; m < 5; ++m) S.Uo[m][c] = uold[m];
#pragma unroll
      for (int m = 0; m < 3; ++m) S.Bo[m][c] = bo[m];
      if (code != kStageNone) {
        fail(st, code, 0, f, i, j, k);
      } else {
        if (active) {
#pragma unroll
          for (int m = 0; m < 5; ++m) S.U[m][c] = u[m];
        }
        if (O.u_mhd) {
#pragma unroll
          for (int m = 0; m < 3; ++m) S.B[m][c] = bn[m];
          if (with_cfl && active && !cfl_step(O, u, bn, b0, G.cflmin[c], &cand))
            fail(st, kStageTimestep, 0, f, i, j, k);
        }
      }
    }
  }
  // every thread of the block reaches the reduction
  if (with_cfl) reduce_cfl(cand, st);
}

#endif  // GCS_SWEEPS_TEMPLATES_ONLY

// ---------------------------------------------------------------------------
// Launchers of the sweeps of one precision over the radial range [i0, i1)
// of the range each sweep covers (clamped to it; empty ranges launch
// nothing).

inline bool clamp_range(int lo, int hi, int i0, int i1, int *a, int *n) {
  *a = lo > i0 ? lo : i0;
  const int b = hi < i1 ? hi : i1;
  *n = b - *a;
  return *n > 0;
}

// Layer range of each family of a sweep over [i0, i1): family q covers
// [lo[q], hi[q]).  Returns the layer groups of the launch (0: nothing to do);
// an empty family has no points.
inline int clamp_boxes(Boxes &X, const int lo[3], const int hi[3], int i0, int i1, Tile t) {
  int groups = 0;
  for (int q = 0; q < 3; ++q) {
    int a = 0, n = 0;
    if (!clamp_range(lo[q], hi[q], i0, i1, &a, &n)) n = 0;
    X.b[q].i0 = a;
    X.b[q].i1 = a + n;
    const int g = (n + t.by - 1) / t.by;
    groups = g > groups ? g : groups;
  }
  return groups;
}
inline dim3 boxes_grid(const Boxes &X, int groups, Tile t) {
  int points = 0;
  for (int q = 0; q < 3; ++q) points = max(points, X.b[q].nj * X.b[q].nk);
  return dim3((unsigned)((points + t.bx - 1) / t.bx), 3u * (unsigned)groups, kFaces);
}
// A sweep's tile: grid.y holds the layer groups of three families in at most
// 65535 blocks, so a grid of more layers than that gets taller tiles.
inline Tile sweep_tile(Tile t, int layers) {
  while (3LL * ((layers + t.by - 1) / t.by) > 65535 && t.bx % 2 == 0) {
    t.bx /= 2;
    t.by *= 2;
  }
  return t;
}
template <typename T>
struct Sweeps {
  static void flux(const Ctx &X, const Bulk<T> &B, const Opts &O, int i0, int i1,
                   cudaStream_t s) {
    const Dims &D = X.D;
    if (X.flux_staged) {
      int a, n;
      if (clamp_range(D.g, D.g + D.nr + 1, i0, i1, &a, &n))
        launch_flux_tma<0, T>(X, B, O, a, a + n, s);
      if (clamp_range(D.g, D.g + D.nr, i0, i1, &a, &n))
        launch_flux_tma<1, T>(X, B, O, a, a + n, s);
      if (clamp_range(D.g, D.g + D.nr, i0, i1, &a, &n))
        launch_flux_tma<2, T>(X, B, O, a, a + n, s);
      return;
    }
    const Tile t = sweep_tile(X.tile[kTileFlux], D.E0 + 1);
    Boxes b;
    for (int d = 0; d < 3; ++d)
      b.b[d] = Box{0, D.g, D.g, D.n + (d == 1), D.n + (d == 2), 0};
    const int lo[3] = {D.g, D.g, D.g}, hi[3] = {D.g + D.nr + 1, D.g + D.nr, D.g + D.nr};
    // FP32 reads the tangents: its rounded frame is not orthonormal to FP32
    constexpr bool kFp64 = sizeof(T) == 8;
    const bool ortho = X.ortho && kFp64;
    const int groups = clamp_boxes(b, lo, hi, i0, i1, t);
    if (groups > 0)
      (ortho ? k_flux<kFp64, T> : k_flux<false, T>)
          <<<boxes_grid(b, groups, t), tile_block(t), 0, s>>>(D, X.S, B, O, X.status, b);
  }
  static void emf(const Ctx &X, const Bulk<T> &B, const Opts &O, int i0, int i1,
                  cudaStream_t s) {
    const Dims &D = X.D;
    // face velocities: family a, edge family e=(a+2)%3 active, a faces, bb all
    const Tile t = sweep_tile(X.tile[kTileFaceVelocity], D.E0 + 1);
    Boxes b;
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      const int e = (a + 2) % 3, bb = (a + 1) % 3;
      int first[3], count[3];
      first[e] = D.g; count[e] = D.act(e);
      first[a] = D.g; count[a] = D.act(a) + 1;
      first[bb] = 0; count[bb] = D.ext(bb);
      lo[a] = first[0];
      hi[a] = first[0] + count[0];
      b.b[a] = Box{0, first[1], first[2], count[1], count[2], 0};
    }
    // all families at once, or one at a time (Ctx::fine_launches)
    for (int only = X.fine_launches ? 0 : -1; only < (X.fine_launches ? 3 : 0); ++only) {
      int l[3], h[3];
      for (int a = 0; a < 3; ++a) {
        const bool on = only < 0 || a == only;
        l[a] = on ? lo[a] : 0;
        h[a] = on ? hi[a] : 0;
      }
      const int groups = clamp_boxes(b, l, h, i0, i1, t);
      if (groups > 0)
        k_face_velocity<T><<<boxes_grid(b, groups, t), tile_block(t), 0, s>>>(D, B, X.status,
                                                                              b);
    }
  }
  static void edge(const Ctx &X, const Bulk<T> &B, const Opts &O, int i0, int i1,
                   cudaStream_t s) {
    const Dims &D = X.D;
    const Tile t = sweep_tile(X.tile[kTileEdgeEmf], D.E0 + 1);
    Boxes b;
    int lo[3], hi[3];
    for (int e = 0; e < 3; ++e) {
      lo[e] = D.g;
      hi[e] = D.g + D.nr + (e != 0);
      b.b[e] = Box{0, D.g, D.g, D.n + (e != 1), D.n + (e != 2), 0};
    }
    const int groups = clamp_boxes(b, lo, hi, i0, i1, t);
    if (groups > 0)
      k_edge_emf<T><<<boxes_grid(b, groups, t), tile_block(t), 0, s>>>(
          D, X.S, X.G, B, O, X.params, X.status, b);
  }
};

}  // namespace gcs
