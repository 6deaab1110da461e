// Device helpers shared by the step kernels: failure recording, box
// iteration and the calibrated B recovery.
#pragma once

#include <cfloat>

#include "gcs_device.cuh"
#include "gcs_physics.cuh"

namespace gcs {

namespace {

__device__ inline void fail(DevStatus *st, int stage, int dir, int face,
                            int i, int j, int k) {
  const unsigned long long mine = pack_failure(stage, dir, face, i, j, k);
  unsigned long long seen = atomicCAS(&st->first, 0ULL, mine);
  while (seen != 0ULL && fails_before(mine, seen)) {
    const unsigned long long was = atomicCAS(&st->first, seen, mine);
    if (was == seen) break;
    seen = was;
  }
  atomicOr(&st->stage_mask, 1u << stage);
}

// The step's failure word.  The sweeps and cell kernels load it first and
// test it before their first store, so the wait for it overlaps their other
// loads; tested at the top it costs every thread a trip to L2 before the
// first useful load.
__device__ inline unsigned long long failure_word(const DevStatus *st) {
  return *(volatile const unsigned long long *)&st->first;
}
__device__ inline bool failed(const DevStatus *st) { return failure_word(st) != 0ULL; }
// Whether a kernel of stage groups [pass, last] has to leave everything as it
// is: a failure of an earlier group or step.  A failure of its own groups
// stops no thread, so the one reported, and what the others store, do not
// depend on the order in which the blocks run.
__device__ inline bool stopped(unsigned long long first, int pass, int last) {
  if (first == 0ULL) return false;
  const int p = stage_pass(failure_stage(first));
  return (first & kEarlierStep) != 0ULL || p < pass || p > last;
}
__device__ inline bool stopped(unsigned long long first, int pass) {
  return stopped(first, pass, pass);
}

// Box iteration over radial layers [i0, i1): a thread block is a tile of
// blockDim.x consecutive points of the flattened (j, k) plane times
// blockDim.y consecutive layers; grid.x over j*k, grid.y over the layer
// groups, grid.z face.
struct Box {
  int i0, j0, k0, nj, nk, i1;
};
// The boxes of the three families of a sweep, one launch for all of them:
// grid.y counts layer groups times three, the family changing fastest, so
// the three families of a layer run together and find its cells in L2.
struct Boxes {
  Box b[3];
};

__device__ inline bool box_coord(const Box &b, int *f, int *i, int *j,
                                 int *k, int group) {
  const int jk = blockIdx.x * blockDim.x + threadIdx.x;
  const int ii = b.i0 + group * (int)blockDim.y + threadIdx.y;
  if (jk >= b.nj * b.nk || ii >= b.i1) return false;
  *f = blockIdx.z;
  *i = ii;
  *j = b.j0 + jk / b.nk;
  *k = b.k0 + jk % b.nk;
  return true;
}
__device__ inline bool box_coord(const Box &b, int *f, int *i, int *j, int *k) {
  return box_coord(b, f, i, j, k, (int)blockIdx.y);
}

// Calibrated recovery, cubedsphere/cubedsphere_recovery.c:69-98, applied as
// the precomputed 3x6 map (response inverse times the moment formula of
// nonorthogonal_operators.c:17-54).  Face order: i-lo, i-hi, j-lo, j-hi,
// k-lo, k-hi.
__device__ inline bool recover_cell(const DevGeom &G, long long c,
                                    const double phi[6], double b[3]) {
  const bool ok = G.cell_ok[c];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    double s = 0.0;
#pragma unroll
    for (int col = 0; col < 6; ++col) s += G.rec[r * 6 + col][c] * phi[col];
    b[r] = s;
  }
  return ok && isfinite(b[0]) && isfinite(b[1]) && isfinite(b[2]);
}

// cubedsphere_halo.c:103-115
__device__ inline bool halo_valid(const double s[5]) {
  const double rho = s[0];
  if (!isfinite(rho) || rho <= 0.0) return false;
  double m2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!isfinite(s[1 + d])) return false;
    m2 += s[1 + d] * s[1 + d];
  }
  return isfinite(s[4]) && s[4] > 0.5 * m2 / rho;
}

// CFL time step of one cell (nonorthogonal_step.c:449-525) from its state,
// residual B and B0; false where the reference fails.
__device__ inline bool cfl_step(const Opts &O, const double u[5], const double bn[3],
                                const double b0[3], double cflmin, double *step) {
  Prim p;
  if (cons_to_prim(u, O.t_gamma, O.t_rho_floor, O.t_p_floor, &p)) return false;
  const double cs = sqrt(O.t_gamma * p.p / p.rho);
  double va = 0.0;
  if (O.t_mhd) {
    double bx = bn[0], by = bn[1], bz = bn[2];
    if (O.t_bg) {
      bx = bn[0] + b0[0];
      by = bn[1] + b0[1];
      bz = bn[2] + b0[2];
    }
    double s2 = 0.0;
    s2 += bx * bx;
    s2 += by * by;
    s2 += bz * bz;
    va = sqrt(s2) / sqrt(p.rho);
    if (O.t_boris) va = O.t_c * va / hypot(O.t_c, va);
  }
  double v2 = 0.0;
  v2 += p.vx * p.vx;
  v2 += p.vy * p.vy;
  v2 += p.vz * p.vz;
  const double speed = sqrt(v2) + hypot(cs, va);
  const double cand = O.t_cfl * cflmin / speed;
  if (!isfinite(cand) || cand <= 0.0) return false;
  *step = cand;
  return true;
}

// Minimum over the block's threads (at most 256), then one atomic (positive
// doubles order as unsigned 64-bit integers).
__device__ inline void reduce_cfl(double cand, DevStatus *st) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    cand = fmin(cand, __shfl_down_sync(0xffffffffu, cand, o));
  __shared__ double wmin[8];
  const int lt = threadIdx.y * blockDim.x + threadIdx.x;
  const int lane = lt & 31, warp = lt >> 5;
  if (lane == 0) wmin[warp] = cand;
  __syncthreads();
  if (warp == 0) {
    cand = lane < (int)((blockDim.x * blockDim.y) >> 5) ? wmin[lane] : DBL_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      cand = fmin(cand, __shfl_down_sync(0xffffffffu, cand, o));
    if (lane == 0 && cand < DBL_MAX)
      atomicMin(&st->cfl_min_bits, (unsigned long long)__double_as_longlong(cand));
  }
}

}  // namespace

}  // namespace gcs
