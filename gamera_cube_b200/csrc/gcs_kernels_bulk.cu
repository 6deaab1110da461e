// FP32-bulk instantiation of the flux, face-velocity and edge-EMF sweeps
// (gcs_sweeps.cuh), built with FMA contraction.  The predictor, seam and
// edge syncs, CT and cell update are the FP64 kernels of gcs_kernels.cu.
#define GCS_SWEEPS_TEMPLATES_ONLY
#include "gcs_sweeps.cuh"

namespace gcs {

void launch_flux_f32(const Ctx &X, const Opts &O, int i0, int i1, cudaStream_t s) {
  if (i1 <= X.D.g || i0 > X.D.g + X.D.nr) return;
  // options outside FP32 fail the step here: the sweep reads 1 / (gamma - 1)
  // and 1 / c^2, not gamma and c
  const float gamma = (float)O.s_gamma, c = (float)O.s_c;
  if (!(gamma > 1.0f) || !isfinite(gamma)) {
    launch_set_failure(X, kStageKineticFluid, 0, s);
    return;
  }
  if (O.s_mhd && O.s_boris && !(c > FLT_MIN && isfinite(c))) {
    launch_set_failure(X, kStageKineticMaxwell, 0, s);
    return;
  }
  Sweeps<float>::flux(X, X.B32, O, i0, i1, s);
}
void launch_face_velocity_f32(const Ctx &X, const Opts &O, int i0, int i1,
                              cudaStream_t s) {
  Sweeps<float>::emf(X, X.B32, O, i0, i1, s);
}
void launch_edge_emf_f32(const Ctx &X, const Opts &O, int i0, int i1, cudaStream_t s) {
  Sweeps<float>::edge(X, X.B32, O, i0, i1, s);
}

int prepare_flux_f32() { return prepare_flux_tma<float>(); }

}  // namespace gcs
