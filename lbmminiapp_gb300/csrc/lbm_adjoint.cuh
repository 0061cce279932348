// Parameters of the adjoint and loss kernels (lbm_adjoint.cu).
#pragma once

#include <cuda_runtime.h>

#include "lbm_aux.cuh"
#include "lbm_step_async.cuh"

namespace lbm {

// Launch constants of the adjoint in its arithmetic, made on the host.
template <typename R>
struct AdjConsts {
   R om, om1, om2, tw, F[3];   // omega, 1 - omega, 1 - omega/2, time weight, uniform force
};

struct AdjParams {
   GridDims g;
   double omega;
   double F[3];
   const uint32_t* links;
   const double* force_field;     // planar [3][plane] or null
   const double* porosity;        // [plane] or null
   // FP32 copies of the fields for the FP32 adjoint, where they hold what it would
   // round the FP64 ones to (the force field only without a uniform force), or null
   const float* force_field_f;
   const float* porosity_f;
   const void* state;             // f^t, the handle's storage, slot s = direction s
   const double* lam_next;        // [Q][plane]
   double* lam;                   // [Q][plane]
   double* grad_force;            // [3][plane] accumulated, or null
   double* grad_porosity;         // [plane] accumulated, or null
   const double* loss_weight;     // velocity: [3][plane]; energy: [plane]; or null
   double time_weight;
   int loss_kind;
   int collide;                   // 0: loss term only (the last state of a rollout)
   const float* lam_next_f;       // FP32 adjoint: [Q][plane]
   float* lam_f;                  // FP32 adjoint: [Q][plane]
   AsyncGeom ag;                  // this and the constants: set by the launch functions
   AdjConsts<double> k;
   AdjConsts<float> kf;
};

cudaError_t launch_adjoint(int Q, int storage, const AdjParams& a, cudaStream_t stream);
cudaError_t launch_adjoint_f32(int Q, int storage, const AdjParams& a, cudaStream_t stream);
cudaError_t launch_loss(int Q, int storage, const AdjParams& a, double* partials, int nblocks, double* out,
                        cudaStream_t stream);

}  // namespace lbm
