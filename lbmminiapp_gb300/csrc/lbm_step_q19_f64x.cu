// D3Q19 step kernels with FP64 population storage and F64X arithmetic (without
// per-cell fields).
#include "lbm_dispatch.cuh"

namespace lbm {

cudaError_t launch_step_q19_f64x(int kind, const Launch& L, const KParams& p, const void* src, void* dst, bool links)
{
   return launch_step_t<19, ST_F64, AR_F64X>(kind, L, p, src, dst, links, false);
}

}  // namespace lbm
