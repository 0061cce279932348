// D3Q19 step kernels with FP64 population storage: exact FP64 arithmetic, and
// the choice between it and F64X.
#include "lbm_dispatch.cuh"

namespace lbm {

cudaError_t launch_step_q19_f64(int arith, int kind, const Launch& L, const KParams& p,
                                const void* src, void* dst, bool links, bool fields)
{
   // per-cell fields use the exact FP64 arithmetic
   if (arith == AR_F64X && !fields) return launch_step_q19_f64x(kind, L, p, src, dst, links);
   return launch_step_t<19, ST_F64, AR_F64>(kind, L, p, src, dst, links, fields);
}

}  // namespace lbm
