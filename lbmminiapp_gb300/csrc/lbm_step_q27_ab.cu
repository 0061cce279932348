// Pipelined D3Q27 AB step kernels for FP64 storage with F64X arithmetic.
#include "lbm_step_async.cuh"

namespace lbm {

template <>
cudaError_t launch_async_ab<27>(int kind, bool links, const KParams& p, const AsyncGeom& ag, const void* src, void* dst,
                                cudaStream_t stream)
{
   return kind == K_AB_PUSH ? launch_async_kind<27, K_AB_PUSH>(links, p, ag, src, dst, stream)
                            : launch_async_kind<27, K_AB_PULL>(links, p, ag, src, dst, stream);
}

}  // namespace lbm
