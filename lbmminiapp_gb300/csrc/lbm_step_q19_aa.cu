// Pipelined D3Q19 AA step kernels for FP64 storage with F64X arithmetic.
#include "lbm_step_async.cuh"

namespace lbm {

template <>
cudaError_t launch_async_aa<19>(int kind, bool links, const KParams& p, const AsyncGeom& ag, const void* src, void* dst,
                                cudaStream_t stream)
{
   return kind == K_AA_EVEN ? launch_async_kind<19, K_AA_EVEN>(links, p, ag, src, dst, stream)
                            : launch_async_kind<19, K_AA_ODD>(links, p, ag, src, dst, stream);
}

}  // namespace lbm
