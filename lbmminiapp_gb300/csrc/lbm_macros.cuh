// Density and velocity readout kernel.
#pragma once

#include "lbm_aux.cuh"
#include "lbm_moments.cuh"
#include "lbm_step.cuh"

namespace lbm {

// rho and u = sum(c f)/rho (no F/2 shift) for the cells [c0, c0+count);
// cell c0+k goes to rho[k] and u[d*out_stride + k]; NaN at solid cells.  mode as
// for export_plane_kernel.  In mode 1 slot s holds direction opp(s): the sums run
// over the slots and the momentum changes sign.
//
// Bound by memory and the rest of its FP64 instructions (a reciprocal and three
// products): the sums are CellMoments'.  At 128^3, D3Q19 FP64: 290 us in chunks
// when the 49 adds per cell ran on the FP64 pipe.
template <int Q, int ST, int MODE>
__global__ void __launch_bounds__(256) macros_kernel(GridDims g, int64_t c0, int64_t count, const void* buf,
                                                     const uint32_t* links, double* rho, double* u, int64_t out_stride)
{
   const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (k >= count) return;
   const int64_t c = c0 + k;
   const uint32_t lk = links ? links[c] : 0u;
   if (lk & kSolidBit) {
      const double nan = __longlong_as_double(0x7FF8000000000000LL);
      rho[k] = nan;
      u[k] = u[out_stride + k] = u[2 * out_stride + k] = nan;
      return;
   }
   CellIndex ci;
   ci.c = c;
   if constexpr (MODE == 2) {
      int x, y, z;
      cell_xyz(g, c, x, y, z);
      ci.dxm = (x == 0) ? g.nx - 1 : -1;
      ci.dxp = (x == g.nx - 1) ? -(g.nx - 1) : 1;
      ci.dym = (y == 0) ? (g.ny - 1) * g.nx : -g.nx;
      ci.dyp = (y == g.ny - 1) ? -(g.ny - 1) * g.nx : g.nx;
      const int nxy = g.nx * g.ny;
      ci.dzm = (z == 0) ? (g.nz - 1) * nxy : -nxy;
      ci.dzp = (z == g.nz - 1) ? -(g.nz - 1) * nxy : nxy;
   }
   const auto load = [&](int s) {
      Access a{s, 0};
      if constexpr (MODE == 2) a = read_access<Q, K_AB_PULL, true>(ci, lk, s);
      return moment_value<ST>(buf, (int64_t)a.slot * g.plane + (c + a.off));
   };
   const CellMoments<Q, ST, decltype(load)> mom(load);
   double r, m[3];
   mom.get(r, m);
   double ir = 1.0 / r;
   rho[k] = r;
   if constexpr (MODE == 1) ir = -ir;
   u[k] = m[0] * ir;
   u[out_stride + k] = m[1] * ir;
   u[2 * out_stride + k] = m[2] * ir;
}

}  // namespace lbm
