// Density and velocity readout kernel.
#pragma once

#include "lbm_aux.cuh"
#include "lbm_moments.cuh"
#include "lbm_step.cuh"

namespace lbm {

// rho and u = sum(c f)/rho (no F/2 shift) for the cells [c0, c0+count);
// cell c0+k goes to rho[k] and u[d*out_stride + k]; NaN at solid cells.  mode as
// for export_plane_kernel: 0 slot s holds direction s, 1 slot opp(s) does, 2 pull
// gather.  FP64 storage: the sums are the reference's, rounded after every
// addition, so that the readout of equal populations is equal text; the shifted
// formats are summed in integers and rounded once (CellMoments).
//
// Bound by the host link for page-locked arrays (67 MB at 189 GB/s for 128^3).
// With the 49 adds per cell on the FP64 pipe the kernel alone took 290 us there.
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
   // stored value of direction s
   const auto load = [&](int s) {
      Access a{MODE == 1 ? lat_opp(Q, s) : s, 0};
      if constexpr (MODE == 2) a = read_access<Q, K_AB_PULL, true>(ci, lk, s);
      return moment_value<ST>(buf, (int64_t)a.slot * g.plane + (c + a.off));
   };
   double r, m[3];
   if constexpr (ST == ST_F64) {
      if (!sums_soft<Q>(load, r, m)) {
         r = m[0] = m[1] = m[2] = 0.0;
#pragma unroll
         for (int s = 0; s < Q; s++) {
            const double f = x64::as_double(load(s));
            r = __dadd_rn(r, f);
#pragma unroll
            for (int d = 0; d < 3; d++) {
               const int cd = lat_c(Q, s, d);
               if (cd > 0) m[d] = __dadd_rn(m[d], f);
               else if (cd < 0) m[d] = __dsub_rn(m[d], f);
            }
         }
      }
   } else {
      const CellMoments<Q, ST, decltype(load)> mom(load);
      mom.get(r, m);
   }
   const double ir = 1.0 / r;
   rho[k] = r;
   u[k] = m[0] * ir;
   u[out_stride + k] = m[1] * ir;
   u[2 * out_stride + k] = m[2] * ir;
}

}  // namespace lbm
