// Host build of the cell moments of the readouts and the loss
// (lbmminiapp_gb300/csrc/lbm_moments.cuh), for tests/test_moments_host.py.
#include <cstdint>

#include "lbm_moments.cuh"

using namespace lbm;

namespace {

template <int Q>
void run_f64(const double* f, int n, double* out, uint8_t* regular)
{
   for (int i = 0; i < n; i++) {
      const auto load = [&](int s) { return x64::double_bits(f[(int64_t)i * Q + s]); };
      const CellMoments<Q, ST_F64, decltype(load)> mom(load);
      double rho, j[3];
      mom.get(rho, j);
      out[4 * (int64_t)i] = rho;
      for (int d = 0; d < 3; d++) out[4 * (int64_t)i + 1 + d] = j[d];
      regular[i] = mom.regular();
   }
}

}  // namespace

// rho and j of n cells (populations in direction order), and whether they took
// the integer sums.
extern "C" void moments_f64(int Q, const double* f, int n, double* out, uint8_t* regular)
{
   if (Q == 19) run_f64<19>(f, n, out, regular);
   else run_f64<27>(f, n, out, regular);
}
