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

template <int Q, int ST>
void run_shifted(const float* g, int n, double* out, uint8_t* regular)
{
   for (int i = 0; i < n; i++) {
      const auto load = [&](int s) { return g[(int64_t)i * Q + s]; };
      const CellMoments<Q, ST, decltype(load)> mom(load);
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

// The same of the deviations f - w as floats; f16: those of FP16 storage.
extern "C" void moments_shifted(int Q, int f16, const float* g, int n, double* out, uint8_t* regular)
{
   if (Q == 19) f16 ? run_shifted<19, ST_F16>(g, n, out, regular) : run_shifted<19, ST_F32>(g, n, out, regular);
   else f16 ? run_shifted<27, ST_F16>(g, n, out, regular) : run_shifted<27, ST_F32>(g, n, out, regular);
}
