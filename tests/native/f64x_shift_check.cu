// Host build of the F64X collision with the launch constants the library makes
// (set_collision_constants), for tests/test_f64x_shift_host.py.
#include <cstdint>
#include <cstring>
#include <limits>

#include "lbm_f64x.cuh"

namespace {

template <int Q>
void run(const double* in, double* out, int n, const lbm::KParams& p, int* fast)
{
   using namespace lbm;
   const x64::Consts k = collide_consts<Q>(p);
   for (int i = 0; i < n; i++) {
      uint64_t bits[Q];
      for (int s = 0; s < Q; s++) bits[s] = x64::double_bits(in[(size_t)i * Q + s]);
      const bool ok = p.forced == 3   ? collide_f64x_fast<Q, 3>(bits, k, p.compat)
                      : p.forced == 2 ? collide_f64x_fast<Q, 2>(bits, k, p.compat)
                      : p.forced == 1 ? collide_f64x_fast<Q, 1>(bits, k, p.compat)
                                      : collide_f64x_fast<Q, 0>(bits, k, p.compat);
      fast[i] = ok;
      for (int s = 0; s < Q; s++)
         out[(size_t)i * Q + s] = ok ? x64::as_double(bits[s]) : std::numeric_limits<double>::quiet_NaN();
   }
}

}  // namespace

// Returns the forcing form that the library picks for this force.
extern "C" int f64x_library_collide(int Q, const double* in, double* out, int n, double omega, const double* F,
                                    int compat, int* fast)
{
   lbm::KParams p;
   std::memset(&p, 0, sizeof(p));
   const double f[3] = {F[0], F[1], F[2]};
   lbm::set_collision_constants(p, Q, omega, f, compat);
   if (Q == 19) run<19>(in, out, n, p, fast);
   else run<27>(in, out, n, p, fast);
   return p.forced;
}
