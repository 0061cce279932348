// Host build of the integer double additions (lbmminiapp_gb300/csrc/lbm_soft.cuh)
// and of the readouts' fixed-point conversion, for tests/test_soft_host.py.
#include <cstdint>

#include "lbm_moments.cuh"
#include "lbm_soft.cuh"

using namespace lbm;

// Running sums of n rows of m signed populations, rounded after every addition:
// out[i] = sum_k sign[i][k] * d[i][k].
extern "C" void soft_sums(const double* d, const int8_t* sign, int n, int m, double* out)
{
   for (int i = 0; i < n; i++) {
      int64_t r = 0;
      for (int k = 0; k < m; k++) {
         const uint64_t X = soft::image(x64::double_bits(d[(int64_t)i * m + k]));
         r = soft::round_signed((int64_t)(sign[(int64_t)i * m + k] > 0 ? (uint64_t)r + X : (uint64_t)r - X));
      }
      out[i] = soft::signed_to_double(r);
   }
}

// The same for positive sums.
extern "C" void soft_positive_sums(const double* d, int n, int m, double* out)
{
   for (int i = 0; i < n; i++) {
      uint64_t r = 0;
      for (int k = 0; k < m; k++) {
         const uint64_t X = soft::image(x64::double_bits(d[(int64_t)i * m + k]));
         r = k == 0 ? X : soft::round_positive(r + X);
      }
      out[i] = soft::positive_to_double(r);
   }
}

// ((1 + c) + q) - h
extern "C" void soft_polynomial(const double* c, const double* q, const double* h, int n, double* out)
{
   for (int i = 0; i < n; i++) {
      const uint64_t cb = x64::double_bits(c[i]);
      const soft::Polynomial poly{soft::image_sticky(x64::double_bits(q[i])), soft::image_sticky(x64::double_bits(h[i]))};
      out[i] = poly(soft::image_sticky(cb), (int64_t)cb < 0);
   }
}

extern "C" void soft_add(const double* a, const double* b, int n, double* out)
{
   for (int i = 0; i < n; i++) out[i] = soft::add_double(a[i], b[i]);
}

// v * 2^-62, rounded
extern "C" void fixed62(const int64_t* v, int n, double* out)
{
   for (int i = 0; i < n; i++) out[i] = fixed62_to_double(v[i]);
}
