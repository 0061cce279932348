// rho and j = sum c f of one cell for the readouts and the loss, without the
// FP64 pipe.
//
// One FP64 instruction holds its pipe for 76 cycles per warp and sub-partition,
// an integer add for one, so sums made there (49 adds per D3Q19 cell) bound a
// kernel that only reads populations.  Here they are made in 64-bit integers, of
// fixed-point images of the populations (FP64 storage) or of the deviations f - w
// (the shifted formats), and rounded once, at the end.  Images that lose no bit,
// or bits below 2^-61 of a deviation, keep the error below that of the sums in
// FP64; a cell outside their ranges is summed in FP64.
#pragma once

#include "lbm_soft.cuh"

namespace lbm {

// (double)x without the FP64 pipe for normal x.
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x)
{
   const uint32_t b = __float_as_uint(x);
   if (((b >> 23) & 0xFFu) - 1u >= 254u) return (double)x;   // zero, subnormal, infinite, NaN
   return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(b << 29));
}

// v * 2^-FRAC rounded to nearest even, in integer instructions.
template <int FRAC>
__host__ __device__ __forceinline__ double fixed_to_double(int64_t v)
{
   if (v == 0) return 0.0;
   const uint64_t m = v < 0 ? (uint64_t)0 - (uint64_t)v : (uint64_t)v;
#ifdef __CUDA_ARCH__
   const int n = __clzll((long long)m);
#else
   const int n = __builtin_clzll(m);
#endif
   const uint64_t t = m << n;                       // leading bit at 63
   const uint64_t r = t + 0x3FFu + ((t >> 11) & 1u);   // half an ulp of the 53 kept bits, ties to even
   // a carry out of bit 63 makes the next power of two
   const uint64_t mant = r < t ? (uint64_t)1 << 53 : r >> 11;
   const uint64_t bits = mant + ((uint64_t)(1023 + 63 - FRAC - n - 1) << 52);
   return x64::as_double(bits | (v < 0 ? 0x8000000000000000ull : 0ull));
}
__host__ __device__ __forceinline__ double fixed62_to_double(int64_t v) { return fixed_to_double<62>(v); }

__device__ __forceinline__ bool finite_bits(double x) { return ((uint32_t)__double2hiint(x) & 0x7FF00000u) != 0x7FF00000u; }

// load(s): the deviation f_s - w_s of direction s as a float (shifted storage) or
// the bit pattern of f_s (FP64 storage).  regular(): the cell took the integer
// sums, so rho and j are finite and rho is not zero.
//
// Shifted formats: a deviation's image is g * 2^kFrac, the bits below dropped.
//   FP16   kFrac = 57: every value lies below 2 and is a multiple of 2^-39, so no
//          bit is lost, and 27 of them stay below 2^6;
//   else   kFrac = 61 for |g| < 1/8 (densities up to 1.3), 27 of them below 2^2.
//          A float from 2^-38 loses no bit, a smaller one at most 2^-61, which is
//          half an ulp of the smallest f = g + w.
template <int Q, int ST, class Load>
struct CellMoments {
   float g[Q];
   int64_t drho, m[3];
   bool fixed;

   static constexpr int kFrac = ST == ST_F16 ? 57 : 61;
   static constexpr uint32_t kBound = ST == ST_F16 ? 128u : 124u;   // exponent field of the least |g| not taken

   // g * 2^kFrac, toward zero
   __host__ __device__ __forceinline__ static uint64_t image(uint32_t b)
   {
      const uint32_t e = (b >> 23) & 0xFFu;
      const uint32_t top = ((b & 0x007FFFFFu) | 0x00800000u) << 2;   // high word of the significand of the largest exponent
      uint32_t k = kBound - 1u - e;
      k = k < 63u ? k : 63u;
      const uint32_t hi = k < 32u ? top >> (k & 31u) : 0u;
      const uint32_t lo = k < 32u ? x64::funnel_r(0u, top, k) : top >> (k & 31u);
      const uint64_t v = ((uint64_t)hi << 32) | lo, sign = (uint64_t)((int64_t)(int32_t)b >> 31);
      return (v ^ sign) - sign;
   }
   __host__ __device__ __forceinline__ explicit CellMoments(const Load& load)
   {
#pragma unroll
      for (int s = 0; s < Q; s++) g[s] = load(s);
      uint32_t most = x64::fbits(g[lat_rest(Q)]) & 0x7FFFFFFFu;
#pragma unroll
      for (int q = 0; q < (Q - 1) / 2; q++) {
         const int a = pair_dir(Q, q);
         most = x64::max3u(most, x64::fbits(g[a]) & 0x7FFFFFFFu, x64::fbits(g[lat_opp(Q, a)]) & 0x7FFFFFFFu);
      }
      fixed = most < kBound << 23;
      drho = m[0] = m[1] = m[2] = 0;
      if (!fixed) return;
      uint64_t r = image(x64::fbits(g[lat_rest(Q)])), j[3] = {0, 0, 0};
#pragma unroll
      for (int q = 0; q < (Q - 1) / 2; q++) {
         const int a = pair_dir(Q, q);
         const uint64_t X = image(x64::fbits(g[a])), Y = image(x64::fbits(g[lat_opp(Q, a)])), D = X - Y;
         r += X + Y;
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, a, d) > 0) j[d] += D;
            if (lat_c(Q, a, d) < 0) j[d] -= D;
         }
      }
      drho = (int64_t)r;
#pragma unroll
      for (int d = 0; d < 3; d++) m[d] = (int64_t)j[d];
      // rho from 1/2, and in 64 bits
      fixed = drho > -((int64_t)1 << (kFrac - 1)) && drho <= INT64_MAX - ((int64_t)1 << kFrac);
   }
   __host__ __device__ __forceinline__ bool regular() const { return fixed; }
   __host__ __device__ __forceinline__ void get(double& rho, double (&j)[3]) const
   {
      if (fixed) {
         rho = fixed_to_double<kFrac>(drho + ((int64_t)1 << kFrac));
#pragma unroll
         for (int d = 0; d < 3; d++) j[d] = fixed_to_double<kFrac>(m[d]);
         return;
      }
      rho = j[0] = j[1] = j[2] = 0.0;
#pragma unroll
      for (int s = 0; s < Q; s++) {
         const double f = (double)g[s] + lat_w(Q, s);
         rho += f;
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, s, d) > 0) j[d] += f;
            if (lat_c(Q, s, d) < 0) j[d] -= f;
         }
      }
   }
};

// FP64 storage: the images f * 2^62 of populations in [2^-10, 1) lose no bit, and
// with rho < 2 their sums do not wrap.
template <int Q, class Load>
struct CellMoments<Q, ST_F64, Load> {
   uint64_t r, m[3];
   bool exact;
   const Load& load;

   __host__ __device__ __forceinline__ explicit CellMoments(const Load& l) : load(l)
   {
      constexpr uint32_t kMin = (uint32_t)(1023 - 10) << 20, kMax = (uint32_t)1023 << 20;
      const uint64_t fr = load(lat_rest(Q));
      uint32_t least = (uint32_t)(fr >> 32), most = least, wrapped = 0u;
      r = soft::image(fr);
      m[0] = m[1] = m[2] = 0;
#pragma unroll
      for (int q = 0; q < (Q - 1) / 2; q++) {
         const int s = pair_dir(Q, q), o = lat_opp(Q, s);
         const uint64_t fs = load(s), fo = load(o);
         least = x64::min3u(least, (uint32_t)(fs >> 32), (uint32_t)(fo >> 32));
         most = x64::max3u(most, (uint32_t)(fs >> 32), (uint32_t)(fo >> 32));
         const uint64_t X = soft::image(fs), Y = soft::image(fo), D = X - Y;
         r += X + Y;
         // rho < 2, looked at after every pair: the sum cannot wrap in between
         wrapped |= (uint32_t)(r >> 32);
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, s, d) > 0) m[d] += D;
            if (lat_c(Q, s, d) < 0) m[d] -= D;
         }
      }
      exact = least >= kMin && most < kMax && !(wrapped & 0x80000000u);
   }
   __host__ __device__ __forceinline__ bool regular() const { return exact; }
   __host__ __device__ __forceinline__ void get(double& rho, double (&j)[3]) const
   {
      if (exact) {
         rho = fixed62_to_double((int64_t)r);
#pragma unroll
         for (int d = 0; d < 3; d++) j[d] = fixed62_to_double((int64_t)m[d]);
         return;
      }
      rho = j[0] = j[1] = j[2] = 0.0;
#pragma unroll
      for (int s = 0; s < Q; s++) {
         const double v = x64::as_double(load(s));
         rho += v;
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, s, d) > 0) j[d] += v;
            if (lat_c(Q, s, d) < 0) j[d] -= v;
         }
      }
   }
};

// Stored value of element idx as CellMoments takes it.
template <int ST>
__device__ __forceinline__ auto moment_value(const void* buf, int64_t idx)
{
   if constexpr (ST == ST_F64) return (uint64_t)static_cast<const unsigned long long*>(buf)[idx];
   else return load_shifted(static_cast<const typename Store<ST>::T*>(buf) + idx);
}

}  // namespace lbm
