// rho and j = sum c f of one cell for the readouts and the loss, without the
// FP64 pipe.
//
// One FP64 instruction holds its pipe for 76 cycles per warp and sub-partition,
// an integer or FP32 add for one, so sums made there (49 adds per D3Q19 cell)
// bound a kernel that only reads populations.  Here FP64 storage is summed
// exactly as 64-bit integers (images f * 2^62 of populations in [2^-10, 1), which
// lose no bit; a cell with another value, or with rho from 2, is summed in FP64),
// and the shifted formats in error-free FP32 additions (TwoSum) of the
// deviations f - w.
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

// v * 2^-62 rounded to nearest even, in integer instructions.
__host__ __device__ __forceinline__ double fixed62_to_double(int64_t v)
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
   const uint64_t bits = mant + ((uint64_t)(1023 + 63 - 62 - n - 1) << 52);
   return x64::as_double(bits | (v < 0 ? 0x8000000000000000ull : 0ull));
}

__device__ __forceinline__ bool finite_bits(double x) { return ((uint32_t)__double2hiint(x) & 0x7FF00000u) != 0x7FF00000u; }

// load(s): the deviation f_s - w_s of direction s as a float (shifted storage) or
// the bit pattern of f_s (FP64 storage).  regular(): rho and j are finite and rho
// is not zero.  Other cells (a diverged state) are summed in FP64.
template <int Q, int ST, class Load>
struct CellMoments {
   x64::df s[4];   // drho, j
   const Load& load;

   __device__ __forceinline__ explicit CellMoments(const Load& l) : load(l)
   {
#pragma unroll
      for (int k = 0; k < 4; k++) s[k] = {0.f, 0.f};
      auto add = [](x64::df& a, float v) {
         const x64::df t = x64::two_sum(a.h, v);
         a = {t.h, x64::fadd(a.l, t.l)};
      };
#pragma unroll
      for (int r = 0; r < Q; r++) {
         const float g = load(r);
         add(s[0], g);
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, r, d) > 0) add(s[1 + d], g);
            if (lat_c(Q, r, d) < 0) add(s[1 + d], -g);
         }
      }
   }
   __device__ __forceinline__ bool regular() const
   {
      return s[0].h > -0.5f && s[0].h < 1e30f && fabsf(s[1].h) < 1e30f && fabsf(s[2].h) < 1e30f &&
             fabsf(s[3].h) < 1e30f;
   }
   __device__ __forceinline__ void get(double& rho, double (&j)[3]) const
   {
      if (regular()) {
         rho = 1.0 + (widen(s[0].h) + widen(s[0].l));
#pragma unroll
         for (int d = 0; d < 3; d++) j[d] = widen(s[1 + d].h) + widen(s[1 + d].l);
         return;
      }
      // TwoSum makes NaN of an infinite population
      rho = j[0] = j[1] = j[2] = 0.0;
#pragma unroll
      for (int r = 0; r < Q; r++) {
         const double f = (double)load(r) + lat_w(Q, r);
         rho += f;
#pragma unroll
         for (int d = 0; d < 3; d++) {
            if (lat_c(Q, r, d) > 0) j[d] += f;
            if (lat_c(Q, r, d) < 0) j[d] -= f;
         }
      }
   }
};

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
