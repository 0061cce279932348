// IEEE double additions in integer instructions, for the exact FP64 collision.
//
// One FP64 instruction holds its pipe for 76 cycles per warp and sub-partition,
// an integer instruction for one or two.  Additions whose operands lie in known
// ranges are therefore made in 64-bit fixed point with 62 fraction bits: the sum
// is exact there, and rounding it to 53 significant bits (ties to even) gives the
// IEEE result.  An operand below the last fraction bit leaves a sticky bit in it,
// which decides ties as the exact value would as long as at least two bits are
// rounded away.
#pragma once

#include "lbm_f64x.cuh"

namespace lbm {
namespace soft {

__host__ __device__ __forceinline__ uint32_t clz32(uint32_t x)
{
#ifdef __CUDA_ARCH__
   return (uint32_t)__clz((int)x);
#else
   return x ? (uint32_t)__builtin_clz(x) : 32u;
#endif
}

// f * 2^62, exact for f in [2^-10, 1).
__host__ __device__ __forceinline__ uint64_t image(uint64_t b)
{
   const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32);
   const uint32_t top = x64::funnel_l(lo, (hi & 0x000FFFFFu) | 0x00100000u, 10), low = lo << 10;
   const uint32_t k = 1023u - (hi >> 20);   // 1 to 10
   return ((uint64_t)x64::funnel_r(top, 0u, k) << 32) | x64::funnel_r(low, top, k);
}

// |x| * 2^62 for |x| < 1, any other bits of x in the last one (sticky).
__host__ __device__ __forceinline__ uint64_t image_sticky(uint64_t b)
{
   const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32) & 0x7FFFFFFFu;
   uint32_t top = x64::funnel_l(lo, (hi & 0x000FFFFFu) | 0x00100000u, 10), low = lo << 10;
   uint32_t k = 1023u - (hi >> 20);
   if ((hi | lo) == 0u) top = low = 0u;
   k = k < 63u ? k : 63u;
   uint32_t lost = 0u;
   if (k & 32u) {
      lost = low;
      low = top;
      top = 0u;
   }
   const uint32_t mask = (1u << (k & 31u)) - 1u;
   lost |= low & mask;
   const uint32_t r = x64::funnel_r(low, top, k);
   return ((uint64_t)x64::funnel_r(top, 0u, k) << 32) | r | (lost != 0u ? 1u : 0u);
}

// Rounds an integer to 53 significant bits, ties to even; k is the number of bits
// rounded away (at most 31; the value's leading bit is 52 + k).
__host__ __device__ __forceinline__ uint64_t round_bits(uint64_t v, uint32_t k)
{
   const uint32_t lo = (uint32_t)v, unit = 1u << k;
   // half an ulp, less one where the kept part is even
   const uint32_t add = (unit - 1u + ((lo >> k) & 1u)) >> 1;
   return (v + add) & ~(uint64_t)(unit - 1u);
}

// A signed sum below 2^63 in magnitude.
__host__ __device__ __forceinline__ int64_t round_signed(int64_t v)
{
   const int32_t hi = (int32_t)((uint64_t)v >> 32);
   // the leading bit of |v| - 1 (v < 0) is that of |v| but for powers of two, which
   // have no bits to round
   const int32_t k = 11 - (int32_t)clz32((uint32_t)(hi ^ (hi >> 31)));
   return (int64_t)round_bits((uint64_t)v, (uint32_t)(k > 0 ? k : 0));
}

// A sum in [2^-8, 4), unsigned.
__host__ __device__ __forceinline__ uint64_t round_positive(uint64_t v)
{
   return round_bits(v, 11u - clz32((uint32_t)(v >> 32)));
}

// v * 2^-62 for v in [2^-8, 4) (times 2^62) of at most 53 significant bits.
__host__ __device__ __forceinline__ double positive_to_double(uint64_t v)
{
   const uint32_t n = clz32((uint32_t)(v >> 32));
   const uint64_t t = v << n;
   return x64::as_double((t >> 11) + ((uint64_t)(1023u + 63u - 62u - 1u - n) << 52));
}

// v * 2^-62 for any v of at most 53 significant bits.
__host__ __device__ __forceinline__ double signed_to_double(int64_t v)
{
   if (v == 0) return 0.0;
   const uint64_t m = v < 0 ? (uint64_t)0 - (uint64_t)v : (uint64_t)v;
   const uint32_t h = (uint32_t)(m >> 32);
   const uint32_t n = h ? clz32(h) : 32u + clz32((uint32_t)m);
   const uint64_t bits = ((m << n) >> 11) + ((uint64_t)(1023u + 63u - 62u - 1u - n) << 52);
   return x64::as_double(bits | ((uint64_t)v & 0x8000000000000000ull));
}

// a + b for b > 0: in integers for |a| < 1/4 and b in [2^-12, 1/4) with a sum in
// [2^-10, 1/2) (64 fraction bits, b exact, a with its sticky bit), else on the
// FP64 pipe.
__host__ __device__ __forceinline__ double add_double(double a, double b)
{
   const uint64_t ab = x64::double_bits(a), bb = x64::double_bits(b);
   const uint32_t ah = (uint32_t)(ab >> 32) & 0x7FFFFFFFu, bh = (uint32_t)(bb >> 32);
   // 4 |a| and 4 b as the images' arguments: exponents two up
   constexpr uint32_t kTwo = 2u << 20;
   const uint64_t A = image_sticky(((uint64_t)(ah > kTwo ? ah + kTwo : 0u) << 32) | (uint32_t)ab);
   const uint64_t B = image(bb + ((uint64_t)kTwo << 32));
   const uint64_t t = (int32_t)(ab >> 32) < 0 ? B - A : B + A;
   const uint32_t h = (uint32_t)(t >> 32);
   constexpr uint32_t kQuarter = (uint32_t)(1023 - 2) << 20, kLeast = (uint32_t)(1023 - 12) << 20;
   const bool ok = ah < kQuarter && bh - kLeast < kQuarter - kLeast && h - (1u << 22) < (1u << 31) - (1u << 22) &&
                   (ah > kTwo || ab << 1 == 0);
   if (!ok) {
#ifdef __CUDA_ARCH__
      return __dadd_rn(a, b);
#else
      return a + b;
#endif
   }
   // v * 2^-64: positive_to_double's with the exponent two down
   const uint64_t v = round_positive(t);
   const uint32_t n = clz32((uint32_t)(v >> 32));
   return x64::as_double(((v << n) >> 11) + ((uint64_t)(1023u + 63u - 64u - 1u - n) << 52));
}

// 1 + c + q - h for |c| < 0.9, 0 <= q <= c^2, 0 <= h < 0.05, each addition rounded.
struct Polynomial {
   uint64_t q, h;
   __host__ __device__ __forceinline__ double operator()(uint64_t c, bool negative) const
   {
      const uint64_t one = (uint64_t)1 << 62;
      const uint64_t s = round_positive(round_positive(negative ? one - c : one + c) + q);
      return positive_to_double(round_positive(s - h));
   }
};

}  // namespace soft
}  // namespace lbm
