// F64X: double-precision BGK collision computed without the FP64 pipe.
//
// GB300's FP64 units run at about 1/60 of its FP32 rate, and double <-> float
// conversions are slow as well, so a collision written in `double` (or in
// float with conversions at load and store) is compute-bound far below the
// HBM roofline.  This path keeps the populations
// in FP64 memory (the reference's Pdf buffers) but:
//
//  * splits each loaded double into an unevaluated float pair (h, l): h is
//    the double truncated to 24 significant bits (integer operations), l the
//    remaining 29 mantissa bits rounded to 24 by an integer-to-float
//    conversion and scaled (|f - (h + l)| <= 2^-48 |f|);
//  * sums rho and j = sum c f exactly from 64-bit fixed-point images of the
//    doubles (integer adds);
//  * evaluates u, the equilibrium and the BGK/Guo update in
//    double-float arithmetic built from the error-free transformations
//    TwoSum (Knuth), Fast2Sum (Dekker 1971) and the FMA two-product, as used
//    in double-double libraries (Hida, Li & Bailey, "Library for double-double
//    and quad-double arithmetic", 2001);
//  * rebuilds the 64-bit pattern of the result (the double nearest to h + l)
//    with integer operations and one float-to-int conversion.
//
// The fast path covers positive populations in [2^-32, 1), the only values a
// physical state holds (with further bounds on the rest population and the
// velocity, checked per cell).  A cell whose inputs or results fall outside
// them is recomputed with the exact IEEE double collision, so any state is
// handled; the fast path's results agree with the exact path to about
// 2^-46 relative per step.
#pragma once

#include <cstdint>
#include <cstring>
#ifndef __CUDA_ARCH__
#include <cfenv>
#include <cmath>
#endif

#include "lbm_packed.cuh"
#include "lbm_physics.cuh"

namespace lbm {
namespace x64 {

// ------------------------------------------------------------ primitives
__host__ __device__ __forceinline__ uint32_t fbits(float f)
{
#ifdef __CUDA_ARCH__
   return __float_as_uint(f);
#else
   uint32_t u;
   std::memcpy(&u, &f, 4);
   return u;
#endif
}

__host__ __device__ __forceinline__ float bitsf(uint32_t u)
{
#ifdef __CUDA_ARCH__
   return __uint_as_float(u);
#else
   float f;
   std::memcpy(&f, &u, 4);
   return f;
#endif
}

__host__ __device__ __forceinline__ float frcp(float a)
{
#ifdef __CUDA_ARCH__
   return __frcp_rn(a);
#else
   volatile float r = 1.0f / a;
   return r;
#endif
}

// High 32 bits of ((hi:lo) << n), n modulo 32.
__host__ __device__ __forceinline__ uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t n)
{
#ifdef __CUDA_ARCH__
   return __funnelshift_l(lo, hi, n);
#else
   const uint64_t v = ((uint64_t)hi << 32) | lo;
   return (uint32_t)((v << (n & 31u)) >> 32);
#endif
}

// Low 32 bits of ((hi:lo) >> n), n modulo 32.
__host__ __device__ __forceinline__ uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t n)
{
#ifdef __CUDA_ARCH__
   return __funnelshift_r(lo, hi, n);
#else
   const uint64_t v = ((uint64_t)hi << 32) | lo;
   return (uint32_t)(v >> (n & 31u));
#endif
}

__host__ __device__ __forceinline__ float i2f_rn(int32_t i)
{
#ifdef __CUDA_ARCH__
   return __int2float_rn(i);
#else
   volatile float r = (float)i;
   return r;
#endif
}

// An integer-valued float (|x| < 2^31) to int32, exactly.
__host__ __device__ __forceinline__ int32_t f2i_exact(float x)
{
#ifdef __CUDA_ARCH__
   return __float2int_rz(x);
#else
   return (int32_t)x;
#endif
}

__host__ __device__ __forceinline__ float u2f_rn(uint32_t u)
{
#ifdef __CUDA_ARCH__
   return __uint2float_rn(u);
#else
   volatile float r = (float)u;
   return r;
#endif
}

// ------------------------------------------------------------ double-float
struct df {
   float h, l;
};

// TwoSum (Knuth): s + e == a + b exactly.
__host__ __device__ __forceinline__ df two_sum(float a, float b)
{
   const float s = fadd(a, b);
   const float bb = fsub(s, a);
   const float e = fadd(fsub(a, fsub(s, bb)), fsub(b, bb));
   return {s, e};
}

// Fast2Sum (Dekker): exact when |a| >= |b|.
__host__ __device__ __forceinline__ df fast_two_sum(float a, float b)
{
   const float s = fadd(a, b);
   return {s, fsub(b, fsub(s, a))};
}

__host__ __device__ __forceinline__ df df_add(df a, df b)
{
   const df s = two_sum(a.h, b.h);
   return fast_two_sum(s.h, fadd(s.l, fadd(a.l, b.l)));
}

__host__ __device__ __forceinline__ df df_neg(df a) { return {-a.h, -a.l}; }

// Product left unnormalised (p + e with |e| <= ~ulp(p)); saves the final Fast2Sum.
__host__ __device__ __forceinline__ df df_mul_u(df a, df b)
{
   const float p = fmul(a.h, b.h);
   float e = ffma(a.h, b.h, -p);
   e = ffma(a.h, b.l, e);
   e = ffma(a.l, b.h, e);
   return {p, e};
}

// ------------------------------------------- two float pairs at a time
struct df2 {
   f2 h, l;
};

__host__ __device__ __forceinline__ df2 dup(df a) { return {dup2(a.h), dup2(a.l)}; }
__host__ __device__ __forceinline__ df2 pack(df a, df b) { return {{a.h, b.h}, {a.l, b.l}}; }
__host__ __device__ __forceinline__ df2 df2_neg(df2 a) { return {neg2(a.h), neg2(a.l)}; }

__host__ __device__ __forceinline__ df2 two_sum2(f2 a, f2 b)
{
   const f2 s = add2(a, b);
   const f2 bb = sub2(s, a);
   return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}

__host__ __device__ __forceinline__ df2 fast_two_sum2(f2 a, f2 b)
{
   const f2 s = add2(a, b);
   return {s, sub2(b, sub2(s, a))};
}

__host__ __device__ __forceinline__ df2 df2_mul_u(df2 a, df2 b)
{
   const f2 p = mul2(a.h, b.h);
   f2 e = fma2(a.h, b.h, neg2(p));
   e = fma2(a.h, b.l, e);
   return {p, fma2(a.l, b.h, e)};
}

__host__ __device__ __forceinline__ df2 df2_sqr_u(df2 a)
{
   const f2 p = mul2(a.h, a.h);
   const f2 e = fma2(a.h, a.h, neg2(p));
   return {p, fma2(mul2(dup2(2.0f), a.h), a.l, e)};
}

__host__ __device__ __forceinline__ uint32_t min3u(uint32_t a, uint32_t b, uint32_t c)
{
#ifdef __CUDA_ARCH__
   return __vimin3_u32(a, b, c);
#else
   const uint32_t m = a < b ? a : b;
   return m < c ? m : c;
#endif
}

__host__ __device__ __forceinline__ uint32_t max3u(uint32_t a, uint32_t b, uint32_t c)
{
#ifdef __CUDA_ARCH__
   return __vimax3_u32(a, b, c);
#else
   const uint32_t m = a > b ? a : b;
   return m > c ? m : c;
#endif
}

// Exact split of a host double constant into a float pair.
__host__ __device__ __forceinline__ df df_from_double(double d)
{
   const float h = (float)d;
   return {h, (float)(d - (double)h)};
}

// ------------------------------------------------ double <-> float pair
// Fast-path range of the double bit patterns: positive, 2^-32 <= f < 1.
constexpr uint32_t kHiMin = (uint32_t)(1023 - 32) << 20;   // high word of 2^-32
constexpr uint32_t kHiMax = (uint32_t)1023 << 20;          // high word of 1.0 (excluded)

// Split a positive double in range (given as its 64-bit pattern) into (h, l).
//   h  = bits 60..29 of the pattern (the low 9 exponent bits above the top
//        23 mantissa bits) plus 2^30, masked to 31 bits: exponent E
//        re-biased to E - 896 in the float's 8-bit field, valid for E in
//        [897, 1150];
//   l  = the low 29 mantissa bits as an integer, rounded to nearest 24 bits
//        by the conversion and scaled by 2^(e(h) - 52) (a power of two, no
//        underflow for e(h) >= -74).  |f - (h + l)| <= 2^-48 |f|.
__host__ __device__ __forceinline__ df split(uint64_t bits)
{
   const uint32_t lo = (uint32_t)bits, hi = (uint32_t)(bits >> 32);
   const uint32_t hb = (funnel_l(lo, hi, 3) + 0x40000000u) & 0x7FFFFFFFu;
   const float scale = bitsf((hb & 0x7F800000u) - (52u << 23));
   return {bitsf(hb), fmul(u2f_rn(lo & 0x1FFFFFFFu), scale)};
}

// split() of two doubles of the fast path's range [2^-32, 1), whose exponents
// (991..1022) have the two bits that the re-biasing takes off both set.
__host__ __device__ __forceinline__ df2 split2(uint64_t b0, uint64_t b1)
{
   const uint32_t lo0 = (uint32_t)b0, lo1 = (uint32_t)b1;
   const uint32_t h0 = funnel_l(lo0, (uint32_t)(b0 >> 32), 3) & 0x3FFFFFFFu;
   const uint32_t h1 = funnel_l(lo1, (uint32_t)(b1 >> 32), 3) & 0x3FFFFFFFu;
   const f2 scale = {bitsf((h0 & 0x7F800000u) - (52u << 23)), bitsf((h1 & 0x7F800000u) - (52u << 23))};
   return {{bitsf(h0), bitsf(h1)}, mul2({u2f_rn(lo0 & 0x1FFFFFFFu), u2f_rn(lo1 & 0x1FFFFFFFu)}, scale)};
}

// Fixed-point image of a positive double f in [2^-32, 1) for the moment
// sums: floor(f * 2^53) as a 64-bit integer, the 53-bit mantissa (with its
// implicit bit) shifted right by k = 1022 - E, in [0, 31] for that range.
// Sums of these images are exact; the truncation loses less than 2^-53 per
// population (its mean, half a unit, is added back to rho).  For an f outside
// that range the result means nothing.
__host__ __device__ __forceinline__ uint64_t fixed53(uint64_t bits)
{
   const uint32_t lo = (uint32_t)bits, hi = (uint32_t)(bits >> 32);
   const uint32_t mh = (hi & 0x000FFFFFu) | 0x00100000u;
   const uint32_t k = 1022u - (hi >> 20);
   return ((uint64_t)funnel_r(mh, 0u, k) << 32) | funnel_r(lo, mh, k);
}

// Float pair of v * 2^-53 for a signed 64-bit v with |v| < 2^54.  The top
// part is v >> 23 rounded to 24 bits (an integer, so the remainder is exact
// and below 2^30), the remainder is rounded to 24 bits: the pair is exact for
// |v| < 2^47 and within 2^-48 |v| above, relative to v however small it is
// (a momentum sum of a slow flow keeps every bit).  Not normalised: h may be
// 0 or below l.
__host__ __device__ __forceinline__ df fixed53_to_pair(int64_t v)
{
   const uint32_t lo = (uint32_t)v, hi = (uint32_t)((uint64_t)v >> 32);
   const float hf = i2f_rn((int32_t)funnel_l(lo, hi, 9));   // v >> 23 (arithmetic), rounded
   const int32_t r = (int32_t)(lo - ((uint32_t)f2i_exact(hf) << 23));   // v - hf * 2^23, |r| < 2^30
   return {fmul(hf, 0x1p-30f), fmul(i2f_rn(r), 0x1p-53f)};
}

// Non-negative float to unsigned int, rounded to nearest even.
__host__ __device__ __forceinline__ uint32_t f2u_rn(float x)
{
#ifdef __CUDA_ARCH__
   return __float2uint_rn(x);
#else
   return (uint32_t)std::nearbyint(x);
#endif
}

// Running check of the result patterns of one cell: the smallest and the
// largest as unsigned integers (a negative or NaN result lands above the
// bound), two results at a time with three-input minima and maxima.
struct JoinRange {
   uint32_t least = 0x3F000000u, most = 0x3F000000u;
   __host__ __device__ __forceinline__ void add(uint32_t s0, uint32_t s1)
   {
      least = min3u(least, s0, s1);
      most = max3u(most, s0, s1);
   }
   // 2^-75 <= S < 1 for every result
   __host__ __device__ __forceinline__ bool ok() const { return least >= 0x1A000000u && most < 0x3F800000u; }
};

// Double pattern of h + l (positive):
//   S  = h + l rounded toward zero; the remainder h + l - S lies in
//        [0, ulp_float(S)); E = l - (S - h) is that remainder rounded to a
//        float (S - h is exact: S and h are within a factor of two).  The
//        remainder of a rounded-toward-zero sum need not be a float: for a
//        tiny negative l, S is h's predecessor and the remainder
//        ulp_float(S) - |l| can round up to ulp_float(S) itself;
//   N  = E in units of one double ulp of S, rounded to the nearest integer,
//        at most 2^29 (one float ulp of S);
//   the pattern of S as a double plus N (an integer add, which carries into
//        the float part and the exponent when N reaches 2^29): within about
//        33 double ulps of h + l.
// S's pattern goes into `range`; the result is valid when range.ok().
__host__ __device__ __forceinline__ uint64_t join_bits(uint32_t sb, float n)
{
   return (((uint64_t)sb << 29) + ((uint64_t)0x38000000u << 32)) + f2u_rn(n);
}

__host__ __device__ __forceinline__ uint64_t join(df v, JoinRange& range)
{
   const float S = fadd_rz(v.h, v.l);
   const float E = fsub(v.l, fsub(S, v.h));
   const uint32_t sb = fbits(S);
   range.add(sb, sb);
   const float scale = bitsf(0x99000000u - (sb & 0x7F800000u));  // 2^(52 - e(S))
   return join_bits(sb, fmul(E, scale));
}

// join() of two results.
struct Pattern2 {
   uint64_t a, b;
};
__host__ __device__ __forceinline__ Pattern2 join2(df2 v, JoinRange& range)
{
   const f2 S = add2_rz(v.h, v.l);
   const f2 E = sub2(v.l, sub2(S, v.h));
   const uint32_t s0 = fbits(S.x), s1 = fbits(S.y);
   range.add(s0, s1);
   const f2 n = mul2(E, {bitsf(0x99000000u - (s0 & 0x7F800000u)), bitsf(0x99000000u - (s1 & 0x7F800000u))});
   return {join_bits(s0, n.x), join_bits(s1, n.y)};
}

__host__ __device__ __forceinline__ double as_double(uint64_t b)
{
   double d;
#ifdef __CUDA_ARCH__
   d = __longlong_as_double((long long)b);
#else
   std::memcpy(&d, &b, 8);
#endif
   return d;
}

__host__ __device__ __forceinline__ uint64_t double_bits(double d)
{
#ifdef __CUDA_ARCH__
   return (uint64_t)__double_as_longlong(d);
#else
   uint64_t b;
   std::memcpy(&b, &d, 8);
   return b;
#endif
}

// Per-launch constants of the double-float collision.
struct Consts {
   df om1;        // 1 - omega
   df omega;
   df ow[4];      // omega * w for |c|^2 = 0, 1, 2, 3
   df F[3];       // uniform body force
   df F3[3];      // 3 F
   df Kf[27];     // (1 - omega/2) w_s 3 c_s.F per direction: the forcing term linear in F
   df om2w[4];    // (1 - omega/2) w per weight class
   df om2w36;     // (1 - omega/2) / 36 (rest weight of the Q19 AA Unroll kernels)
   float om2;
   // small-force form (FORCE 3): F / omega, (1 - omega/2) / omega, and per
   // direction 3/2 F.F - (3 c.F)^2 / 2
   df Fshift[3];
   float kappa, E[27];
};

}  // namespace x64

// Forcing form of the F64X fast path: 0 no force; 1 any force (the forcing
// terms are added after the equilibrium with error-free sums); 2 a force small
// enough, sum |F_d| <= 0.004 omega, for the terms to be folded into the
// equilibrium's symmetric and antisymmetric parts.  The fast path's inputs
// give rho >= 1/4, |3 v_d| < 0.3, hence omega w rho (Q+ - |3 c.v|) >=
// 0.11 omega w, while the folded terms stay below 6.2 w sum |F_d|, so the
// Fast2Sum operand order still holds (with a 4.5x margin at the bound).
inline int force_mode(const double force[3], double omega)
{
   double fsum = 0.0;
   for (int d = 0; d < 3; d++) fsum += force[d] < 0.0 ? -force[d] : force[d];
   if (fsum == 0.0) return 0;
   return fsum <= 0.004 * omega ? 2 : 1;
}

// Form 3 of the step kernels: the force shifts the velocity.  With
// k = (1 - omega/2) / (omega rho) and v' = (j + F/omega) / rho = v + k F,
//   omega eq_s(v) + (1 - omega/2) fdist_s = omega eq_s(v') + omega w rho k^2 E_s,
//   E_s = 3/2 F.F - (3 c.F)^2 / 2,
// exactly: the forcing costs one multiply-add per pair instead of about 25
// double-float operations.  The E term is single precision: with
// sum |F_d| (1 - omega/2) / omega <= 1e-5 and rho >= 1/4 it is below 2^-27 of the
// equilibrium (|E| <= 4 (sum |F_d|)^2, at a diagonal force), and its error, from the
// roundings of kappa, 1/rho, their product, its square and E, below 2^-48.  That is
// at the limit and rho = 1/4; at rho = 1 both are 16 times smaller.  The whole
// collision's error is below that of form 2, whose forcing terms are float pairs, at
// any force up to the limit: rms over flow cells 8.2e-15 against 9.0e-15 (D3Q19,
// tau = 0.55), 9.6e-15 against 1.07e-14 (D3Q27).  Not for the rest weight of the
// Unroll kernels (compat), which breaks the identity.
inline bool force_shifts(const double force[3], double omega)
{
   double fsum = 0.0;
   for (int d = 0; d < 3; d++) fsum += force[d] < 0.0 ? -force[d] : force[d];
   return fsum > 0.0 && fsum * (1.0 - 0.5 * omega) <= 1e-5 * omega;
}

// Host: the collision constants of a launch (relaxation rate, uniform force,
// the Q19 AA Unroll rest-weight switch) in double, float and float-pair form.
inline void set_collision_constants(KParams& p, int Q, double omega, const double force[3], int compat)
{
   p.omega = omega;
   p.om1 = 1.0 - omega;
   p.om2 = 1.0 - 0.5 * omega;
   p.omegaf = (float)p.omega;
   p.om1f = (float)p.om1;
   p.om2f = (float)p.om2;
   for (int d = 0; d < 3; d++) {
      p.F[d] = force[d];
      p.Ff[d] = (float)force[d];
   }
   p.compat = compat;
   for (int d = 0; d < 3; d++) p.half_F[d] = 0.5 * force[d];
   for (int q = 0, s = 0; s < Q; s++) {
      if (s >= lat_opp(Q, s)) continue;
      // c_s.F as the reference sums it (its zero terms add +-0), then times 3
      double acc = 0.0;
      for (int d = 0; d < 3; d++) acc += lat_c(Q, s, d) * force[d];
      p.cf3[q++] = 3.0 * acc;
   }
   auto split = [](double d, float* out) {
      const float hi = (float)d;
      out[0] = hi;
      out[1] = (float)(d - (double)hi);
   };
   split(p.om1, p.x_om1);
   split(p.omega, p.x_omega);
   for (int k = 0; k < 4; k++) {
      double w;
      if (Q == 19) w = k == 0 ? 1.0 / 3.0 : (k == 1 ? 1.0 / 18.0 : 1.0 / 36.0);
      else w = k == 0 ? 8.0 / 27.0 : (k == 1 ? 2.0 / 27.0 : (k == 2 ? 1.0 / 54.0 : 1.0 / 216.0));
      split(omega * w, p.x_ow[k]);
      split(p.om2 * w, p.x_om2w[k]);
   }
   for (int d = 0; d < 3; d++) split(force[d], p.x_F[d]);
   for (int s = 0; s < Q; s++) {
      const double cf = 3.0 * (lat_c(Q, s, 0) * force[0] + lat_c(Q, s, 1) * force[1] + lat_c(Q, s, 2) * force[2]);
      split(p.om2 * lat_w(Q, s) * cf, p.x_Kf[s]);
   }
   for (int d = 0; d < 3; d++) split(3.0 * force[d], p.x_F3[d]);
   split(p.om2 / 36.0, p.x_om2w36);
   p.forced = force_mode(force, omega);
   if (!compat && force_shifts(force, omega)) p.forced = 3;
   for (int d = 0; d < 3; d++) split(force[d] / omega, p.x_Fshift[d]);
   p.x_kappa = (float)((1.0 - 0.5 * omega) / omega);
   for (int s = 0; s < Q; s++) {
      const double cf = 3.0 * (lat_c(Q, s, 0) * force[0] + lat_c(Q, s, 1) * force[1] + lat_c(Q, s, 2) * force[2]);
      const double ff = force[0] * force[0] + force[1] * force[1] + force[2] * force[2];
      p.x_E[s] = (float)(1.5 * ff - 0.5 * cf * cf);
   }
}

// Representative s < opp(s) of the p-th opposite pair (direction order of
// the reference: pairs are (0,1), (2,3), ... with the rest direction last).
__host__ __device__ constexpr int pair_dir(int Q, int p)
{
   int seen = 0;
   for (int s = 0; s < Q; s++) {
      if (s < lat_opp(Q, s)) {
         if (seen == p) return s;
         seen++;
      }
   }
   return -1;
}

// Fast-path validity thresholds (high words of the doubles).
constexpr uint32_t kHiQuarter = (uint32_t)(1023 - 2) << 20;   // 0.25

// Input policy of the fast path that keeps the input patterns in registers.
struct KeepInputs {
   static constexpr bool kRefetch = false;
   __host__ __device__ __forceinline__ uint64_t raw(int) const { return 0; }
};

// Pattern of input s: kept, or read again.
template <int Q, class Again>
__host__ __device__ __forceinline__ uint64_t input_bits(const uint64_t (&bits)[Q], const Again& again, int s)
{
   if constexpr (Again::kRefetch) return again.raw(s);
   else return bits[s];
}

// Parts of the update that two opposite pairs (s, opp(s)) share, the two pairs
// in the halves: A +- B is omega eq plus the folded forcing, K and sym the
// forcing added afterwards (FORCE 1).
struct PairParts {
   x64::df2 A, B, K, sym;
};

// cu = 3 c_s.v; owc = omega w rho, om2wc = (1 - omega/2) w of the pairs' class;
// K = (1 - omega/2) w 3 c_s.F.  Forcing om2 w (+-cf - fu + cu cf) =
// +-K + (K cu - om2 w fu); FORCE 3: kk E = k^2 E_s joins the quadratic term.
template <int FORCE>
__host__ __device__ __forceinline__ PairParts pair_parts(x64::df2 cu, x64::df2 base, x64::df2 owc, x64::df2 K,
                                                         x64::df2 om2wc, x64::df2 fu, x64::f2 kk, x64::f2 E)
{
   using namespace x64;
   PairParts r;
   const f2 half = dup2(0.5f);
   // Qp = base + cu^2 / 2
   const df2 c2h = df2_sqr_u(cu);
   const df2 qs = fast_two_sum2(base.h, mul2(half, c2h.h));
   f2 low = fma2(half, c2h.l, base.l);
   if constexpr (FORCE == 3) low = fma2(kk, E, low);
   const df2 Qp = {qs.h, add2(qs.l, low)};
   r.A = df2_mul_u(owc, Qp);   // omega * eq, symmetric part
   r.B = df2_mul_u(owc, cu);   // omega * eq, antisymmetric part
   r.K = K;
   if constexpr (FORCE == 1 || FORCE == 2) {
      const df2 gc = df2_mul_u(K, cu);
      const df2 wf = df2_mul_u(om2wc, fu);
      const df2 t3 = two_sum2(gc.h, neg2(wf.h));
      r.sym = {t3.h, add2(t3.l, sub2(gc.l, wf.l))};
   }
   if constexpr (FORCE == 2) {
      // small force: sym joins the symmetric part (far below it) and K the
      // antisymmetric part (which may vanish, hence TwoSum)
      const df2 as = fast_two_sum2(r.A.h, r.sym.h);
      r.A = {as.h, add2(as.l, add2(r.A.l, r.sym.l))};
      const df2 bs = two_sum2(r.B.h, K.h);
      r.B = {bs.h, add2(bs.l, add2(r.B.l, K.l))};
   }
   return r;
}

// Patterns of A + B + (1 - omega) f for two directions (B, K negated for the
// opposite ones), f their inputs.
template <int FORCE>
__host__ __device__ __forceinline__ x64::Pattern2 pair_out(const PairParts& q, x64::df2 B, x64::df2 K, x64::df2 f,
                                                           x64::df2 om1, x64::JoinRange& range)
{
   using namespace x64;
   const df2 tp = fast_two_sum2(q.A.h, B.h);
   const df2 a = df2_mul_u(om1, f);
   const df2 t = two_sum2(tp.h, a.h);
   df2 out = {t.h, add2(t.l, add2(tp.l, add2(add2(q.A.l, B.l), a.l)))};
   if constexpr (FORCE == 1) {
      const df2 fr = two_sum2(K.h, q.sym.h);
      const df2 t2 = two_sum2(out.h, fr.h);
      out = {t2.h, add2(t2.l, add2(out.l, add2(fr.l, add2(K.l, q.sym.l))))};
   }
   return join2(out, range);
}

// The fast-path collision on one cell.  bits[] holds the Q input patterns in
// direction order; each output pattern is handed to emit(s, pattern).
// Returns false when the cell must take the exact path (nothing is emitted
// when an input check fails; after an output check fails every output has
// been emitted, possibly wrong):
//   * inputs: rest population in [0.25, 1), the others in [2^-32, 0.25), and
//     rho < 2;
//   * |3 v_d| < 0.3: |c.u| stays well below 1 - uu/2, so the pair sums
//     (1 - uu/2 + cu^2/2) +- cu keep their larger operand first;
//   * outputs inside [2^-75, 1).
// Work is organised by opposite pairs (s, opp(s)): cu, the quadratic term and
// the omega*w*rho products are shared, since cu(opp) = -cu(s).  Two pairs of one
// weight class go through the packed instructions together; the third axis pair
// (z) runs alone, its two directions in the halves.
// FORCE is the forcing form (0 none, 1 added after the equilibrium, 2 folded
// into it, 3 a velocity shift: force_mode(), force_shifts()); Again supplies the inputs of the
// (1 - omega) f term (KeepInputs, or a second read from shared memory).
//
// ROLLED: the planar and body diagonals run in loops over their packed pairs
// instead of unrolled, with the same operations in the same order, so the same
// bits.  The direction and its velocity are then run-time values: outputs go to
// emit.put(s, opp(s), c_s, pattern), and Kf (float pairs) and E point at the
// per-direction forcing constants.  The step kernels run the unrolled form (the
// loops' smaller code paid only while the scalar form overran the instruction
// cache: D3Q27 AA even step, 256x128x128: 293 us rolled, 283 us unrolled); the
// rolled one is its cross-check on the host.
template <int Q, int FORCE, class Emit, class Again, bool ROLLED = false>
__host__ __device__ __forceinline__ bool collide_f64x_fast_emit(const uint64_t (&bits)[Q], const x64::Consts& k,
                                                               int compat, Emit& emit, const Again& again,
                                                               const float (*Kf)[2] = nullptr,
                                                               const float* E = nullptr)
{
   using namespace x64;
   constexpr int R = lat_rest(Q);
   constexpr int NP = (Q - 1) / 2;
   // One pass over the inputs: the range of their high words, and rho and
   // j = sum c_s f_s from the exact sums of the fixed-point images
   // floor(f * 2^53), j by each pair's difference.  An input outside the range
   // makes meaningless sums, which are not used: so no input has to stay in a
   // register until the checks are done.
   uint32_t hmin = 0xFFFFFFFFu, hmax = 0;
   uint64_t rho_x = fixed53(bits[R]) + (uint64_t)(Q / 2);   // mean truncation loss, half a unit per population
   int64_t jx[3] = {0, 0, 0};
#pragma unroll
   for (int q = 0; q < NP; q++) {
      const int s = pair_dir(Q, q);
      const uint64_t bs = bits[s], bo = bits[lat_opp(Q, s)];
      hmin = min3u(hmin, (uint32_t)(bs >> 32), (uint32_t)(bo >> 32));
      hmax = max3u(hmax, (uint32_t)(bs >> 32), (uint32_t)(bo >> 32));
      const uint64_t X = fixed53(bs), Y = fixed53(bo);
      const uint64_t D = X - Y;
      rho_x += X + Y;
#pragma unroll
      for (int d = 0; d < 3; d++) {
         const int c = lat_c(Q, s, d);
         if (c > 0) jx[d] = (int64_t)((uint64_t)jx[d] + D);
         if (c < 0) jx[d] = (int64_t)((uint64_t)jx[d] - D);
      }
   }
   const uint32_t hr = (uint32_t)(bits[R] >> 32);
   // rho < 2: its top word is below 2^22
   if (hmin < kHiMin || hmax >= kHiQuarter || hr < kHiQuarter || hr >= kHiMax || (rho_x >> 32) >= (1u << 22))
      return false;
   df j[3];
#pragma unroll
   for (int d = 0; d < 3; d++) {
      // Fast2Sum is exact here: t.h is 0 or at least ulp-aligned above |t.l|.
      const df t = fixed53_to_pair(jx[d]);
      j[d] = fast_two_sum(t.h, t.l);
   }
   // rho >= 1/4 (the rest population alone): Fast2Sum normalises the pair.
   const df rho0 = fixed53_to_pair((int64_t)rho_x);
   const df rho = fast_two_sum(rho0.h, rho0.l);

   // v = (j + F/2) / rho, left unnormalised (p + e); 3v normalised
   const float r0 = frcp(rho.h);
   float e = ffma(-rho.h, r0, 1.0f);
   e = ffma(-rho.l, r0, e);
   const df inv = {r0, fmul(r0, e)};
   df v[3], v3[3];
#pragma unroll
   for (int d = 0; d < 3; d++) {
      df jf = j[d];
      if constexpr (FORCE == 3) jf = df_add(j[d], k.Fshift[d]);
      else if constexpr (FORCE != 0) jf = df_add(j[d], {0.5f * k.F[d].h, 0.5f * k.F[d].l});
      v[d] = df_mul_u(jf, inv);
      const float p = fmul(3.0f, v[d].h);
      v3[d] = fast_two_sum(p, ffma(3.0f, v[d].h, -p) + 3.0f * v[d].l);
   }
   if (!(fabsf(v3[0].h) < 0.3f && fabsf(v3[1].h) < 0.3f && fabsf(v3[2].h) < 0.3f)) return false;
   // base = 1 - uu/2 with uu = 3 v.v, as a Fast2Sum chain from 1 (each
   // term 3 v_d^2 / 2 < 0.045 stays below the running value); left
   // unnormalised (its low part is a few ulps of its high part at most).
   df base;
   {
      const df p0 = df_mul_u(v3[0], v[0]), p1 = df_mul_u(v3[1], v[1]), p2 = df_mul_u(v3[2], v[2]);
      const df b0 = fast_two_sum(1.0f, -0.5f * p0.h);
      const df b1 = fast_two_sum(b0.h, -0.5f * p1.h);
      const df b2 = fast_two_sum(b1.h, -0.5f * p2.h);
      const float lows = ffma(-0.5f, p2.l, ffma(-0.5f, p1.l, ffma(-0.5f, p0.l, fadd(b0.l, b1.l))));
      base = {b2.h, fadd(b2.l, lows)};
   }
   // fu = 3 F.v (float pair; zero without a force)
   df fu = {0.f, 0.f};
   if constexpr (FORCE == 1 || FORCE == 2) {
      fu = df_mul_u(k.F3[0], v[0]);
      fu = df_add(fu, df_mul_u(k.F3[1], v[1]));
      fu = df_add(fu, df_mul_u(k.F3[2], v[2]));
   }

   // Each output goes to emit(s, pattern) as soon as it is made; the return
   // value says whether all of them passed the range check (if not, the
   // caller overwrites every one with the exact result).
   JoinRange range;
   float kk = 0.f;   // k^2 of the velocity shift
   if constexpr (FORCE == 3) {
      const float kr = fmul(k.kappa, r0);
      kk = fmul(kr, kr);
   }
   // rest direction: P = base
   {
      df A = df_mul_u(df_mul_u(k.ow[0], rho), FORCE == 3 ? df{base.h, ffma(kk, k.E[R], base.l)} : base);
      if (FORCE == 2) {
         // -(1 - omega/2) wf fu (wf = 1/36 with the Unroll-kernel weights),
         // folded into the equilibrium term
         const df fr = df_mul_u(compat ? k.om2w36 : k.om2w[0], fu);
         const df t2 = fast_two_sum(A.h, -fr.h);
         A = {t2.h, fadd(t2.l, fsub(A.l, fr.l))};
      }
      const df a = df_mul_u(k.om1, split(input_bits(bits, again, R)));
      const df t = two_sum(A.h, a.h);
      df out = {t.h, fadd(t.l, fadd(A.l, a.l))};
      if (FORCE == 1) {
         // -(1 - omega/2) wf fu, wf = 1/36 with the Unroll-kernel weights
         const df fr = df_mul_u(compat ? k.om2w36 : k.om2w[0], fu);
         const df t2 = two_sum(out.h, -fr.h);
         out = {t2.h, fadd(t2.l, fsub(out.l, fr.l))};
      }
      emit(R, join(out, range));
   }

   const df2 base2 = dup(base), fu2 = dup(fu), om1 = dup(k.om1);
   auto inputs = [&](int a, int b) { return split2(input_bits(bits, again, a), input_bits(bits, again, b)); };
   auto forcing = [&](int s) {
      if constexpr (FORCE == 0 || FORCE == 3) return df{0.f, 0.f};
      else if constexpr (ROLLED) return df{Kf[s][0], Kf[s][1]};
      else return k.Kf[s];
   };
   auto shift = [&](int s) {
      if constexpr (FORCE != 3) return 0.f;
      else if constexpr (ROLLED) return E[s];
      else return k.E[s];
   };
   // Patterns of the pairs (s1, o1), (s2, o2) of one class with cu = (3 c_s1.v,
   // 3 c_s2.v): out(sign) gives those of s1, s2 (+) or o1, o2 (-).
   struct Outs {
      Pattern2 s, o;
   };
   auto pairs = [&](const df2 cu, const df2 owc, const df om2wc, int s1, int o1, int s2, int o2) {
      const PairParts q = pair_parts<FORCE>(cu, base2, owc, pack(forcing(s1), forcing(s2)), dup(om2wc), fu2,
                                            dup2(kk), {shift(s1), shift(s2)});
      Outs r;
      r.s = pair_out<FORCE>(q, q.B, q.K, inputs(s1, s2), om1, range);
      r.o = pair_out<FORCE>(q, df2_neg(q.B), df2_neg(q.K), inputs(o1, o2), om1, range);
      return r;
   };
   // axes: (0,1) and (2,3) together, (4,5) with its two directions in the halves
   {
      const df2 ow1 = dup(df_mul_u(k.ow[1], rho));
      const Outs r = pairs(pack(v3[0], v3[1]), ow1, k.om2w[1], 0, 1, 2, 3);
      const df K = forcing(4);
      const PairParts q = pair_parts<FORCE>(pack(v3[2], df_neg(v3[2])), base2, ow1, pack(K, df_neg(K)),
                                            dup(k.om2w[1]), fu2, dup2(kk), dup2(shift(4)));
      const Pattern2 z = pair_out<FORCE>(q, q.B, q.K, inputs(4, 5), om1, range);
      if constexpr (ROLLED) {
         emit.put(0, 1, 1, 0, 0, r.s.a);
         emit.put(2, 3, 0, 1, 0, r.s.b);
         emit.put(1, 0, -1, 0, 0, r.o.a);
         emit.put(3, 2, 0, -1, 0, r.o.b);
         emit.put(4, 5, 0, 0, 1, z.a);
         emit.put(5, 4, 0, 0, -1, z.b);
      } else {
         emit(0, r.s.a);
         emit(2, r.s.b);
         emit(1, r.o.a);
         emit(3, r.o.b);
         emit(4, z.a);
         emit(5, z.b);
      }
   }
   // cu = a + b in float pairs (TwoSum-based, left unnormalised)
   auto sum = [](const df2 a, const df2 b) {
      const df2 t = two_sum2(a.h, b.h);
      return df2{t.h, add2(t.l, add2(a.l, b.l))};
   };
   // planar diagonals (6,11) (7,10), (8,13) (9,12), (14,17) (15,16):
   // c = e_a + e_b and e_a - e_b, a < b
   const df2 ow2 = dup(df_mul_u(k.ow[2], rho));
   if constexpr (ROLLED) {
#pragma unroll 1
      for (int j = 0; j < 3; j++) {
         const int a = j < 2 ? 0 : 1, b = j == 0 ? 1 : 2;
         const df va = a == 0 ? v3[0] : v3[1], vb = b == 1 ? v3[1] : v3[2];
         const int s1 = j == 0 ? 6 : (j == 1 ? 8 : 14), o1 = j == 0 ? 11 : (j == 1 ? 13 : 17);
         const int s2 = s1 + 1, o2 = o1 - 1;
         const int ax = a == 0, ay = a == 1, by = b == 1, bz = b == 2;
         const Outs r = pairs(sum(dup(va), pack(vb, df_neg(vb))), ow2, k.om2w[2], s1, o1, s2, o2);
         emit.put(s1, o1, ax, ay + by, bz, r.s.a);
         emit.put(s2, o2, ax, ay - by, -bz, r.s.b);
         emit.put(o1, s1, -ax, -ay - by, -bz, r.o.a);
         emit.put(o2, s2, -ax, by - ay, bz, r.o.b);
      }
   } else {
#pragma unroll
      for (int j = 0; j < 3; j++) {
         const int a = j < 2 ? 0 : 1, b = j == 0 ? 1 : 2;
         const int s1 = j == 0 ? 6 : (j == 1 ? 8 : 14), o1 = lat_opp(Q, s1);
         const int s2 = s1 + 1, o2 = lat_opp(Q, s2);
         const Outs r = pairs(sum(dup(v3[a]), pack(v3[b], df_neg(v3[b]))), ow2, k.om2w[2], s1, o1, s2, o2);
         emit(s1, r.s.a);
         emit(s2, r.s.b);
         emit(o1, r.o.a);
         emit(o2, r.o.b);
      }
   }
   // body diagonals (18,25) (20,23), then (19,24) (21,22): c = (1, +-1, 1), (1, +-1, -1)
   if constexpr (Q == 27) {
      const df2 ow3 = dup(df_mul_u(k.ow[3], rho));
      if constexpr (ROLLED) {
#pragma unroll 1
         for (int j = 0; j < 2; j++) {
            const df2 xy = sum(dup(v3[0]), pack(v3[1], df_neg(v3[1])));
            const df2 z = dup(j == 0 ? v3[2] : df_neg(v3[2]));
            const int s1 = 18 + j, o1 = 25 - j, s2 = 20 + j, o2 = 23 - j, cz = j == 0 ? 1 : -1;
            const Outs r = pairs(sum(xy, z), ow3, k.om2w[3], s1, o1, s2, o2);
            emit.put(s1, o1, 1, 1, cz, r.s.a);
            emit.put(s2, o2, 1, -1, cz, r.s.b);
            emit.put(o1, s1, -1, -1, -cz, r.o.a);
            emit.put(o2, s2, -1, 1, -cz, r.o.b);
         }
      } else {
         const df2 xy = sum(dup(v3[0]), pack(v3[1], df_neg(v3[1])));
#pragma unroll
         for (int j = 0; j < 2; j++) {
            const int s1 = 18 + j, o1 = 25 - j, s2 = 20 + j, o2 = 23 - j;
            const Outs r = pairs(sum(xy, dup(j == 0 ? v3[2] : df_neg(v3[2]))), ow3, k.om2w[3], s1, o1, s2, o2);
            emit(s1, r.s.a);
            emit(s2, r.s.b);
            emit(o1, r.o.a);
            emit(o2, r.o.b);
         }
      }
   }
   return range.ok();
}

// Emitter that collects the outputs in registers.
template <int Q>
struct EmitToArray {
   uint64_t res[Q];
   __host__ __device__ __forceinline__ void operator()(int s, uint64_t v) { res[s] = v; }
   __host__ __device__ __forceinline__ void put(int s, int, int, int, int, uint64_t v) { res[s] = v; }
};


// The fast path on bits[] in place: returns false, leaving bits[] untouched,
// when the cell must take the exact path.
template <int Q, int FORCE>
__host__ __device__ __forceinline__ bool collide_f64x_fast(uint64_t (&bits)[Q], const x64::Consts& k,
                                                          int compat)
{
   EmitToArray<Q> out;
   if (!collide_f64x_fast_emit<Q, FORCE>(bits, k, compat, out, KeepInputs{})) return false;
#pragma unroll
   for (int s = 0; s < Q; s++) bits[s] = out.res[s];
   return true;
}

// The fast path's constants from the launch parameters.
template <int Q>
__host__ __device__ __forceinline__ x64::Consts collide_consts(const KParams& p)
{
   x64::Consts k;
   k.om1 = {p.x_om1[0], p.x_om1[1]};
   k.omega = {p.x_omega[0], p.x_omega[1]};
#pragma unroll
   for (int c = 0; c < 4; c++) k.ow[c] = {p.x_ow[c][0], p.x_ow[c][1]};
#pragma unroll
   for (int d = 0; d < 3; d++) k.F[d] = {p.x_F[d][0], p.x_F[d][1]};
#pragma unroll
   for (int d = 0; d < 3; d++) k.F3[d] = {p.x_F3[d][0], p.x_F3[d][1]};
#pragma unroll
   for (int s = 0; s < Q; s++) k.Kf[s] = {p.x_Kf[s][0], p.x_Kf[s][1]};
#pragma unroll
   for (int c = 0; c < 4; c++) k.om2w[c] = {p.x_om2w[c][0], p.x_om2w[c][1]};
   k.om2w36 = {p.x_om2w36[0], p.x_om2w36[1]};
   k.om2 = p.om2f;
#pragma unroll
   for (int d = 0; d < 3; d++) k.Fshift[d] = {p.x_Fshift[d][0], p.x_Fshift[d][1]};
   k.kappa = p.x_kappa;
#pragma unroll
   for (int s = 0; s < Q; s++) k.E[s] = p.x_E[s];
   return k;
}

}  // namespace lbm
