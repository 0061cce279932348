// Exact FP64 collision: the reference's operations, each rounded as IEEE double.
#pragma once

#include "lbm_soft.cuh"

namespace lbm {

// ------------------------------------------------- exact FP64 collision
// Operation order and association of KernelAA_SOA_Base.cpp:186-247 with every
// operation an explicitly rounded IEEE double op (no FMA contraction), so the
// result is bit-identical to the reference CPU build.
//
// The FP64 pipe bounds it: one FP64 instruction holds it for 76 cycles per warp
// and sub-partition (measured; an FP32 or integer add: 1).  So every operation
// whose result is known without it is left out, each time with the same bits:
//   * terms whose stencil component is zero (the reference adds d * 0.0 = +-0.0,
//     which leaves every non-zero partial sum unchanged) and the first add to 0;
//   * opposite directions share 3 c.v, its square and 3 c.F up to the sign
//     (negation is exact), and w rho is one product per weight class;
//   * products with 0.5 are exponent decrements (half_exact);
//   * 3 c.F and F/2 of a uniform force are the same for all cells and come from
//     the host;
//   * without a force every forcing term is +-0 and leaves the result unchanged,
//     unless v is not finite, which makes every result NaN (F.v = 0 inf).
// The step kernels (SOFT) then move additions to the integer pipes, which are idle:
// the sums, 1 + cu + cu^2/2 - uu/2 and the last addition (lbm_soft.cuh), for cells in
// the ranges checked there; others take the plain form.  Additions and products left
// in FP64 per D3Q19 cell: 215 without a force and 330 with one in the plain form, 94
// without a force in the integer one (136 executed with the reciprocal, by the
// counter; the pipe is 78 % busy).  Two steps of a 128^3 D3Q19 box: 3375 us with
// every operation of the reference, 1803 us in the plain form, 1182 us in the integer
// one, whose integer work is about 3,500 instructions.
template <int Q, int S>
__device__ __forceinline__ double cdot_exact(double a0, double a1, double a2)
{
   constexpr int c0 = lat_c(Q, S, 0), c1 = lat_c(Q, S, 1), c2 = lat_c(Q, S, 2);
   double acc = 0.0;
   bool any = false;
   if (c0 != 0) { acc = c0 > 0 ? a0 : -a0; any = true; }
   if (c1 != 0) { acc = any ? (c1 > 0 ? __dadd_rn(acc, a1) : __dsub_rn(acc, a1)) : (c1 > 0 ? a1 : -a1); any = true; }
   if (c2 != 0) { acc = any ? (c2 > 0 ? __dadd_rn(acc, a2) : __dsub_rn(acc, a2)) : (c2 > 0 ? a2 : -a2); any = true; }
   return acc;
}

// 0.5 x by the exponent field.  Where that is not exact x is below 2^-1021: the
// result is 0 then, which the callers multiply by x (a product that underflows
// to zero either way) or subtract from a value near 1.  An infinite or NaN x
// gives a finite value, which the callers multiply by x or guard against.
__device__ __forceinline__ double half_exact(double x)
{
   const uint32_t hi = (uint32_t)__double2hiint(x);
   const bool tiny = (hi & 0x7FE00000u) == 0u;
   return __hiloint2double((int)(tiny ? 0u : hi - 0x00100000u), tiny ? 0 : __double2loint(x));
}

__device__ __forceinline__ bool finite_exact(double x) { return ((uint32_t)__double2hiint(x) & 0x7FF00000u) != 0x7FF00000u; }

// Forcing of the exact collision: none, a uniform force (3 c.F from the host),
// or a force of the cell.
enum ExactForce { XF_NONE = 0, XF_UNIFORM = 1, XF_CELL = 2 };

// Per-cell values of the exact collision (hq: hvv as a fixed-point image, SOFT).
struct ExactCell {
   uint64_t hq;
   double v[3], F[3];
   double wr[4];          // w rho per weight class
   double hvv, fdotv;     // vdotv / 2, fdotv
   double sp, keep;
};

// (1 - sp) out + sp f_opp: partial bounce-back with solid fraction sp.
__device__ __forceinline__ double bounce_exact(double o, double f_opp, const ExactCell& c)
{
   return c.sp != 0.0 ? __dadd_rn(__dmul_rn(c.keep, o), __dmul_rn(c.sp, f_opp)) : o;
}

// Pairs P, P + 1, ...: in(s) gives population s, emit(s, out) takes its result
// as soon as it is made.
template <int Q, int FORM, bool SOFT, int P = 0, class In, class Emit>
__device__ __forceinline__ void pairs_exact(const ExactCell& c, const In& in, Emit& emit, const KParams& p)
{
   if constexpr (P < (Q - 1) / 2) {
      constexpr int s = pair_rep<Q, P>();
      constexpr int ob = lat_opp(Q, s);
      constexpr int cls = lat_norm2(Q, s);
      constexpr double w = lat_w(Q, s);
      const double cv = __dmul_rn(3.0, cdot_exact<Q, s>(c.v[0], c.v[1], c.v[2]));
      const double q = __dmul_rn(half_exact(cv), cv);
      double ps, po;
      if constexpr (SOFT) {
         const uint64_t cb = x64::double_bits(cv), ci = soft::image_sticky(cb);
         const bool neg = (int64_t)cb < 0;
         const soft::Polynomial poly{soft::image_sticky(x64::double_bits(q)), c.hq};
         ps = poly(ci, neg);
         po = poly(ci, !neg);
      } else {
         ps = __dsub_rn(__dadd_rn(__dadd_rn(1.0, cv), q), c.hvv);
         po = __dsub_rn(__dadd_rn(__dsub_rn(1.0, cv), q), c.hvv);
      }
      const double ds = in(s), dob = in(ob);
      const double as = __dmul_rn(p.om1, ds), ao = __dmul_rn(p.om1, dob);
      const double bs = __dmul_rn(p.omega, __dmul_rn(c.wr[cls], ps)), bo = __dmul_rn(p.omega, __dmul_rn(c.wr[cls], po));
      double os, oob;
      if constexpr (SOFT) {
         os = soft::add_double(as, bs);
         oob = soft::add_double(ao, bo);
      } else {
         os = __dadd_rn(as, bs);
         oob = __dadd_rn(ao, bo);
      }
      if constexpr (FORM != XF_NONE) {
         double cf;
         if constexpr (FORM == XF_UNIFORM) cf = p.cf3[P];
         else cf = __dmul_rn(3.0, cdot_exact<Q, s>(c.F[0], c.F[1], c.F[2]));
         const double vf = __dmul_rn(cv, cf);
         const double fs = __dmul_rn(w, __dadd_rn(__dsub_rn(cf, c.fdotv), vf));
         const double fo = __dmul_rn(w, __dadd_rn(__dsub_rn(-cf, c.fdotv), vf));
         os = __dadd_rn(os, __dmul_rn(p.om2, fs));
         oob = __dadd_rn(oob, __dmul_rn(p.om2, fo));
      }
      emit(s, bounce_exact(os, dob, c));
      emit(ob, bounce_exact(oob, ds, c));
      pairs_exact<Q, FORM, SOFT, P + 1>(c, in, emit, p);
   }
}

// rho and sum c f, added up direction by direction as the reference does and
// rounded after every addition, in integer instructions; in(s) gives the pattern
// of population s.  False (the results mean nothing) unless the populations lie in
// [2^-10, 1/4), the rest one below 1, and rho < 2.
template <int Q, class In>
__device__ __forceinline__ bool sums_soft(const In& in, double& rho, double (&v)[3])
{
   constexpr uint32_t kLeast = (uint32_t)(1023 - 10) << 20, kQuarter = (uint32_t)(1023 - 2) << 20,
                      kOne = (uint32_t)1023 << 20;
   uint32_t least = kQuarter, most = 0u, wrapped = 0u;
   uint64_t r = 0;
   int64_t j[3] = {0, 0, 0};
#pragma unroll
   for (int s = 0; s < Q; s++) {
      const uint64_t b = in(s);
      const uint32_t hi = (uint32_t)(b >> 32);
      least = least < hi ? least : hi;
      if (s != lat_rest(Q)) most = most > hi ? most : hi;
      else wrapped |= hi >= kOne ? 0x80000000u : 0u;
      const uint64_t X = soft::image(b);
      r = s == 0 ? X : soft::round_positive(r + X);
      // rho < 2: looked at often enough that the sum cannot wrap in between
      if (s % 6 == 5 || s == Q - 1) wrapped |= (uint32_t)(r >> 32);
#pragma unroll
      for (int k = 0; k < 3; k++) {
         const int cs = lat_c(Q, s, k);
         const bool first = s == 2 * k;   // the axis pairs come first, +e_k at 2k
         if (cs > 0) j[k] = first ? (int64_t)X : soft::round_signed((int64_t)((uint64_t)j[k] + X));
         else if (cs < 0) j[k] = soft::round_signed((int64_t)((uint64_t)j[k] - X));
      }
   }
   if (least < kLeast || most >= kQuarter || (wrapped & 0x80000000u)) return false;
   rho = soft::positive_to_double(r);
#pragma unroll
   for (int k = 0; k < 3; k++) v[k] = soft::signed_to_double(j[k]);
   return true;
}

// One cell: in(s) gives population s (called twice per direction), emit(s, out)
// takes the results.  F is read for XF_CELL only.  SOFT: returns false, with
// nothing emitted, for a cell outside the integer additions' ranges.
template <int Q, int FORM, bool SOFT, class In, class Emit>
__device__ __forceinline__ bool collide_f64_form(const In& in, Emit& emit, double F0, double F1, double F2, double sp,
                                                 const KParams& p)
{
   ExactCell c;
   c.F[0] = F0; c.F[1] = F1; c.F[2] = F2;
   double rho = 0.0;
   c.v[0] = c.v[1] = c.v[2] = 0.0;
   if constexpr (SOFT) {
      if (!sums_soft<Q>([&](int s) { return x64::double_bits(in(s)); }, rho, c.v)) return false;
   } else {
#pragma unroll
      for (int s = 0; s < Q; s++) {
         const double d = in(s);
         rho = s == 0 ? d : __dadd_rn(rho, d);
#pragma unroll
         for (int k = 0; k < 3; k++) {
            const int cs = lat_c(Q, s, k);
            const bool first = s == 2 * k;
            if (cs > 0) c.v[k] = first ? d : __dadd_rn(c.v[k], d);
            else if (cs < 0) c.v[k] = __dsub_rn(c.v[k], d);
         }
      }
   }
   if constexpr (FORM != XF_NONE) {
#pragma unroll
      for (int k = 0; k < 3; k++)
         c.v[k] = __dadd_rn(c.v[k], FORM == XF_UNIFORM ? p.half_F[k] : __dmul_rn(0.5, c.F[k]));
   }
   const double invRho = __drcp_rn(rho);
#pragma unroll
   for (int k = 0; k < 3; k++) c.v[k] = __dmul_rn(c.v[k], invRho);
   if constexpr (SOFT) {
      // |v_d| < 0.1 (its high word): |3 c.v| < 0.9, uu/2 < 0.05
      constexpr uint32_t kTenth = 0x3FB99999u;
      const uint32_t h0 = (uint32_t)__double2hiint(c.v[0]) & 0x7FFFFFFFu, h1 = (uint32_t)__double2hiint(c.v[1]) & 0x7FFFFFFFu,
                     h2 = (uint32_t)__double2hiint(c.v[2]) & 0x7FFFFFFFu;
      if (h0 >= kTenth || h1 >= kTenth || h2 >= kTenth) return false;
   }
   const double vdotv = __dmul_rn(
      3.0, __dadd_rn(__dadd_rn(__dmul_rn(c.v[0], c.v[0]), __dmul_rn(c.v[1], c.v[1])), __dmul_rn(c.v[2], c.v[2])));
   c.hvv = half_exact(vdotv);
   if (!finite_exact(vdotv)) {
      c.hvv = vdotv;
      // F.v of a force of zero is NaN for such a v
      if (FORM == XF_NONE && !(finite_exact(c.v[0]) && finite_exact(c.v[1]) && finite_exact(c.v[2])))
         c.hvv = __longlong_as_double(0x7FF8000000000000LL);
   }
   c.hq = 0;
   if constexpr (SOFT) c.hq = soft::image_sticky(x64::double_bits(c.hvv));
   c.fdotv = 0.0;
   if constexpr (FORM != XF_NONE) {
      const double G0 = FORM == XF_UNIFORM ? p.F[0] : c.F[0], G1 = FORM == XF_UNIFORM ? p.F[1] : c.F[1],
                   G2 = FORM == XF_UNIFORM ? p.F[2] : c.F[2];
      c.fdotv = __dmul_rn(
         3.0, __dadd_rn(__dadd_rn(__dmul_rn(G0, c.v[0]), __dmul_rn(G1, c.v[1])), __dmul_rn(G2, c.v[2])));
   }
   c.sp = sp;
   c.keep = __dsub_rn(1.0, sp);
   constexpr int kClasses = Q == 19 ? 3 : 4;
   constexpr double wc[4] = {lat_w(Q, lat_rest(Q)), lat_w(Q, 0), lat_w(Q, 6), lat_w(Q, Q == 27 ? 18 : 6)};
#pragma unroll
   for (int k = 0; k < kClasses; k++) c.wr[k] = __dmul_rn(wc[k], rho);
   // rest direction: c.v = c.F = 0
   constexpr int R = lat_rest(Q);
   const double dr = in(R);
   double o = __dadd_rn(__dmul_rn(p.om1, dr), __dmul_rn(p.omega, __dmul_rn(c.wr[0], __dsub_rn(1.0, c.hvv))));
   if constexpr (FORM != XF_NONE) {
      const double wf = (Q == 19 && p.compat) ? 1.0 / 36.0 : lat_w(Q, R);
      o = __dadd_rn(o, __dmul_rn(p.om2, __dmul_rn(wf, -c.fdotv)));
   }
   emit(R, bounce_exact(o, dr, c));
   pairs_exact<Q, FORM, SOFT>(c, in, emit, p);
   return true;
}

// SOFT: the integer additions where the cell allows them.
template <int Q, int FORM, bool SOFT, class In, class Emit>
__device__ __forceinline__ void collide_f64_emit(const In& in, Emit& emit, double F0, double F1, double F2, double sp,
                                                 const KParams& p)
{
   if constexpr (SOFT)
      if (collide_f64_form<Q, FORM, true>(in, emit, F0, F1, F2, sp, p)) return;
   collide_f64_form<Q, FORM, false>(in, emit, F0, F1, F2, sp, p);
}

// The same for a uniform force, none or not.
template <int Q, bool SOFT, class In, class Emit>
__device__ __forceinline__ void collide_f64_uniform(const In& in, Emit& emit, double sp, const KParams& p)
{
   if (p.forced) collide_f64_emit<Q, XF_UNIFORM, SOFT>(in, emit, 0.0, 0.0, 0.0, sp, p);
   else collide_f64_emit<Q, XF_NONE, SOFT>(in, emit, 0.0, 0.0, 0.0, sp, p);
}

}  // namespace lbm
