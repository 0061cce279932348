// Collision arithmetic and population storage for the collide-stream kernels.
//
// The physics is the reference's BGK collision with Guo forcing
// (src/kernels/KernelAA_SOA_Base.cpp:186-247):
//   rho = sum f_s,  v = (sum c_s f_s + F/2) / rho
//   eq_s    = w_s rho (1 + cu + cu^2/2 - uu/2),   cu = 3 c_s.v, uu = 3 v.v
//   fdist_s = w_s (cf - fu + cu cf),              cf = 3 c_s.F, fu = 3 F.v
//   f_s'    = (1-omega) f_s + omega eq_s + (1-omega/2) fdist_s
// optionally followed by partial bounce-back with solid fraction sp:
//   post_s  = (1-sp) f_s' + sp f_opp(s)
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "lbm_lattice.cuh"
#include "lbm_packed.cuh"

namespace lbm {

enum StoreKind { ST_F64 = 0, ST_F32 = 1, ST_BF16 = 2, ST_F16 = 3 };
enum ArithKind { AR_F64 = 1, AR_F64X = 2, AR_F32 = 3 };
enum StepKind { K_AA_EVEN = 0, K_AA_ODD = 1, K_AB_PUSH = 2, K_AB_PULL = 3 };

// Scale applied to shifted FP16 populations so that small deviations stay in
// the normal range of binary16 (as in the FP16S format of Lehmann et al.
// 2022, "Accuracy and performance of the lattice Boltzmann method with 64-bit,
// 32-bit, and customized 16-bit number formats").
constexpr float kF16Scale = 32768.0f;

// Everything a step kernel needs, passed by value.
struct KParams {
   int nx, ny, nz;
   int z0;               // first z plane covered by the launch
   int64_t ncell;
   int64_t plane;        // elements between direction planes
   int64_t cstart, cend; // cell range handled by this launch
   double omega, om1, om2;        // omega, 1-omega, 1-0.5*omega (as the reference folds them)
   float omegaf, om1f, om2f;
   double F[3];                   // uniform body force
   float Ff[3];
   int compat;                    // Q19 AA Unroll rest forcing weight
   const uint32_t* links;         // per-cell link word or null
   const double* force_field;     // planar [3][plane] (FP64 arithmetic) or null
   const float* force_field_f;    // planar [3][plane] (FP32 arithmetic) or null
   const double* porosity;        // [plane] or null
   const float* porosity_f;
   // Float-pair (hi, lo) splits of the launch constants for the F64X path,
   // made on the host so no thread converts doubles.
   float x_om1[2], x_omega[2];
   float x_ow[4][2];              // omega * w per weight class (|c|^2 = 0..3)
   float x_F[3][2];               // uniform force
   float x_Kf[27][2];             // (1 - omega/2) w_s 3 c_s.F per direction
   float x_F3[3][2];              // 3 F
   float x_om2w[4][2];            // (1 - omega/2) w per weight class
   float x_om2w36[2];             // (1 - omega/2) / 36
   float x_Fshift[3][2];          // F / omega
   float x_kappa, x_E[27];        // (1 - omega/2) / omega; 3/2 F.F - (3 c_s.F)^2 / 2 per direction
   int forced;                    // forcing form of the F64X fast path, 0 without a uniform force
   // Exact FP64 arithmetic: F/2 and 3 c_s.F of the uniform force for the first
   // direction s of each opposite pair, rounded as the reference rounds them.
   double half_F[3];
   double cf3[13];
   uint32_t* sched;               // [kFeedWords] tile counters of the persistent kernels, zero between launches
};

// Link word: bit s set when the neighbour at x + c_s is solid or outside a
// non-periodic face (half-way bounce-back); bit 31 set when x itself is solid.
constexpr uint32_t kSolidBit = 0x80000000u;

// ---------------------------------------------------------------- storage
template <int ST> struct Store;
template <> struct Store<ST_F64> { using T = double; static constexpr int bytes = 8; };
template <> struct Store<ST_F32> { using T = float; static constexpr int bytes = 4; };
template <> struct Store<ST_BF16> { using T = __nv_bfloat16; static constexpr int bytes = 2; };
template <> struct Store<ST_F16> { using T = __half; static constexpr int bytes = 2; };

// Shifted storage: the stored value is (f - w) (times kF16Scale for FP16).
__device__ __forceinline__ float load_shifted(const float* p) { return *p; }
__device__ __forceinline__ float load_shifted(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float load_shifted(const __half* p)
{
   return __half2float(*p) * (1.0f / kF16Scale);
}
__device__ __forceinline__ void store_shifted(float* p, float g) { *p = g; }
__device__ __forceinline__ void store_shifted(__nv_bfloat16* p, float g) { *p = __float2bfloat16_rn(g); }
__device__ __forceinline__ void store_shifted(__half* p, float g) { *p = __float2half_rn(g * kF16Scale); }

// Representative s < opp(s) of the P-th opposite pair (the reference's
// direction order: pairs (0,1), (2,3), ..., the rest direction last).
template <int Q, int P>
__host__ __device__ constexpr int pair_rep()
{
   int seen = 0;
   for (int t = 0; t < Q; t++)
      if (t < lat_opp(Q, t)) {
         if (seen == P) return t;
         seen++;
      }
   return -1;
}

// ------------------------------------------- FP32 shifted collision
// Stored values are G = S (f - w) with S = 2^15 for FP16 and 1 otherwise.
// With drho = sum (f - w) (sum w = 1) and j = sum c (f - w) (sum c w = 0):
//   eq_s - w_s = w_s (drho + rho (cu + cu^2/2 - uu/2))
//   G_s'       = (1-omega) G_s + omega S (eq_s - w_s) + (1-omega/2) S fdist_s
// which keeps the large constant w out of the single-precision arithmetic;
// S enters only through per-cell factors.  Opposite directions share
// cu(opp) = -cu, so S (eq - w) = A +- B with A = w (S drho + S rho (cu^2 - uu)/2)
// and B = w S rho cu.
// Every operation has a rounding of its own, whatever the compiler contracts:
// products are joined to sums by explicit multiply-adds, and sums of values that
// are products themselves (3u, 3F) are intrinsics.  So the one-cell and the
// two-cell forms, in any kernel, give the same bits.
template <int ST> struct ShiftScale { static constexpr float S = 1.0f; };
template <> struct ShiftScale<ST_F16> { static constexpr float S = kF16Scale; };

__device__ __forceinline__ float load_raw(const float* p) { return *p; }
__device__ __forceinline__ float load_raw(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float load_raw(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ void store_raw(float* p, float g) { *p = g; }
__device__ __forceinline__ void store_raw(__nv_bfloat16* p, float g) { *p = __float2bfloat16_rn(g); }
__device__ __forceinline__ void store_raw(__half* p, float g) { *p = __float2half_rn(g); }

template <int Q, int S_>
__device__ __forceinline__ float cdot_f(const float (&v)[3])
{
   constexpr int c0 = lat_c(Q, S_, 0), c1 = lat_c(Q, S_, 1), c2 = lat_c(Q, S_, 2);
   float r = 0.0f;
   bool any = false;
   if (c0 != 0) { r = c0 > 0 ? v[0] : -v[0]; any = true; }
   if (c1 != 0) { r = any ? (c1 > 0 ? x64::fadd(r, v[1]) : x64::fsub(r, v[1])) : (c1 > 0 ? v[1] : -v[1]); any = true; }
   if (c2 != 0) { r = any ? (c2 > 0 ? x64::fadd(r, v[2]) : x64::fsub(r, v[2])) : (c2 > 0 ? v[2] : -v[2]); }
   return r;
}

// Per-cell quantities of the shifted collision: 3u, 3F, fu = 3 F.u, uu = 3 u.u
// and the weight-class factors w S drho, w S rho.
struct ShiftedCell {
   float u3[3], F3[3], fu, uu, wSd[4], wSr[4];
};

template <int Q, int ST, bool FORCE>
__device__ __forceinline__ ShiftedCell shifted_cell(const float (&G)[Q], float F0, float F1, float F2)
{
   constexpr float S = ShiftScale<ST>::S;
   constexpr float iS = 1.0f / S;
   ShiftedCell c;
   float Sd = 0.f, j0 = 0.f, j1 = 0.f, j2 = 0.f;
#pragma unroll
   for (int s = 0; s < Q; s++) {
      Sd += G[s];
      const int c0 = lat_c(Q, s, 0), c1 = lat_c(Q, s, 1), c2 = lat_c(Q, s, 2);
      if (c0 > 0) j0 += G[s]; else if (c0 < 0) j0 -= G[s];
      if (c1 > 0) j1 += G[s]; else if (c1 < 0) j1 -= G[s];
      if (c2 > 0) j2 += G[s]; else if (c2 < 0) j2 -= G[s];
   }
   const float rho = fmaf(Sd, iS, 1.0f);
   const float ir = __frcp_rn(rho);
   // 3u and 3F
   const float ir3 = 3.0f * ir;
   c.u3[0] = fmaf(j0, iS, 0.5f * F0) * ir3;
   c.u3[1] = fmaf(j1, iS, 0.5f * F1) * ir3;
   c.u3[2] = fmaf(j2, iS, 0.5f * F2) * ir3;
   c.uu = fmaf(c.u3[2], c.u3[2], fmaf(c.u3[0], c.u3[0], x64::fmul(c.u3[1], c.u3[1]))) * (1.0f / 3.0f);   // 3 u.u
   c.F3[0] = 3.0f * F0;
   c.F3[1] = 3.0f * F1;
   c.F3[2] = 3.0f * F2;
   c.fu = FORCE ? fmaf(c.F3[2], c.u3[2], fmaf(c.F3[0], c.u3[0], x64::fmul(c.F3[1], c.u3[1]))) * (1.0f / 3.0f) : 0.0f;
   const float Sr = S * rho;
#pragma unroll
   for (int k = 0; k < 4; k++) {
      float w;
      if (Q == 19) w = k == 0 ? (float)(1.0 / 3.0) : (k == 1 ? (float)(1.0 / 18.0) : (float)(1.0 / 36.0));
      else w = k == 0 ? (float)(8.0 / 27.0) : (k == 1 ? (float)(2.0 / 27.0) : (k == 2 ? (float)(1.0 / 54.0) : (float)(1.0 / 216.0)));
      c.wSd[k] = w * Sd;
      c.wSr[k] = w * Sr;
   }
   return c;
}

// Outputs of the P-th pair (s, opp(s)) from the inputs Gs, Gob.
template <int Q, int ST, bool FORCE, int P>
__device__ __forceinline__ void shifted_pair(const ShiftedCell& c, float Gs, float Gob, float om1, float omega,
                                             float Som2, float& os, float& oob)
{
   constexpr int s = pair_rep<Q, P>();
   constexpr int cls = lat_norm2(Q, s);
   const float cu = cdot_f<Q, s>(c.u3);
   const float A = fmaf(c.wSr[cls], 0.5f * fmaf(cu, cu, -c.uu), c.wSd[cls]);
   float fs = 0.0f, fo = 0.0f;
   if (FORCE) {
      constexpr float w = (float)lat_w(Q, s);
      const float cf = cdot_f<Q, s>(c.F3);
      const float sym = fmaf(cu, cf, -c.fu);
      fs = Som2 * w * x64::fadd(cf, sym);
      fo = Som2 * w * x64::fsub(sym, cf);
   }
   os = fmaf(om1, Gs, fmaf(omega, fmaf(c.wSr[cls], cu, A), fs));
   oob = fmaf(om1, Gob, fmaf(omega, fmaf(-c.wSr[cls], cu, A), fo));
}

// Output of the rest direction: A = w (S drho + S rho (-uu/2)), forcing -wf fu.
template <int Q, int ST, bool FORCE>
__device__ __forceinline__ float shifted_rest(const ShiftedCell& c, float GR, const KParams& p, float Som2)
{
   const float A = fmaf(c.wSr[0], -0.5f * c.uu, c.wSd[0]);
   float fr = 0.0f;
   if (FORCE) {
      const float wf = (Q == 19 && p.compat) ? (float)(1.0 / 36.0) : (float)lat_w(Q, lat_rest(Q));
      fr = -Som2 * wf * c.fu;
   }
   return fmaf(p.om1f, GR, fmaf(p.omegaf, A, fr));
}

template <int Q, int ST, bool FORCE, int P = 0>
__device__ __forceinline__ void collide_pairs_f32(const float (&G)[Q], float (&o)[Q], const ShiftedCell& c, float om1,
                                                  float omega, float Som2)
{
   if constexpr (P < (Q - 1) / 2) {
      constexpr int s = pair_rep<Q, P>();
      constexpr int ob = lat_opp(Q, s);
      shifted_pair<Q, ST, FORCE, P>(c, G[s], G[ob], om1, omega, Som2, o[s], o[ob]);
      collide_pairs_f32<Q, ST, FORCE, P + 1>(G, o, c, om1, omega, Som2);
   }
}

template <int Q, int ST, bool FORCE>
__device__ __forceinline__ void collide_f32(const float (&G)[Q], float (&o)[Q], float F0, float F1, float F2,
                                            float sp, const KParams& p)
{
   const ShiftedCell c = shifted_cell<Q, ST, FORCE>(G, F0, F1, F2);
   const float Som2 = ShiftScale<ST>::S * p.om2f;
   collide_pairs_f32<Q, ST, FORCE>(G, o, c, p.om1f, p.omegaf, Som2);
   constexpr int R = lat_rest(Q);
   o[R] = shifted_rest<Q, ST, FORCE>(c, G[R], p, Som2);
   if (sp != 0.0f) {
      const float keep = 1.0f - sp;
#pragma unroll
      for (int s = 0; s < Q; s++) o[s] = fmaf(keep, o[s], x64::fmul(sp, G[lat_opp(Q, s)]));
   }
}

// ------------------------------------- two cells in the packed halves
// The arithmetic of collide_f32 for two cells with a uniform force, operation for
// operation: inputs G[s] = (cell 0, cell 1); each direction's two outputs go to
// emit(s, (o0, o1)) as soon as they are made, so no output array stays in
// registers.
struct ShiftedCell2 {
   x64::f2 u3[3], fu, uu, wSd[4], wSr[4];
   float F3[3];
};

template <int Q, int S_>
__device__ __forceinline__ x64::f2 cdot_f2(const x64::f2 (&v)[3])
{
   constexpr int c0 = lat_c(Q, S_, 0), c1 = lat_c(Q, S_, 1), c2 = lat_c(Q, S_, 2);
   x64::f2 r = {0.0f, 0.0f};
   bool any = false;
   if (c0 != 0) { r = c0 > 0 ? v[0] : x64::neg2(v[0]); any = true; }
   if (c1 != 0) { r = any ? (c1 > 0 ? x64::add2(r, v[1]) : x64::sub2(r, v[1])) : (c1 > 0 ? v[1] : x64::neg2(v[1])); any = true; }
   if (c2 != 0) { r = any ? (c2 > 0 ? x64::add2(r, v[2]) : x64::sub2(r, v[2])) : (c2 > 0 ? v[2] : x64::neg2(v[2])); }
   return r;
}

template <int Q, int ST, bool FORCE>
__device__ __forceinline__ ShiftedCell2 shifted_cell2(const x64::f2 (&G)[Q], const KParams& p)
{
   using namespace x64;
   constexpr float S = ShiftScale<ST>::S;
   constexpr float iS = 1.0f / S;
   ShiftedCell2 c;
   f2 Sd = {0.f, 0.f}, j[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
   for (int s = 0; s < Q; s++) {
      Sd = add2(Sd, G[s]);
#pragma unroll
      for (int d = 0; d < 3; d++) {
         if (lat_c(Q, s, d) > 0) j[d] = add2(j[d], G[s]);
         if (lat_c(Q, s, d) < 0) j[d] = sub2(j[d], G[s]);
      }
   }
   const f2 rho = fma2(Sd, dup2(iS), dup2(1.0f));
   const f2 ir3 = {3.0f * __frcp_rn(rho.x), 3.0f * __frcp_rn(rho.y)};
#pragma unroll
   for (int d = 0; d < 3; d++) c.u3[d] = mul2(fma2(j[d], dup2(iS), dup2(FORCE ? 0.5f * p.Ff[d] : 0.0f)), ir3);
   const f2 third = dup2(1.0f / 3.0f);
   c.uu = mul2(fma2(c.u3[2], c.u3[2], fma2(c.u3[0], c.u3[0], mul2(c.u3[1], c.u3[1]))), third);
   c.fu = {0.f, 0.f};
   if constexpr (FORCE) {
#pragma unroll
      for (int d = 0; d < 3; d++) c.F3[d] = 3.0f * p.Ff[d];
      c.fu = mul2(fma2(dup2(c.F3[2]), c.u3[2], fma2(dup2(c.F3[0]), c.u3[0], mul2(dup2(c.F3[1]), c.u3[1]))), third);
   }
   const f2 Sr = mul2(dup2(S), rho);
#pragma unroll
   for (int k = 0; k < 4; k++) {
      float w;
      if (Q == 19) w = k == 0 ? (float)(1.0 / 3.0) : (k == 1 ? (float)(1.0 / 18.0) : (float)(1.0 / 36.0));
      else w = k == 0 ? (float)(8.0 / 27.0) : (k == 1 ? (float)(2.0 / 27.0) : (k == 2 ? (float)(1.0 / 54.0) : (float)(1.0 / 216.0)));
      c.wSd[k] = mul2(dup2(w), Sd);
      c.wSr[k] = mul2(dup2(w), Sr);
   }
   return c;
}

template <int Q, int ST, bool FORCE, int P = 0, class Emit2>
__device__ __forceinline__ void shifted_pairs2(const x64::f2 (&G)[Q], const ShiftedCell2& c, const KParams& p, float Som2,
                                               Emit2& emit)
{
   using namespace x64;
   if constexpr (P < (Q - 1) / 2) {
      constexpr int s = pair_rep<Q, P>();
      constexpr int ob = lat_opp(Q, s);
      constexpr int cls = lat_norm2(Q, s);
      const f2 cu = cdot_f2<Q, s>(c.u3);
      const f2 A = fma2(c.wSr[cls], mul2(dup2(0.5f), fma2(cu, cu, neg2(c.uu))), c.wSd[cls]);
      f2 fs = {0.f, 0.f}, fo = {0.f, 0.f};
      if constexpr (FORCE) {
         constexpr float w = (float)lat_w(Q, s);
         const f2 cf = dup2(cdot_f<Q, s>(c.F3));
         const f2 sym = fma2(cu, cf, neg2(c.fu));
         const f2 Sw = dup2(Som2 * w);
         fs = mul2(Sw, add2(cf, sym));
         fo = mul2(Sw, sub2(sym, cf));
      }
      const f2 om1 = dup2(p.om1f), om = dup2(p.omegaf);
      emit(s, fma2(om1, G[s], fma2(om, fma2(c.wSr[cls], cu, A), fs)));
      emit(ob, fma2(om1, G[ob], fma2(om, fma2(neg2(c.wSr[cls]), cu, A), fo)));
      shifted_pairs2<Q, ST, FORCE, P + 1>(G, c, p, Som2, emit);
   }
}

template <int Q, int ST, bool FORCE, class Emit2>
__device__ __forceinline__ void collide2_f32_emit(const x64::f2 (&G)[Q], const KParams& p, Emit2& emit)
{
   using namespace x64;
   const ShiftedCell2 c = shifted_cell2<Q, ST, FORCE>(G, p);
   const float Som2 = ShiftScale<ST>::S * p.om2f;
   shifted_pairs2<Q, ST, FORCE>(G, c, p, Som2, emit);
   constexpr int R = lat_rest(Q);
   const f2 A = fma2(c.wSr[0], mul2(dup2(-0.5f), c.uu), c.wSd[0]);
   f2 fr = {0.f, 0.f};
   if constexpr (FORCE) {
      const float wf = (Q == 19 && p.compat) ? (float)(1.0 / 36.0) : (float)lat_w(Q, R);
      fr = mul2(dup2(-Som2 * wf), c.fu);
   }
   emit(R, fma2(dup2(p.om1f), G[R], fma2(dup2(p.omegaf), A, fr)));
}

}  // namespace lbm
