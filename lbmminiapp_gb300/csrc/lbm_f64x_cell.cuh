// F64X cell updates: the fast path, and the exact IEEE double collision for cells
// outside its range.
#pragma once

#include "lbm_exact.cuh"
#include "lbm_f64x.cuh"

namespace lbm {

// F64X cell update with a uniform force: fast path, else the exact IEEE
// double collision.
template <int Q>
__device__ __forceinline__ void collide_f64x(uint64_t (&bits)[Q], const KParams& p)
{
   const x64::Consts k = collide_consts<Q>(p);
   const bool fast = p.forced == 3   ? collide_f64x_fast<Q, 3>(bits, k, p.compat)
                     : p.forced == 2 ? collide_f64x_fast<Q, 2>(bits, k, p.compat)
                     : p.forced    ? collide_f64x_fast<Q, 1>(bits, k, p.compat)
                                   : collide_f64x_fast<Q, 0>(bits, k, p.compat);
   if (fast) return;
   double o[Q];
   auto in = [&](int s) { return x64::as_double(bits[s]); };
   auto keep = [&](int s, double v) { o[s] = v; };
   collide_f64_uniform<Q, false>(in, keep, 0.0, p);
#pragma unroll
   for (int s = 0; s < Q; s++) bits[s] = x64::double_bits(o[s]);
}

// Input pattern s read again from shared memory (direction s at byte 256 s
// from the lane's first).  The load is volatile so that the compiler does not
// keep the first load's value live in registers instead.  REST: the rest
// population is in a register.
template <int Q, bool REST>
struct AgainFromShared {
   static constexpr bool kRefetch = true;
   uint32_t addr;
   uint64_t rest;
   __device__ __forceinline__ uint64_t raw(int s) const
   {
      if (REST && s == lat_rest(Q)) return rest;
      unsigned long long v;
      asm volatile("ld.shared.u64 %0, [%1];\n" : "=l"(v) : "r"(addr + 256u * (uint32_t)s));
      return v;
   }
};

// collide_f64x for inputs that stay in shared memory (direction s at in[32 s]; with
// REST the last one, the rest direction, is `rest`),
// with each output handed to emit(s, pattern) as it is made, so neither the
// input nor the output patterns stay in registers through the fast path: the
// moment sums read the inputs once, the update reads them again.  If
// the fast path fails after emitting, the exact results are emitted again
// over them (the fallback reads its inputs from shared memory): a caller's
// emit must let a later emit of the same s win, as stores from one thread to
// one address do.
// FORCE: the launch's forcing form (p.forced), compile-time for no force and for
// the velocity shift, the forms that nearly every run has: a kernel that holds
// all four forms' code allocates registers for the worst of them (D3Q19 AA odd
// step, 256x128x128: 219 us against 211).  kForceOther holds forms 1 and 2.
constexpr int kForceOther = 1;
template <int Q, int FORCE, bool REST, class Emit>
__device__ __forceinline__ void collide_f64x_shared_emit(const unsigned long long* in, uint64_t rest, const KParams& p,
                                                         Emit& emit)
{
   uint64_t bits[Q];
#pragma unroll
   for (int s = 0; s < Q; s++) bits[s] = REST && s == lat_rest(Q) ? rest : in[s * 32];
   const x64::Consts k = collide_consts<Q>(p);
   const AgainFromShared<Q, REST> again{(uint32_t)__cvta_generic_to_shared(in), rest};
   bool fast;
   if constexpr (FORCE == kForceOther)
      fast = p.forced == 2 ? collide_f64x_fast_emit<Q, 2>(bits, k, p.compat, emit, again)
                           : collide_f64x_fast_emit<Q, 1>(bits, k, p.compat, emit, again);
   else fast = collide_f64x_fast_emit<Q, FORCE>(bits, k, p.compat, emit, again);
   if (fast) return;
   auto input = [&](int s) { return x64::as_double(again.raw(s)); };
   auto out = [&](int s, double v) { emit(s, x64::double_bits(v)); };
   collide_f64_emit<Q, FORCE == 0 ? XF_NONE : XF_UNIFORM, false>(input, out, 0.0, 0.0, 0.0, 0.0, p);
}

}  // namespace lbm
