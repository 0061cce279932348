// FP32 operations with defined rounding, one at a time and two at a time.
//
// sm_103a's packed FP32 instructions do two independent IEEE operations on a
// 64-bit register pair: the same FP32 rate (2 cycles per warp instruction and
// sub-partition instead of 1) from half the issue slots, with negations folded
// into the operands.  The step kernels run short of issue slots, so the F64X
// collision runs two directions at a time and the two-cells-per-thread kernels of
// the shifted storage run their two cells together.  Each half rounds as the
// scalar instruction does: the results are the scalar form's, bit for bit.
#pragma once

#include <cstdint>
#ifndef __CUDA_ARCH__
#include <cfenv>
#include <cmath>
#endif

namespace lbm {
namespace x64 {

__host__ __device__ __forceinline__ float ffma(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
   return __fmaf_rn(a, b, c);
#else
   return std::fmaf(a, b, c);
#endif
}

// Plain rounded-to-nearest FP32 ops that the compiler must not contract.
__host__ __device__ __forceinline__ float fadd(float a, float b)
{
#ifdef __CUDA_ARCH__
   return __fadd_rn(a, b);
#else
   volatile float r = a + b;
   return r;
#endif
}

__host__ __device__ __forceinline__ float fsub(float a, float b)
{
#ifdef __CUDA_ARCH__
   return __fsub_rn(a, b);
#else
   volatile float r = a - b;
   return r;
#endif
}

__host__ __device__ __forceinline__ float fmul(float a, float b)
{
#ifdef __CUDA_ARCH__
   return __fmul_rn(a, b);
#else
   volatile float r = a * b;
   return r;
#endif
}

// a + b rounded toward zero.
__host__ __device__ __forceinline__ float fadd_rz(float a, float b)
{
#ifdef __CUDA_ARCH__
   return __fadd_rz(a, b);
#else
   const int old = std::fegetround();
   std::fesetround(FE_TOWARDZERO);
   volatile float va = a, vb = b;
   volatile float r = va + vb;
   std::fesetround(old);
   return r;
#endif
}

struct f2 {
   float x, y;
};

__host__ __device__ __forceinline__ f2 dup2(float a) { return {a, a}; }
__host__ __device__ __forceinline__ f2 neg2(f2 a) { return {-a.x, -a.y}; }

#define LBM_PACKED_BINARY(NAME, OP, SCALAR)                                                                     \
   __host__ __device__ __forceinline__ f2 NAME(f2 a, f2 b)                                                      \
   {                                                                                                            \
      LBM_PACKED_BODY(OP, SCALAR)                                                                               \
   }
#ifdef __CUDA_ARCH__
#define LBM_PACKED_BODY(OP, SCALAR)                                                                             \
   f2 r;                                                                                                        \
   asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t" OP " d, a, b;\n\t"        \
       "mov.b64 {%0, %1}, d;\n\t}"                                                                              \
       : "=f"(r.x), "=f"(r.y)                                                                                   \
       : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                               \
   return r;
#else
#define LBM_PACKED_BODY(OP, SCALAR) return {SCALAR(a.x, b.x), SCALAR(a.y, b.y)};
#endif
LBM_PACKED_BINARY(add2, "add.rn.f32x2", fadd)
LBM_PACKED_BINARY(sub2, "sub.rn.f32x2", fsub)
LBM_PACKED_BINARY(mul2, "mul.rn.f32x2", fmul)
LBM_PACKED_BINARY(add2_rz, "add.rz.f32x2", fadd_rz)
#undef LBM_PACKED_BINARY
#undef LBM_PACKED_BODY

__host__ __device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
#ifdef __CUDA_ARCH__
   f2 r;
   asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
       "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
       : "=f"(r.x), "=f"(r.y)
       : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
   return r;
#else
   return {ffma(a.x, b.x, c.x), ffma(a.y, b.y, c.y)};
#endif
}

}  // namespace x64
}  // namespace lbm
