// f32x2.cuh - pairs of floats on sm_100a's packed FP32 instructions, which
// round each half as the scalar operation does and take one issue slot for
// both.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace shb {

using f32x2 = uint64_t;

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 dup2(float a) { return pack2(a, a); }
__device__ __forceinline__ float2 unpack2(f32x2 r) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(r));
  return f;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// Both halves -0, in constant memory so that the assembler cannot know them.
static __constant__ f32x2 c_neg_zero2 = 0x8000000080000000ull;

// A product by the multiply-add instruction with -0 added, which rounds the
// same and keeps the sign of zero.  ptxas contracts a packed multiplication
// and a packed addition into one multiply-add although both say .rn and
// whatever -fmad says (measured), also through a literal -0.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { return fma2(a, b, c_neg_zero2); }

// a / b rounded to nearest in both halves, given nb = -b and y = 1 / b
// rounded to nearest (__frcp_rn), so that several numerators share one
// reciprocal.  The first correction makes the quotient faithful; the second
// makes it the correctly rounded one by Markstein's theorem (P. Markstein,
// Computation of elementary functions on the IBM RISC System/6000
// processor, 1990): with y = RN(1/b), q a faithful a/b and r = a - b q
// exact, RN(q + r y) = RN(a/b).  Operands must keep quotient and residual
// clear of overflow and underflow; a zero numerator gives a zero of either
// sign.
__device__ __forceinline__ f32x2 div2(f32x2 a, f32x2 nb, f32x2 y) {
  const f32x2 q0 = mul2(a, y);
  const f32x2 q1 = fma2(fma2(nb, q0, a), y, q0);
  return fma2(fma2(nb, q1, a), y, q1);
}

}  // namespace shb
