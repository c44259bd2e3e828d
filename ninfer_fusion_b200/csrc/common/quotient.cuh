// a / (1 + exp(-x)) for gates and activations.
#pragma once

namespace nfb {

// a / b for b >= 1.  Markstein's correction: the quotient by an approximate reciprocal, then its residual a - b q, which one fused
// operation yields exactly, times the reciprocal on top.  With a reciprocal good to 2^-23 the sum is within 2^-45 of a / b before its
// rounding, so it is the rounded quotient but where that lies closer to halfway between two floats.  Five instructions without a
// branch, where the general division tests exponents and calls a slow path.  An infinite a or b makes the residual a NaN: the first
// quotient (an infinity, a zero, or the NaN that it has to be) stands then.  b above 2^126 gives zero (a gate of x below -87.3 loses a value
// of some 1e-36).  The kernels for one or few tokens divide: there a unit may differ by the last bit before its rounding to bf16.
__device__ __forceinline__ float quotient(float a, float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r;
  const float c = fmaf(fmaf(-b, q, a), r, q);
  return c == c ? c : q;
}
__device__ __forceinline__ float gate_by(float a, float x) { return quotient(a, 1.f + __expf(-x)); }   // a sigmoid(x)

}  // namespace nfb
