// Correctly rounded quotients, reciprocals and roots without the range checks and branches of the IEEE operators: the hardware
// approximation with one Newton step, then the quotient's or root's residual, exact in an FMA, as its correction (P. W.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). They
// equal the operators for every normal operand whose result, reciprocal and residual are normal too; tested against the
// operators on all mantissas (reciprocals and roots) and on the quotients nearest to a tie. For a zero, infinite or NaN operand
// they give a value that is not finite where the operator's may be, so a caller tests its results with all_finite() and
// takes the operators (out of line: hardly ever called) where one is not. Divisors are below 2^126.
#pragma once
#include "common.cuh"

namespace hush {

HD_INL float rcp_rn(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(fmaf(-x, r, 1.0f), r, r);
}
HD_INL float quot_rn(float a, float d, float rcp_d) {
  const float q = __fmul_rn(a, rcp_d);
  return fmaf(-fmaf(d, q, -a), rcp_d, q);  // (the residual negated: a zero keeps its sign)
}
static __device__ __noinline__ float quot_any(float a, float d) { return __fdiv_rn(a, d); }
static __device__ __noinline__ float sqrt_any(float x) { return __fsqrt_rn(x); }

HD_INL bool all_finite(float sum) { return fabsf(sum) < INFINITY; }  // of the results' sum (false too if it overflows)

// c / d
HD_INL float3 div3(float3 c, float d) {
  const float r = rcp_rn(d);
  const float3 q = make_float3(quot_rn(c.x, d, r), quot_rn(c.y, d, r), quot_rn(c.z, d, r));
  if (all_finite(q.x + q.y + q.z)) return q;
  return make_float3(quot_any(c.x, d), quot_any(c.y, d), quot_any(c.z, d));
}
HD_INL float sqrt_rn(float x) {
  if (!(x > 1e-30f && x < 1e30f)) return sqrt_any(x);
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float s = __fmul_rn(x, r);
  return fmaf(fmaf(-s, s, x), 0.5f * r, s);
}

}  // namespace hush
