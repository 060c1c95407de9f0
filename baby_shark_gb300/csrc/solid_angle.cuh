// The reference's solid angle of a triangle, float32 operation for operation.
#pragma once

#include "bs_internal.cuh"

namespace bs {

// v / len for the three components of v, correctly rounded, with one
// reciprocal (mdiv) where the operands allow it.
__device__ __forceinline__ F3 div3(F3 v, float len) {
  if (mdiv_range(len) && (v.x == 0.0f || mdiv_range(v.x)) && (v.y == 0.0f || mdiv_range(v.y)) &&
      (v.z == 0.0f || mdiv_range(v.z))) {
    const float y = __frcp_rn(len);
    // a zero component keeps its sign (0 / len = 0 * (1 / len))
    return f3(v.x == 0.0f ? fmul(v.x, y) : mdiv(v.x, len, y), v.y == 0.0f ? fmul(v.y, y) : mdiv(v.y, len, y),
              v.z == 0.0f ? fmul(v.z, y) : mdiv(v.z, len, y));
  }
  return f3(fdiv(v.x, len), fdiv(v.y, len), fdiv(v.z, len));
}

// solid_angle (aabb_tree.rs:582-615): Van Oosterom–Strackee, unfused.
__device__ __forceinline__ float solid_angle(float4 A, float4 Bv, float4 C, F3 q) {
  F3 qa = sub3(f3(A.x, A.y, A.z), q), qb = sub3(f3(Bv.x, Bv.y, Bv.z), q), qc = sub3(f3(C.x, C.y, C.z), q);
  const float la = fsqrt(dot3(qa, qa)), lb = fsqrt(dot3(qb, qb)), lc = fsqrt(dot3(qc, qc));
  if (la == 0.f || lb == 0.f || lc == 0.f) return 0.f;
  qa = div3(qa, la);
  qb = div3(qb, lb);
  qc = div3(qc, lc);
  const float num = dot3(qa, cross3(sub3(qb, qa), sub3(qc, qa)));
  if (num == 0.f) return 0.f;
  const float den = fadd(fadd(fadd(1.0f, dot3(qa, qb)), dot3(qa, qc)), dot3(qb, qc));
  return fmul(atan2f(num, den), 2.0f);
}

}  // namespace bs
