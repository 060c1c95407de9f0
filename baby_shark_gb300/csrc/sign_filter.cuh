// Arithmetic of the certified sign filters (sign_filter.cu on the reference's
// tree, fast_sign.cu on this library's): a winding number's far fields and
// solid angles in cheap arithmetic, with a bound on how far the sum can be
// from the float32 value of the traversal that it stands for.
//
// Error bound (everything times 4 pi; u = 2^-24).  A node's field is the
// dipole a . r / |r|^3 and the quadrupole 3 r^T S r / |r|^5 of the traceless
// symmetric part S of its order-2 matrix B (the reference's Frobenius product
// sees nothing else), r = p - q.  Both are derivatives of the harmonic
// 1 / |r|.  With x = rho / D (rho the group's radius, D the distance of its
// centre), the degree-n part of the expansion of 1 / |r| is a solid harmonic
// bounded by rho^n / D^(n+1); by Szego's form of Bernstein's inequality on
// great circles a first derivative of a harmonic of degree m and sup norm M
// on the unit sphere is at most m M, so the dipole's terms from degree 3 on
// sum to at most |a| / D^2 * 4 x^3 / (1 - x)^2 and the quadrupole's from
// degree 2 on to at most sqrt(3) |B| / D^3 * 12 x^2 / (1 - x)^3 (a second
// derivative, the nuclear norm of S).  Rounding, of the reference's formula
// (15 u of the dipole's and 150 u of the quadrupole's magnitude), of this
// one's (below 60 u) and of both sums (45 u for 40 levels of additions, the
// number of additions here), is bounded through the accumulated magnitudes
// mag = sum (|a| + 5 |B| / |r|) / |r|^2 (doubled and more for expanded nodes,
// whose voxels may be (1 - x) as far).  A solid angle's numerator and
// denominator, as fractions of |a||b||c|, differ by less than 256 u from the
// reference's, which moves the angle by at most 1.5 * 256 u / max(|num|,
// |den|); with the arctangent's 1e-5 that is below 1.4e-4 / max(..) for twice
// the angle.  Where that argument ends, near the branch cut (den < 0, |num|
// small) and at a vertex or edge, the callers take the exact formula or a wider
// bound.  A voxel is left undecided outside the range of distances where no
// float32 product of either formula over- or underflows, or where any value is
// NaN.
#pragma once

#include "bs_internal.cuh"

namespace bs {
namespace sign_filter {

constexpr unsigned FULLM = 0xffffffffu;
constexpr float FOURPI = 12.566370614359172f;
constexpr float X_MAX = 0.5f;        // group radius over distance below which a node may be expanded
constexpr float E_MAX = 0.045f;      // most truncation error (times 4 pi) of one expanded node in a group,
constexpr float E_BRICK = 0.03f;     // in a brick,
constexpr float E_FINE = 0.004f;     // and in the second attempt at a group
constexpr float R2_MIN = 0x1p-48f;   // squared distances outside [R2_MIN, R2_MAX] are left to the exact pass
constexpr float R2_MAX = 0x1p40f;

// ---------------------------------------------------------- arithmetic ----
// Taylor polynomial around a centre: c0 + L . d + Qxx (dx^2 - dz^2) + Qyy
// (dy^2 - dz^2) + Qxy dx dy + Qxz dx dz + Qyz dy dz; [9] truncation bound,
// [10] magnitude.
struct Taylor {
  float c[11];
};

__device__ __forceinline__ void taylor_clear(Taylor& t) {
#pragma unroll
  for (int k = 0; k < 11; ++k) t.c[k] = 0.0f;
}

__device__ __forceinline__ void taylor_add(Taylor& t, const Taylor& p) {
#pragma unroll
  for (int k = 0; k < 11; ++k) t.c[k] += p.c[k];
}

// Truncation bound of a node expanded at distance 1 / iD, x = rho iD < 1
// (12 sqrt(3) / 5 < 4.16).
__device__ __forceinline__ float taylor_error(float iD, float x, float na, float nb5) {
  const float om = __frcp_rn(1.0f - x), iD2 = iD * iD;
  const float x2 = x * x * om * om;
  return x2 * iD2 * (na * 4.0f * x + nb5 * 4.16f * iD * om);
}

// Polynomial of the node at s = p - centre, distance 1 / iD; err its truncation bound.
__device__ __forceinline__ Taylor taylor_of(float sx, float sy, float sz, float iD, float err, float4 A, float4 S,
                                            float na, float nb5) {
  Taylor t;
  const float iD2 = iD * iD, iD3 = iD2 * iD, iD4 = iD2 * iD2;
  const float nx = sx * iD, ny = sy * iD, nz = sz * iD;
  const float an = A.x * nx + A.y * ny + A.z * nz;
  const float X = A.w, Y = S.x, XY = S.y, XZ = S.z, YZ = S.w;
  const float gx = 2.0f * X * nx + XY * ny + XZ * nz;  // 6 S n
  const float gy = 2.0f * Y * ny + XY * nx + YZ * nz;
  const float gz = XZ * nx + YZ * ny - 2.0f * (X + Y) * nz;
  const float tn = 0.5f * (gx * nx + gy * ny + gz * nz);  // 3 n^T S n
  t.c[0] = an * iD2 - tn * iD3;
  const float m = 3.0f * an * iD3 - 5.0f * tn * iD4;
  t.c[1] = nx * m - A.x * iD3 + gx * iD4;
  t.c[2] = ny * m - A.y * iD3 + gy * iD4;
  t.c[3] = nz * m - A.z * iD3 + gz * iD4;
  const float k = 1.5f * iD4, k5 = 5.0f * an;
  t.c[4] = k * ((k5 * nx - 2.0f * A.x) * nx - an);
  t.c[5] = k * ((k5 * ny - 2.0f * A.y) * ny - an);
  t.c[6] = 2.0f * k * (k5 * nx * ny - (nx * A.y + ny * A.x));
  t.c[7] = 2.0f * k * (k5 * nx * nz - (nx * A.z + nz * A.x));
  t.c[8] = 2.0f * k * (k5 * ny * nz - (ny * A.z + nz * A.y));
  t.c[9] = err;
  t.c[10] = 8.0f * (na * iD2 + nb5 * iD3);
  return t;
}

__device__ __forceinline__ float taylor_at(const float* c, float dx, float dy, float dz) {
  const float zz = dz * dz;
  return c[0] + (c[1] * dx + c[2] * dy + c[3] * dz) + (c[4] * (dx * dx - zz) + c[5] * (dy * dy - zz)) +
         (c[6] * dx * dy + c[7] * dx * dz + c[8] * dy * dz);
}

struct Lane {  // one voxel's sums
  float w, mag, etri;
  bool bad;
};

// Far field of a node (order-1 vector and S in A, S) at r = p - q.
__device__ __forceinline__ void far_add(Lane& s, float4 A, float4 S, float na, float nb5, float rx, float ry, float rz,
                                        float r2) {
  const float i = rsqrtf(r2), i2 = i * i;
  const float ar = A.x * rx + A.y * ry + A.z * rz;
  const float zz = rz * rz;
  const float tr = A.w * (rx * rx - zz) + S.x * (ry * ry - zz) + rx * (S.y * ry + S.z * rz) + S.w * ry * rz;
  s.w += (ar - tr * i2) * (i2 * i);
  s.mag += i2 * (na + nb5 * i);
}

// Solid angle of a triangle at q: 2 atan2(num, den), Van Oosterom
// and Strackee's formula on the unnormalised corner vectors.  The arctangent
// on [0, 1] is Abramowitz and Stegun 4.4.47 (|error| <= 1e-5).  Where the
// bound above ends (fine false; NaN too), unsettled(an, P, 1 / max(an, |den|),
// min length^2, this value) gives the value and raises the bounds.
template <class Unsettled>
__device__ __forceinline__ void angle_add(Lane& s, float4 A, float4 B, float4 C, F3 q, Unsettled unsettled) {
  const float ax = A.x - q.x, ay = A.y - q.y, az = A.z - q.z;
  const float bx = B.x - q.x, by = B.y - q.y, bz = B.z - q.z;
  const float cx = C.x - q.x, cy = C.y - q.y, cz = C.z - q.z;
  const float la2 = ax * ax + ay * ay + az * az, lb2 = bx * bx + by * by + bz * bz, lc2 = cx * cx + cy * cy + cz * cz;
  const float la = la2 * rsqrtf(la2), lb = lb2 * rsqrtf(lb2), lc = lc2 * rsqrtf(lc2);
  const float num = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
  const float ab = ax * bx + ay * by + az * bz, ac = ax * cx + ay * cy + az * cz, bc = bx * cx + by * cy + bz * cz;
  const float P = la * lb * lc;
  const float den = P + ab * lc + ac * lb + bc * la;
  const float an = fabsf(num), ad = fabsf(den);
  const float mx = fmaxf(an, ad), mn = fminf(an, ad);
  const float im = __frcp_rn(mx);
  const float t = mn * im, t2 = t * t;
  float p = t * (0.9998660f + t2 * (-0.3302995f + t2 * (0.1801410f + t2 * (-0.0851330f + t2 * 0.0208351f))));
  p = an > ad ? 1.57079633f - p : p;
  p = den < 0.0f ? 3.14159265f - p : p;
  float w = copysignf(2.0f * p, num);
  // written so that NaN is not fine
  const float l2 = fminf(fminf(la2, lb2), lc2);
  const bool fine = l2 >= 0x1p-60f && mx >= 0.0078125f * P && (den >= 0.0f || an > 4e-5f * P);
  if (fine)
    s.etri += 1.4e-4f * (P * im);
  else
    w = unsettled(an, P, im, l2, w);
  s.w += w;
  s.mag += fabsf(w);
}

// How a node (dipole centre and far threshold H) stands to a group of voxels
// within rho of c.  The reference's test per voxel is r2 > tau with r2 the
// float32 squared distance, within 5 u of the true one; the margins here are
// 1e-5.
struct NodeTest {
  float sx, sy, sz, iD, err;
  bool all_far, all_near, poly;  // poly: its polynomial is good enough
};

__device__ __forceinline__ NodeTest test_node(float4 H, float na, float nb5, float cx, float cy, float cz, float rho,
                                              float e_max) {
  NodeTest n;
  n.sx = H.x - cx;
  n.sy = H.y - cy;
  n.sz = H.z - cz;
  const float D2 = n.sx * n.sx + n.sy * n.sy + n.sz * n.sz;
  n.iD = rsqrtf(D2);
  const float D = D2 * n.iD, x = rho * n.iD;
  const float lo = D * 0.99999f - rho, hi = D * 1.00001f + rho;
  n.all_far = lo > 0.0f && lo * lo * 0.99999f > fmaxf(H.w, R2_MIN) && H.w == H.w;
  n.all_near = hi * hi * 1.00001f <= H.w;  // also where D2 = 0: iD = inf, D = NaN, neither holds
  n.err = taylor_error(n.iD, x, na, nb5);
  n.poly = x <= X_MAX && n.err <= e_max && lo * lo >= R2_MIN;  // false for NaN
  return n;
}

}  // namespace sign_filter
}  // namespace bs
