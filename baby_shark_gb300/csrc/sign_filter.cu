// Signs of band voxels on the reference's tree, decided by a certified filter.
//
// A band voxel needs only the side of the threshold its winding number lies
// on (mesh_to_volume.rs:264-271).  The reference's value (fast_wn,
// aabb_tree.rs:662-691) is a sum over one cut of the tree per voxel: far
// fields of the nodes with |q - p| > beta r, exact solid angles of the
// triangles in the leaves that are near.  This pass evaluates the same cut —
// every far / near decision is the reference's own float32 comparison or
// provably equal to it — in cheaper arithmetic together with a bound E on how
// far its sum W can be from the reference's float32 value.  |W - threshold|
// > E settles the sign; the voxels it does not settle go to the exact
// traversal (ref_tree.cu), so signs equal the reference's bit for bit.
//
// What makes it cheap.  Nodes are tested 32 at a time, one per lane, against
// the bounding sphere of a whole group of voxels (first a brick's voxels,
// then each 32 of them in Morton order), not one by one for 32 voxels:
//   * far for every voxel and the group small against the distance (radius
//     below X_MAX of it): the node's field enters one Taylor polynomial
//     around the group's centre (lane by lane, summed over the warp once);
//   * near for every voxel: opened, or a leaf whose triangles every voxel sums;
//   * far for every voxel but close: its far field per voxel;
//   * the rest: the reference's test per voxel, descending with lane masks.
// The brick's polynomial and its undecided nodes (the frontier) are shared by
// its groups.
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
// the angle.  A voxel is left undecided where that argument ends: near the
// branch cut (den < 0, |num| small), at a vertex or edge, outside the range
// of distances where no float32 product of either formula over- or
// underflows, or where any value is NaN.
#include <algorithm>

#include "ref_tree.cuh"
#include "solid_angle.cuh"

namespace bs {
namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr float FOURPI = 12.566370614359172f;
constexpr float X_MAX = 0.5f;        // group radius over distance below which a node may be expanded
constexpr float E_MAX = 0.045f;      // most truncation error (times 4 pi) of one expanded node in a group,
constexpr float E_BRICK = 0.03f;     // in a brick,
constexpr float E_FINE = 0.004f;     // and in the second attempt at a group
constexpr float R2_MIN = 0x1p-48f;   // squared distances outside [R2_MIN, R2_MAX] are left to the exact pass
constexpr float R2_MAX = 0x1p40f;
constexpr int FRONT = 512;           // frontier nodes of a brick
constexpr int GSTACK = 256;          // pending (node, lanes) pairs of a group (a brick's own phase uses all warps' stacks)
constexpr int SLOT = 5;              // float4 per lane's broadcast slot: 4 and one that keeps the banks apart

__device__ __forceinline__ int mesh_index(const uint32_t* __restrict__ base, int K, uint64_t i) {
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (uint64_t(base[mid]) <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------ records -----
// Filter record of a node: 4 float4
//   [0] dipole centre, far threshold            [1] order-1 vector, 3 Sxx
//   [2] 3 Syy, 6 Sxy, 6 Sxz, 6 Syz              [3] |a|, 5 |B| (rounded up), left, right child
// (a leaf's: triangle count in place of the left child).  Internal node id at
// id, leaf p at nt + p.
__device__ __forceinline__ void filter_record(const float4* __restrict__ r, float4* __restrict__ o, int left,
                                              int right) {
  const float4 P = r[0], c1 = r[1], c2 = r[2], c3 = r[3];
  // column-major order-2 matrix: B[3 j + i]
  const float b0 = c1.w, b1 = c2.x, b2 = c2.y, b3 = c2.z, b4 = c2.w, b5 = c3.x, b6 = c3.y, b7 = c3.z, b8 = c3.w;
  const float tr = b0 + b4 + b8;
  const float na = sqrtf(c1.x * c1.x + c1.y * c1.y + c1.z * c1.z) * 1.00001f;
  const float bb = b0 * b0 + b1 * b1 + b2 * b2 + b3 * b3 + b4 * b4 + b5 * b5 + b6 * b6 + b7 * b7 + b8 * b8;
  const float nb = sqrtf(bb) * 1.00001f;
  o[0] = P;
  o[1] = make_float4(c1.x, c1.y, c1.z, 3.0f * b0 - tr);
  o[2] = make_float4(3.0f * b4 - tr, 3.0f * (b1 + b3), 3.0f * (b2 + b6), 3.0f * (b5 + b7));
  o[3] = make_float4(na, 5.0f * nb, __int_as_float(left), __int_as_float(right));
}

__global__ void k_rt_filter_records(uint64_t nt, const int* __restrict__ flags, const int2* __restrict__ topo,
                                    const uint32_t* __restrict__ leaf_cnt, const float4* __restrict__ rec_i,
                                    const float4* __restrict__ rec_l, float4* __restrict__ frec) {
  const uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (p >= nt) return;
  if (flags[p] == 2) {
    const int2 ch = topo[p];
    filter_record(rec_i + 4 * p, frec + 4 * p, ch.x, ch.y);
  }
  const uint32_t c = leaf_cnt[p];
  if (c) filter_record(rec_l + 4 * p, frec + 4 * (nt + p), int(c), 0);
}

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

// The reference's solid angle, out of line: few voxels need it.
__device__ __noinline__ float exact_angle(float4 A, float4 B, float4 C, F3 q) { return solid_angle(A, B, C, q); }

// Solid angle of a triangle at q: 2 atan2(num, den), Van Oosterom
// and Strackee's formula on the unnormalised corner vectors.  The arctangent
// on [0, 1] is Abramowitz and Stegun 4.4.47 (|error| <= 1e-5).
__device__ __forceinline__ void angle_add(Lane& s, float4 A, float4 B, float4 C, F3 q) {
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
  // written so that NaN takes the reference's own formula
  const bool fine = fminf(fminf(la2, lb2), lc2) >= 0x1p-60f && mx >= 0.0078125f * P && (den >= 0.0f || an > 4e-5f * P);
  if (fine)
    s.etri += 1.4e-4f * (P * im);
  else
    w = exact_angle(A, B, C, q);
  s.w += w;
  s.mag += fabsf(w);
}

struct WorkCounts {  // per lane, but visits per warp
  uint32_t visits = 0, far_sec = 0, exact_sec = 0, far = 0;
  unsigned long long exact = 0;
};

__device__ __forceinline__ int rec_index(int ref, int nt) { return ref >= 0 ? ref : nt + ~ref; }

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

template <int WARPS>
struct SignSmem {
  float4 slot[WARPS][32 * SLOT];
  int2 stack[WARPS][GSTACK];
  int front[FRONT];
  float taylor[11];
  uint32_t rho2;     // float bits, by atomicMax
  int n_front;
  int next_group;
  unsigned long long cnt[6];
};

// One CTA per brick: its first warp runs the brick's phase, then every warp
// takes the next 32 voxels.  Issue-bound (like the exact traversal): 62.6 ms
// with the exact traversal of every voxel, 15.1 ms here, on a torus of 1 M
// triangles and 35.6 M band voxels; 38.2 and 10.4 ms on a scan of 1.2 M
// triangles with holes and 19.2 M band voxels, 0.25 ms of it the exact pass
// over 0.02 % of the voxels (0.3 % and 2.8 ms without the second attempt).
// E_MAX between 0.03 and 0.06 changes it by 1 %; 0.1 spends the second
// attempt on 3 to 16 % of the voxels.
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_rt_sign(
    const uint32_t* __restrict__ act, const uint32_t* __restrict__ voff, const uint32_t* __restrict__ leaf_base, int K,
    const RefSignMesh* __restrict__ meshes, const int4* __restrict__ origins, float* __restrict__ values,
    const float4* __restrict__ frec, int nt, const float* __restrict__ rad_i, const float* __restrict__ rad_l,
    const float4* __restrict__ tri, const uint32_t* __restrict__ act_base, uint32_t* __restrict__ undecided,
    uint32_t* __restrict__ n_undecided, unsigned long long* __restrict__ counters) {
  __shared__ SignSmem<WARPS> sm;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t b = blockIdx.x;
  const int4 org = origins[b];
  const int mesh = K > 1 ? mesh_index(leaf_base, K, b) : 0;
  const RefSignMesh M = meshes[mesh];
  const uint32_t v0 = voff[b], nv = voff[b + 1] - v0;
  const float bcx = (float(org.x) + 3.5f) * M.h, bcy = (float(org.y) + 3.5f) * M.h, bcz = (float(org.z) + 3.5f) * M.h;
  auto point = [&](uint32_t o) {
    return f3(fmul(__int2float_rn(org.x + int(o >> 6)), M.h), fmul(__int2float_rn(org.y + int((o >> 3) & 7)), M.h),
              fmul(__int2float_rn(org.z + int(o & 7)), M.h));
  };
  if (threadIdx.x == 0) {
    sm.rho2 = 0;
    sm.n_front = 0;
    sm.next_group = 0;
  }
  if (threadIdx.x < 6) sm.cnt[threadIdx.x] = 0;
  __syncthreads();
  {
    float r2 = 0.0f;
    for (uint32_t i = threadIdx.x; i < nv; i += 32 * WARPS) {
      const F3 q = point(act[v0 + i] & 511u);
      const float dx = q.x - bcx, dy = q.y - bcy, dz = q.z - bcz;
      r2 = fmaxf(r2, dx * dx + dy * dy + dz * dz);
    }
    const uint32_t m = __reduce_max_sync(FULLM, __float_as_uint(r2));
    if (lane == 0) atomicMax(&sm.rho2, m);
  }
  __syncthreads();
  // Distances from any voxel to any vertex or dipole centre of the mesh stay
  // below R2_MAX when the root's sphere and this brick do.
  WorkCounts wc;
  float4 Hroot = frec[4 * uint64_t(rec_index(M.root, nt))];
  const float root_r = M.root >= 0 ? rad_i[M.root] : rad_l[~M.root];
  const float reach = root_r + (fabsf(Hroot.x - bcx) + fabsf(Hroot.y - bcy) + fabsf(Hroot.z - bcz)) + 16.0f * M.h;
  const bool in_range = reach * reach < R2_MAX;  // false for NaN

  // ---- brick phase: warp 0 ----
  if (w == 0) {
    const float rho = sqrtf(__uint_as_float(sm.rho2)) * 1.00001f;
    int* stk = &sm.stack[0][0].x;
    constexpr int CAP = 2 * WARPS * GSTACK;
    Taylor T;
    taylor_clear(T);
    int sp = 1, nf = 0;
    uint32_t n_far = 0;
    bool over = false;
    if (lane == 0) stk[0] = M.root;
    __syncwarp();
    while (sp > 0) {
      const int n = min(sp, 32);
      const bool have = lane < n;
      const int ref = have ? stk[sp - n + lane] : 0;
      sp -= n;
      __syncwarp();
      int left = 0, right = 0;
      bool expand = false, open = false;
      if (have) {
        const float4* R = frec + 4 * uint64_t(rec_index(ref, nt));
        const float4 H = __ldg(R), Mr = __ldg(R + 3);
        left = __float_as_int(Mr.z);
        right = __float_as_int(Mr.w);
        const NodeTest t = test_node(H, Mr.x, Mr.y, bcx, bcy, bcz, rho, E_BRICK);
        expand = t.all_far && t.poly;
        open = t.all_near && ref >= 0;
        if (expand) taylor_add(T, taylor_of(t.sx, t.sy, t.sz, t.iD, t.err, __ldg(R + 1), __ldg(R + 2), Mr.x, Mr.y));
      }
      const bool keep = have && !expand && !open;
      const unsigned m_t = __ballot_sync(FULLM, expand), m_o = __ballot_sync(FULLM, open);
      const unsigned m_f = __ballot_sync(FULLM, keep);
      wc.visits += n;
      n_far += __popc(m_t);
      if (nf + __popc(m_f) > FRONT || sp + 2 * __popc(m_o) > CAP) {
        over = true;
        break;
      }
      if (keep) sm.front[nf + __popc(m_f & lt)] = ref;
      nf += __popc(m_f);
      if (open) {
        const int at = sp + 2 * __popc(m_o & lt);
        stk[at] = left;
        stk[at + 1] = right;
      }
      sp += 2 * __popc(m_o);
      __syncwarp();
    }
    if (over) {  // no room: every group starts at the root
      taylor_clear(T);
      n_far = 0;
      nf = 1;
      if (lane == 0) sm.front[0] = M.root;
    }
#pragma unroll
    for (int k = 0; k < 11; ++k) {
      float v = T.c[k];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULLM, v, d);
      if (lane == 0) sm.taylor[k] = v;
    }
    if (lane == 0) {
      wc.far += n_far * nv;
      wc.far_sec += n_far;
      sm.n_front = nf;
    }
  }
  __syncthreads();

  // ---- group phase: 32 voxels per warp at a time ----
  const int n_front = sm.n_front;
  int2* stk = sm.stack[w];
  float4* slot = sm.slot[w];
  const float thr4 = M.thresh * FOURPI;
  for (;;) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(&sm.next_group, 1);
    g = __shfl_sync(FULLM, g, 0);
    if (32 * g >= nv) break;
    const bool ok = 32 * g + lane < nv;
    const uint32_t vox = act[v0 + (ok ? 32 * g + lane : nv - 1)];
    const uint32_t o = vox & 511u;
    const F3 q = point(o);
    unsigned lanes = __ballot_sync(FULLM, ok);
    // centre of the voxels' bounding box and the largest distance from it
    const int ix = int(o >> 6), iy = int((o >> 3) & 7), iz = int(o & 7);
    const float cx = (float(org.x) + 0.5f * float(__reduce_min_sync(FULLM, ix) + __reduce_max_sync(FULLM, ix))) * M.h;
    const float cy = (float(org.y) + 0.5f * float(__reduce_min_sync(FULLM, iy) + __reduce_max_sync(FULLM, iy))) * M.h;
    const float cz = (float(org.z) + 0.5f * float(__reduce_min_sync(FULLM, iz) + __reduce_max_sync(FULLM, iz))) * M.h;
    const float dx = q.x - cx, dy = q.y - cy, dz = q.z - cz;
    const float zz = dz * dz, d4 = dx * dx - zz, d5 = dy * dy - zz, d6 = dx * dy, d7 = dx * dz, d8 = dy * dz;
    const float rho =
        sqrtf(__uint_as_float(__reduce_max_sync(FULLM, __float_as_uint(dx * dx + dy * dy + zz)))) * 1.00001f;
    // the polynomial in lane src's slot at this lane's voxel
    auto poly_at = [&](const float4* P) {
      const float4 a = P[1], b2 = P[2];
      const float c8 = P[3].x;
      return a.x + (a.y * dx + a.z * dy + a.w * dz) + (b2.x * d4 + b2.y * d5) + (b2.z * d6 + b2.w * d7 + c8 * d8);
    };
    // first with the brick's polynomial and frontier; the voxels this does not
    // settle once more from the root with a finer bound
    for (int attempt = 0; attempt < 2; ++attempt) {
      const float e_max = attempt ? E_FINE : E_MAX;
      Taylor T;
      taylor_clear(T);
      Lane s;
      s.w = s.mag = s.etri = 0.0f;
      s.bad = !in_range;
      uint32_t n_add = 0;
      bool over = false;
      int sp = 0, pos = 0;
      if (attempt) {
        if (lane == 0) stk[0] = make_int2(M.root, int(lanes));
        __syncwarp();
        sp = 1;
        pos = n_front;
      }
      while (sp > 0 || pos < n_front) {
        const int n1 = min(sp, 32), n2 = min(32 - n1, n_front - pos), n = n1 + n2;
        const bool have = lane < n;
        int2 it = make_int2(0, 0);
        if (lane < n1) it = stk[sp - n1 + lane];
        else if (have) it = make_int2(sm.front[pos + lane - n1], int(lanes));
        sp -= n1;
        pos += n2;
        __syncwarp();
        const int ref = it.x;
        const unsigned who = unsigned(it.y);
        int left = 0, right = 0;
        unsigned far = 0;  // lanes that take this lane's node as far
        bool poly = false, direct = false, mixed = false;
        if (have) {
          const float4* R = frec + 4 * uint64_t(rec_index(ref, nt));
          const float4 H = __ldg(R), Mr = __ldg(R + 3);
          left = __float_as_int(Mr.z);
          right = __float_as_int(Mr.w);
          const NodeTest t = test_node(H, Mr.x, Mr.y, cx, cy, cz, rho, e_max);
          mixed = !t.all_far && !t.all_near;
          if (t.all_far) far = who;
          if (!t.all_near) {
            const float4 A = __ldg(R + 1), S = __ldg(R + 2);
            float4* P4 = slot + SLOT * lane;
            P4[0] = H;
            if (t.poly) {
              const Taylor P = taylor_of(t.sx, t.sy, t.sz, t.iD, t.err, A, S, Mr.x, Mr.y);
              if (t.all_far && who == lanes) {
                taylor_add(T, P);
              } else {
                T.c[9] += P.c[9];
                T.c[10] += P.c[10];
                P4[1] = make_float4(P.c[0], P.c[1], P.c[2], P.c[3]);
                P4[2] = make_float4(P.c[4], P.c[5], P.c[6], P.c[7]);
                P4[3] = make_float4(P.c[8], __int_as_float(int(who)), 0.0f, 0.0f);
                poly = true;
              }
            } else {
              P4[1] = A;
              P4[2] = S;
              P4[3] = make_float4(0.0f, __int_as_float(int(who)), Mr.x, Mr.y);
              direct = true;
            }
          }
        }
        __syncwarp();
        // far for the lanes of its mask, expanded
        for (unsigned m = __ballot_sync(FULLM, poly && !mixed); m; m &= m - 1u) {
          const float4* P = slot + SLOT * (__ffs(m) - 1);
          const float v = poly_at(P);
          ++n_add;
          if ((__float_as_uint(P[3].y) >> lane) & 1u) s.w += v;
        }
        // the reference's test per voxel, expanded
        for (unsigned m = __ballot_sync(FULLM, poly && mixed); m; m &= m - 1u) {
          const int src = __ffs(m) - 1;
          const float4* P = slot + SLOT * src;
          const float4 H = P[0];
          // the reference's r2, operation for operation (its q - p)
          const float ex = fsub(q.x, H.x), ey = fsub(q.y, H.y), ez = fsub(q.z, H.z);
          const float r2 = fadd(fadd(fmul(ex, ex), fmul(ey, ey)), fmul(ez, ez));
          const unsigned f = __ballot_sync(FULLM, r2 > H.w) & __float_as_uint(P[3].y);
          const float v = poly_at(P);
          ++n_add;
          if ((f >> lane) & 1u) s.w += v;
          if (lane == src) far = f;
        }
        // the same with the node's far field itself
        for (unsigned m = __ballot_sync(FULLM, direct); m; m &= m - 1u) {
          const int src = __ffs(m) - 1;
          const float4* P = slot + SLOT * src;
          const float4 H = P[0];
          const float ex = fsub(q.x, H.x), ey = fsub(q.y, H.y), ez = fsub(q.z, H.z);
          const float r2 = fadd(fadd(fmul(ex, ex), fmul(ey, ey)), fmul(ez, ez));
          const float4 M4 = P[3];
          const unsigned f = __ballot_sync(FULLM, r2 > H.w) & __float_as_uint(M4.y);
          ++n_add;
          if ((f >> lane) & 1u) {
            far_add(s, P[1], P[2], M4.z, M4.w, -ex, -ey, -ez, r2);
            s.bad |= !(r2 >= R2_MIN);
          }
          if (lane == src) far = f;
        }
        // the lanes that do not: triangles of a leaf, or the children
        const unsigned near = who & ~far;
        if (attempt == 0) {
          wc.visits += n;
          wc.far += __popc(far);
          wc.far_sec += far != 0;
          if (near && ref < 0) {
            wc.exact += uint64_t(__popc(near)) * uint32_t(left);
            wc.exact_sec += uint32_t(left);
          }
        }
        const bool open = near && ref >= 0;
        const unsigned m_o = __ballot_sync(FULLM, open);
        if (sp + 2 * __popc(m_o) > GSTACK) {
          over = true;
          break;
        }
        if (open) {
          const int at = sp + 2 * __popc(m_o & lt);
          stk[at] = make_int2(left, int(near));
          stk[at + 1] = make_int2(right, int(near));
        }
        sp += 2 * __popc(m_o);
        for (unsigned m = __ballot_sync(FULLM, near && ref < 0); m; m &= m - 1u) {
          const int src = __ffs(m) - 1;
          const uint32_t p = uint32_t(~__shfl_sync(FULLM, ref, src)), c = uint32_t(__shfl_sync(FULLM, left, src));
          const unsigned l = __shfl_sync(FULLM, near, src);
          n_add += c;
          const float4* tp = tri + 3 * uint64_t(p);
          if ((l >> lane) & 1u)
            for (uint32_t k = 0; k < c; ++k) angle_add(s, __ldg(tp + 3 * k), __ldg(tp + 3 * k + 1), __ldg(tp + 3 * k + 2), q);
        }
        __syncwarp();
      }
      // the group's polynomial, summed over the warp
  #pragma unroll
      for (int k = 0; k < 11; ++k) {
  #pragma unroll
        for (int d = 16; d > 0; d >>= 1) T.c[k] += __shfl_xor_sync(FULLM, T.c[k], d);
      }
      float W = s.w + taylor_at(T.c, dx, dy, dz), mag = s.mag + T.c[10], err = T.c[9];
      if (attempt == 0) {
        W += taylor_at(sm.taylor, q.x - bcx, q.y - bcy, q.z - bcz);
        err += sm.taylor[9];
        mag += sm.taylor[10];
      }
      const float E = 1.01f * err + 5.9604645e-8f * (float(n_add) + 400.0f) * mag + s.etri + 1e-3f;
      const float d = W - thr4;
      const bool outside = d < -E, inside = d > E;
      const bool mine = (lanes >> lane) & 1u;
      const bool settled = !s.bad && !over && (outside || inside);
      if (mine && settled) {
        const uint64_t at = uint64_t(b) * 512 + o;
        const float dist = values[at];
        values[at] = outside ? copysignf(dist, 1.0f) : copysignf(dist, -1.0f);
      }
      __syncwarp();
      lanes = __ballot_sync(FULLM, mine && !settled);
      if (!lanes) break;
    }
    if (lanes) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(n_undecided + mesh, uint32_t(__popc(lanes)));
      base = __shfl_sync(FULLM, base, 0);
      if ((lanes >> lane) & 1u) undecided[act_base[mesh] + base + __popc(lanes & lt)] = vox;
    }
    __syncwarp();
  }
  const uint32_t far_all = __reduce_add_sync(FULLM, wc.far), fs = __reduce_add_sync(FULLM, wc.far_sec),
                 es = __reduce_add_sync(FULLM, wc.exact_sec);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) wc.exact += __shfl_xor_sync(FULLM, wc.exact, d);
  if (lane == 0) {
    atomicAdd(&sm.cnt[0], (unsigned long long)wc.visits);
    atomicAdd(&sm.cnt[1], (unsigned long long)far_all);
    atomicAdd(&sm.cnt[2], wc.exact);
    atomicAdd(&sm.cnt[4], (unsigned long long)fs);
    atomicAdd(&sm.cnt[5], (unsigned long long)es);
  }
  __syncthreads();
  if (threadIdx.x < 6 && sm.cnt[threadIdx.x]) atomicAdd(counters + threadIdx.x, sm.cnt[threadIdx.x]);
}

// Work split of the exact pass: base[m] = first warp of mesh m, base[K + 1] =
// voxels per warp.  A warp walks the union of its voxels' cuts, and the few
// undecided voxels are scattered over the mesh, so as long as warps are free a
// warp takes fewer voxels (one, when n_warps suffice for all).
__global__ void k_undecided_warps(const uint32_t* __restrict__ n_undecided, int K, uint32_t n_warps,
                                  uint32_t* __restrict__ base) {
  const int lane = threadIdx.x;
  unsigned long long total = 0;
  for (int m = lane; m < K; m += 32) total += n_undecided[m];
  for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(FULLM, total, d);
  const uint32_t per = uint32_t(min((unsigned long long)32, max(1ull, (total + n_warps - 1) / n_warps)));
  if (lane) return;
  uint32_t at = 0;
  for (int m = 0; m < K; ++m) {
    base[m] = at;
    at += (n_undecided[m] + per - 1) / per;
  }
  base[K] = at;
  base[K + 1] = per;
}

}  // namespace

void ref_tree_sign(bs_ctx* ctx, const RefTrees& t, const uint32_t* act, const uint32_t* voff, uint64_t n_bricks,
                   uint64_t n_act, const uint32_t* d_act_base, const uint32_t* d_leaf_base, int K,
                   const RefSignMesh* d_meshes, const int4* origins, float* values, unsigned long long* d_counters) {
  if (n_act == 0) return;
  cudaStream_t s = ctx->stream;
  DBuf<uint32_t> und(ctx, n_act), n_und(ctx, K), warps(ctx, K + 2);
  DBuf<float4> frec(ctx, 8 * t.nt);
  BS_CUDA(cudaMemsetAsync(n_und.p, 0, K * sizeof(uint32_t), s));
  BS_KERNEL(ctx, "k_rt_filter_records", (k_rt_filter_records<<<unsigned((t.nt + 255) / 256), 256, 0, s>>>(
                                            t.nt, t.flags.p, t.topo.p, t.leaf_cnt.p, t.rec_i.p, t.rec_l.p, frec.p)));
#define BS_RT_SIGN(W)                                                                                                  \
  BS_KERNEL(ctx, "k_rt_sign", (k_rt_sign<W><<<unsigned(n_bricks), 32 * W, 0, s>>>(                                     \
                                  act, voff, d_leaf_base, K, d_meshes, origins, values, frec.p, int(t.nt), t.rad_i.p, \
                                  t.rad_l.p, t.tri.p, d_act_base, und.p, n_und.p, d_counters)))
  if (ctx->tune_wn_warps == 2)
    BS_RT_SIGN(2);
  else if (ctx->tune_wn_warps == 8)
    BS_RT_SIGN(8);
  else
    BS_RT_SIGN(4);
#undef BS_RT_SIGN
  const unsigned grid = ref_tree_sign_exact_grid(ctx, n_act);
  BS_KERNEL(ctx, "k_undecided_warps",
            (k_undecided_warps<<<1, 32, 0, s>>>(n_und.p, K, grid * REF_SIGN_WARPS, warps.p)));
  ref_tree_sign_exact(ctx, t, grid, und.p, d_act_base, n_und.p, warps.p, K, d_meshes, origins, values, d_counters);
}

}  // namespace bs
