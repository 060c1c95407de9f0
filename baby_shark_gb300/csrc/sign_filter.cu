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
// The error bound is in sign_filter.cuh.
#include <algorithm>

#include "ref_tree.cuh"
#include "sign_filter.cuh"
#include "solid_angle.cuh"

namespace bs {
namespace {

using namespace sign_filter;

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

// ---------------------------------------------------------------- pass ----
// The reference's solid angle, out of line: few voxels need it.
__device__ __noinline__ float exact_angle(float4 A, float4 B, float4 C, F3 q) { return solid_angle(A, B, C, q); }

struct WorkCounts {  // per lane, but visits per warp
  uint32_t visits = 0, far_sec = 0, exact_sec = 0, far = 0;
  unsigned long long exact = 0;
};

__device__ __forceinline__ int rec_index(int ref, int nt) { return ref >= 0 ? ref : nt + ~ref; }

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

// All of a brick's voxels to the traversal, in warps of their own: `end` is where its mesh's room ends.
__device__ __noinline__ void hand_over(const uint32_t* __restrict__ act, uint32_t nv, uint64_t end, uint32_t* n_uncounted,
                                       uint32_t* __restrict__ undecided, uint32_t* at) {
  const uint32_t n = (nv + 31u) & ~31u;
  if (threadIdx.x == 0) *at = atomicAdd(n_uncounted, n);
  __syncthreads();
  end -= *at + uint64_t(n);
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) undecided[end + i] = i < nv ? act[i] : NO_VOXEL;
}

// One CTA per brick: its first warp runs the brick's phase, then every warp
// takes the next 32 voxels.  Issue-bound (like the exact traversal): 62.6 ms
// with the exact traversal of every voxel, 15.2 ms here, on a torus of 1 M
// triangles and 35.6 M band voxels; 38.2 and 10.4 ms on a scan of 1.2 M
// triangles with holes and 19.2 M band voxels, 0.25 ms of it the exact pass
// over 0.02 % of the voxels (0.3 % and 2.8 ms without the second attempt).
// E_MAX between 0.03 and 0.06 changes it by 1 %; 0.1 spends the second
// attempt on 3 to 16 % of the voxels.  80 registers and a few spilled bytes, as
// the compiler chooses; held to other numbers it took 1 to 7 % longer.
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
  // below R2_MAX (past which the bound does not hold) when the root's sphere and this brick do.
  WorkCounts wc;
  float4 Hroot = frec[4 * uint64_t(rec_index(M.root, nt))];
  const float root_r = M.root >= 0 ? rad_i[M.root] : rad_l[~M.root];
  const float reach = root_r + (fabsf(Hroot.x - bcx) + fabsf(Hroot.y - bcy) + fabsf(Hroot.z - bcz)) + 16.0f * M.h;
  if (!(reach * reach < R2_MAX)) {  // NaN too
    hand_over(act + v0, nv, uint64_t(act_base[mesh + 1]) + 32 * uint64_t(leaf_base[mesh + 1]),
              n_undecided + 2 * mesh + 1, undecided, &sm.rho2);
    return;
  }

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
      s.bad = false;
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
        // fewer where the stack fills: with RT_MAX_DEPTH left it goes one node
        // at a time, deepest first, and needs one more entry per level
        const int most = min(32, max(1, GSTACK - RT_MAX_DEPTH - sp));
        const int n1 = min(sp, most), n2 = min(most - n1, n_front - pos), n = n1 + n2;
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
        if (sp + 2 * __popc(m_o) > GSTACK) {  // only in a tree deeper than RT_MAX_DEPTH
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
            for (uint32_t k = 0; k < c; ++k) {
              const float4 A = __ldg(tp + 3 * k), B = __ldg(tp + 3 * k + 1), C = __ldg(tp + 3 * k + 2);
              angle_add(s, A, B, C, q, [&](float, float, float, float, float) { return exact_angle(A, B, C, q); });
            }
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
      if (lane == 0) base = atomicAdd(n_undecided + 2 * mesh, uint32_t(__popc(lanes)));
      base = __shfl_sync(FULLM, base, 0);
      if ((lanes >> lane) & 1u)
        undecided[uint64_t(act_base[mesh]) + 32 * uint64_t(leaf_base[mesh]) + base + __popc(lanes & lt)] = vox;
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

// Work split of the exact pass over n lists: base[l] = first warp of list l,
// base[n + 1] = voxels per warp, base[n + 2] = 0.  A warp walks the union of its
// voxels' cuts, and the few undecided voxels are scattered over the mesh, so as
// long as warps are free a warp takes fewer voxels (one, when n_warps suffice
// for all).  A power of two, which keeps 32 voxels that were listed together
// together.
__global__ void k_undecided_warps(const uint32_t* __restrict__ n_undecided, int n, uint32_t n_warps,
                                  uint32_t* __restrict__ base) {
  const int lane = threadIdx.x;
  unsigned long long total = 0;
  for (int l = lane; l < n; l += 32) total += n_undecided[l];
  for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(FULLM, total, d);
  uint32_t per = 1;
  while (per < 32 && uint64_t(per) * n_warps < total) per *= 2;
  uint32_t at = 0;
  for (int l0 = 0; l0 < n; l0 += 32) {
    const uint32_t mine = l0 + lane < n ? (n_undecided[l0 + lane] + per - 1) / per : 0u;
    uint32_t end = mine;
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(FULLM, end, d);
      if (lane >= d) end += v;
    }
    if (l0 + lane < n) base[l0 + lane] = at + end - mine;
    at += __shfl_sync(FULLM, end, 31);
  }
  if (lane == 0) {
    base[n] = at;
    base[n + 1] = per;
    base[n + 2] = 0;
  }
}

}  // namespace

void ref_tree_sign(bs_ctx* ctx, const RefTrees& t, const uint32_t* act, const uint32_t* voff, uint64_t n_bricks,
                   uint64_t n_act, const uint32_t* d_act_base, const uint32_t* d_leaf_base, int K,
                   const RefSignMesh* d_meshes, const int4* origins, float* values, unsigned long long* d_counters) {
  if (n_act == 0) return;
  cudaStream_t s = ctx->stream;
  DBuf<uint32_t> und(ctx, n_act + 32 * n_bricks), n_und(ctx, 2 * K), warps(ctx, 2 * K + 3);
  DBuf<float4> frec(ctx, 8 * t.nt);
  BS_CUDA(cudaMemsetAsync(n_und.p, 0, 2 * K * sizeof(uint32_t), s));
  BS_KERNEL(ctx, "k_rt_filter_records", (k_rt_filter_records<<<unsigned((t.nt + 255) / 256), 256, 0, s>>>(
                                            t.nt, t.flags.p, t.topo.p, t.leaf_cnt.p, t.rec_i.p, t.rec_l.p, frec.p)));
#define BS_RT_SIGN(W)                                                                                                  \
  BS_KERNEL(ctx, "k_rt_sign", (k_rt_sign<W><<<unsigned(n_bricks), 32 * W, 0, s>>>(                                     \
                                  act, voff, d_leaf_base, K, d_meshes, origins, values, frec.p, int(t.nt), t.rad_i.p, \
                                  t.rad_l.p, t.tri.p, d_act_base, und.p, n_und.p, d_counters)))
  int n_sm = 0;
  BS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, ctx->device));
  // A brick's warps take its groups in turn, and the busiest brick's turns set
  // the time, so where the bricks are few they get more warps, up to one per
  // group, while there are 64 warps or fewer to an SM.  With 4 / 8 / 16 warps:
  // 124 bricks of a torus (accuracy scale 8) 8.7 / 5.0 / 3.5 ms; 543 of random
  // triangles 9.7 / 5.8 / 3.6; 512 of small boxes 1.65 / 1.05 / -; 545 of a torus
  // 0.415 / 0.346 / 0.395; 960 of a torus 0.409 / 0.426 / -; 1,451 (past the
  // line) 0.436 / 0.524 / -.  (24 warps fit an SM at a time; a line there: a
  // batch of eight meshes, two of them crowded, 648 bricks, 2.32 against 1.31 ms.)
  int warps_of = ctx->tune_wn_warps;
  while (warps_of < 16 && n_bricks * 2 * warps_of <= uint64_t(n_sm) * 64) warps_of *= 2;
  if (warps_of == 2)
    BS_RT_SIGN(2);
  else if (warps_of == 8)
    BS_RT_SIGN(8);
  else if (warps_of == 16)
    BS_RT_SIGN(16);
  else
    BS_RT_SIGN(4);
#undef BS_RT_SIGN
  const unsigned grid = ref_tree_sign_exact_grid(ctx, n_act);
  const uint32_t enough = std::min(grid * REF_SIGN_WARPS, unsigned(n_sm) * 32);
  BS_KERNEL(ctx, "k_undecided_warps",
            (k_undecided_warps<<<1, 32, 0, s>>>(n_und.p, 2 * K, enough, warps.p)));
  ref_tree_sign_exact(ctx, t, grid, und.p, d_act_base, d_leaf_base, n_und.p, warps.p, K, d_meshes, origins, values,
                      d_counters);
}

}  // namespace bs
