// Signs of band voxels on this library's tree, decided by a certified filter.
//
// The traversal (wn_traverse in m2v.cu) sums, for 32 consecutive active
// voxels together, one cut of the tree: the far field of every node that is
// far for all 32, the solid angles of the leaves that are not.  A band voxel
// needs only the side of the threshold its sum lies on
// (mesh_to_volume.rs:264-271).  This pass walks the same cut and evaluates it
// in cheaper arithmetic with a bound on how far the traversal's float32 sum
// can be (sign_filter.cuh).  The warps whose voxels' sides it cannot settle, or
// whose cut it has no room for, are listed and traversed (k_wn_sign_rest), as
// are those of a mesh out of its range or that it gives up, so the signs are the
// traversal's.
//
// What makes it cheap: nodes are tested 32 at a time, one per lane, against
// the bounding sphere and box of the voxels (of up to 256 consecutive ones
// first, then of each 32), and where these leave a node open its lane
// goes through the voxels; far nodes with a small enough truncation error
// enter one Taylor polynomial, lane by lane; only close far nodes and the near
// triangles are evaluated by every voxel.
#include "fast_sign.cuh"
#include "sign_filter.cuh"
#include "solid_angle.cuh"

namespace bs {
namespace {

using namespace sign_filter;

constexpr int FRONT = 448;   // nodes a warp's first phase leaves to its groups
constexpr int STACK = 256;   // pending nodes
constexpr float E_GROUP = 0.02f;  // truncation error of one expanded node in a group's first attempt
// A mesh of whose groups the filter has left more than one in TALLY_SHARE goes
// to the traversal from there on, but for one span in TALLY_SAMPLE.  The filter
// takes about 0.4 of the traversal's time, twice that with the second attempt,
// so it pays below a third: with 40 % left (a torus, threshold 0) 11.5 ms with it
// and 8.8 given up; below the line (20 k needles) 53.9 with it, 73.2 without.
constexpr uint32_t TALLY_FROM = 64, TALLY_SHARE = 3, TALLY_SAMPLE = 32;
constexpr int SLOT = 5;      // float4 per lane's broadcast slot: 4 and one that keeps the banks apart
// the float32 squared distances are within 4 u: outside of this the traversal's test is certain
constexpr float TAU_LO = 0.999999f, TAU_HI = 1.000001f;

__device__ __forceinline__ int segment(const uint32_t* __restrict__ base, int K, uint32_t i) {
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------ records -----
//   [0] dipole centre, far threshold            [1] order-1 vector, 3 Sxx
//   [2] 3 Syy, 6 Sxy, 6 Sxz, 6 Syz              [3] |a|, 5 |B| (rounded up), left, right child
// A leaf has the dipole alone.  Children >= 0 are internal nodes, ~leaf else,
// counted within the mesh.
__global__ void k_wn_filter_records(const float4* __restrict__ inode, uint64_t ni,
                                    const uint32_t* __restrict__ inode_base, const float4* __restrict__ leaf,
                                    uint64_t nt, const uint32_t* __restrict__ tri_base, int K,
                                    const FastSignMesh* __restrict__ meshes, float4* __restrict__ frec) {
  const uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  auto tau = [&](float r, const uint32_t* base) {
    const float b = meshes[K > 1 ? segment(base, K, uint32_t(p)) : 0].beta;
    return fmul(fmul(r, r), fmul(b, b));
  };
  if (p < ni) {
    const float4 P = inode[5 * p], A = inode[5 * p + 1], B0 = inode[5 * p + 2], B1 = inode[5 * p + 3],
                 B2 = inode[5 * p + 4];
    const float tr = B0.x + B1.x + B2.x;
    const float na = sqrtf(A.x * A.x + A.y * A.y + A.z * A.z) * 1.00001f;
    const float bb = B0.x * B0.x + B0.y * B0.y + B0.z * B0.z + B0.w * B0.w + B1.x * B1.x + B1.y * B1.y + B1.z * B1.z +
                     B1.w * B1.w + B2.x * B2.x;
    float4* o = frec + 4 * p;
    o[0] = make_float4(P.x, P.y, P.z, tau(P.w, inode_base));
    o[1] = make_float4(A.x, A.y, A.z, 3.0f * B0.x - tr);
    o[2] = make_float4(3.0f * B1.x - tr, 3.0f * (B0.y + B0.w), 3.0f * (B0.z + B1.z), 3.0f * (B1.y + B1.w));
    o[3] = make_float4(na, 5.0f * sqrtf(bb) * 1.00001f, B2.y, B2.z);
  }
  if (p < nt) {
    const float4 P = leaf[5 * p], A = leaf[5 * p + 1];
    float4* o = frec + 4 * (ni + p);
    o[0] = make_float4(P.x, P.y, P.z, tau(P.w, tri_base));
    o[1] = make_float4(A.x, A.y, A.z, 0.0f);
    o[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    o[3] = make_float4(sqrtf(A.x * A.x + A.y * A.y + A.z * A.z) * 1.00001f, 0.0f, 0.0f, 0.0f);
  }
}

// ---------------------------------------------------------------- pass ----
// The traversal's solid angle near a triangle's plane (tri_wn_exact is this
// over 4 pi), out of line: few voxels need it.
__device__ __noinline__ float exact_angle(float4 A, float4 B, float4 C, F3 q) { return solid_angle(A, B, C, q); }

struct FastSmem {  // of a warp
  float4 slot[32 * SLOT];
  float4 pos[32];  // a group's voxels
  int stack[STACK];
  int front[FRONT];
  float taylor[11];  // the span's polynomial
};

// Every warp takes a span of voxels by itself.  Issue-bound: about 12 k
// instructions per 32 voxels on a torus of 1 M triangles (35.7 M band voxels,
// 15.0 ms), of which the far fields per voxel take a quarter and the tests, the
// polynomials and the triangles (27) a fifth each.  On a scan of 1.2 M triangles
// with holes and 14.7 M band voxels: 13.8 ms with the traversal of every warp,
// 8.1 ms here, 0.37 ms of it the traversal of the warps left over.  80 registers
// without a spill: 36 spilled bytes took 10 % longer.  Blocks that share one first phase behind
// a barrier: 9.1 ms; spans of 64, 128, 512 voxels: +0.6, +0.1, +0.2 ms; 28 or
// 32 warps per SM with spills: +0.1, +0.2 ms; testing a node with a vote of
// all voxels instead of in a loop over them on its lane: +0.6 ms; E_GROUP
// 0.045: +0.3 ms (5 % of the groups take the second attempt).
constexpr int WARPS_PER_SM = 24, SPAN_WAVES = 4;

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS_PER_SM / WARPS) k_wn_filter(
    const uint32_t* __restrict__ act, const uint32_t* __restrict__ act_base, const uint32_t* __restrict__ span_base,
    uint32_t span_size, int K, const FastSignMesh* __restrict__ meshes, const int4* __restrict__ origins,
    float* __restrict__ values, const float4* __restrict__ frec0, uint64_t ni, const float4* __restrict__ inode, const float4* __restrict__ leaf0,
    uint32_t* __restrict__ rest, uint32_t n_warps, uint32_t* __restrict__ n_rest, uint8_t* __restrict__ done,
    unsigned long long* __restrict__ tally, unsigned long long* __restrict__ counts, uint32_t count_stride) {
  __shared__ FastSmem smem[WARPS];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t span = blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (span >= span_base[K]) return;  // whole warp
  FastSmem& sm = smem[threadIdx.x >> 5];
  const int mesh = K > 1 ? segment(span_base, K, span) : 0;
  const FastSignMesh M = meshes[mesh];
  const uint32_t i0 = act_base[mesh] + (span - span_base[mesh]) * span_size;
  const uint32_t nv = min(span_size, act_base[mesh + 1] - i0);
  const uint32_t n_groups = (nv + 31) / 32;
  // whether the filter has left too many of the mesh's groups to be worth its time
  auto wasted = [&] {
    const uint2 t = __ldcg(reinterpret_cast<const uint2*>(tally + mesh));  // groups tried, of them left
    return __any_sync(FULLM, t.x >= TALLY_FROM && TALLY_SHARE * t.y > t.x && span % TALLY_SAMPLE != 0) != 0;
  };
  {
    // Distances from any band voxel to any vertex or dipole centre of the mesh
    // stay below R2_MAX, past which the bound does not hold, when the root's
    // diameter and the band do.
    const float r = (M.n_tri > 1 ? inode[5 * uint64_t(M.inode_base)] : leaf0[5 * uint64_t(M.tri_base)]).w;
    const float reach = 2.0f * r + M.band;
    if (!(reach * reach < R2_MAX) || wasted()) return;  // NaN too
  }
  const float4* frec_i = frec0 + 4 * uint64_t(M.inode_base);
  const float4* frec_l = frec0 + 4 * (ni + M.tri_base);
  const float4* leaf = leaf0 + 5 * uint64_t(M.tri_base);
  const int root = M.n_tri > 1 ? 0 : ~0;
  auto record = [&](int ref) { return ref >= 0 ? frec_i + 4 * uint64_t(ref) : frec_l + 4 * uint64_t(~ref); };
  auto grid = [&](uint32_t v) {
    const int4 org = origins[v >> 9];
    return make_int3(org.x + int((v >> 6) & 7u), org.y + int((v >> 3) & 7u), org.z + int(v & 7u));
  };
  auto point = [&](int3 g) {
    return f3(fmul(__int2float_rn(g.x), M.h), fmul(__int2float_rn(g.y), M.h), fmul(__int2float_rn(g.z), M.h));
  };
  int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-0x7fffffff, -0x7fffffff, -0x7fffffff};
  for (uint32_t j = 0; j < nv; j += 32) {
    const int3 g = grid(act[i0 + min(j + lane, nv - 1)]);
    lo[0] = min(lo[0], g.x); lo[1] = min(lo[1], g.y); lo[2] = min(lo[2], g.z);
    hi[0] = max(hi[0], g.x); hi[1] = max(hi[1], g.y); hi[2] = max(hi[2], g.z);
  }
  auto middle = [&](int l, int u) {
    return 0.5f * (float(__reduce_min_sync(FULLM, l)) + float(__reduce_max_sync(FULLM, u))) * M.h;
  };
  const float bcx = middle(lo[0], hi[0]), bcy = middle(lo[1], hi[1]), bcz = middle(lo[2], hi[2]);
  float brho = 0.0f;
  for (uint32_t j = 0; j < nv; j += 32) {
    const F3 q = point(grid(act[i0 + min(j + lane, nv - 1)]));
    const float dx = q.x - bcx, dy = q.y - bcy, dz = q.z - bcz;
    brho = fmaxf(brho, dx * dx + dy * dy + dz * dz);
  }
  brho = sqrtf(__uint_as_float(__reduce_max_sync(FULLM, __float_as_uint(brho)))) * 1.00001f;
  // Work of the groups whose cut was walked to its end.  Every visit opens a
  // node, takes its far field or its solid angle, and opening gives two more:
  // (visits + 1) / 2 of a cut are not openings.
  uint32_t c_visit = 0, c_cuts = 0, c_exact = 0;

  // ---- first phase, all voxels of the span ----
  int* stk = sm.stack;
  int n_front = 0;
  uint32_t n_shared = 0;  // visits of every group's cut in this phase
  {
    Taylor TB;
    taylor_clear(TB);
    int sp = 1;
    bool over = false;
    if (lane == 0) stk[0] = root;
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
        const float4* R = record(ref);
        const float4 H = __ldg(R), Mr = __ldg(R + 3);
        left = __float_as_int(Mr.z);
        right = __float_as_int(Mr.w);
        const NodeTest t = test_node(H, Mr.x, Mr.y, bcx, bcy, bcz, brho, E_BRICK);
        expand = t.all_far && t.poly;
        open = t.all_near && ref >= 0;
        if (expand) taylor_add(TB, taylor_of(t.sx, t.sy, t.sz, t.iD, t.err, __ldg(R + 1), __ldg(R + 2), Mr.x, Mr.y));
      }
      const bool keep = have && !expand && !open;
      const unsigned m_o = __ballot_sync(FULLM, open), m_f = __ballot_sync(FULLM, keep);
      n_shared += __popc(__ballot_sync(FULLM, expand || open));
      if (n_front + __popc(m_f) > FRONT || sp + 2 * __popc(m_o) > STACK) {
        over = true;
        break;
      }
      if (keep) sm.front[n_front + __popc(m_f & lt)] = ref;
      n_front += __popc(m_f);
      if (open) {
        const int at = sp + 2 * __popc(m_o & lt);
        stk[at] = left;
        stk[at + 1] = right;
      }
      sp += 2 * __popc(m_o);
      __syncwarp();
    }
    if (over) {  // no room: every group starts at the root
      taylor_clear(TB);
      n_shared = 0;
      n_front = 1;
      if (lane == 0) sm.front[0] = root;
    }
#pragma unroll
    for (int k = 0; k < 11; ++k) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) TB.c[k] += __shfl_xor_sync(FULLM, TB.c[k], d);
      if (lane == 0) sm.taylor[k] = TB.c[k];
    }
    __syncwarp();
  }

  // ---- groups: the traversal's 32 voxels ----
  float4* slot = sm.slot;
  const float thr4 = M.thresh * FOURPI;
  uint32_t g = 0;
  for (; g < n_groups; ++g) {
    if (g && wasted()) break;
    const bool ok = 32 * g + lane < nv;
    const uint32_t vox = act[i0 + (ok ? 32 * g + lane : nv - 1)];
    const int3 gr = grid(vox);
    const F3 q = point(gr);
    const F3 blo = point(make_int3(__reduce_min_sync(FULLM, gr.x), __reduce_min_sync(FULLM, gr.y), __reduce_min_sync(FULLM, gr.z)));
    const F3 bhi = point(make_int3(__reduce_max_sync(FULLM, gr.x), __reduce_max_sync(FULLM, gr.y), __reduce_max_sync(FULLM, gr.z)));
    sm.pos[lane] = make_float4(q.x, q.y, q.z, 0.0f);
    __syncwarp();
    const float cx = 0.5f * (blo.x + bhi.x), cy = 0.5f * (blo.y + bhi.y), cz = 0.5f * (blo.z + bhi.z);
    const float dx = q.x - cx, dy = q.y - cy, dz = q.z - cz;
    const float rho =
        sqrtf(__uint_as_float(__reduce_max_sync(FULLM, __float_as_uint(dx * dx + dy * dy + dz * dz)))) * 1.00001f;
    unsigned open_lanes = __ballot_sync(FULLM, ok);  // voxels without a sign yet
    bool counted = false;
    // first with the span's polynomial and frontier; the voxels this does not
    // settle once more from the root with a finer bound
    for (int attempt = 0; attempt < 2; ++attempt) {
      const float e_max = attempt ? E_FINE : E_GROUP;
      Taylor T;
      taylor_clear(T);
      Lane s;
      s.w = s.mag = s.etri = 0.0f;
      s.bad = false;
      uint32_t n_add = 0, n_visit = 0, n_exact = 0;
      bool lost = false;  // no room for the cut
      int sp = 0, pos = 0;
      if (attempt) {
        if (lane == 0) stk[0] = root;
        __syncwarp();
        sp = 1;
        pos = n_front;
      }
      while (sp > 0 || pos < n_front) {
        const int n1 = min(sp, 32), n2 = min(32 - n1, n_front - pos), n = n1 + n2;
        const bool have = lane < n;
        int ref = 0;
        if (lane < n1) ref = stk[sp - n1 + lane];
        else if (have) ref = sm.front[pos + lane - n1];
        sp -= n1;
        pos += n2;
        __syncwarp();
        int left = 0, right = 0;
        float tau_lo = 0.0f, tau_hi = 0.0f;
        bool mixed = false;
        NodeTest t;
        t.all_far = t.all_near = t.poly = false;
        float4 H = make_float4(0.f, 0.f, 0.f, 0.f), Mr = H;
        const float4* R = nullptr;
        bool far = false;
        if (have) {
          R = record(ref);
          H = __ldg(R);
          Mr = __ldg(R + 3);
          left = __float_as_int(Mr.z);
          right = __float_as_int(Mr.w);
          t = test_node(H, Mr.x, Mr.y, cx, cy, cz, rho, e_max);
          // where the sphere leaves it open: far if it is from the voxels' box
          const float bx = fmaxf(fmaxf(blo.x - H.x, H.x - bhi.x), 0.0f), by = fmaxf(fmaxf(blo.y - H.y, H.y - bhi.y), 0.0f),
                      bz = fmaxf(fmaxf(blo.z - H.z, H.z - bhi.z), 0.0f);
          // below R2_MIN float32 squares lose their relative bound: never surely near there
          tau_lo = H.w < R2_MIN ? -1.0f : H.w * TAU_LO;
          tau_hi = fmaxf(H.w * TAU_HI, R2_MIN) + 0.0f * (H.x + H.y + H.z + H.w);  // NaN if any is
          far = t.all_far || bx * bx + by * by + bz * bz >= tau_hi * TAU_HI;
          mixed = !far && !t.all_near;
        }
        // the traversal's test of every voxel, on this lane's node
        float r2min = INFINITY;
        for (int j = 0; j < 8; ++j) {
          if (!__any_sync(FULLM, mixed && !(r2min <= tau_lo))) break;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 v = sm.pos[j + 8 * k];
            const float ex = H.x - v.x, ey = H.y - v.y, ez = H.z - v.z;
            r2min = fminf(r2min, ex * ex + ey * ey + ez * ez);
          }
        }
        bool near = r2min <= tau_lo;
        // too close to call, or a NaN: the traversal's own comparison
        for (unsigned m = __ballot_sync(FULLM, mixed && !near && !(r2min >= tau_hi)); m; m &= m - 1u) {
          const int src = __ffs(m) - 1;
          const float hx = __shfl_sync(FULLM, H.x, src), hy = __shfl_sync(FULLM, H.y, src),
                      hz = __shfl_sync(FULLM, H.z, src), hw = __shfl_sync(FULLM, H.w, src);
          const bool opens = !__all_sync(FULLM, cut_dist2(hx - q.x, hy - q.y, hz - q.z) > hw);
          if (lane == src) near = opens;
        }
        if (mixed) far = !near;
        const bool direct = far && !t.poly;
        if (far) {
          const float4 A = __ldg(R + 1), S = __ldg(R + 2);
          if (t.poly) {
            taylor_add(T, taylor_of(t.sx, t.sy, t.sz, t.iD, t.err, A, S, Mr.x, Mr.y));
          } else {
            float4* P4 = slot + SLOT * lane;
            P4[0] = H;
            P4[1] = A;
            P4[2] = S;
            P4[3] = Mr;
          }
        }
        __syncwarp();
        for (unsigned m = __ballot_sync(FULLM, direct); m; m &= m - 1u) {
          const float4* P = slot + SLOT * (__ffs(m) - 1);
          const float4 H4 = P[0], M4 = P[3];
          const float rx = H4.x - q.x, ry = H4.y - q.y, rz = H4.z - q.z;
          const float r2 = rx * rx + ry * ry + rz * rz;
          ++n_add;
          far_add(s, P[1], P[2], M4.x, M4.y, rx, ry, rz, r2);
          s.bad |= !(r2 >= R2_MIN);
        }
        const bool tri = have && !far && ref < 0, open = have && !far && ref >= 0;
        const unsigned m_o = __ballot_sync(FULLM, open);
        n_visit += n;
        if (sp + 2 * __popc(m_o) > STACK) {
          lost = true;
          break;
        }
        if (open) {
          const int at = sp + 2 * __popc(m_o & lt);
          stk[at] = left;
          stk[at + 1] = right;
        }
        sp += 2 * __popc(m_o);
        unsigned m = __ballot_sync(FULLM, tri);
        n_exact += __popc(m);
        for (; m; m &= m - 1u) {
          const float4* L = leaf + 5 * uint64_t(~__shfl_sync(FULLM, ref, __ffs(m) - 1)) + 2;
          const float4 A = __ldg(L), B = __ldg(L + 1), C = __ldg(L + 2);
          ++n_add;
          // the traversal's own formula where it takes the unfused one for
          // certain: below its minimal length, or |num| < 1e-4 (256 u and
          // more below that).  Else, near an edge or vertex, num and den are
          // off by 256 u each and 0.8e-4 or more from 0 together, which moves
          // twice the angle by at most 2 asin(sqrt(2) 256 u / max(..)) and the
          // arctangents' errors: below 5e-5 / max(..).
          angle_add(s, A, B, C, q, [&](float an, float P, float im, float l2, float w) {
            if (l2 < 0x1p-100f || (l2 >= 0x1p-60f && an < 0.8e-4f * P)) return exact_angle(A, B, C, q);
            s.bad |= !(l2 >= 0x1p-60f);
            s.etri += 5e-5f * (P * im);
            return w;
          });
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
      if (attempt == 0 && !lost) {
        c_visit += n_visit + n_shared;
        ++c_cuts;
        c_exact += n_exact;
        counted = true;
      }
      if (attempt == 0) {
        W += taylor_at(sm.taylor, q.x - bcx, q.y - bcy, q.z - bcz);
        err += sm.taylor[9];
        mag += sm.taylor[10];
      }
      const float E = 1.01f * err + 5.9604645e-8f * (float(n_add) + 400.0f) * mag + s.etri + 1e-3f;
      const float d = W - thr4;
      const bool outside = d < -E, inside = d > E;
      const bool mine = (open_lanes >> lane) & 1u;
      const bool settled = !s.bad && !lost && (outside || inside);
      if (mine && settled) {
        const uint64_t at = uint64_t(vox >> 9) * 512 + (vox & 511u);
        const float dist = values[at];
        values[at] = outside ? copysignf(dist, 1.0f) : copysignf(dist, -1.0f);
      }
      __syncwarp();
      open_lanes = __ballot_sync(FULLM, mine && !settled);
      if (!open_lanes || lost) break;
    }
    if (lane == 0) {
      atomicAdd(tally + mesh, open_lanes ? (1ull << 32) + 1ull : 1ull);
      if (open_lanes) rest[counted ? atomicAdd(n_rest, 1u) : n_warps - 1u - atomicAdd(n_rest + 1, 1u)] = i0 + 32 * g;
    }
    __syncwarp();
  }
  if (lane == 0) {
    done[span] = uint8_t(g);
    atomicAdd(n_rest + 2, g);
    unsigned long long* c = counts + uint64_t(mesh) * count_stride;
    atomicAdd(c, (unsigned long long)c_visit);
    atomicAdd(c + 1, (unsigned long long)((c_visit + c_cuts) / 2 - c_exact));
    atomicAdd(c + 2, (unsigned long long)c_exact);
  }
}

}  // namespace

void fast_filter_records(bs_ctx* ctx, const float4* inode, uint64_t n_internal, const uint32_t* d_inode_base,
                         const float4* leaf, uint64_t nt, const uint32_t* d_tri_base, int K,
                         const FastSignMesh* d_meshes, float4* frec) {
  BS_KERNEL(ctx, "k_wn_filter_records",
            (k_wn_filter_records<<<unsigned((nt + 255) / 256), 256, 0, ctx->stream>>>(
                inode, n_internal, d_inode_base, leaf, nt, d_tri_base, K, d_meshes, frec)));
}

// Consecutive active voxels of a mesh that one warp takes, for n_act of them in
// all: 32, 64, 128 or 256.  The longer a span, the more its groups share; but
// a warp takes its groups one after another, so the spans must fill the SMs
// several times over (1, 2, 4, 8 times: 1.34, 1.21, 1.19, 1.23 ms for 1 M voxels;
// 1,944 voxels of an icosphere: 0.51 ms in spans of 256, 0.12 of 32).
uint32_t fast_sign_span(bs_ctx* ctx, uint64_t n_act) {
  int n_sm = 0;
  BS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, ctx->device));
  uint32_t span = 256;
  while (span > 32 && n_act < uint64_t(span) * SPAN_WAVES * WARPS_PER_SM * unsigned(n_sm)) span /= 2;
  return span;
}

void fast_sign(bs_ctx* ctx, const uint32_t* act, const uint32_t* d_act_base, const uint32_t* d_span_base,
               uint32_t span, uint32_t n_spans, int K, const FastSignMesh* d_meshes, const int4* origins, float* values,
               const float4* frec, uint64_t n_internal, const float4* inode, const float4* leaf, uint32_t* rest,
               uint32_t n_warps, uint32_t* n_rest, uint8_t* done, unsigned long long* d_tally,
               unsigned long long* d_counts, uint32_t count_stride) {
  if (n_spans == 0) return;
#define BS_WN_FILTER(W)                                                                                            \
  BS_KERNEL(ctx, "k_wn_filter", (k_wn_filter<W><<<(n_spans + W - 1) / W, 32 * W, 0, ctx->stream>>>(                                \
                                  act, d_act_base, d_span_base, span, K, d_meshes, origins, values, frec, n_internal,    \
                                  inode, leaf, rest, n_warps, n_rest, done, d_tally, \
                                  d_counts, count_stride)))
  if (ctx->tune_wn_warps == 2)
    BS_WN_FILTER(2);
  else if (ctx->tune_wn_warps == 8)
    BS_WN_FILTER(8);
  else
    BS_WN_FILTER(4);
#undef BS_WN_FILTER
}

}  // namespace bs
