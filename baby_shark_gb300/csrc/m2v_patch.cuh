// Distance pass over patches of sub-triangles, for triangles that are cut into
// many sub-triangles under a wide band (m2v.cu picks it): a triangle's
// sub-triangles are congruent cells of a flat grid, so one test against a
// patch's outline stands for up to nine of theirs.  Included by m2v.cu.
#pragma once

#include "bs_internal.cuh"

namespace bs {

// Patch record, 144 B.  (rho, kappa, C) are signed distances within the plane,
// all linear in the point: rho across the rows from the patch's middle, kappa
// across the columns, C past the triangle's diagonal edge (k = r).  A point at
// height w over the plane is at least sqrt(w^2 + max(0, |rho| - hr, |kappa| -
// hk, C)^2) from every sub-triangle of the patch, up to the rounding covered
// by the culling margin.
struct Patch {
  __device__ int mesh() const { return int(uint32_t(lo.w) & 0x0fffffffu); }
  __device__ int rows() const { return int(uint32_t(lo.w) >> 28) & 3; }
  __device__ int cols() const { return int(uint32_t(lo.w) >> 30); }
  float4 n4;  // unit normal, reference point x
  float4 m1;  // gradient of rho, reference point y
  float4 m2;  // gradient of kappa, reference point z
  float4 m3;  // gradient of C, C at the reference point
  float4 g;   // hr, hk, culling coefficients c2 and E0 (times the square root of 513)
  float4 h;   // widths of a row, a column, a diagonal strip; bits of first row | first column << 16
  float4 ih;  // 1 / row width, 1 / column width, bits of the inner box: what the sub-triangles' boxes share,
              // as six nibbles (union box low side + nibble x, y, z; high side - nibble x, y, z), -
  int4 lo;    // union of the widened boxes (x, y, z); mesh | rows << 28 | columns << 30
  int4 hi;    // ..., index of the triangle's first sub-triangle
};

// Sub-triangles of a patch: calls f(position within the triangle, row, column, inverted).
template <class F>
__device__ __forceinline__ void for_each_sub(int rows, int cols, uint32_t r0, uint32_t k0, F f) {
  for (int i = 0; i < rows; ++i)
    for (int j = 0; j < cols; ++j) {
      const uint32_t r = r0 + i, k = k0 + j;
      if (k <= r) f(sub_index(r, k, false), i, j, false);
      if (k < r) f(sub_index(r, k, true), i, j, true);
    }
}

// Culling margin of a patch.  With D the distance from a voxel to the ideal
// (affine) patch, every sub-triangle lies at least D - delta away, delta
// bounding how far the accumulated float32 vertices stray from the affine grid
// (2 n additions of coordinates below M on three axes, the roundings of the
// steps, 3 u of an edge L) and the rounding of the linear functions (R: the
// patch's reach; the frame's directions are off by a few u times longest edge^2
// / area) and of their reference point; its float32
// distance is then at least D - t, t = c2 / 4 D^2 + E1 + delta with the largest
// coefficients of cull_coeffs in the patch (d - eps(d) increases, so a larger
// distance only helps).  D^2 > cur * 513/512 + 513 t^2 implies D - t > sqrt(cur)
// (2 t sqrt(cur) <= cur / 512 + 512 t^2), so such a pair cannot lower the
// voxel's minimum.  CULL_FACTOR is 513/512 with room for the squares' rounding.
constexpr float CULL_FACTOR = 1.00196f;

__global__ void k_patches(const float4* __restrict__ T, const uint32_t* __restrict__ nsub,
                          const uint32_t* __restrict__ off, const uint32_t* __restrict__ poff, uint64_t nt, uint64_t np,
                          const MeshInfo* __restrict__ mi, const SubTri* __restrict__ S, Patch* __restrict__ out,
                          M2VStats* st) {
  const uint64_t first = blockIdx.x * uint64_t(blockDim.x), p = first + threadIdx.x;
  const uint64_t i = owner_of(poff, nt, first, p);
  const unsigned live = __ballot_sync(0xffffffffu, p < np);
  if (p >= np) return;
  const uint32_t n = isqrt(nsub[i]), b = uint32_t(p - poff[i]);
  uint32_t r0 = 0, k0 = 0, rows = n, cols = n;
  if (n > 3) {  // block row I holds columns 0 .. I: b = I (I + 1) / 2 + J
    uint32_t I = uint32_t((sqrtf(8.0f * float(b) + 1.0f) - 1.0f) * 0.5f);
    while (uint64_t(I) * (I + 1) / 2 > b) --I;
    while (uint64_t(I + 1) * (I + 2) / 2 <= b) ++I;
    r0 = 2 * I;
    k0 = 2 * (b - uint32_t(uint64_t(I) * (I + 1) / 2));
    rows = min(2u, n - r0);
    cols = min(2u, n - k0);
  }
  const SubTri* base = S + off[i];
  Patch P;
  P.lo = make_int4(INT_MAX, INT_MAX, INT_MAX, 0);
  P.hi = make_int4(INT_MIN, INT_MIN, INT_MIN, int(off[i]));
  int4 ilo = make_int4(INT_MIN, INT_MIN, INT_MIN, 0), ihi = make_int4(INT_MAX, INT_MAX, INT_MAX, 0);
  float c2 = 0.0f, E0 = 0.0f;
  unsigned long long pairs = 0, vpairs = 0;
  for_each_sub(int(rows), int(cols), r0, k0, [&](uint32_t q, int, int, bool) {
    const SubTri s = base[q];
    P.lo = make_int4(min(P.lo.x, s.lo.x), min(P.lo.y, s.lo.y), min(P.lo.z, s.lo.z), s.lo.w);
    P.hi = make_int4(max(P.hi.x, s.hi.x), max(P.hi.y, s.hi.y), max(P.hi.z, s.hi.z), P.hi.w);
    ilo = make_int4(max(ilo.x, s.lo.x), max(ilo.y, s.lo.y), max(ilo.z, s.lo.z), 0);
    ihi = make_int4(min(ihi.x, s.hi.x), min(ihi.y, s.hi.y), min(ihi.z, s.hi.z), 0);
    c2 = fmaxf(c2, s.p2.y);
    E0 = fmaxf(E0, s.p2.w);
    pairs += uint64_t((s.hi.x >> 3) - (s.lo.x >> 3) + 1) * ((s.hi.y >> 3) - (s.lo.y >> 3) + 1) *
             ((s.hi.z >> 3) - (s.lo.z >> 3) + 1);
    vpairs += uint64_t(s.hi.x - s.lo.x + 1) * (s.hi.y - s.lo.y + 1) * (s.hi.z - s.lo.z + 1);
  });
  const int mesh = P.lo.w;
  __syncwarp(live);
  warp_add(&st[mesh].n_pairs, pairs, mesh, live);
  warp_add(&st[mesh].n_vpairs, vpairs, mesh, live);
  // the affine frame
  const float4 a4 = T[3 * i], b4 = T[3 * i + 1], c4 = T[3 * i + 2];
  const float inv = 1.0f / float(n);
  const float s1[3] = {(b4.x - a4.x) * inv, (b4.y - a4.y) * inv, (b4.z - a4.z) * inv};
  const float s2[3] = {(c4.x - b4.x) * inv, (c4.y - b4.y) * inv, (c4.z - b4.z) * inv};
  const float d[3] = {s1[0] + s2[0], s1[1] + s2[1], s1[2] + s2[2]};
  auto dot = [](const float* u, const float* v) { return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]; };
  const float N[3] = {s1[1] * s2[2] - s1[2] * s2[1], s1[2] * s2[0] - s1[0] * s2[2], s1[0] * s2[1] - s1[1] * s2[0]};
  const float l1 = dot(s1, s1), l2 = dot(s2, s2), ld = dot(d, d), ia = rsqrtf(dot(N, N)), area = dot(N, N) * ia;
  const float rm = float(r0) + 0.5f * float(rows), km = float(k0) + 0.5f * float(cols);
  const float h1 = area * rsqrtf(l2), h2 = area * rsqrtf(l1), h3 = area * rsqrtf(ld);
  // unit in-plane normals of the three edge directions: s2 x N, N x s1, N x d, normalised
  float ref[3], m1[3], m2[3], m3[3];
  const float i1 = ia * rsqrtf(l2), i2 = ia * rsqrtf(l1), i3 = ia * rsqrtf(ld);
  for (int k = 0; k < 3; ++k) {
    const int x = (k + 1) % 3, y = (k + 2) % 3;
    (&ref[0])[k] = (&a4.x)[k] + rm * s1[k] + km * s2[k];
    m1[k] = (s2[x] * N[y] - s2[y] * N[x]) * i1;
    m2[k] = (N[x] * s1[y] - N[y] * s1[x]) * i2;
    m3[k] = (N[x] * d[y] - N[y] * d[x]) * i3;
  }
  const float hh = mi[mesh].h;
  const float ex = float(P.hi.x - P.lo.x), ey = float(P.hi.y - P.lo.y), ez = float(P.hi.z - P.lo.z);
  const float R = hh * (sqrtf(ex * ex + ey * ey + ez * ez) + 2.0f);
  const float gm = hh * float(max(max(max(abs(P.lo.x), abs(P.hi.x)), max(abs(P.lo.y), abs(P.hi.y))),
                                  max(abs(P.lo.z), abs(P.hi.z))) + 1);
  const float M = fmaxf(gm, fmaxf(fmaxf(fmaxf(fabsf(a4.x), fabsf(a4.y)), fmaxf(fabsf(a4.z), fabsf(b4.x))),
                                  fmaxf(fmaxf(fabsf(b4.y), fabsf(b4.z)),
                                        fmaxf(fmaxf(fabsf(c4.x), fabsf(c4.y)), fabsf(c4.z)))));
  const float u = 5.9604645e-8f;
  const float e2 = fmaxf(l1, fmaxf(l2, ld)), L = sqrtf(e2) * float(n);  // the triangle's longest edge
  const float delta = (4.0f * float(n) + 8.0f) * u * M + 16.0f * u * L + (32.0f + 64.0f * e2 * ia) * u * R;
  const float sc = 22.66f;  // above sqrt(513)
  const float cs = sc * (0.25f * c2), es = sc * (E0 + delta);
  // a degenerate triangle has no frame: its patch is never culled
  if (cs < __int_as_float(0x7f800000) && es < __int_as_float(0x7f800000) && area > 0.0f && h3 > 0.0f && delta < __int_as_float(0x7f800000)) {
    P.n4 = make_float4(N[0] * ia, N[1] * ia, N[2] * ia, ref[0]);
    P.m1 = make_float4(m1[0], m1[1], m1[2], ref[1]);
    P.m2 = make_float4(m2[0], m2[1], m2[2], ref[2]);
    P.m3 = make_float4(m3[0], m3[1], m3[2], (km - rm) * h3);
    P.g = make_float4(0.5f * float(rows) * h1, 0.5f * float(cols) * h2, cs, es);
    P.h = make_float4(h1, h2, h3, 0.0f);
    P.ih = make_float4(1.0f / h1, 1.0f / h2, 0.0f, 0.0f);
  } else {
    P.n4 = P.m1 = P.m2 = P.m3 = P.h = P.ih = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    P.g = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0x7f800000));
  }
  P.lo.w = int(uint32_t(mesh) | (rows << 28) | (cols << 30));
  P.h.w = __int_as_float(int(r0 | (k0 << 16)));
  const int in[6] = {ilo.x - P.lo.x, ilo.y - P.lo.y, ilo.z - P.lo.z, P.hi.x - ihi.x, P.hi.y - ihi.y, P.hi.z - ihi.z};
  uint32_t nib = 0;
  for (int k = 0; k < 6; ++k) nib |= uint32_t(min(in[k], 15)) << (4 * k);  // 15: past every box's far side or unused
  P.ih.z = __uint_as_float(nib);
  out[p] = P;
}

// Calls f(directory entry, class) for every brick that some sub-triangle's
// box of the patch meets (the patch's own box meets a few more); of the
// bricks in question every `split`th (a power of two) from number `part` on.
template <bool SPLIT, class F>
__device__ __forceinline__ bool for_each_brick(const Patch& P, const SubTri* __restrict__ S, const Dir& d,
                                               uint32_t split, uint32_t part, F f) {
  int lo[3], hi[3];
  if (!brick_range(P.lo, P.hi, d, lo, hi)) return false;
  const int rows = P.rows(), cols = P.cols(), at = __float_as_int(P.h.w);
  const uint32_t r0 = uint32_t(at) & 0xffffu, k0 = uint32_t(at) >> 16;
  const SubTri* base = S + uint32_t(P.hi.w);
  const uint32_t nib = __float_as_uint(P.ih.z);
  const int ulo[3] = {P.lo.x, P.lo.y, P.lo.z}, uhi[3] = {P.hi.x, P.hi.y, P.hi.z};
  int ilo[3], ihi[3];
  for (int k = 0; k < 3; ++k) {
    const int a = int(nib >> (4 * k)) & 15, b = int(nib >> (4 * k + 12)) & 15;
    const bool none = a == 15 || b == 15 || ulo[k] + a > uhi[k] - b;
    ilo[k] = none ? INT_MAX : ulo[k] + a;
    ihi[k] = none ? INT_MIN : uhi[k] - b;
  }
  uint32_t turn = 0;
  for (int x = lo[0]; x <= hi[0]; ++x)
    for (int y = lo[1]; y <= hi[1]; ++y)
      for (int z = lo[2]; z <= hi[2]; ++z) {
        if (SPLIT && (turn++ & (split - 1u)) != part) continue;
        const int bx = x + d.bx0, by = y + d.by0, bz = z + d.bz0;
        // the box that all sub-triangles share, else one by one
        bool hit = (ilo[0] >> 3) <= bx && (ihi[0] >> 3) >= bx && (ilo[1] >> 3) <= by && (ihi[1] >> 3) >= by &&
                   (ilo[2] >> 3) <= bz && (ihi[2] >> 3) >= bz;
        if (!hit)
          for_each_sub(rows, cols, r0, k0, [&](uint32_t q, int, int, bool) {
            if (hit) return;
            const int4 l = base[q].lo, h = base[q].hi;
            hit = (l.x >> 3) <= bx && (h.x >> 3) >= bx && (l.y >> 3) <= by && (h.y >> 3) >= by && (l.z >> 3) <= bz &&
                  (h.z >> 3) >= bz;
          });
        if (hit) f(((uint64_t(x) * d.dy + y) * d.dz + z), pair_class(P.lo, P.hi, bx, by, bz));
      }
  return true;
}

// `split` threads per patch, 32 where patches are few, 1 from 256 per SM on: a
// patch of a few large triangles meets dozens of bricks, which one thread would
// test in turn (80 triangles, boxes of 10 voxels: both passes 0.120 ms with one
// thread, 0.076 with 32; 5,120 triangles 0.120 against 0.098 ms).  SPLIT: more
// than one (counting the bricks costs 0.1 of 1.4 ms where patches are many).
template <bool SPLIT>
__global__ void k_count_patches(const Patch* __restrict__ P, uint64_t np, const SubTri* __restrict__ S,
                              const Dir* __restrict__ dirs, const uint64_t* __restrict__ dir_base,
                              uint32_t* __restrict__ cnt, M2VStats* st, uint32_t split) {
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, i = SPLIT ? t / split : t;
  if (i >= np) return;
  const Patch p = P[i];
  const int mesh = p.mesh();
  uint32_t* C = cnt + dir_base[mesh] * LIST_CLASSES;
  if (!for_each_brick<SPLIT>(p, S, dirs[mesh], split, SPLIT ? uint32_t(t % split) : 0u,
                             [&](uint64_t e, int c) { atomicAdd(&C[e * LIST_CLASSES + c], 1u); }))
    atomicExch(&st[mesh].error, 2);
}

template <bool SPLIT>
__global__ void k_fill_patches(const Patch* __restrict__ P, uint64_t np, const SubTri* __restrict__ S,
                             const Dir* __restrict__ dirs, const uint64_t* __restrict__ dir_base,
                             uint32_t* __restrict__ cursor, uint32_t* __restrict__ list, uint32_t split) {
  const uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, i = SPLIT ? t / split : t;
  if (i >= np) return;
  const Patch p = P[i];
  uint32_t* C = cursor + dir_base[p.mesh()] * LIST_CLASSES;
  for_each_brick<SPLIT>(p, S, dirs[p.mesh()], split, SPLIT ? uint32_t(t % split) : 0u,
                 [&](uint64_t e, int c) { list[atomicAdd(&C[e * LIST_CLASSES + c], 1u)] = uint32_t(i); });
}

// One CTA per brick.  Each warp stages BATCH patches of the brick's list;
// the per-voxel minimum of the squared distance is kept in shared memory with
// atomicMin on the float bits (distances are >= 0, so unsigned order is float
// order; NaN distances are skipped, as `dist < cur` never holds for NaN in the
// reference).
//
// Pairs that cannot lower the voxel's minimum are culled before the exact
// point-triangle distance is evaluated, in two steps: (voxel, patch) pairs by
// the distance to the patch's flat outline, then the sub-triangles of a
// surviving pair by the distance to each one's outline, both against the
// voxel's running minimum with the margin of k_patches.  The running minimum
// is a value some evaluated pair produced, so the minimum over the surviving
// pairs equals the minimum over all pairs, bit for bit, whatever the order; a
// voxel whose minimum is still +inf keeps all its pairs, so the active set is
// unchanged too.
//
// Lanes take (patch, y, z) columns of the staged patches: height and in-plane
// distances at the column's first voxel, then one addition each per voxel, the
// running minima as two float4 loads.  Surviving pairs go through a per-warp
// queue; 32 at a time each lane evaluates the sub-triangle nearest to its
// voxel, which tightens the minimum, and queues the others that may still be
// nearer; these are evaluated 32 at a time too.  A sub-triangle counts only
// where its own widened box holds the voxel.
//
// Issue-bound (83 % of cycles issue): 10.9 G warp instructions and 12.0 ms
// beside the tree build (10.5 alone) on a torus of 1 M triangles, 10.7 M
// sub-triangles and 35.7 M band voxels, where the pass over sub-triangles takes
// 16.8 G and 15.6 ms; it evaluates 12 exact distances per voxel instead of 28.  (Work units of 64 voxels with their own
// nearest-first order: no fewer evaluations, 15.5 G instructions, 19.0 ms.)
//
// Threads per brick: 64, 128 or 256 (bs_autotune_mesh_to_volume); a warp
// stages 8 patches at a time (16: 12.7 against 12.3 ms on the torus, 0.23
// against 0.18 ms on an icosphere of 1,500 bricks).
constexpr int BATCH = 8;
constexpr int PATCH_QUEUE = 32 + 8 * 32;  // < 32 left over + 8 per lane

struct __align__(16) PatchTile {
  float4 n4, m1, m2, m3, g, h;  // as in Patch
  float4 ih;  // 1 / row width, 1 / column width, bits of the inner box's x | y << 8 | z << 16 in the brick, -
  int4 box;   // first y and z of (box) x (brick) within the brick, its z extent, index of the first sub-triangle
  int4 box1;  // mask of the brick x covered by the box, bits of 1 / z extent, rows, columns
  // 144 B apart: eight lanes' float4 loads of eight patches fall on different banks
};

// Out of line: the kernel's hot code then fits the instruction cache (inlined
// at its call sites, 3 of 13 warps' stall cycles waited for instructions).
__device__ __noinline__ float sub_distance2(const SubTri* s, F3 p) {
  const float4 p0 = __ldg(&s->p0), p1 = __ldg(&s->p1);
  const float p2x = __ldg(&s->p2.x);
  return point_triangle_dist2(f3(p0.x, p0.y, p0.z), f3(p0.w, p1.x, p1.y), f3(p1.z, p1.w, p2x), p);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_patch_distance(
    const int4* __restrict__ origins, const uint32_t* __restrict__ list_off, const uint32_t* __restrict__ list,
    const Patch* __restrict__ patches, const SubTri* __restrict__ S, const MeshInfo* __restrict__ mi,
    const uint32_t* __restrict__ leaf_base, int K, float* __restrict__ values, uint32_t* __restrict__ masks,
    M2VStats* st) {
  // per-voxel running minimum of d^2, x fastest: index (y << 6) | (z << 3) | x,
  // so a (y, z) column's eight voxels are two float4 loads
  __shared__ __align__(16) uint32_t dmin[512];
  __shared__ PatchTile bt[THREADS / 32][BATCH];
  __shared__ int pre[THREADS / 32][BATCH + 1];
  __shared__ uint32_t queue[THREADS / 32][PATCH_QUEUE];   // patch << 9 | voxel
  __shared__ uint2 queue2[THREADS / 32][PATCH_QUEUE];     // sub-triangle, voxel
  __shared__ float gtab[3][8];  // grid coordinates x * h of the brick's voxels, per axis
  __shared__ uint32_t evaluated, next_tile;
  const int b = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int4 org = origins[b];
  const int mesh = find_seg(leaf_base, K, uint64_t(b));
  const float h = mi[mesh].h;
  for (int o = t; o < 512; o += THREADS) dmin[o] = 0x7f800000u;  // +inf
  if (t < 24) {
    const int ax = t >> 3, i = t & 7;
    gtab[ax][i] = fmul(__int2float_rn((ax == 0 ? org.x : ax == 1 ? org.y : org.z) + i), h);
  }
  if (t == 0) evaluated = next_tile = 0;
  __syncthreads();
  const uint32_t beg = list_off[b], end = list_off[b + 1];
  PatchTile* W = bt[warp];
  int* P = pre[warp];
  uint32_t* Q = queue[warp];
  uint2* Q2 = queue2[warp];
  uint32_t n_eval = 0;
  int qn = 0, qn2 = 0;

  // exact distance of voxel o (column-major) to sub-triangle idx; `outer`: its box may not hold the voxel
  auto eval = [&](uint32_t idx, int o, bool outer) {
    const SubTri* s = S + idx;
    if (outer) {
      const int4 lo = __ldg(&s->lo), hi = __ldg(&s->hi);
      const int vx = org.x + (o & 7), vy = org.y + (o >> 6), vz = org.z + ((o >> 3) & 7);
      if (vx < lo.x || vx > hi.x || vy < lo.y || vy > hi.y || vz < lo.z || vz > hi.z) return;
    }
    ++n_eval;
    const float d2 = sub_distance2(s, f3(gtab[0][o & 7], gtab[1][o >> 6], gtab[2][(o >> 3) & 7]));
    if (d2 < __int_as_float(0x7f800000))  // false for NaN and +inf
      atomicMin(&dmin[o], __float_as_uint(d2));
  };
  // the last `cnt` queued sub-triangles
  auto drain2 = [&](int cnt) {
    __syncwarp();
    qn2 -= cnt;
    if (lane < cnt) {
      const uint2 e = Q2[qn2 + lane];
      eval(e.x, int(e.y & 511u), e.y >> 9);
    }
    __syncwarp();
  };
  // the last `cnt` queued (voxel, patch) pairs
  auto drain = [&](int cnt) {
    __syncwarp();
    qn -= cnt;
    uint32_t bits = 0, off = 0, r0 = 0, k0 = 0;
    int o = 0, cols = 1;
    bool outer = false;
    if (lane < cnt) {
      const uint32_t ent = Q[qn + lane];
      const PatchTile& q = W[ent >> 9];
      o = int(ent & 511u);
      const float4 n4 = q.n4, m1 = q.m1, m2 = q.m2, m3 = q.m3, g = q.g, hw = q.h;
      const float dx = gtab[0][o & 7] - n4.w, dy = gtab[1][o >> 6] - m1.w, dz = gtab[2][(o >> 3) & 7] - m2.w;
      const float w = n4.x * dx + n4.y * dy + n4.z * dz;
      const float rho = m1.x * dx + m1.y * dy + m1.z * dz;
      const float kap = m2.x * dx + m2.y * dy + m2.z * dz;
      const float C = m3.x * dx + m3.y * dy + m3.z * dz + m3.w;
      const int at = __float_as_int(hw.w), rows = q.box1.z;
      cols = q.box1.w;
      r0 = uint32_t(at) & 0xffffu;
      k0 = uint32_t(at) >> 16;
      off = uint32_t(q.box.w);
      const int dk = int(r0) - int(k0);
      const float fr = 0.5f * float(rows), fk = 0.5f * float(cols);
      const float4 ih = q.ih;
      const uint32_t inner = __float_as_uint(ih.z);
      outer = !(((inner >> (o & 7)) & (inner >> (8 + (o >> 6))) & (inner >> (16 + ((o >> 3) & 7)))) & 1u);
      // the cell below the voxel, and which of its halves (a good first guess
      // is all that is needed: clamped into the patch)
      const float rl = fmaf(rho, ih.x, fr), kl = fmaf(kap, ih.y, fk);
      const int bi = min(max(int(rl), 0), rows - 1), bj = min(min(max(int(kl), 0), cols - 1), bi + dk);
      const bool bd = bj < bi + dk && kl - float(bj) > rl - float(bi);
      eval(off + sub_index(r0 + bi, k0 + bj, bd), o, outer);
      if (rows * cols > 1) {  // the others that may be nearer than what the voxel has now
        const float lim = CULL_FACTOR * __uint_as_float(*reinterpret_cast<volatile uint32_t*>(&dmin[o])), w2 = w * w;
        auto may = [&](float e) {  // e: largest in-plane distance past an edge
          e = fmaxf(e, 0.0f);
          const float lb = fmaf(e, e, w2), tm = fmaf(g.z, lb, g.w);
          return !(lb > fmaf(tm, tm, lim));
        };
        for (int i = 0; i < rows; ++i) {
          const float ra = fmaf(fr - float(i), hw.x, rho);  // past row r
          const int last = min(cols - 1, i + dk);
          for (int j = 0; j <= last; ++j) {
            const float ka = fmaf(fk - float(j), hw.y, kap);             // past column k
            const float cd = fmaf(float(dk + i - j), hw.z, C);           // past the cell's diagonal
            const int c = 2 * (i * cols + j);
            if (may(fmaxf(fmaxf(ra - hw.x, -ka), cd))) bits |= 1u << c;
            if (j < i + dk && may(fmaxf(fmaxf(-ra, ka - hw.y), -cd))) bits |= 2u << c;
          }
        }
        bits &= ~((bd ? 2u : 1u) << (2 * (bi * cols + bj)));
      }
    }
    // at most 8 per lane (a patch has nine sub-triangles, the nearest is taken),
    // which PATCH_QUEUE has room for beside fewer than 32 left over
    const int n = __popc(bits);
    if (__any_sync(0xffffffffu, n)) {
      int pos = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pos, d);
        if (lane >= d) pos += v;
      }
      const int added = __shfl_sync(0xffffffffu, pos, 31);
      pos += qn2 - n;
      while (bits) {
        const int c = __ffs(bits) - 1;
        bits &= bits - 1u;
        const int cell = c >> 1, i = cell / cols, j = cell - i * cols;
        Q2[pos++] = make_uint2(off + sub_index(r0 + i, k0 + j, c & 1), uint32_t(o) | (outer ? 512u : 0u));
      }
      qn2 += added;
      while (qn2 >= 32) drain2(32);
    }
  };

  for (;;) {
    // the next tile of the list, nearest class first, to whichever warp is free
    uint32_t e0 = 0;
    if (lane == 0) e0 = atomicAdd(&next_tile, BATCH);
    e0 = beg + __shfl_sync(0xffffffffu, e0, 0);
    if (e0 >= end) break;
    // lanes 0..BATCH-1: stage one patch each and count its (y, z) columns of
    // voxels in this brick
    int cols = 0;
    if (lane < BATCH && e0 + lane < end) {
      const Patch* sp = patches + list[e0 + lane];
      const int4 lo = __ldg(&sp->lo), hi = __ldg(&sp->hi);
      const int x0 = max(lo.x, org.x), y0 = max(lo.y, org.y), z0 = max(lo.z, org.z);
      const int nx = min(hi.x, org.x + 7) - x0 + 1, ny = min(hi.y, org.y + 7) - y0 + 1,
                nz = min(hi.z, org.z + 7) - z0 + 1;
      if (nx > 0 && ny > 0 && nz > 0) {
        PatchTile& q = W[lane];
        q.n4 = __ldg(&sp->n4);
        q.m1 = __ldg(&sp->m1);
        q.m2 = __ldg(&sp->m2);
        q.m3 = __ldg(&sp->m3);
        q.g = __ldg(&sp->g);
        q.h = __ldg(&sp->h);
        const float4 ih = __ldg(&sp->ih);
        const uint32_t nib = __float_as_uint(ih.z);
        auto span = [](int a, int b) {  // bits a .. b of a byte
          a = max(a, 0);
          b = min(b, 7);
          return a > b ? 0u : ((1u << (b - a + 1)) - 1u) << a;
        };
        auto inner = [&](int k, int l, int u, int o0) {
          const int d0 = int(nib >> (4 * k)) & 15, d1 = int(nib >> (4 * k + 12)) & 15;
          return (d0 == 15 || d1 == 15) ? 0u : span(l + d0 - o0, u - d1 - o0);
        };
        const uint32_t in = inner(0, lo.x, hi.x, org.x) | (inner(1, lo.y, hi.y, org.y) << 8) |
                            (inner(2, lo.z, hi.z, org.z) << 16);
        q.ih = make_float4(ih.x, ih.y, __uint_as_float(in), 0.0f);
        q.box = make_int4(y0 - org.y, z0 - org.z, nz, hi.w);
        q.box1 = make_int4(int(((1u << nx) - 1u) << (x0 - org.x)), __float_as_int(1.0f / float(nz)),
                           int(uint32_t(lo.w) >> 28) & 3, int(uint32_t(lo.w) >> 30));
        cols = ny * nz;
      }
    }
    // inclusive prefix of the column counts over the batch lanes
    int inc = cols;
#pragma unroll
    for (int d = 1; d < BATCH; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += v;
    }
    if (lane < BATCH) P[lane + 1] = inc;
    if (lane == 0) P[0] = 0;
    const int total = __shfl_sync(0xffffffffu, inc, BATCH - 1);
    __syncwarp();
    int j = 0;
    for (int base = 0; base < total; base += 32) {
      // one lane per (patch, y, z) column: an 8-bit mask of the column's
      // voxels (x within the brick) that survive the cull test
      const int k = base + lane;
      uint32_t bits = 0, colb = 0;
      if (k < total) {
        while (k >= P[j + 1]) ++j;  // P[BATCH] = total > k
        const PatchTile& q = W[j];
        const int4 bx = q.box, b1 = q.box1;
        const float4 n4 = q.n4, m1 = q.m1, m2 = q.m2, m3 = q.m3, g = q.g;
        const int c = k - P[j];
        // c -> (iy, iz) by reciprocal multiply: c < 64 and nz <= 8 keep the
        // product at least 0.5/8 away from the next integer
        const int iy = int((float(c) + 0.5f) * __int_as_float(b1.y)), iz = c - iy * bx.z;
        const int oy = bx.x + iy, oz = bx.y + iz;
        const float dx = gtab[0][0] - n4.w, dy = gtab[1][oy] - m1.w, dz = gtab[2][oz] - m2.w;
        float w = n4.x * dx + n4.y * dy + n4.z * dz;
        float rho = m1.x * dx + m1.y * dy + m1.z * dz;
        float kap = m2.x * dx + m2.y * dy + m2.z * dz;
        float C = m3.x * dx + m3.y * dy + m3.z * dz + m3.w;
        const float iw = n4.x * h, ir = m1.x * h, ik = m2.x * h, ic = m3.x * h;
        colb = uint32_t((oy << 6) | (oz << 3));
        const float4 ca = *reinterpret_cast<const float4*>(&dmin[colb]);
        const float4 cc = *reinterpret_cast<const float4*>(&dmin[colb + 4]);
        const float cur[8] = {ca.x, ca.y, ca.z, ca.w, cc.x, cc.y, cc.z, cc.w};
#pragma unroll
        for (int ix = 0; ix < 8; ++ix) {
          const float e = fmaxf(fmaxf(fabsf(rho) - g.x, fabsf(kap) - g.y), fmaxf(C, 0.0f));
          const float lb = fmaf(e, e, w * w), tm = fmaf(g.z, lb, g.w);
          bits |= (lb > fmaf(tm, tm, CULL_FACTOR * cur[ix])) ? 0u : (1u << ix);
          w += iw;
          rho += ir;
          kap += ik;
          C += ic;
        }
        bits &= uint32_t(b1.x);  // the voxels of (box) x (brick) in this column
      }
      // survivors to the queue: warp prefix of the per-lane counts
      const int cnt = __popc(bits);
      int pos = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pos, d);
        if (lane >= d) pos += v;
      }
      const int added = __shfl_sync(0xffffffffu, pos, 31);
      pos += qn - cnt;
      while (bits) {
        const int ix = __ffs(bits) - 1;
        bits &= bits - 1u;
        Q[pos++] = (uint32_t(j) << 9) | colb | uint32_t(ix);
      }
      qn += added;
      const bool last = base + 32 >= total;  // the tile's entries refer to it
      while (qn >= 32 || (last && qn > 0)) drain(min(qn, 32));
      __syncwarp();
    }
  }
  if (qn2 > 0) drain2(qn2);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) n_eval += __shfl_xor_sync(0xffffffffu, n_eval, d);
  if (lane == 0 && n_eval) atomicAdd(&evaluated, n_eval);
  __syncthreads();
  if (t == 0 && evaluated) atomicAdd(&st[mesh].n_eval, (unsigned long long)evaluated);
#pragma unroll
  for (int k = 0; k < 512 / THREADS; ++k) {
    const int o = t + THREADS * k;  // (x << 6) | (y << 3) | z
    const uint32_t u = dmin[((o & 0x38) << 3) | ((o & 7) << 3) | (o >> 6)];
    const float dist = fsqrt(__uint_as_float(u));
    const bool act = dist < __int_as_float(0x7f800000);  // sqrt of a finite square can overflow to inf
    const uint32_t m = __ballot_sync(0xffffffffu, act);
    values[uint64_t(b) * 512 + o] = act ? dist : 0.0f;
    if (lane == 0) masks[uint64_t(b) * 16 + warp + (THREADS / 32) * k] = m;
  }
}

}  // namespace bs
