// Dual contouring on the GPU (voxel/meshing/dual_contouring.rs:16-473).
//
// Leaves are handled by a warp each, on bit masks where only activity and
// signs matter, and on compacted work lists where values are computed:
//   0. the sign bits of every leaf's values, and its 27 neighbour leaves;
//   1. masks of edge crossings (active voxels whose +1 neighbour along an axis
//      is active with the other sign, dual_contouring.rs:249-387) and of cells
//      (8 active corners, not all of one sign, dual_contouring.rs:193-217),
//      eight voxels of a z-line at a time with shifts of 9-bit lines;
//   2. per crossing the point and the normal from interpolated central /
//      one-sided differences;
//   3. per cell the particle solver over its crossings (find_feature_point,
//      dual_contouring.rs:429-458, 50 damped iterations);
//   4. per crossing whose 4 surrounding cells have vertices, two triangles,
//      flipped when the first end is inside, scaled by the voxel size; exactly
//      degenerate triangles are dropped (dual_contouring.rs:62-79, 93-174):
//      counted, scanned, written.
// Masks are stored with each word's rank (the set bits before it), so a
// crossing or cell is found with one 8-byte load.  What bounds it: latency of
// dependent gathers (points of a cell, vertices of a quad) and, in the solver,
// its chain of float operations.  One CTA of 128 threads per leaf tested all
// 512 voxels in every pass before, with a hash probe of 27 neighbours in each:
// on a torus of 57 k leaves (1.3 M crossings) the kernels took 2.81 ms, now 0.55.
// Every float operation follows the reference's order without fused
// multiply-adds, so the vertices are bit-identical to the reference's.  The
// face order is deterministic (leaves in volume order, voxels, axes); the
// reference's own order depends on thread scheduling.
#include <cub/device/device_scan.cuh>

#include "bs_internal.cuh"
#include "dc.cuh"
#include "leaf_hash.cuh"
#include "volume_upper.cuh"

namespace bs {

template <class T>
static void scan_e(bs_ctx* ctx, const T* in, T* out, size_t n) {
  size_t tmp = 0;
  BS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, n, ctx->stream));
  DBuf<uint8_t> t(ctx, tmp);
  BS_CUDA(cub::DeviceScan::ExclusiveSum(t.p, tmp, in, out, n, ctx->stream));
}

constexpr int DC_WARPS = 4;
constexpr unsigned DC_FULL = 0xffffffffu;

// 27 neighbour leaves around every leaf, index (dx+1)*9 + (dy+1)*3 + (dz+1).
__global__ void k_dc_neighbours(const int4* __restrict__ org, LeafHash hash, uint64_t n, int* __restrict__ nbr) {
  const uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= 27 * n) return;
  const uint64_t l = i / 27;
  const int k = int(i - 27 * l);
  const int4 o = org[l];
  nbr[i] = k == 13 ? int(l) : hash.find(o.x + 8 * (k / 9 - 1), o.y + 8 * ((k / 3) % 3 - 1), o.z + 8 * (k % 3 - 1));
}

// Sign bits of every leaf's values, one warp per leaf: lane's float4 j is
// voxels 4 (lane + 32 j) .. + 3, a nibble of word (lane + 32 j) / 8.
__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_signs(const float* __restrict__ val, uint64_t n,
                                                            uint32_t* __restrict__ sgn) {
  const uint64_t l = blockIdx.x * uint64_t(DC_WARPS) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (l >= n) return;
  const float4* v4 = reinterpret_cast<const float4*>(val + l * 512);
  float4 r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) r[j] = v4[lane + 32 * j];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t nib = (signbit(r[j].x) ? 1u : 0u) | (signbit(r[j].y) ? 2u : 0u) | (signbit(r[j].z) ? 4u : 0u) |
                   (signbit(r[j].w) ? 8u : 0u);
    nib <<= 4 * (lane & 7);
    nib |= __shfl_xor_sync(DC_FULL, nib, 1);
    nib |= __shfl_xor_sync(DC_FULL, nib, 2);
    nib |= __shfl_xor_sync(DC_FULL, nib, 4);
    if ((lane & 7) == 0) sgn[l * 16 + (lane >> 3) + 4 * j] = nib;
  }
}

// Value at voxel (x, y, z) given relative to the leaf origin (in [-8, 16)),
// as the tree's `at` returns it: an active leaf voxel, or, for a voxel
// outside every leaf, its active tile's value.  Inactive voxels of a leaf
// have no value.
// TILES: the volume has active tiles (the kernels reading neighbour values
// come in both forms, so tile-free volumes run without the lookup).
template <bool TILES>
__device__ __forceinline__ bool at(const DcVol& V, const int* nb, int4 org, int x, int y, int z, float& v) {
  const int k = ((x >> 3) + 1) * 9 + ((y >> 3) + 1) * 3 + ((z >> 3) + 1);
  const int l = nb[k];
  if (l < 0) return TILES && tile_value(V.tiles, org.x + x, org.y + y, org.z + z, v);
  const int o = ((x & 7) << 6) | ((y & 7) << 3) | (z & 7);
  if (!((V.msk[uint64_t(l) * 16 + (o >> 5)] >> (o & 31)) & 1u)) return false;
  v = V.val[uint64_t(l) * 512 + o];
  return true;
}

// dual_contouring.rs:362-386
template <bool TILES>
__device__ __forceinline__ bool grad(const DcVol& V, const int* nb, int4 org, int x, int y, int z, int axis,
                                     float& g) {
  const int lx = axis == 0 ? 1 : 0, ly = axis == 1 ? 1 : 0, lz = axis == 2 ? 1 : 0;
  float vp, vl, vr;
  const bool hp = at<TILES>(V, nb, org, x, y, z, vp);
  const bool hl = at<TILES>(V, nb, org, x - lx, y - ly, z - lz, vl);
  const bool hr = at<TILES>(V, nb, org, x + lx, y + ly, z + lz, vr);
  if (hp && hl && hr) { g = fmul(fsub(vr, vl), 0.5f); return true; }
  if (hp && hr) { g = fsub(vr, vp); return true; }
  if (hp && hl) { g = fsub(vp, vl); return true; }
  return false;  // the reference stops with unreachable!() here
}

// Masks of crossings and cells with their ranks: em[(l*3 + dir)*16 + w] and
// cellm[l*16 + w] = (mask word, set bits in the words before it), and their
// counts per leaf and direction (ccount) and per leaf (cellc).
template <bool TILES>
__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_masks(DcVol V, uint64_t n, uint2* __restrict__ em,
                                                            uint32_t* __restrict__ ccount, uint2* __restrict__ cellm,
                                                            uint32_t* __restrict__ cellc) {
  __shared__ uint32_t line[DC_WARPS][81];       // z-lines (x, y) of 9 x 9: 9 active bits | 9 sign bits << 16
  __shared__ uint32_t words[DC_WARPS][4][16];   // crossings x, y, z; cells
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint64_t l = blockIdx.x * uint64_t(DC_WARPS) + wi;
  if (l >= n) return;
  const int* nb = V.nbr + l * 27;
  const int4 org = V.org[l];
  // active and sign byte of the z-line (x, y) of the neighbour leaf (bx, by, bz) in {0, 1}
  auto bits = [&](int x, int y, int bx, int by, int bz) -> uint32_t {
    const int k = nb[(bx + 1) * 9 + (by + 1) * 3 + bz + 1];
    if (k >= 0) {
      const uint64_t w = uint64_t(k) * 16 + (x << 1) + (y >> 2);
      const int sh = 8 * (y & 3);
      return ((V.msk[w] >> sh) & 0xffu) | (((V.sgn[w] >> sh) & 0xffu) << 16);
    }
    float v;
    // a missing leaf's block lies in one tile whole
    if (TILES && tile_value(V.tiles, org.x + 8 * bx, org.y + 8 * by, org.z + 8 * bz, v))
      return signbit(v) ? 0x00ff00ffu : 0x000000ffu;
    return 0u;
  };
  for (int i = lane; i < 81; i += 32) {
    const int x = i / 9, y = i - 9 * x, bx = x >> 3, by = y >> 3;
    const uint32_t lo = bits(x & 7, y & 7, bx, by, 0), hi = bits(x & 7, y & 7, bx, by, 1);
    line[wi][i] = lo | ((hi & 0x00010001u) << 8);
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int j = lane + 32 * h, x = j >> 3, y = j & 7;
    const uint32_t* L = line[wi] + 9 * x + y;
    const uint32_t a = L[0], b = L[9], c = L[1], d = L[10];  // (x, y), (x+1, y), (x, y+1), (x+1, y+1)
    const uint32_t A = a & 0x1ffu, B = b & 0x1ffu, C = c & 0x1ffu, D = d & 0x1ffu;
    const uint32_t S = a >> 16, SB = b >> 16, SC = c >> 16, SD = d >> 16;
    uint32_t all = A & B & C & D, neg = S | SB | SC | SD, nall = S & SB & SC & SD;
    all &= all >> 1;
    neg |= neg >> 1;
    nall &= nall >> 1;
    const uint32_t m[4] = {A & B & (S ^ SB), A & C & (S ^ SC), A & (A >> 1) & (S ^ (S >> 1)), all & neg & ~nall};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t v = (m[t] & 0xffu) << (8 * (lane & 3));
      v |= __shfl_xor_sync(DC_FULL, v, 1);
      v |= __shfl_xor_sync(DC_FULL, v, 2);
      if ((lane & 3) == 0) words[wi][t][8 * h + (lane >> 2)] = v;
    }
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // two masks at a time, 16 lanes each
    const int t = 2 * h + (lane >> 4), w = lane & 15;
    const uint32_t v = words[wi][t][w];
    uint32_t inc = __popc(v);
#pragma unroll
    for (int s = 1; s < 16; s <<= 1) {
      const uint32_t u = __shfl_up_sync(DC_FULL, inc, s, 16);
      if (w >= s) inc += u;
    }
    const uint2 e = make_uint2(v, inc - __popc(v));
    if (t < 3) em[(l * 3 + t) * 16 + w] = e;
    else cellm[l * 16 + w] = e;
    if (w == 15) {
      if (t < 3) ccount[l * 3 + t] = inc;
      else cellc[l] = inc;
    }
  }
  if (l == n - 1 && lane == 0) {
    ccount[n * 3] = 0;
    cellc[n] = 0;
  }
}

// Position of voxel o in a mask with ranks, or -1.
__device__ __forceinline__ int ranked(const uint2* __restrict__ m, int o) {
  const uint2 e = __ldg(m + (o >> 5));
  const uint32_t bit = 1u << (o & 31);
  return (e.x & bit) ? int(e.y + __popc(e.x & (bit - 1u))) : -1;
}

// Crossing points and normals (dual_contouring.rs:249-313): `split` warps per
// leaf, its crossings (directions, then voxels in ascending order) listed and
// taken 32 at a time, so points are written in order.
template <bool TILES>
__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_edge_points(DcVol V, uint64_t n, const uint2* __restrict__ em,
                                                                  const uint32_t* __restrict__ coff,
                                                                  float* __restrict__ pts, DcStats* st,
                                                                  uint32_t split) {
  __shared__ uint16_t list[DC_WARPS][3 * 512];
  __shared__ int nbs[DC_WARPS][27];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint64_t gw = blockIdx.x * uint64_t(DC_WARPS) + wi, l = gw / split;
  if (l >= n) return;
  const uint32_t c0 = coff[l * 3], cnt = coff[l * 3 + 3] - c0, first = 32 * uint32_t(gw % split);
  if (cnt <= first) return;
  if (lane < 27) nbs[wi][lane] = V.nbr[l * 27 + lane];
  for (int k = lane; k < 48; k += 32) {
    const uint2 e = em[l * 48 + k];
    uint32_t at = coff[l * 3 + (k >> 4)] - c0 + e.y;
    for (uint32_t m = e.x; m; m &= m - 1u) list[wi][at++] = uint16_t((k << 5) | (__ffs(m) - 1));
  }
  __syncwarp();
  const int* nb = nbs[wi];
  const int4 org = V.org[l];
  for (uint32_t i = first + lane; i < cnt; i += 32 * split) {
    const int code = list[wi][i], dir = code >> 9, o = code & 511;
    const int x = o >> 6, y = (o >> 3) & 7, z = o & 7;
    const int x2 = x + (dir == 0), y2 = y + (dir == 1), z2 = z + (dir == 2);
    float v1, v2;
    at<TILES>(V, nb, org, x, y, z, v1);
    at<TILES>(V, nb, org, x2, y2, z2, v2);
    const float t = (v1 == v2) ? 0.5f : fdiv(v1, fsub(v1, v2));
    float p[3] = {__int2float_rn(org.x + x), __int2float_rn(org.y + y), __int2float_rn(org.z + z)};
    if (dir == 0) p[0] = fadd(p[0], t);
    else if (dir == 1) p[1] = fadd(p[1], t);
    else p[2] = fadd(p[2], t);
    float nrm[3];
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float g1, g2;
      ok = ok && grad<TILES>(V, nb, org, x, y, z, a, g1) && grad<TILES>(V, nb, org, x2, y2, z2, a, g2);
      if (ok) nrm[a] = fadd(fmul(fsub(1.0f, t), g1), fmul(t, g2));
    }
    if (!ok) {
      atomicExch(&st->error, 1);
      continue;
    }
    const float len = fsqrt(fadd(fadd(fmul(nrm[0], nrm[0]), fmul(nrm[1], nrm[1])), fmul(nrm[2], nrm[2])));
    float2* q = reinterpret_cast<float2*>(pts + uint64_t(c0 + i) * 6);
    q[0] = make_float2(p[0], p[1]);
    q[1] = make_float2(p[2], fdiv(nrm[0], len));
    q[2] = make_float2(fdiv(nrm[1], len), fdiv(nrm[2], len));
  }
}

// voxel/utils.rs:88-97 and dual_contouring.rs:410-423
__constant__ int8_t c_edges[12][4] = {{0, 0, 0, 0}, {0, 0, 0, 1}, {0, 0, 0, 2}, {1, 0, 0, 1},
                                      {1, 0, 0, 2}, {0, 0, 1, 0}, {0, 0, 1, 1}, {0, 1, 0, 0},
                                      {0, 1, 0, 2}, {1, 0, 1, 1}, {0, 1, 1, 0}, {1, 1, 0, 2}};
__constant__ int8_t c_cells[3][4][3] = {{{0, 0, 0}, {0, 0, -1}, {0, -1, -1}, {0, -1, 0}},
                                        {{0, 0, 0}, {-1, 0, 0}, {-1, 0, -1}, {0, 0, -1}},
                                        {{0, -1, 0}, {-1, -1, 0}, {-1, 0, 0}, {0, 0, 0}}};

// The crossing stored for edge (x, y, z, dir) of the leaf's neighbourhood.
__device__ __forceinline__ const float* edge_point(const int* nb, const uint2* em, const uint32_t* coff,
                                                   const float* pts, int x, int y, int z, int dir) {
  const int k = ((x >> 3) + 1) * 9 + ((y >> 3) + 1) * 3 + ((z >> 3) + 1);
  const int l = nb[k];
  if (l < 0) return nullptr;
  const int o = ((x & 7) << 6) | ((y & 7) << 3) | (z & 7);
  const uint64_t d = uint64_t(l) * 3 + dir;
  const int r = ranked(em + d * 16, o);
  return r < 0 ? nullptr : pts + uint64_t(coff[d] + uint32_t(r)) * 6;
}

// The cells of a leaf as a list in ascending order; returns their number.
__device__ __forceinline__ uint32_t list_cells(const uint2* __restrict__ cellm, uint64_t l, uint16_t* list) {
  const int lane = threadIdx.x & 31;
  uint32_t end = 0;
  if (lane < 16) {
    const uint2 e = cellm[l * 16 + lane];
    uint32_t at = e.y;
    for (uint32_t m = e.x; m; m &= m - 1u) list[at++] = uint16_t((lane << 5) | (__ffs(m) - 1));
    end = e.y + __popc(e.x);
  }
  __syncwarp();
  return __shfl_sync(DC_FULL, end, 15);
}

// The particle solver (dual_contouring.rs:429-458), a lane per cell and
// `split` warps per leaf.  Its 50 dependent iterations set the time, so
// the quotients by the number of crossings share one reciprocal and a leaf's
// cells are spread over two warps or more.  (Crossings copied to shared memory instead
// of read through L1: 0.40 against 0.14 ms on 57 k leaves, the 9 KB per warp
// leave too few warps resident.)
__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_cell_points(DcVol V, uint64_t n, const uint2* __restrict__ em,
                                                                  const uint32_t* __restrict__ coff,
                                                                  const float* __restrict__ pts,
                                                                  const uint2* __restrict__ cellm,
                                                                  const uint32_t* __restrict__ celloff,
                                                                  float* __restrict__ cells, uint32_t split) {
  __shared__ uint16_t list[DC_WARPS][512];
  __shared__ int nbs[DC_WARPS][27];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint64_t gw = blockIdx.x * uint64_t(DC_WARPS) + wi, l = gw / split;
  if (l >= n) return;
  const uint32_t cnt = list_cells(cellm, l, list[wi]), first = 32 * uint32_t(gw % split);
  if (cnt <= first) return;
  if (lane < 27) nbs[wi][lane] = V.nbr[l * 27 + lane];
  __syncwarp();
  const int* nb = nbs[wi];
  for (uint32_t ci = first + lane; ci < cnt; ci += 32 * split) {
    const int o = list[wi][ci];
    const int x = o >> 6, y = (o >> 3) & 7, z = o & 7;
    const float2* ip[12];
    int np = 0;
    float c0 = 0.f, c1 = 0.f, c2 = 0.f;
    for (int e = 0; e < 12; ++e) {
      const float* q = edge_point(nb, em, coff, pts, x + c_edges[e][0], y + c_edges[e][1], z + c_edges[e][2],
                                  c_edges[e][3]);
      if (!q) continue;
      ip[np++] = reinterpret_cast<const float2*>(q);
      c0 = fadd(c0, q[0]);
      c1 = fadd(c1, q[1]);
      c2 = fadd(c2, q[2]);
    }
    const float len = __int2float_rn(np), inv = __frcp_rn(len);
    auto over = [&](float a) {  // a / len
      return a == 0.0f ? a : mdiv_range(a) ? mdiv(a, len, inv) : fdiv(a, len);
    };
    c0 = over(c0);
    c1 = over(c1);
    c2 = over(c2);
    for (int it = 0; it < 50; ++it) {
      float f0 = 0.f, f1 = 0.f, f2 = 0.f;
#pragma unroll 2
      for (int i = 0; i < np; ++i) {
        const float2 a = __ldg(ip[i]), b = __ldg(ip[i] + 1), c = __ldg(ip[i] + 2);
        const float n0 = b.y, n1 = c.x, n2 = c.y;
        const float d = fadd(fadd(fmul(n0, fsub(c0, a.x)), fmul(n1, fsub(c1, a.y))), fmul(n2, fsub(c2, b.x)));
        f0 = fadd(f0, fmul(fmul(n0, -1.0f), d));
        f1 = fadd(f1, fmul(fmul(n1, -1.0f), d));
        f2 = fadd(f2, fmul(fmul(n2, -1.0f), d));
      }
      const float damping = fsub(1.0f, fdiv(__int2float_rn(it), 50.0f));
      c0 = fadd(c0, over(fmul(f0, damping)));
      c1 = fadd(c1, over(fmul(f1, damping)));
      c2 = fadd(c2, over(fmul(f2, damping)));
      if (fadd(fadd(fmul(f0, f0), fmul(f1, f1)), fmul(f2, f2)) < 1e-6f) break;
    }
    float* out = cells + uint64_t(celloff[l] + ci) * 3;
    out[0] = c0;
    out[1] = c1;
    out[2] = c2;
  }
}

// Eigen-decomposition of a symmetric 3x3 matrix by cyclic Jacobi rotations
// (Jacobi 1846; Rutishauser's update): a is overwritten, w = eigenvalues,
// columns of V = eigenvectors.
__device__ __forceinline__ void sym3_jacobi(double a[3][3], double V[3][3], double w[3]) {
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) V[r][c] = r == c ? 1.0 : 0.0;
  const int P[3] = {0, 0, 1}, Q[3] = {1, 2, 2};
  for (int sweep = 0; sweep < 24; ++sweep) {
    const double off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
    const double dia = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
    if (off <= 1e-30 * dia || off == 0.0) break;
    for (int k = 0; k < 3; ++k) {
      const int p = P[k], q = Q[k];
      const double apq = a[p][q];
      if (apq == 0.0) continue;
      const double theta = (a[q][q] - a[p][p]) / (2.0 * apq);
      const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
      const double c = 1.0 / sqrt(t * t + 1.0), s = t * c, tau = s / (1.0 + c);
      a[p][p] -= t * apq;
      a[q][q] += t * apq;
      a[p][q] = a[q][p] = 0.0;
      for (int r = 0; r < 3; ++r) {
        if (r != p && r != q) {
          const double arp = a[r][p], arq = a[r][q];
          a[r][p] = a[p][r] = arp - s * (arq + tau * arp);
          a[r][q] = a[q][r] = arq + s * (arp - tau * arq);
        }
        const double vrp = V[r][p], vrq = V[r][q];
        V[r][p] = vrp - s * (vrq + tau * vrp);
        V[r][q] = vrq + s * (vrp - tau * vrq);
      }
    }
  }
  for (int k = 0; k < 3; ++k) w[k] = a[k][k];
}

// QEF mode (no reference counterpart): the point minimising
// sum_i (n_i . (x - p_i))^2 over the cell's crossings p_i with normals n_i,
// taken as m + pinv(A^T A) (A^T b - A^T A m) around the crossings' mass
// point m, with eigenvalues below QEF_TRUNC of the largest dropped; all in
// double.
constexpr double QEF_TRUNC = 0.1;

__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_cell_qef(DcVol V, uint64_t n, const uint2* __restrict__ em,
                                                               const uint32_t* __restrict__ coff,
                                                               const float* __restrict__ pts,
                                                               const uint2* __restrict__ cellm,
                                                               const uint32_t* __restrict__ celloff,
                                                               float* __restrict__ cells, uint32_t split) {
  __shared__ uint16_t list[DC_WARPS][512];
  __shared__ int nbs[DC_WARPS][27];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint64_t gw = blockIdx.x * uint64_t(DC_WARPS) + wi, l = gw / split;
  if (l >= n) return;
  const uint32_t cnt = list_cells(cellm, l, list[wi]), first = 32 * uint32_t(gw % split);
  if (cnt <= first) return;
  if (lane < 27) nbs[wi][lane] = V.nbr[l * 27 + lane];
  __syncwarp();
  const int* nb = nbs[wi];
  for (uint32_t ci = first + lane; ci < cnt; ci += 32 * split) {
    const int o = list[wi][ci];
    const int x = o >> 6, y = (o >> 3) & 7, z = o & 7;
    double mp[3] = {0.0, 0.0, 0.0}, ata[3][3] = {{0.0}}, atb[3] = {0.0, 0.0, 0.0};
    int np = 0;
    for (int e = 0; e < 12; ++e) {
      const float* q = edge_point(nb, em, coff, pts, x + c_edges[e][0], y + c_edges[e][1], z + c_edges[e][2],
                                  c_edges[e][3]);
      if (!q) continue;
      ++np;
      const double p[3] = {q[0], q[1], q[2]}, nn[3] = {q[3], q[4], q[5]};
      const double d = nn[0] * p[0] + nn[1] * p[1] + nn[2] * p[2];
      for (int r = 0; r < 3; ++r) {
        mp[r] += p[r];
        atb[r] += nn[r] * d;
        for (int c = 0; c < 3; ++c) ata[r][c] += nn[r] * nn[c];
      }
    }
    for (int r = 0; r < 3; ++r) mp[r] /= double(np);
    double rhs[3];
    for (int r = 0; r < 3; ++r) rhs[r] = atb[r] - (ata[r][0] * mp[0] + ata[r][1] * mp[1] + ata[r][2] * mp[2]);
    double a[3][3], Vm[3][3], w[3];
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) a[r][c] = ata[r][c];
    sym3_jacobi(a, Vm, w);
    const double wmax = fmax(fabs(w[0]), fmax(fabs(w[1]), fabs(w[2])));
    double xs[3] = {mp[0], mp[1], mp[2]};
    for (int k = 0; k < 3; ++k) {
      if (!(fabs(w[k]) > QEF_TRUNC * wmax)) continue;
      const double proj = (Vm[0][k] * rhs[0] + Vm[1][k] * rhs[1] + Vm[2][k] * rhs[2]) / w[k];
      for (int r = 0; r < 3; ++r) xs[r] += proj * Vm[r][k];
    }
    float* out = cells + uint64_t(celloff[l] + ci) * 3;
    out[0] = float(xs[0]);
    out[1] = float(xs[1]);
    out[2] = float(xs[2]);
  }
}

__device__ __forceinline__ const float* cell_point(const int* nb, const uint2* cellm, const uint32_t* celloff,
                                                   const float* cells, int x, int y, int z) {
  const int k = ((x >> 3) + 1) * 9 + ((y >> 3) + 1) * 3 + ((z >> 3) + 1);
  const int l = nb[k];
  if (l < 0) return nullptr;
  const int r = ranked(cellm + uint64_t(l) * 16, ((x & 7) << 6) | ((y & 7) << 3) | (z & 7));
  return r < 0 ? nullptr : cells + uint64_t(celloff[l] + uint32_t(r)) * 3;
}

__device__ __forceinline__ bool degenerate(const float* a, const float* b, const float* c) {
  const float e0 = fsub(b[0], a[0]), e1 = fsub(b[1], a[1]), e2 = fsub(b[2], a[2]);
  const float f0 = fsub(c[0], a[0]), f1 = fsub(c[1], a[1]), f2 = fsub(c[2], a[2]);
  const float x = fsub(fmul(e1, f2), fmul(e2, f1)), y = fsub(fmul(e2, f0), fmul(e0, f2)),
              z = fsub(fmul(e0, f1), fmul(e1, f0));
  return fadd(fadd(fmul(x, x), fmul(y, y)), fmul(z, z)) == 0.0f;
}

// The two triangles of every quad around a sign-change edge
// (dual_contouring.rs:93-139), scaled by the voxel size, minus exactly
// degenerate ones (dual_contouring.rs:62-79).  One warp per leaf lists its
// crossings by voxel, then direction, and takes them 32 at a time.  Count
// pass (WRITE false): vcount[l] = triangles of leaf l.  Write pass: they go
// out from tris + voff[l] in list order, a round's triangles through shared
// memory so that the stores are coalesced.
template <bool WRITE>
__global__ void __launch_bounds__(32 * DC_WARPS) k_dc_quads(DcVol V, uint64_t n, const uint2* __restrict__ em,
                                                            const uint32_t* __restrict__ coff,
                                                            const uint2* __restrict__ cellm,
                                                            const uint32_t* __restrict__ celloff,
                                                            const float* __restrict__ cells, float h,
                                                            uint64_t* __restrict__ vcount,
                                                            const uint64_t* __restrict__ voff,
                                                            float* __restrict__ tris) {
  __shared__ uint16_t list[DC_WARPS][3 * 512];
  __shared__ int nbs[DC_WARPS][27];
  __shared__ float stage[WRITE ? DC_WARPS : 1][WRITE ? 64 * 9 : 1];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const uint64_t l = blockIdx.x * uint64_t(DC_WARPS) + wi;
  if (l >= n) return;
  if (!WRITE && l == n - 1 && lane == 0) vcount[n] = 0;
  const uint32_t cnt = coff[l * 3 + 3] - coff[l * 3];
  if (cnt == 0) {
    if (!WRITE && lane == 0) vcount[l] = 0;
    return;
  }
  if (lane < 27) nbs[wi][lane] = V.nbr[l * 27 + lane];
  if (lane < 16) {
    const uint2 e0 = em[l * 48 + lane], e1 = em[l * 48 + 16 + lane], e2 = em[l * 48 + 32 + lane];
    uint32_t at = e0.y + e1.y + e2.y;
    for (uint32_t m = e0.x | e1.x | e2.x; m; m &= m - 1u) {
      const int b = __ffs(m) - 1, o = (lane << 5) | b;
      if ((e0.x >> b) & 1u) list[wi][at++] = uint16_t(o << 2);
      if ((e1.x >> b) & 1u) list[wi][at++] = uint16_t((o << 2) | 1);
      if ((e2.x >> b) & 1u) list[wi][at++] = uint16_t((o << 2) | 2);
    }
  }
  __syncwarp();
  const int* nb = nbs[wi];
  const uint32_t sg = lane < 16 ? V.sgn[l * 16 + lane] : 0u;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t run = WRITE ? voff[l] : 0;
  uint32_t total = 0;
  for (uint32_t base = 0; base < cnt; base += 32) {
    const bool have = base + lane < cnt;
    const int code = have ? list[wi][base + lane] : 0, o = code >> 2, dir = code & 3;
    const bool neg = (__shfl_sync(DC_FULL, sg, o >> 5) >> (o & 31)) & 1u;
    const int x = o >> 6, y = (o >> 3) & 7, z = o & 7;
    float q[4][3];
    bool ok = have;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float* p = ok ? cell_point(nb, cellm, celloff, cells, x + c_cells[dir][c][0], y + c_cells[dir][c][1],
                                       z + c_cells[dir][c][2])
                          : nullptr;
      ok = ok && p != nullptr;
      if (ok)
        for (int i = 0; i < 3; ++i) q[c][i] = fmul(p[i], h);
    }
    // [p0, p1, p2, p2, p3, p0], with (1,2) and (4,5) swapped when the first end is inside
    const float* t0[3] = {q[0], neg ? q[2] : q[1], neg ? q[1] : q[2]};
    const float* t1[3] = {q[2], neg ? q[0] : q[3], neg ? q[3] : q[0]};
    const bool k0 = ok && !degenerate(t0[0], t0[1], t0[2]), k1 = ok && !degenerate(t1[0], t1[1], t1[2]);
    const unsigned m0 = __ballot_sync(DC_FULL, k0), m1 = __ballot_sync(DC_FULL, k1);
    const uint32_t sum = __popc(m0) + __popc(m1);
    if (WRITE) {
      float* d = stage[WRITE ? wi : 0] + 9 * (__popc(m0 & lt) + __popc(m1 & lt));
      if (k0) {
        for (int v = 0; v < 3; ++v)
          for (int i = 0; i < 3; ++i) d[3 * v + i] = t0[v][i];
        d += 9;
      }
      if (k1)
        for (int v = 0; v < 3; ++v)
          for (int i = 0; i < 3; ++i) d[3 * v + i] = t1[v][i];
      __syncwarp();
      for (uint32_t i = lane; i < 9 * sum; i += 32) tris[run * 9 + i] = stage[WRITE ? wi : 0][i];
      __syncwarp();
      run += sum;
    } else {
      total += sum;
    }
  }
  if (!WRITE && lane == 0) vcount[l] = total;
}

// Launches shared with dc_noalloc.cu (tiles: the volume has active tiles).
static inline unsigned dc_blocks(uint64_t n) { return unsigned((n + DC_WARPS - 1) / DC_WARPS); }

// Warps per leaf of the passes that compute values: `least` where the leaves
// fill the SMs, doubled up to 16 (all 512 cells of a leaf at once) while there
// are 64 warps or fewer to an SM, since a warp goes through a crowded leaf's
// cells 32 at a time.  With one warp (two for the particles) throughout
// against this, cell pass in ms, QEF / particles: 64 crowded leaves 0.774 /
// 0.304 against 0.071 / 0.055; 1,440 of a surface 0.301 / 0.096 against 0.200 /
// 0.069; 5,858 (above the line) 0.66 / 0.10 on both sides.
static uint32_t dc_split(uint64_t n, uint32_t least) {
  int device = 0, n_sm = 0;
  BS_CUDA(cudaGetDevice(&device));
  BS_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device));
  uint32_t split = least;
  while (split < 16 && n * split * 2 <= uint64_t(n_sm) * 64) split *= 2;
  return split;
}

void launch_dc_prepare(const DcVol& V, LeafHash hash, uint64_t n, int* nbr, uint32_t* sgn, cudaStream_t s) {
  k_dc_neighbours<<<unsigned((27 * n + 255) / 256), 256, 0, s>>>(V.org, hash, n, nbr);
  k_dc_signs<<<dc_blocks(n), 32 * DC_WARPS, 0, s>>>(V.val, n, sgn);
}
void launch_dc_masks(bool tiles, const DcVol& V, uint64_t n, uint2* em, uint32_t* ccnt, uint2* cellm, uint32_t* cellc,
                     cudaStream_t s) {
  if (tiles)
    k_dc_masks<true><<<dc_blocks(n), 32 * DC_WARPS, 0, s>>>(V, n, em, ccnt, cellm, cellc);
  else
    k_dc_masks<false><<<dc_blocks(n), 32 * DC_WARPS, 0, s>>>(V, n, em, ccnt, cellm, cellc);
}
void launch_dc_edge_points(bool tiles, const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff, float* pts,
                           DcStats* st, cudaStream_t s) {
  const uint32_t split = dc_split(n, 1);
  if (tiles)
    k_dc_edge_points<true><<<dc_blocks(n * split), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, pts, st, split);
  else
    k_dc_edge_points<false><<<dc_blocks(n * split), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, pts, st, split);
}
void launch_dc_cell_points(int mode, const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff,
                           const float* pts, const uint2* cellm, const uint32_t* celloff, float* cells,
                           cudaStream_t s) {
  const uint32_t split = dc_split(n, mode == 1 ? 1 : 2);
  if (mode == 1)
    k_dc_cell_qef<<<dc_blocks(n * split), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, pts, cellm, celloff, cells, split);
  else
    k_dc_cell_points<<<dc_blocks(n * split), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, pts, cellm, celloff, cells, split);
}
void launch_dc_quads(const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff, const uint2* cellm,
                     const uint32_t* celloff, const float* cells, float h, uint64_t* vcount, const uint64_t* voff,
                     float* tris, cudaStream_t s) {
  if (tris)
    k_dc_quads<true><<<dc_blocks(n), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, cellm, celloff, cells, h, nullptr, voff,
                                                           tris);
  else
    k_dc_quads<false><<<dc_blocks(n), 32 * DC_WARPS, 0, s>>>(V, n, em, coff, cellm, celloff, cells, h, vcount, nullptr,
                                                            nullptr);
}

static bool has_active_tiles(const bs_volume* v) { return v->n_tiles != 0; }

void dual_contour_impl(bs_ctx* ctx, bs_volume* v, float voxel_size, int mode) {
  if (v->dc_valid && v->dc_h == voxel_size && v->dc_mode == mode) return;
  cudaStream_t s = ctx->stream;
  dfree(ctx, v->d_dc_tris);
  v->d_dc_tris = nullptr;
  v->n_dc_tris = 0;
  const uint64_t n = v->n_leaves;
  if (n == 0) {
    v->dc_valid = true;
    v->dc_h = voxel_size;
    v->dc_mode = mode;
    return;
  }
  LeafHashBuf hb, h1, h2;
  hb.build(ctx, v->d_origins, n, n);
  DBuf<int> nbr(ctx, 27 * n);
  DBuf<uint32_t> sgn(ctx, 16 * n);
  DcVol V{v->d_origins, v->d_values, v->d_masks, sgn.p, nbr.p, TileLookup{}};
  if (has_active_tiles(v)) {
    // The reference stops at active tiles (todo!(), dual_contouring.rs:139,
    // 186, 347).  Here the passes still visit the leaves only and read every
    // neighbour, cell corner and gradient stencil voxel as the tree's `at`
    // returns it, so a voxel of an active tile has the tile's value.
    const Upper* u = v->upper;
    if (!u) fail(BS_ERR_UNSUPPORTED, "dual contouring: tiles without internal levels");
    h1.build(ctx, u->l1.d_key, u->l1.n, u->l1.n);
    h2.build(ctx, u->l2.d_key, u->l2.n, u->l2.n);
    V.tiles = TileLookup{h1.h, h2.h, u->l1.d_state, u->l1.d_tile, u->l2.d_state, u->l2.d_tile, 1};
  }
  DBuf<DcStats> st(ctx, 1);
  BS_CUDA(cudaMemsetAsync(st.p, 0, sizeof(DcStats), s));
  ctx->launches++;  // two kernels
  BS_KERNEL(ctx, "k_dc_prepare", launch_dc_prepare(V, hb.h, n, nbr.p, sgn.p, s));
  // crossings and cells
  DBuf<uint2> em(ctx, n * 3 * 16), cellm(ctx, n * 16);
  DBuf<uint32_t> ccnt(ctx, n * 3 + 1), coff(ctx, n * 3 + 1), cellc(ctx, n + 1), celloff(ctx, n + 1);
  BS_KERNEL(ctx, "k_dc_masks", launch_dc_masks(V.tiles.any, V, n, em.p, ccnt.p, cellm.p, cellc.p, s));
  scan_e(ctx, ccnt.p, coff.p, n * 3 + 1);
  scan_e(ctx, cellc.p, celloff.p, n + 1);
  uint32_t* sizes = static_cast<uint32_t*>(ctx->h_pinned);
  BS_CUDA(cudaMemcpyAsync(sizes, coff.p + n * 3, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  BS_CUDA(cudaMemcpyAsync(sizes + 1, celloff.p + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  BS_CUDA(cudaStreamSynchronize(s));
  const uint32_t ne = sizes[0], nc = sizes[1];
  DBuf<float> pts(ctx, uint64_t(ne) * 6), cells(ctx, uint64_t(nc) * 3);
  BS_KERNEL(ctx, "k_dc_edge_points", launch_dc_edge_points(V.tiles.any, V, n, em.p, coff.p, pts.p, st.p, s));
  BS_KERNEL(ctx, mode == 1 ? "k_dc_cell_qef" : "k_dc_cell_points",
            launch_dc_cell_points(mode, V, n, em.p, coff.p, pts.p, cellm.p, celloff.p, cells.p, s));
  // quads
  DBuf<uint64_t> vcnt(ctx, n + 1), voff(ctx, n + 1);
  BS_KERNEL(ctx, "k_dc_quads_count", launch_dc_quads(V, n, em.p, coff.p, cellm.p, celloff.p, cells.p, voxel_size, vcnt.p, nullptr, nullptr, s));
  scan_e(ctx, vcnt.p, voff.p, n + 1);
  uint64_t* nt_h = static_cast<uint64_t*>(ctx->h_pinned);
  DcStats* st_h = reinterpret_cast<DcStats*>(nt_h + 1);
  BS_CUDA(cudaMemcpyAsync(nt_h, voff.p + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  BS_CUDA(cudaMemcpyAsync(st_h, st.p, sizeof(DcStats), cudaMemcpyDeviceToHost, s));
  BS_CUDA(cudaStreamSynchronize(s));
  const uint64_t nt = *nt_h;
  if (st_h->error == 1)
    fail(BS_ERR_UNSUPPORTED, "dual contouring: gradient at a voxel with no active neighbour on an axis (the reference stops with unreachable!())");
  v->d_dc_tris = dalloc<float>(ctx, nt * 9);
  if (nt)
    BS_KERNEL(ctx, "k_dc_quads", launch_dc_quads(V, n, em.p, coff.p, cellm.p, celloff.p, cells.p, voxel_size, nullptr, voff.p, v->d_dc_tris, s));
  v->n_dc_tris = nt;
  v->dc_valid = true;
  v->dc_h = voxel_size;
  v->dc_mode = mode;
  ctx->last_stats[6] = ne;
  ctx->last_stats[7] = nc;
  ctx->last_stats[8] = BS_STATS_DUAL_CONTOURING;
}

}  // namespace bs
