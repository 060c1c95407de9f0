// Filter pass of the signs on this library's tree (fast_sign.cu).
#pragma once

#include "bs_internal.cuh"

namespace bs {

struct FastSignMesh {
  uint32_t inode_base, tri_base, n_tri;
  float h, beta, thresh;
  float band;  // twice the most that a band voxel is from the mesh
};

// Filter records of K meshes' trees: 4 float4 per node (fast_sign.cu), the
// n_internal internal nodes first, then the leaves.
void fast_filter_records(bs_ctx* ctx, const float4* inode, uint64_t n_internal, const uint32_t* d_inode_base,
                         const float4* leaf, uint64_t nt, const uint32_t* d_tri_base, int K,
                         const FastSignMesh* d_meshes, float4* frec);

// Squared distance of the far test of the order-2 traversal, the same float32
// operations wherever its cut is taken (the order-3 traversal has no filter).
__device__ __forceinline__ float cut_dist2(float rx, float ry, float rz) {
  return __fmaf_rn(rz, rz, __fmaf_rn(rx, rx, __fmul_rn(ry, ry)));
}

// Consecutive active voxels of a mesh that one warp takes, for n_act of them
// in all.
uint32_t fast_sign_span(bs_ctx* ctx, uint64_t n_act);

// Signs the active voxels of K meshes as wn_warp would (m2v.cu), except those
// of the warps that it does not come to, done[s] of span s's being behind it
// (a mesh out of the filter's range, or one of which it settles too little),
// and of those that it lists (by their first index into act) in rest: n_rest[0] of
// them from rest[0] up, n_rest[1] from rest[n_warps - 1] down.  span_base[m] ..
// span_base[m + 1] are mesh m's spans of `span` voxels of
// act[act_base[m], act_base[m + 1]).  Mesh m's node visits, far fields and
// solid angles of the warps' cuts are added to counts[m * count_stride] and
// the two after it; those of the n_rest[1] warps and of the ones that it did
// not come to are left to their traversal.  n_rest[2] counts those that it
// came to; n_rest, done and d_tally (one per mesh) are zero before.
void fast_sign(bs_ctx* ctx, const uint32_t* act, const uint32_t* d_act_base, const uint32_t* d_span_base,
               uint32_t span, uint32_t n_spans, int K, const FastSignMesh* d_meshes, const int4* origins, float* values,
               const float4* frec, uint64_t n_internal, const float4* inode, const float4* leaf, uint32_t* rest,
               uint32_t n_warps, uint32_t* n_rest, uint8_t* done, unsigned long long* d_tally,
               unsigned long long* d_counts, uint32_t count_stride);

}  // namespace bs
