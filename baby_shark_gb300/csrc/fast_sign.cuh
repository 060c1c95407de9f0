// Filter pass of the signs on this library's tree (fast_sign.cu).
#pragma once

#include "bs_internal.cuh"

namespace bs {

struct FastSignMesh {
  uint32_t inode_base, tri_base, n_tri;
  float h, beta, thresh;
};

// Filter records of K meshes' trees: 4 float4 per node (fast_sign.cu), the
// n_internal internal nodes first, then the leaves.
void fast_filter_records(bs_ctx* ctx, const float4* inode, uint64_t n_internal, const uint32_t* d_inode_base,
                         const float4* leaf, uint64_t nt, const uint32_t* d_tri_base, int K,
                         const FastSignMesh* d_meshes, float4* frec);

// Consecutive active voxels of a mesh that one warp takes.
constexpr int FAST_SIGN_SPAN = 256;

// Signs the active voxels of K meshes as wn_warp would (m2v.cu), except those
// of the warps it lists in rest (by their first index into act; count in
// *n_rest): span_base[m] .. span_base[m + 1] are mesh m's spans of
// FAST_SIGN_SPAN voxels of act[act_base[m], act_base[m + 1]).  Mesh m's node
// visits, far fields and solid angles of the warps' cuts are added to
// counts[m * count_stride] and the two after it.
void fast_sign(bs_ctx* ctx, const uint32_t* act, const uint32_t* d_act_base, const uint32_t* d_span_base,
               uint32_t n_spans, int K, const FastSignMesh* d_meshes, const int4* origins, float* values,
               const float4* frec, uint64_t n_internal, const float4* inode, const float4* leaf, uint32_t* rest,
               uint32_t* n_rest, unsigned long long* d_counts, uint32_t count_stride);

}  // namespace bs
