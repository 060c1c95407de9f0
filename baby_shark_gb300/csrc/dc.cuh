// Shared declarations of the dual-contouring kernels (defined in dc.cu, also
// launched by the allocation-free entry point in dc_noalloc.cu).
#pragma once

#include "leaf_hash.cuh"
#include "tiles.cuh"

namespace bs {

struct DcVol {
  const int4* org;
  const float* val;
  const uint32_t* msk;
  const uint32_t* sgn;  // [n][16] sign bits of the values
  const int* nbr;       // [n][27] neighbour leaves
  TileLookup tiles;  // active tiles, read where a voxel lies outside every leaf (tiles.any == 0: none)
};

struct DcStats {
  int error;  // 1: gradient with no neighbours
};

// The passes (tiles: the volume has active tiles, read through the tree's
// `at`).  Masks come with ranks: (word, set bits in the words before it).
void launch_dc_prepare(const DcVol& V, LeafHash hash, uint64_t n, int* nbr, uint32_t* sgn, cudaStream_t s);
void launch_dc_masks(bool tiles, const DcVol& V, uint64_t n, uint2* em, uint32_t* ccnt, uint2* cellm, uint32_t* cellc,
                     cudaStream_t s);
void launch_dc_edge_points(bool tiles, const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff, float* pts,
                           DcStats* st, cudaStream_t s);
// mode 0: the particle solver; 1: the float64 QEF vertex
void launch_dc_cell_points(int mode, const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff,
                           const float* pts, const uint2* cellm, const uint32_t* celloff, float* cells,
                           cudaStream_t s);
// counts triangles per leaf (tris null) or writes them from voff
void launch_dc_quads(const DcVol& V, uint64_t n, const uint2* em, const uint32_t* coff, const uint2* cellm,
                     const uint32_t* celloff, const float* cells, float h, uint64_t* vcount, const uint64_t* voff,
                     float* tris, cudaStream_t s);

}  // namespace bs
