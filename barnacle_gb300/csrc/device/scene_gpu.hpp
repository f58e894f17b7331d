// Device side of bn_scene_upload (k_scene.cu): triangle boxes, permuted triangles and areas of a mesh
// whose BLAS is built on the GPU, and the wide records of every BLAS.
#pragma once
#include <cuda_runtime.h>

#include "../../../include/barnacle_gpu.h"

namespace bn {

// bounds[6 t]: the box of triangle t, MinNative/MaxNative over its vertices
cudaError_t scene_launch_boxes(const float* vertices, const int* indices, int n, float* bounds, cudaStream_t st);
// tris[3 k], areas[k]: triangle perm[k] as the walk reads it (dev_types.cuh) and its object-space area
cudaError_t scene_launch_tris(const float* vertices, const int* indices, const int* tri_material, const int* perm, int n,
                              float4* tris, float* areas, cudaStream_t st);
// areas[k] -> areas[k] / sum (1 / n where the sum is zero), in place
cudaError_t scene_launch_pdf(float* areas, int n, float sum, cudaStream_t st);

// The wide records of the BLASes in nodes[base .. base + n): their meshes' first nodes are
// mesh_base[0 .. n_meshes), ascending; odd[i] is the parity of node base + i's depth.
struct WideParams {
  const float4* nodes;
  int base, n;
  const unsigned char* odd;
  const int* mesh_base;
  int n_meshes;
  int leaf_bits;    // leaf_count_bits of the largest BVH
  int* rank;        // n: records before the node in its block of 1,024 nodes
  int* sums;        // n / 1,024 + 2: records before each block, then their number
  int* flags;       // bit 0: some box does not contain its children's; bit 1: some leaf does not fit its code
  int* roots;       // n_meshes: record of the mesh's root, -1 where it is a leaf
  float4* records;  // 8 per record
  int first_record; // index of the first of them
};
// rank and sums (sums[blocks] = the number of records)
cudaError_t scene_launch_wide_count(const WideParams& p, cudaStream_t st);
// records, roots, flags
cudaError_t scene_launch_wide_fill(const WideParams& p, cudaStream_t st);

}  // namespace bn
