// lbvh.h -- linear BVH over triangles or sphere AABBs (see lbvh.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

struct PrimBox { float lo[3], hi[3]; };

// 64-byte node: a = (c0.lo.xyz, c0.hi.x), b = (c0.hi.yz, c1.lo.xy),
// c = (c1.lo.z, c1.hi.xyz), d = (child0, child1); child < 0 is leaf ~child.
struct __align__(16) BvhNode { float4 a, b, c; int4 d; };

struct Lbvh {
  int n = 0;               // primitives
  BvhNode *nodes = nullptr;  // n-1 internal nodes, root = 0
  int *perm = nullptr;     // sorted position -> original primitive index
  float4 *prims = nullptr; // 3 float4 per sorted primitive (see lbvh.cu)
  const float *wide = nullptr;  // 32-wide nodes (wide_bvh_build), root = 0
  int n_wide = 0;
};

// 32-wide form of a binary hierarchy, one node per warp-wide visit: six
// planes of 32 floats (lo.x, hi.x, lo.y, hi.y, lo.z, hi.z of each child) and
// 32 child references (>= 0 wide node, < 0 leaf of sorted primitive ~c; an
// unused slot has an inverted box).
#define AMS_WIDE_WORDS (7 * 32)
#define AMS_WIDE_LEVELS 64
// device memory of the wide nodes of n primitives and of their build
size_t wide_bvh_bytes(int n);
size_t wide_bvh_scratch_bytes(int n);
// enqueue the passes first .. last - 1 (one per level) of the collapse of
// `b`; scratch starts with AMS_WIDE_LEVELS + 1 node counts (per level, then an
// overflow flag), which the caller reads back to see whether a level is left
cudaError_t wide_bvh_build(const Lbvh &b, int first, int last, float *wide, char *scratch,
                           cudaStream_t st);
int wide_bvh_cap(int n);

size_t lbvh_scratch_bytes(int n);
size_t lbvh_output_bytes(int n);
cudaError_t lbvh_build_triangles(Lbvh &out, const float *tris, int n, char *scratch,
                                 char *outbuf, cudaStream_t st);
// with `skip` (device) and a value other than 0 there, nothing is built
cudaError_t lbvh_build_spheres(Lbvh &out, const float *pos, const float *aabb, int n,
                               char *scratch, char *outbuf, const int *skip, cudaStream_t st);
// adopts a hierarchy built on the host (bvh_sah.h) for triangles already on
// the device: copies nodes and perm into outbuf (the caller keeps the host
// arrays alive until the stream has run) and packs the sorted triangles
cudaError_t lbvh_from_host(Lbvh &out, const float *tris, int n, const BvhNode *h_nodes,
                           const int *h_perm, char *outbuf, cudaStream_t st);
cudaError_t sphere_aabbs(const float *pos, int n, float r, float *aabb, cudaStream_t st);
