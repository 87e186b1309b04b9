// lbvh.cu -- linear BVH builder (Karras 2012, "Maximizing parallelism in
// the construction of BVHs, octrees and k-d trees"), GB300 version.
//
// Replaces the OptiX GAS builds of the reference (optixPathTracer.cpp:382-546:
// one triangle GAS, one custom-AABB GAS per sphere set) with:
//   1. centroid bounds (one CTA reduction),
//   2. 30-bit Morton codes of the centroids scaled to a cube, with the
//      primitive index in the low word (bit 30 set for primitives larger
//      than a quarter of the scene),
//   3. a sort of the keys: bitonic in shared memory up to 16,384 keys, else
//      a stable LSD radix sort (one 1024-thread CTA, 4-bit digits, warp
//      ballots for the in-tile ranks),
//   4. the Karras hierarchy, one thread per internal node,
//   5. a bottom-up refit with per-node arrival counters.
// Node layout: both children's boxes live in the parent (64 bytes per node,
// four 16-byte loads), boxes widened outward so that node culling is
// conservative.  Leaves hold one primitive; a child reference c < 0 is the
// leaf of sorted primitive ~c.
#include <algorithm>

#include "ams_common.cuh"
#include "lbvh.h"

namespace {

__device__ __forceinline__ float widen_lo(float v) {
  return nextafterf(v - (1e-6f + 1e-6f * fabsf(v)), -3.0e38f);
}
__device__ __forceinline__ float widen_hi(float v) {
  return nextafterf(v + (1e-6f + 1e-6f * fabsf(v)), 3.0e38f);
}

// centroid bounds of the boxes, by one CTA of up to 1024 threads
__device__ __forceinline__ void centroid_bounds(const PrimBox *boxes, int n, float *out6) {
  __shared__ float s[6][32];
  float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const PrimBox b = boxes[i];
    for (int k = 0; k < 3; k++) {
      float c = 0.5f * (b.lo[k] + b.hi[k]);
      lo[k] = fminf(lo[k], c);
      hi[k] = fmaxf(hi[k], c);
    }
  }
  for (int k = 0; k < 3; k++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
    }
  }
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0)
    for (int k = 0; k < 3; k++) { s[k][w] = lo[k]; s[3 + k][w] = hi[k]; }
  __syncthreads();
  if (w == 0) {
    int nw = blockDim.x >> 5;
    for (int k = 0; k < 6; k++) {
      float v = l < nw ? s[k][l] : (k < 3 ? 3.0e38f : -3.0e38f);
      for (int o = 16; o > 0; o >>= 1) {
        float u = __shfl_xor_sync(0xffffffffu, v, o);
        v = k < 3 ? fminf(v, u) : fmaxf(v, u);
      }
      if (l == 0) out6[k] = v;
    }
  }
}

__global__ void k_bounds(const PrimBox *boxes, int n, float *out6, const int *skip) {
  if (skip && *skip) return;
  centroid_bounds(boxes, n, out6);
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__device__ __forceinline__ uint64_t morton_key(const PrimBox &b, int i, const float *b6) {
  uint32_t q[3];
  // one scale for all axes (the largest centroid extent): a flat room or
  // building gets its first splits across its long sides instead of cutting
  // its 3 m height as finely as its 45 m width
  const float cube = fmaxf(fmaxf(b6[3] - b6[0], b6[4] - b6[1]), b6[5] - b6[2]);
  for (int k = 0; k < 3; k++) {
    float c = 0.5f * (b.lo[k] + b.hi[k]);
    float u = cube > 0.0f ? (c - b6[k]) / cube : 0.5f;
    u = fminf(fmaxf(u, 0.0f), 1.0f);
    q[k] = (uint32_t)fminf(u * 1024.0f, 1023.0f);
  }
  uint32_t m = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
  // Primitives larger than a quarter of the scene (floors, walls) get a bit
  // above the Morton code, so the root splits them off into their own
  // subtree instead of inflating the boxes of every node on the way to the
  // small ones around their centroids.  Culling only: results do not change.
  float bext = 0.0f, sext = 0.0f;
  for (int k = 0; k < 3; k++) {
    bext = fmaxf(bext, b.hi[k] - b.lo[k]);
    sext = fmaxf(sext, b6[3 + k] - b6[k]);
  }
  if (sext > 0.0f && bext > 0.25f * sext) m |= 1u << 30;
  return ((uint64_t)m << 32) | (uint32_t)i;
}
__global__ void k_morton(const PrimBox *boxes, int n, const float *b6, uint64_t *keys,
                         const int *skip) {
  if (skip && *skip) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) keys[i] = morton_key(boxes[i], i, b6);
}

// Stable LSD radix sort of 64-bit items on their upper 32 bits (30 used),
// one CTA of 1024 threads, tiles of 1024 items in order.
__global__ void __launch_bounds__(1024) k_sort(uint64_t *a, uint64_t *b, int n, const int *skip) {
  if (skip && *skip) return;
  __shared__ int hist[16];
  __shared__ int base[16];
  __shared__ int wcnt[32][16];
  __shared__ int woff[32][16];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t *in = a, *out = b;
  for (int pass = 0; pass < 8; pass++) {
    const int shift = 32 + 4 * pass;
    if (tid < 16) hist[tid] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += 1024) atomicAdd(&hist[(int)((in[i] >> shift) & 15u)], 1);
    __syncthreads();
    if (tid == 0) {
      int s = 0;
      for (int v = 0; v < 16; v++) { base[v] = s; s += hist[v]; }
    }
    __syncthreads();
    for (int t0 = 0; t0 < n; t0 += 1024) {
      int i = t0 + tid;
      bool valid = i < n;
      uint64_t key = valid ? in[i] : 0ull;
      int d = valid ? (int)((key >> shift) & 15u) : 16;
      int rank = 0;
      for (int v = 0; v < 16; v++) {
        unsigned bal = __ballot_sync(0xffffffffu, d == v);
        if (d == v) rank = __popc(bal & lt);
        if (lane == 0) wcnt[w][v] = __popc(bal);
      }
      __syncthreads();
      if (tid < 16) {
        int s = 0;
        for (int ww = 0; ww < 32; ww++) { woff[ww][tid] = s; s += wcnt[ww][tid]; }
        hist[tid] = s;  // tile count of digit tid
      }
      __syncthreads();
      if (valid) out[base[d] + woff[w][d] + rank] = key;
      __syncthreads();
      if (tid < 16) base[tid] += hist[tid];
      __syncthreads();
    }
    uint64_t *t = in; in = out; out = t;
  }
  // 8 passes: the sorted data is back in `a`
}

// ascending bitonic sort of np (a power of two) keys in shared memory
__device__ __forceinline__ void bitonic_sort(uint64_t *sk, int np) {
  // each step visits its np / 2 compare-exchange pairs (i, i + j) directly
  for (int k = 2; k <= np; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int q = threadIdx.x; q < (np >> 1); q += blockDim.x) {
        const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
        const int l = i + j;
        const uint64_t x = sk[i], y = sk[l];
        const bool up = (i & k) == 0;
        if ((x > y) == up) { sk[i] = y; sk[l] = x; }
      }
      __syncthreads();
    }
  }
}
// Up to kSmemSortMax keys: bitonic sort in shared memory, one CTA of 1024
// threads (log2(n) (log2(n) + 1) / 2 compare-exchange steps).  The keys are
// unique (primitive index in the low word), so the order equals the stable
// radix sort's.  Padding slots hold ~0, which sorts last.
constexpr int kSmemSortMax = 16384;
__global__ void __launch_bounds__(1024) k_sort_smem(uint64_t *a, int n, const int *skip) {
  if (skip && *skip) return;
  extern __shared__ uint64_t sk[];
  int np = 1;
  while (np < n) np <<= 1;
  for (int i = threadIdx.x; i < np; i += blockDim.x) sk[i] = i < n ? a[i] : ~0ull;
  __syncthreads();
  bitonic_sort(sk, np);
  for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = sk[i];
}

__device__ __forceinline__ int delta(const uint64_t *k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  return __clzll(k[i] ^ k[j]);  // keys are unique (index in the low word)
}

// internal node i of the hierarchy over the sorted keys
__device__ __forceinline__ void karras_node(const uint64_t *keys, int n, int i, BvhNode *nodes,
                                            int *parent) {
  // parent[0 .. n-2]: internal nodes, parent[n-1 .. 2n-2]: leaves
  int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = delta(keys, n, i, i - d);
  int lmax = 2;
  while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int dnode = delta(keys, n, i, j);
  int s = 0;
  int len = l;
  int t = (len + 1) >> 1;
  while (true) {
    if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    if (t == 1) break;
    t = (t + 1) >> 1;
  }
  int g = i + s * d + min(d, 0);
  int lo = min(i, j), hi = max(i, j);
  int left = (lo == g) ? ~g : g;
  int right = (hi == g + 1) ? ~(g + 1) : g + 1;
  nodes[i].d = make_int4(left, right, 0, 0);
  if (left >= 0) parent[left] = i; else parent[(n - 1) + ~left] = i;
  if (right >= 0) parent[right] = i; else parent[(n - 1) + ~right] = i;
  if (i == 0) parent[0] = -1;
}
__global__ void k_karras(const uint64_t *keys, int n, BvhNode *nodes, int *parent,
                         const int *skip) {
  if (skip && *skip) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n - 1) karras_node(keys, n, i, nodes, parent);
}

__device__ __forceinline__ void store_child(BvhNode &nd, int which, const float lo[3],
                                            const float hi[3]) {
  float wl[3], wh[3];
  for (int k = 0; k < 3; k++) { wl[k] = widen_lo(lo[k]); wh[k] = widen_hi(hi[k]); }
  if (which == 0) {
    nd.a = make_float4(wl[0], wl[1], wl[2], wh[0]);
    nd.b.x = wh[1]; nd.b.y = wh[2];
  } else {
    nd.b.z = wl[0]; nd.b.w = wl[1];
    nd.c = make_float4(wl[2], wh[0], wh[1], wh[2]);
  }
}

// boxes from sorted leaf j upwards, as far as it is the second to arrive
__device__ __forceinline__ void refit_from(const uint64_t *keys, const PrimBox *boxes, int n, int j,
                                           BvhNode *nodes, const int *parent, int *flags,
                                           float *node_box, int *perm) {
  int orig = (int)(keys[j] & 0xffffffffu);
  perm[j] = orig;
  if (n == 1) return;
  int p = parent[(n - 1) + j];
  while (p >= 0) {
    __threadfence();
    if (atomicAdd(&flags[p], 1) == 0) return;  // the sibling finishes this node
    __threadfence();
    int4 ch = nodes[p].d;
    float lo[2][3], hi[2][3];
    for (int c = 0; c < 2; c++) {
      int r = c == 0 ? ch.x : ch.y;
      if (r < 0) {
        const PrimBox b = boxes[(int)(keys[~r] & 0xffffffffu)];
        for (int k = 0; k < 3; k++) { lo[c][k] = b.lo[k]; hi[c][k] = b.hi[k]; }
      } else {
        const volatile float *nb = node_box + 6 * r;
        for (int k = 0; k < 3; k++) { lo[c][k] = nb[k]; hi[c][k] = nb[3 + k]; }
      }
    }
    BvhNode nd = nodes[p];
    store_child(nd, 0, lo[0], hi[0]);
    store_child(nd, 1, lo[1], hi[1]);
    nodes[p] = nd;
    float *ob = node_box + 6 * p;
    for (int k = 0; k < 3; k++) {
      ob[k] = fminf(lo[0][k], lo[1][k]);
      ob[3 + k] = fmaxf(hi[0][k], hi[1][k]);
    }
    p = parent[p];
  }
}
__global__ void k_refit(const uint64_t *keys, const PrimBox *boxes, int n, BvhNode *nodes,
                        const int *parent, int *flags, float *node_box, int *perm,
                        const int *skip) {
  if (skip && *skip) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) refit_from(keys, boxes, n, j, nodes, parent, flags, node_box, perm);
}

__device__ __forceinline__ PrimBox tri_box(const float *tris, int i) {
  const float *v = tris + (size_t)i * 9;
  PrimBox b;
  for (int k = 0; k < 3; k++) {
    b.lo[k] = fminf(fminf(v[k], v[3 + k]), v[6 + k]);
    b.hi[k] = fmaxf(fmaxf(v[k], v[3 + k]), v[6 + k]);
  }
  return b;
}
__global__ void k_tri_boxes(const float *tris, int n, PrimBox *boxes) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) boxes[i] = tri_box(tris, i);
}

__device__ __forceinline__ PrimBox aabb_box(const float *aabb, int i) {
  PrimBox b;
  for (int k = 0; k < 3; k++) { b.lo[k] = aabb[6 * i + k]; b.hi[k] = aabb[6 * i + 3 + k]; }
  return b;
}
__global__ void k_aabb_boxes(const float *aabb, int n, PrimBox *boxes, const int *skip) {
  if (skip && *skip) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) boxes[i] = aabb_box(aabb, i);
}

// sorted triangle data: v0 (w = original index), v1, v2
__device__ __forceinline__ void pack_tri(const float *tris, int o, int j, float4 *out) {
  const float *v = tris + (size_t)o * 9;
  out[3 * j + 0] = make_float4(v[0], v[1], v[2], __int_as_float(o));
  out[3 * j + 1] = make_float4(v[3], v[4], v[5], 0.0f);
  out[3 * j + 2] = make_float4(v[6], v[7], v[8], 0.0f);
}
__global__ void k_pack_tris(const float *tris, const int *perm, int n, float4 *out) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) pack_tri(tris, perm[j], j, out);
}

// sorted sphere data: centre (w = original index), box lo, box hi
__device__ __forceinline__ void pack_sphere(const float *pos, const float *aabb, int o, int j,
                                            float4 *out) {
  out[3 * j + 0] = make_float4(pos[3 * o], pos[3 * o + 1], pos[3 * o + 2], __int_as_float(o));
  out[3 * j + 1] = make_float4(aabb[6 * o], aabb[6 * o + 1], aabb[6 * o + 2], 0.0f);
  out[3 * j + 2] = make_float4(aabb[6 * o + 3], aabb[6 * o + 4], aabb[6 * o + 5], 0.0f);
}
__global__ void k_pack_spheres(const float *pos, const float *aabb, const int *perm, int n,
                               float4 *out, const int *skip) {
  if (skip && *skip) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) pack_sphere(pos, aabb, perm[j], j, out);
}

// The whole build for up to kSmallMax primitives in one CTA: every step above
// with barriers between (a Tx array took seven launches and a memset, 20 us of
// launch gaps and 60 us of host time for both sphere sets).  TRI: pos holds
// the triangles, aabb nothing.
constexpr int kSmallMax = 2048;
template <bool TRI>
__global__ void __launch_bounds__(1024) k_lbvh_small(const float *pos, const float *aabb, int n,
                                                     PrimBox *boxes, int *parent, int *flags,
                                                     float *node_box, BvhNode *nodes, int *perm,
                                                     float4 *prims, const int *skip) {
  if (skip && *skip) return;
  __shared__ uint64_t key[kSmallMax];
  __shared__ float b6[6];
  const int t = threadIdx.x;
  for (int i = t; i < n; i += blockDim.x) {
    boxes[i] = TRI ? tri_box(pos, i) : aabb_box(aabb, i);
    flags[i] = 0;
  }
  __syncthreads();
  centroid_bounds(boxes, n, b6);
  __syncthreads();
  int np = 1;
  while (np < n) np <<= 1;
  for (int i = t; i < np; i += blockDim.x) key[i] = i < n ? morton_key(boxes[i], i, b6) : ~0ull;
  __syncthreads();
  bitonic_sort(key, np);
  for (int i = t; i < n - 1; i += blockDim.x) karras_node(key, n, i, nodes, parent);
  __syncthreads();
  for (int i = t; i < n; i += blockDim.x)
    refit_from(key, boxes, n, i, nodes, parent, flags, node_box, perm);
  for (int i = t; i < n; i += blockDim.x) {
    const int o = (int)(key[i] & 0xffffffffu);
    if (TRI) pack_tri(pos, o, i, prims);
    else pack_sphere(pos, aabb, o, i, prims);
  }
}

__global__ void k_sphere_aabbs(const float *pos, int n, float r, float *aabb) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = 0; k < 3; k++) {
    aabb[6 * i + k] = pos[3 * i + k] - r;
    aabb[6 * i + 3 + k] = pos[3 * i + k] + r;
  }
}

// One level of the collapse of a binary hierarchy into 32-wide nodes: a warp
// per wide node.  The warp's list starts with the two children of the wide
// node's binary root; every round replaces inner children by their own two
// (all of them while they fit, else those with the largest surface) until the
// list holds 32 or only leaves.  Wide nodes of level l + 1 are numbered after
// those of level l through the level's counter.  Latency-bound (one dependent
// node load per round, at most six full rounds).
__global__ void __launch_bounds__(128) k_wide_pass(const BvhNode *nodes, int level, int cap,
                                                   float *wide, int *src, int *cnt) {
  __shared__ float box[4][6][32];
  __shared__ int ref[4][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int base = 0;
  for (int l = 0; l < level; l++) base += cnt[l];
  const int count = level == 0 ? 1 : cnt[level];
  const int nbase = base + count;
  if (nbase > cap) {  // a previous level did not fit
    if (threadIdx.x == 0) cnt[AMS_WIDE_LEVELS] = 1;
    return;
  }
  const int nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < count; i += nwarp) {
    if (lane == 0) ref[w][0] = level == 0 ? 0 : src[base + i];
    int c = 1;
    __syncwarp();
    while (true) {
      const bool in = lane < c && ref[w][lane] >= 0;
      const int ni = __popc(__ballot_sync(0xffffffffu, in)), room = 32 - c;
      if (ni == 0 || room == 0) break;
      bool ex = in;
      if (ni > room) {  // only the largest fit
        const float dx = box[w][1][lane] - box[w][0][lane], dy = box[w][3][lane] - box[w][2][lane],
                    dz = box[w][5][lane] - box[w][4][lane];
        const float area = in ? dx * dy + dy * dz + dz * dx : -1.0f;
        int rank = 0;
        for (int k = 0; k < 32; k++) {
          const float o = __shfl_sync(0xffffffffu, area, k);
          rank += (o > area || (o == area && k < lane)) ? 1 : 0;
        }
        ex = in && rank < room;
      }
      const unsigned me = __ballot_sync(0xffffffffu, ex);
      const int at = c + __popc(me & lt);
      const int node = ex ? ref[w][lane] : 0;
      __syncwarp();
      if (ex) {
        const BvhNode nd = nodes[node];
        box[w][0][lane] = nd.a.x; box[w][2][lane] = nd.a.y; box[w][4][lane] = nd.a.z;
        box[w][1][lane] = nd.a.w; box[w][3][lane] = nd.b.x; box[w][5][lane] = nd.b.y;
        box[w][0][at] = nd.b.z; box[w][2][at] = nd.b.w; box[w][4][at] = nd.c.x;
        box[w][1][at] = nd.c.y; box[w][3][at] = nd.c.z; box[w][5][at] = nd.c.w;
        ref[w][lane] = nd.d.x;
        ref[w][at] = nd.d.y;
      }
      c += __popc(me);
      __syncwarp();
    }
    const bool used = lane < c, inner = used && ref[w][lane] >= 0;
    const unsigned mi = __ballot_sync(0xffffffffu, inner);
    int first = 0;
    if (lane == 0 && mi) first = nbase + atomicAdd(cnt + level + 1, __popc(mi));
    first = __shfl_sync(0xffffffffu, first, 0);
    const int id = first + __popc(mi & lt);
    const bool fits = first + __popc(mi) <= cap;
    if (!fits && lane == 0) cnt[AMS_WIDE_LEVELS] = 1;  // the caller drops the wide form
    if (inner && fits) src[id] = ref[w][lane];
    float *out = wide + (size_t)(base + i) * AMS_WIDE_WORDS + lane;
#pragma unroll
    for (int k = 0; k < 6; k++)
      out[32 * k] = used ? box[w][k][lane] : ((k & 1) ? -3.0e38f : 3.0e38f);
    reinterpret_cast<int *>(out)[32 * 6] =
        !used ? (int)0x80000000 : (inner ? (fits ? id : (int)0x80000000) : ref[w][lane]);
    __syncwarp();
  }
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

// A wide node with inner children is full, so the number of wide nodes is
// at most n / 2 (every bottom node holding two leaves); a third covers any
// hierarchy met in practice, and beyond it the wide form is not used.
int wide_bvh_cap(int n) { return n / 3 + 64; }
size_t wide_bvh_bytes(int n) {
  return sizeof(float) * AMS_WIDE_WORDS * (size_t)wide_bvh_cap(n);
}
size_t wide_bvh_scratch_bytes(int n) {
  return sizeof(int) * ((size_t)wide_bvh_cap(n) + AMS_WIDE_LEVELS + 1);
}
cudaError_t wide_bvh_build(const Lbvh &b, int first, int last, float *wide, char *scratch,
                           cudaStream_t st) {
  int *cnt = reinterpret_cast<int *>(scratch), *src = cnt + AMS_WIDE_LEVELS + 1;
  if (first == 0) {
    // level 0 is the root alone; its count is 1
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int) * (AMS_WIDE_LEVELS + 1), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 1, 1, st);  // little-endian int 1
    if (e != cudaSuccess) return e;
  }
  const int cap = wide_bvh_cap(b.n);
  for (int l = first; l < last && l < AMS_WIDE_LEVELS - 1; l++) {
    // level l has at most 32^l nodes
    const long long most = l < 4 ? (1ll << (5 * l)) : (1ll << 20);
    const int blocks = (int)std::min<long long>((std::min<long long>(most, cap) + 3) / 4, 1216);
    k_wide_pass<<<blocks, 128, 0, st>>>(b.nodes, l, cap, wide, src, cnt);
  }
  return cudaGetLastError();
}

size_t lbvh_scratch_bytes(int n) {
  size_t s = 0;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  s += al(sizeof(PrimBox) * (size_t)n);      // boxes
  s += al(sizeof(uint64_t) * (size_t)n) * 2;  // keys ping-pong
  s += al(sizeof(int) * (size_t)(2 * n));     // parent
  s += al(sizeof(int) * (size_t)n);           // flags
  s += al(sizeof(float) * 6 * (size_t)n);     // node boxes
  s += al(sizeof(float) * 8);                 // bounds
  return s;
}

size_t lbvh_output_bytes(int n) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  return al(sizeof(BvhNode) * (size_t)(n > 1 ? n - 1 : 1)) + al(sizeof(int) * (size_t)n) +
         al(sizeof(float4) * 3 * (size_t)n);
}

// pos / aabb as k_lbvh_small takes them; beyond kSmallMax primitives the boxes
// are in scratch already
static cudaError_t build_common(Lbvh &out, const float *pos, const float *aabb, int n,
                                char *scratch, char *outbuf, const int *skip, cudaStream_t st) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  PrimBox *boxes = (PrimBox *)scratch;
  char *p = scratch + al(sizeof(PrimBox) * (size_t)n);
  uint64_t *ka = (uint64_t *)p; p += al(sizeof(uint64_t) * (size_t)n);
  uint64_t *kb = (uint64_t *)p; p += al(sizeof(uint64_t) * (size_t)n);
  int *parent = (int *)p; p += al(sizeof(int) * (size_t)(2 * n));
  int *flags = (int *)p; p += al(sizeof(int) * (size_t)n);
  float *nbox = (float *)p; p += al(sizeof(float) * 6 * (size_t)n);
  float *b6 = (float *)p;
  out.n = n;
  out.nodes = (BvhNode *)outbuf;
  out.perm = (int *)(outbuf + al(sizeof(BvhNode) * (size_t)(n > 1 ? n - 1 : 1)));
  out.prims = (float4 *)((char *)out.perm + al(sizeof(int) * (size_t)n));
  if (n == 0) return cudaSuccess;
  if (n <= kSmallMax) {
    if (aabb)
      k_lbvh_small<false><<<1, 1024, 0, st>>>(pos, aabb, n, boxes, parent, flags, nbox, out.nodes,
                                              out.perm, out.prims, skip);
    else
      k_lbvh_small<true><<<1, 1024, 0, st>>>(pos, aabb, n, boxes, parent, flags, nbox, out.nodes,
                                             out.perm, out.prims, skip);
    return cudaGetLastError();
  }
  k_bounds<<<1, 1024, 0, st>>>(boxes, n, b6, skip);
  k_morton<<<nblk(n, 256), 256, 0, st>>>(boxes, n, b6, ka, skip);
  if (n <= kSmemSortMax) {
    static size_t attr_set[AMS_MAX_DEVICES] = {0};
    cudaError_t e = ams_set_smem_atleast(attr_set, k_sort_smem, kSmemSortMax * sizeof(uint64_t));
    if (e != cudaSuccess) return e;
    int np = 1;
    while (np < n) np <<= 1;
    k_sort_smem<<<1, 1024, np * sizeof(uint64_t), st>>>(ka, n, skip);
  } else {
    k_sort<<<1, 1024, 0, st>>>(ka, kb, n, skip);
  }
  if (n > 1) {
    k_karras<<<nblk(n - 1, 256), 256, 0, st>>>(ka, n, out.nodes, parent, skip);
    cudaMemsetAsync(flags, 0, sizeof(int) * (size_t)n, st);
  }
  k_refit<<<nblk(n, 256), 256, 0, st>>>(ka, boxes, n, out.nodes, parent, flags, nbox, out.perm,
                                        skip);
  return cudaGetLastError();
}

cudaError_t lbvh_build_triangles(Lbvh &out, const float *tris, int n, char *scratch,
                                 char *outbuf, cudaStream_t st) {
  if (n > kSmallMax) k_tri_boxes<<<nblk(n, 256), 256, 0, st>>>(tris, n, (PrimBox *)scratch);
  cudaError_t e = build_common(out, tris, nullptr, n, scratch, outbuf, nullptr, st);
  if (e != cudaSuccess || n <= kSmallMax) return e;
  k_pack_tris<<<nblk(n, 256), 256, 0, st>>>(tris, out.perm, n, out.prims);
  return cudaGetLastError();
}

cudaError_t lbvh_build_spheres(Lbvh &out, const float *pos, const float *aabb, int n,
                               char *scratch, char *outbuf, const int *skip, cudaStream_t st) {
  if (n > kSmallMax)
    k_aabb_boxes<<<nblk(n, 256), 256, 0, st>>>(aabb, n, (PrimBox *)scratch, skip);
  cudaError_t e = build_common(out, pos, aabb, n, scratch, outbuf, skip, st);
  if (e != cudaSuccess || n <= kSmallMax) return e;
  k_pack_spheres<<<nblk(n, 256), 256, 0, st>>>(pos, aabb, out.perm, n, out.prims, skip);
  return cudaGetLastError();
}

cudaError_t lbvh_from_host(Lbvh &out, const float *tris, int n, const BvhNode *h_nodes,
                           const int *h_perm, char *outbuf, cudaStream_t st) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  out.n = n;
  out.nodes = (BvhNode *)outbuf;
  out.perm = (int *)(outbuf + al(sizeof(BvhNode) * (size_t)(n > 1 ? n - 1 : 1)));
  out.prims = (float4 *)((char *)out.perm + al(sizeof(int) * (size_t)n));
  if (n == 0) return cudaSuccess;
  cudaError_t e;
  if (n > 1 && (e = cudaMemcpyAsync(out.nodes, h_nodes, sizeof(BvhNode) * (size_t)(n - 1),
                                    cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return e;
  if ((e = cudaMemcpyAsync(out.perm, h_perm, sizeof(int) * (size_t)n, cudaMemcpyHostToDevice,
                           st)) != cudaSuccess)
    return e;
  k_pack_tris<<<nblk(n, 256), 256, 0, st>>>(tris, out.perm, n, out.prims);
  return cudaGetLastError();
}

cudaError_t sphere_aabbs(const float *pos, int n, float r, float *aabb, cudaStream_t st) {
  if (n > 0) k_sphere_aabbs<<<nblk(n, 256), 256, 0, st>>>(pos, n, r, aabb);
  return cudaGetLastError();
}
