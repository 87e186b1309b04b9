// trace.h -- device-side parameter block and launchers of the channel tracer.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/ams.h"
#include "lbvh.h"

// device error flags (bits of TraceDev::err)
#define AMS_DERR_PATH_TABLE 1u    // path table full
#define AMS_DERR_HASH 2u          // a path-table slot's key words never appeared
#define AMS_DERR_STACK 4u         // traversal stack overflow
#define AMS_DERR_ACC_RANGE 8u     // contribution outside the fixed-point range
#define AMS_DERR_TASKS 16u        // task list overflow
#define AMS_DERR_BVH 32u          // BVH node index out of range
#define AMS_DERR_LOOP 64u         // a ray exceeded the segment cap

// division of 32-bit numbers by a constant: n / d = (((n - q) >> 1) + q) >> shift
// with q the high word of n * mul; mul 0 stands for d = 1
struct FastDiv { unsigned mul, shift; };
FastDiv make_fast_div(unsigned d);

// counts of one stage-2 round: new tasks found, tasks and chunks listed
struct RoundCount { unsigned long long tasks, listed, chunks, pad; };
#define AMS_ROUND_SLOTS 16  // ring of them (a power of two)

struct TraceDev {
  // scene triangles: original order [n_tri, 9] and sorted (3 float4 each)
  const float *tris;
  const BvhNode *tri_nodes;
  const float4 *tri_prims;
  int n_tri;
  const float *tri_wide;  // 32-wide form of tri_nodes (NULL: none)
  int n_tri_wide;
  const float4 *tri_attr;  // trace_tri_attr, original order
  const int *mat;
  const float *mat_prop;
  // Tx spheres (instance 1) and Rx spheres (instance 2)
  const BvhNode *tx_nodes;
  const float4 *tx_prims;
  int n_src;
  const float *src;  // original order [n_src, 3]
  const float *src_aabb;  // original order [n_src, 6]
  const float4 *tx_info;  // trace_tx_info
  float src_r;
  const BvhNode *rx_nodes;
  const float4 *rx_prims;
  int n_dst;
  const float *dst;  // original order [n_dst, 3]
  const float *dst_aabb;  // original order [n_dst, 6]
  const float *rx_grid;   // trace_rx_grid
  float dst_r;
  // Rx grid and cells
  int n0_dst, n1_dst, n0g, n1g, ng, gs;
  int strict_grid;
  // stage-2 items: groups of 32 (Rx within the cell, Tx) pairs of a chunk
  unsigned s2_groups;
  FastDiv div_groups, div_src, div_gs, div_n1g;
  // launch parameters
  int L, reserve, spl, launch_x, launch_y;
  float lam_f;
  double lam_d;
  double two_pi_over_lam;  // 2 pi / lam_d
  float src_dir[3], dst_dir[3];
  int src_bp, dst_bp;
  // path table (open addressing, slot = path id)
  unsigned long long *tab_h;
  int32_t *tab_key;  // 14 words per slot, sign bits flipped (0 = not written yet)
  unsigned tab_mask;
  unsigned tab_limit;  // occupied slots above this -> grow and retry
  // task bitmaps [ng][W]: stage 1 sets T in table-slot space (W = slots /
  // 32); stage 2 runs on dense path ids (W = ceil(n_paths / 32))
  unsigned *T;  // traced
  unsigned *N;  // new this round
  unsigned *S;  // succeeded this round
  unsigned *S_next;  // cleared for the next round
  int W;
  // stage-2 path ids: dense id -> table slot
  int *slot_of;
  int n_paths;
  // tasks of the current round: runs of dense path ids in task_path, one run
  // per cell, cut into chunks of up to kpi paths
  int2 *task_path;  // (dense path id, table slot)
  int4 *chunk_at;   // (cell, first task, end task, 0)
  unsigned long long task_cap;  // entries of task_path and of chunk_at
  RoundCount *rounds;  // [AMS_ROUND_SLOTS]
  unsigned round_slot;
  // lists in cell order (trace_list_ordered)
  int *cell_cnt;   // [ng] tasks per cell
  int *cell_off;   // [ng + 1]
  int *chunk_off;  // [ng + 1]
  int kpi;         // paths per stage-2 item this round
  // fixed-point channel accumulators, Rx-major: acc[(dst * n_src + s) * 2]
  unsigned long long *acc;
  // counters: 0 records, 1 overflow threads, 2 occupied slots, 3 ok rays,
  // 4 failed rays, 6 unique records,
  // 8 stage-1 closest-hit queries, 9 stage-2 closest-hit queries,
  // 10 stage-1 launch-index fetch, 12 dense path ids, 13 int64 adds into acc
  unsigned long long *ctr;
  unsigned *err;
  // per-ray records of stage 2 (ams_trace_channel_export): record of ray r
  // of the round at rec[rec_base + r] while below rec_cap
  ams_ray_record *rec;
  unsigned long long rec_cap, rec_base;
};

// per-triangle values of the hit programs, 2 float4 a triangle
cudaError_t trace_tri_attr(const float *tris, int n, float4 *attr, cudaStream_t st);
// shape of the Tx array, 16 floats (k_tx_info in trace.cu), zero before
cudaError_t trace_tx_info(const float *src, const float *aabb, int n, float *info,
                          cudaStream_t st);
// how the Rx set fits an axis-aligned grid, 9 words (RxGrid in trace.cu), zero
// before; word 7 is 1 where it does
cudaError_t trace_rx_grid(const float *dst, const float *aabb, int n0, int n1, float radius,
                          float *out, cudaStream_t st);
cudaError_t trace_stage1(const TraceDev &P, cudaStream_t st);
// dense path ids (dense_of [slots], P.slot_of) and the stage-1 bitmap
// T_slots [ng][w_slots] turned into dense ids in `out` [ng][P.W], zeroed before
cudaError_t trace_dense_paths(const TraceDev &P, const unsigned *T_slots, int w_slots,
                              int *dense_of, unsigned *out, cudaStream_t st);
// paths per stage-2 item for a round of n_tasks tasks (set P.kpi before
// listing the round's tasks)
int trace_paths_per_item(const TraceDev &P, unsigned long long n_tasks);
// Flood-fill step (the new tasks' bits N, T and the count in P.rounds) and
// the list of a round's tasks, in one kernel when both are asked for.
cudaError_t trace_round(const TraceDev &P, bool expand, bool list, cudaStream_t st);
// the list in cell order
cudaError_t trace_list_ordered(const TraceDev &P, cudaStream_t st);
// The listed round; n_tasks = 0 when the host does not know their number.
// With P.rec set every ray's record is written (P.kpi must be 1 then).
cudaError_t trace_stage2(const TraceDev &P, unsigned long long n_tasks, cudaStream_t st);
// whether a round is so small that its kernels run without the host looking
bool trace_round_is_small(const TraceDev &P, unsigned long long n_tasks);
cudaError_t trace_count_bits(const TraceDev &P, const unsigned *bits, unsigned long long *out,
                             cudaStream_t st);
cudaError_t trace_finalize(const TraceDev &P, float *result, cudaStream_t st);
cudaError_t trace_export_paths(const TraceDev &P, int32_t *out_keys, unsigned long long *n_out,
                               cudaStream_t st);
