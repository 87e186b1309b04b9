// gemm_tc.h -- tcgen05 BF16 GEMM with a fused epilogue (gemm_tc.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

// Epilogue of C = A . B^T (row-major C with leading dimension ldc):
//   x = acc (+ bias[col]) ; relu ; x *= (mask[row, col] > 0) ; store.
struct GemmEpilogue {
  const float *bias = nullptr;
  bool relu = false;
  const __nv_bfloat16 *mask = nullptr;  // same shape as C
  float *out32 = nullptr;               // rows below rows32 only
  __nv_bfloat16 *out16 = nullptr;
  int ldc = 0;
  int rows32 = 0x7fffffff;
  __nv_bfloat16 *out16t = nullptr;  // C^T, leading dimension ldt
  int ldt = 0;
};

// One GEMM of a launch: tensor maps of A [M, K] and B [N, K] (bf16, K
// contiguous; gemm_map_a, gemm_map_b), M % 128 == 0, N % 64 == 0, K % 64 == 0.
struct GemmOne {
  CUtensorMap a, b;
  GemmEpilogue ep;
  int M, N, K;
};
constexpr int kGemmGroup = 8;

// maps over a row-major bf16 matrix of `rows` rows, `ld` elements apart (16-byte
// multiples); false when the driver refuses
bool gemm_map_a(CUtensorMap *m, const __nv_bfloat16 *p, long long rows, long long ld);
bool gemm_map_b(CUtensorMap *m, const __nv_bfloat16 *p, long long rows, long long ld);
// n <= kGemmGroup independent GEMMs in one launch.  err: flag word (device or
// mapped host memory), bits set on a timed-out wait inside the kernel.  With
// `chained` the kernel may start before the one in front of it has ended (it
// waits for it before it reads anything).
cudaError_t gemm_bf16_group(const GemmOne *g, int n, unsigned *err, bool chained, cudaStream_t st);

// A [M, K], B [N, K] bf16 row-major (K contiguous).
cudaError_t gemm_bf16_tc(const __nv_bfloat16 *A, const __nv_bfloat16 *B, int M, int N, int K,
                         const GemmEpilogue &ep, unsigned *err, cudaStream_t st);
