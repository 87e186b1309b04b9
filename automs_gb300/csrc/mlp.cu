// mlp.cu -- surrogate MLP: training and inference on the tcgen05 GEMM.
//
// No counterpart in the reference (it searches hyper-configs with NNI's
// annealer, physical_exp_nni_main.py:11-29, running the full tracer +
// optimiser per trial).  The surrogate maps a placement descriptor to a
// coverage-gain map and screens candidates so that the tracer only judges the
// best few.
//
// Network: H_l = relu(H_{l-1} W_l^T + b_l), l < L; Y = H_{L-1} W_L^T + b_L.
// Compute is BF16 on the tensor cores with FP32 accumulation; master
// weights, gradients and Adam moments are FP32.  Each weight is kept in two
// BF16 copies, W [out, in] for the forward pass and W^T [in, out] for the
// input gradient, both K-major as the GEMM wants.
//   forward   H_l  = gemm(H_{l-1}, W_l)            epilogue: bias, relu -> bf16
//   loss      dY   = 2 (Y - T) / (B d_L)          rows >= B are zero
//   backward  dZ_{l-1} = gemm(dZ_l, W_l^T) o (H_{l-1} > 0)   epilogue mask -> bf16
//             dW_l = gemm(dZ_l^T, H_{l-1}^T)       fp32, all layers in one launch
//             db_l = column sums of dZ_l           all layers in one launch
//   update    Adam on the FP32 masters, both BF16 copies refreshed, one launch.
// The producers write H and dZ transposed as well (the epilogues have a column's
// 32 rows in 32 lanes), so nothing is turned in a pass of its own.  A training
// step of the surrogate (72, 4 x 512, 4096; batch 64) is bound by the latency
// of its chain of nine GEMMs: 14 launches, the GEMMs launched early
// (programmatic dependent launch), instead of 42.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "gemm_tc.h"
#include "mlp.h"

namespace {

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}

// W ~ U(-sqrt(6/fan_in), sqrt(6/fan_in)) (He-uniform), b = 0
__global__ void k_init(float *W, int rows, int cols, int cols_used, uint32_t seed, float bound) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)rows * cols) return;
  int c = (int)(i % cols);
  float u = (hash32((uint32_t)i * 2654435761u ^ seed) >> 8) * (1.0f / 16777216.0f);
  W[i] = c < cols_used ? (2.0f * u - 1.0f) * bound : 0.0f;
}

// fp32 [B, d] -> bf16 [Bp, dp] with zero padding, and its transpose (or NULL);
// 32 x 32 tiles, block (32, 8), grid (ceil(dp / 32), Bp / 32)
__global__ void __launch_bounds__(256) k_pack_input(const float *X, int B, int d, int dp,
                                                    __nv_bfloat16 *out, __nv_bfloat16 *out_t,
                                                    int ldt) {
  __shared__ __nv_bfloat16 t[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int r = r0 + j;
    const __nv_bfloat16 v =
        __float2bfloat16_rn((r < B && c < d) ? X[(size_t)r * d + c] : 0.0f);
    if (c < dp) out[(size_t)r * dp + c] = v;
    t[j][threadIdx.x] = v;
  }
  if (!out_t) return;
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int cc = blockIdx.x * 32 + j;
    if (cc < dp) out_t[(size_t)cc * ldt + r0 + threadIdx.x] = t[threadIdx.x][j];
  }
}

// MSE loss over the first B rows, dY (bf16, zero for padded rows) and dY^T.
// A CTA takes 32 rows x 64 columns; the last one adds the CTAs' FP64 partial
// sums (thread t those with index t mod 256, then a tree: a fixed order) into
// *loss, if given.
__global__ void __launch_bounds__(256) k_loss(const float *Y, const float *T, int B, int d,
                                              float scale, double loss_scale, __nv_bfloat16 *dY,
                                              __nv_bfloat16 *dYt, int ldt, double *part,
                                              unsigned *done, float *loss) {
  __shared__ __nv_bfloat16 t[kMlpLossCols][kMlpLossRows + 1];
  __shared__ double s[8];
  __shared__ bool last;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c0 = blockIdx.x * kMlpLossCols, r0 = blockIdx.y * kMlpLossRows;
  double acc = 0.0;
  for (int j = ty; j < kMlpLossRows; j += 8) {
    const int r = r0 + j;
#pragma unroll
    for (int h = 0; h < kMlpLossCols; h += 32) {
      const int c = c0 + h + tx;
      float g = 0.0f;
      if (r < B) {
        const float e = Y[(size_t)r * d + c] - T[(size_t)r * d + c];
        acc += (double)e * e;
        g = 2.0f * e * scale;
      }
      const __nv_bfloat16 v = __float2bfloat16_rn(g);
      dY[(size_t)r * d + c] = v;
      t[h + tx][j] = v;
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (tx == 0) s[ty] = acc;
  __syncthreads();
  for (int j = ty; j < kMlpLossCols; j += 8) dYt[(size_t)(c0 + j) * ldt + r0 + tx] = t[j][tx];
  const int n = gridDim.x * gridDim.y;
  if (threadIdx.x == 0) {
    double x = 0;
    for (int w = 0; w < 8; w++) x += s[w];
    part[blockIdx.y * gridDim.x + blockIdx.x] = x;
    __threadfence();
    last = atomicAdd(done, 1u) == (unsigned)n - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) acc += __ldcg(part + i);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (tx == 0) s[ty] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0;
    for (int w = 0; w < 8; w++) x += s[w];
    if (loss) *loss = (float)(x * loss_scale);
    *done = 0u;  // ready for the next call
  }
}

// db of every layer: a warp sums one row of dZ^T
struct ColsumArgs {
  int L, ld, Bp;
  int first[kMlpMaxLayers + 1];  // first row of layer l + 1
  const __nv_bfloat16 *dZt[kMlpMaxLayers];
  float *gb[kMlpMaxLayers];
};
__global__ void __launch_bounds__(256) k_colsum(const ColsumArgs a) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= a.first[a.L]) return;
  int l = 0;
  while (row >= a.first[l + 1]) l++;
  const int c = row - a.first[l];
  const __nv_bfloat162 *z = reinterpret_cast<const __nv_bfloat162 *>(a.dZt[l] + (size_t)c * a.ld);
  float s = 0.0f;
  for (int i = lane; i < a.Bp / 2; i += 32) {
    const float2 v = __bfloat1622float2(z[i]);
    s += v.x + v.y;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) a.gb[l][c] = s;
}

// One layer of the kernels over all parameters.
struct LayerArgs {
  float *W, *b;
  const float *gW, *gb;
  float *mW, *vW, *mb, *vb;
  int rows, cols, used;  // d_out, stored and true d_in
  __nv_bfloat16 *Wb, *Wt;
  int tile0;             // first 32 x 32 tile; the bias follows the layer's tiles
  long long flat0;       // first element in the flat array
};
struct AdamArgs {
  int L;
  float lr, b1, b2, eps, c1, c2;
  LayerArgs l[kMlpMaxLayers];
};
__device__ __forceinline__ float adam_step(const AdamArgs &a, float w, float g, float &m,
                                           float &v) {
  m = a.b1 * m + (1.0f - a.b1) * g;
  v = a.b2 * v + (1.0f - a.b2) * g * g;
  return w - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
}
// Adam on the fp32 masters of every layer, W bf16 [rows, cols] and W^T bf16
// [cols, rows] refreshed: a CTA takes a 32 x 32 tile (turned through shared
// memory), or 1024 entries of a bias
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ AdamArgs a) {
  cudaGridDependencySynchronize();
  int l = 0;
  while (l + 1 < a.L && (int)blockIdx.x >= a.l[l + 1].tile0) l++;
  const LayerArgs &y = a.l[l];
  const int tiles_c = (y.cols + 31) / 32, tile = (int)blockIdx.x - y.tile0,
            tiles = tiles_c * (y.rows / 32);
  if (tile >= tiles) {
    for (int i = (tile - tiles) * 1024 + threadIdx.x, k = 0; k < 4; k++, i += 256)
      if (i < y.rows) {
        float m = y.mb[i], v = y.vb[i];
        y.b[i] = adam_step(a, y.b[i], y.gb[i], m, v);
        y.mb[i] = m;
        y.vb[i] = v;
      }
    return;
  }
  __shared__ __nv_bfloat16 t[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int r0 = tile / tiles_c * 32, c = tile % tiles_c * 32 + tx;
#pragma unroll
  for (int j = ty; j < 32; j += 8) {
    const size_t i = (size_t)(r0 + j) * y.cols + c;
    if (c < y.cols) {
      float w = y.W[i];
      if (c < y.used) {
        float m = y.mW[i], v = y.vW[i];
        w = adam_step(a, w, y.gW[i], m, v);
        y.mW[i] = m;
        y.vW[i] = v;
        y.W[i] = w;
      }
      const __nv_bfloat16 h = __float2bfloat16_rn(w);
      y.Wb[i] = h;
      t[j][tx] = h;
    }
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    const int cc = tile % tiles_c * 32 + j;
    if (cc < y.cols) y.Wt[(size_t)cc * y.rows + r0 + tx] = t[tx][j];
  }
}

// the flat array from (or into) the layers' arrays, one launch
struct FlatArgs {
  int L;
  long long n;
  struct { float *W, *b; int rows, cols, used; long long first; } l[kMlpMaxLayers];
};
__global__ void __launch_bounds__(256) k_flat(const __grid_constant__ FlatArgs a, float *flat,
                                              bool to_flat) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n;
       i += (long long)gridDim.x * blockDim.x) {
    int l = 0;
    while (l + 1 < a.L && i >= a.l[l + 1].first) l++;
    const int k = (int)(i - a.l[l].first), nw = a.l[l].rows * a.l[l].used;
    float *p = k < nw ? a.l[l].W + (size_t)(k / a.l[l].used) * a.l[l].cols + k % a.l[l].used
                      : a.l[l].b + (k - nw);
    if (to_flat) flat[i] = *p;
    else *p = flat[i];
  }
}

__global__ void k_to_bf16_pair(const float *W, long long n, int rows, int cols, __nv_bfloat16 *Wb,
                               __nv_bfloat16 *Wt) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int r = (int)(i / cols), c = (int)(i % cols);
  __nv_bfloat16 h = __float2bfloat16_rn(W[i]);
  Wb[i] = h;
  Wt[(size_t)c * rows + r] = h;
}

inline int nb(long long n, int b) { return (int)((n + b - 1) / b); }

}  // namespace

cudaError_t mlp_init(MlpDev &m, uint32_t seed, cudaStream_t st) {
  for (int l = 1; l <= m.L; l++) {
    const int rows = m.d[l], cols = m.dp[l - 1], used = m.d[l - 1];
    const float bound = sqrtf(6.0f / (float)used);
    k_init<<<nb((long long)rows * cols, 256), 256, 0, st>>>(m.W[l], rows, cols, used,
                                                             seed * 7919u + (uint32_t)l, bound);
    cudaMemsetAsync(m.b[l], 0, sizeof(float) * rows, st);
    cudaMemsetAsync(m.mW[l], 0, sizeof(float) * (size_t)rows * cols, st);
    cudaMemsetAsync(m.vW[l], 0, sizeof(float) * (size_t)rows * cols, st);
    cudaMemsetAsync(m.mb[l], 0, sizeof(float) * rows, st);
    cudaMemsetAsync(m.vb[l], 0, sizeof(float) * rows, st);
    GemmOne &f = m.fwd[l], &d = m.dgrad[l], &w = m.wgrad[l];
    const bool ok = gemm_map_a(&f.a, m.H[l - 1], m.max_bp, cols) &&
                    gemm_map_b(&f.b, m.Wb[l], rows, cols) &&
                    gemm_map_a(&d.a, m.dZ[l], m.max_bp, rows) &&
                    gemm_map_b(&d.b, m.Wt[l], cols, rows) &&
                    gemm_map_a(&w.a, m.dZt[l], rows, m.max_bp) &&
                    gemm_map_b(&w.b, m.Ht[l - 1], cols, m.max_bp);
    if (!ok) return cudaErrorInvalidValue;
    f.N = rows; f.K = cols;
    f.ep.bias = m.b[l];
    f.ep.relu = l < m.L;
    f.ep.ldc = rows;
    d.N = cols; d.K = rows;
    d.ep.ldc = cols;
    d.ep.ldt = m.max_bp;
    if (l > 1) {
      d.ep.mask = m.H[l - 1];
      d.ep.out16 = m.dZ[l - 1];
      d.ep.out16t = m.dZt[l - 1];
    }
    w.M = rows; w.N = cols;
    w.ep.out32 = m.gW[l];
    w.ep.ldc = cols;
  }
  cudaMemsetAsync(m.done, 0, sizeof(unsigned), st);
  return mlp_refresh_bf16(m, st);
}

cudaError_t mlp_refresh_bf16(MlpDev &m, cudaStream_t st) {
  for (int l = 1; l <= m.L; l++) {
    const long long n = (long long)m.d[l] * m.dp[l - 1];
    k_to_bf16_pair<<<nb(n, 256), 256, 0, st>>>(m.W[l], n, m.d[l], m.dp[l - 1], m.Wb[l], m.Wt[l]);
  }
  return cudaGetLastError();
}

namespace {
// a launch that may start before the kernel in front of it has ended (the
// kernel waits for it)
template <class... P, class... A>
cudaError_t launch_chained(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}
}  // namespace

cudaError_t mlp_forward(MlpDev &m, const float *X, int B, float *Y_out, cudaStream_t st) {
  const int Bp = (B + 127) / 128 * 128;
  const bool train = Y_out == nullptr;
  k_pack_input<<<dim3((m.dp[0] + 31) / 32, Bp / 32), dim3(32, 8), 0, st>>>(
      X, B, m.d[0], m.dp[0], m.H[0], train ? m.Ht[0] : nullptr, m.max_bp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // the last layer writes the caller's rows itself where they are aligned
  const bool direct = Y_out && (reinterpret_cast<uintptr_t>(Y_out) & 15) == 0;
  for (int l = 1; l <= m.L; l++) {
    GemmOne g = m.fwd[l];
    g.M = Bp;
    if (l < m.L) {
      g.ep.out16 = m.H[l];
      if (train) { g.ep.out16t = m.Ht[l]; g.ep.ldt = m.max_bp; }
    } else {
      g.ep.out32 = direct ? Y_out : m.Y;
      if (direct) g.ep.rows32 = B;
    }
    e = gemm_bf16_group(&g, 1, m.err, true, st);
    if (e != cudaSuccess) return e;
  }
  if (Y_out && !direct)
    e = cudaMemcpyAsync(Y_out, m.Y, sizeof(float) * (size_t)B * m.d[m.L],
                        cudaMemcpyDeviceToDevice, st);
  return e;
}

cudaError_t mlp_backward(MlpDev &m, const float *T, int B, float *loss, cudaStream_t st) {
  const int Bp = (B + 127) / 128 * 128;
  const int L = m.L;
  const int dl = m.d[L];
  // targets arrive as [B, d_L]; the output buffer has the same width
  cudaError_t e = launch_chained(
      k_loss, dim3(dl / kMlpLossCols, Bp / kMlpLossRows), dim3(256), st, (const float *)m.Y, T, B,
      dl, 1.0f / ((float)B * dl), 1.0 / ((double)B * dl), m.dZ[L], m.dZt[L], m.max_bp, m.part,
      m.done, loss);
  if (e != cudaSuccess) return e;
  for (int l = L; l > 1; l--) {
    GemmOne g = m.dgrad[l];
    g.M = Bp;
    if ((e = gemm_bf16_group(&g, 1, m.err, true, st)) != cudaSuccess) return e;
  }
  GemmOne w[kMlpMaxLayers];
  ColsumArgs c{};
  c.L = L;
  c.ld = m.max_bp;
  c.Bp = Bp;
  for (int l = 1; l <= L; l++) {
    w[l - 1] = m.wgrad[l];
    w[l - 1].K = Bp;
    c.first[l] = c.first[l - 1] + m.d[l];
    c.dZt[l - 1] = m.dZt[l];
    c.gb[l - 1] = m.gb[l];
  }
  if ((e = gemm_bf16_group(w, L, m.err, true, st)) != cudaSuccess) return e;
  return launch_chained(k_colsum, dim3((c.first[L] + 7) / 8), dim3(256), st, c);
}

cudaError_t mlp_adam(MlpDev &m, float lr, cudaStream_t st) {
  m.step++;
  AdamArgs a{};
  a.L = m.L;
  a.lr = lr;
  a.b1 = 0.9f; a.b2 = 0.999f; a.eps = 1e-8f;
  a.c1 = 1.0f - powf(a.b1, (float)m.step);
  a.c2 = 1.0f - powf(a.b2, (float)m.step);
  int tiles = 0;
  for (int l = 1; l <= m.L; l++) {
    LayerArgs &y = a.l[l - 1];
    y.W = m.W[l]; y.b = m.b[l]; y.gW = m.gW[l]; y.gb = m.gb[l];
    y.mW = m.mW[l]; y.vW = m.vW[l]; y.mb = m.mb[l]; y.vb = m.vb[l];
    y.rows = m.d[l]; y.cols = m.dp[l - 1]; y.used = m.d[l - 1];
    y.Wb = m.Wb[l]; y.Wt = m.Wt[l];
    y.tile0 = tiles;
    tiles += (y.cols + 31) / 32 * (y.rows / 32) + (y.rows + 1023) / 1024;
  }
  return launch_chained(k_adam, dim3(tiles), dim3(256), st, a);
}

cudaError_t mlp_flat_copy(MlpDev &m, float *flat, bool to_flat, int which, cudaStream_t st) {
  FlatArgs a{};
  a.L = m.L;
  for (int l = 1; l <= m.L; l++) {
    float *const Ws[4] = {m.W[l], m.gW[l], m.mW[l], m.vW[l]};
    float *const bs[4] = {m.b[l], m.gb[l], m.mb[l], m.vb[l]};
    auto &y = a.l[l - 1];
    y.W = Ws[which]; y.b = bs[which];
    y.rows = m.d[l]; y.cols = m.dp[l - 1]; y.used = m.d[l - 1];
    y.first = a.n;
    a.n += (long long)y.rows * y.used + y.rows;
  }
  k_flat<<<(int)((a.n + 1023) / 1024), 256, 0, st>>>(a, flat, to_flat);
  return cudaGetLastError();
}
