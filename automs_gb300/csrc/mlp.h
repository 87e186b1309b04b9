// mlp.h -- device state and launchers of the surrogate MLP (mlp.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "gemm_tc.h"

constexpr int kMlpMaxLayers = 8;
static_assert(kMlpMaxLayers <= kGemmGroup, "the weight gradients are one launch");
// tile of the loss kernel, whose CTAs write one FP64 partial sum each (a fixed
// work split, so the loss is summed in the same order on every device)
constexpr int kMlpLossRows = 32, kMlpLossCols = 64;

struct MlpDev {
  int L = 0;                       // weight layers
  int d[kMlpMaxLayers + 1] = {};   // logical widths d[0..L]
  int dp[kMlpMaxLayers + 1] = {};  // stored widths (d[0] padded to 64)
  int max_bp = 0;                  // batch capacity (multiple of 128)
  int step = 0;                    // Adam step count
  float *W[kMlpMaxLayers + 1] = {}, *b[kMlpMaxLayers + 1] = {};
  float *mW[kMlpMaxLayers + 1] = {}, *vW[kMlpMaxLayers + 1] = {};
  float *mb[kMlpMaxLayers + 1] = {}, *vb[kMlpMaxLayers + 1] = {};
  float *gW[kMlpMaxLayers + 1] = {}, *gb[kMlpMaxLayers + 1] = {};
  __nv_bfloat16 *Wb[kMlpMaxLayers + 1] = {}, *Wt[kMlpMaxLayers + 1] = {};
  __nv_bfloat16 *H[kMlpMaxLayers + 1] = {};   // H[0] packed input, H[l] activations
  __nv_bfloat16 *dZ[kMlpMaxLayers + 1] = {};  // gradients of the pre-activations
  // transposes for the weight gradients [width, max_bp]
  __nv_bfloat16 *Ht[kMlpMaxLayers + 1] = {}, *dZt[kMlpMaxLayers + 1] = {};
  float *Y = nullptr;
  double *part = nullptr;
  unsigned *done = nullptr;  // CTAs of the loss kernel that are done (zero between calls)
  unsigned *err = nullptr;   // wait-timeout flags, mapped host memory
  // the layers' GEMMs (mlp_init; M or K = the padded batch is set per call)
  GemmOne fwd[kMlpMaxLayers + 1], dgrad[kMlpMaxLayers + 1], wgrad[kMlpMaxLayers + 1];
};

cudaError_t mlp_init(MlpDev &m, uint32_t seed, cudaStream_t st);
cudaError_t mlp_refresh_bf16(MlpDev &m, cudaStream_t st);
// X [B, d0] fp32; Y_out [B, dL] fp32.  NULL: a training pass, whose output stays
// in m.Y and which keeps the activations transposed too.
cudaError_t mlp_forward(MlpDev &m, const float *X, int B, float *Y_out, cudaStream_t st);
// after mlp_forward on the same batch: gradients into gW/gb, loss (device) if given
cudaError_t mlp_backward(MlpDev &m, const float *T, int B, float *loss, cudaStream_t st);
cudaError_t mlp_adam(MlpDev &m, float lr, cudaStream_t st);
// the network's state as one array (per layer W [d_out, d_in], then b [d_out]):
// which 0 parameters, 1 gradients, 2 Adam first moments, 3 second moments
cudaError_t mlp_flat_copy(MlpDev &m, float *flat, bool to_flat, int which, cudaStream_t st);
