// objective.cu -- phase-map coverage objective and its adjoint on GB300.
//
// Reference: Model.get_channel (go.py:107-157, one metasurface hop) and
// Model.forward with loss mode "capacity" (go.py:159-245), differentiated by
// hand instead of autograd.  Channels in the reference orientation:
// H_d [S,R], H_a [S,M], H_r [M,R], code weights W [C,S], complex64.
//
//   U   = (W H_a) o exp(j (phi mod max_phase))            k_prep
//   Y   = W H_d + U H_r        (one streaming pass)        k_pass1
//   per Rx: |Y|, capacity, dropout, max over codes, mask, and the two
//   gradient parts G1 (max term) and G2 (norm term, before 1/||.||)
//   loss = -w sum max + ||masked||                          k_scalars
//   G_U = (G1 + G2/||.||) [H_r; H_d]^H  (second pass)       k_pass2
//   dphi = -Im(conj(G_U) o U) summed over codes,
//   G_W  = G_Wd + (G_U o exp(-j phi')) H_a^H                k_final
//
// Accumulation is FP32 with FP64 for the loss scalars.  When H_r fits in L2
// the second pass reads it from L2, so one evaluation moves H_r from HBM
// once.  Scratch lives in a per-device buffer kept across calls; calls on
// one device must not overlap.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <vector>

#include "../../include/ams.h"
#include "objective.h"
#include "tc_ptx.cuh"

namespace {

constexpr float kN0 = 1e-9f;                 // 10^(-90/10) mW, go.py:183-184
constexpr float kEps = 1.1920928955078125e-07f;  // float32 eps, go.py:181
constexpr float kInvLn2 = 1.4426950408889634f;
// the value of every output of a call whose bounded wait ran out
__device__ __forceinline__ float obj_nan() { return __int_as_float(0x7fc00000); }
// a bounded wait of this call ran out (err may be NULL: a path without waits)
__device__ __forceinline__ bool obj_failed(const unsigned *err) {
  return err != nullptr && __ldcg(err) != 0u;
}

struct c2 { float x, y; };
__device__ __forceinline__ c2 ld2(const float *p, size_t i) {
  float2 v = __ldg(reinterpret_cast<const float2 *>(p) + i);
  return {v.x, v.y};
}
__device__ __forceinline__ void mac(c2 &acc, c2 a, c2 b) {  // acc += a*b
  acc.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x));
  acc.y = fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y));
}
__device__ __forceinline__ void macc(c2 &acc, c2 a, c2 b) {  // acc += a*conj(b)
  acc.x = fmaf(a.x, b.x, fmaf(a.y, b.y, acc.x));
  acc.y = fmaf(a.y, b.x, fmaf(-a.x, b.y, acc.y));
}

// Python/torch remainder: result has the sign of the divisor
__device__ __forceinline__ float py_mod(float a, float b) {
  float r = fmodf(a, b);
  if (r != 0.f && ((r < 0.f) != (b < 0.f))) r += b;
  return r;
}

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi); a pair of values goes to
// element `pair` of the bf16x2 views of the hi and lo arrays
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}
__device__ __forceinline__ void put_pair(__nv_bfloat16 *hi, __nv_bfloat16 *lo, size_t pair,
                                         float a, float b) {
  __nv_bfloat16 h0, l0, h1, l1;
  split_bf16(a, h0, l0);
  split_bf16(b, h1, l1);
  reinterpret_cast<__nv_bfloat162 *>(hi)[pair] = __halves2bfloat162(h0, h1);
  reinterpret_cast<__nv_bfloat162 *>(lo)[pair] = __halves2bfloat162(l0, l1);
}

// ------------------------------------------------------------------
// Virtual rows k in [0, K), K = M + S: row k < M is H_r[k, :] with
// coefficient U[c, k]; row k >= M is H_d[k - M, :] with coefficient
// W[c, k - M].  Y[c, r] = sum_k coef[c, k] row_k[r].

__device__ __forceinline__ const float *row_ptr(const float *Hr, const float *Hd, int M, int R,
                                                int k) {
  return k < M ? Hr + (size_t)k * R * 2 : Hd + (size_t)(k - M) * R * 2;
}

constexpr int KCHUNK = 256;

// U[c, m] for the streaming path: 8 lanes per (m, c) split the sum over the
// AP elements; the dependent streaming kernel may start before this one ends
// (programmatic dependent launch) and waits for it only before reading U.
__global__ void __launch_bounds__(256) k_prep_wide(ObjArgs a, int M, float *U, unsigned *err) {
  // let the streaming kernel launch now; it waits for this grid before reading U
  cudaTriggerProgrammaticLaunchCompletion();
  // the call's wait-timeout word starts clear (a streaming kernel can set it
  // only after its grid-dependency wait on this grid)
  if (err && blockIdx.x == 0 && threadIdx.x == 0) *err = 0u;
  const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  const bool live = e < (long long)M * a.C;
  const int c = live ? (int)(e / M) : 0, m = live ? (int)(e % M) : 0;
  c2 v = {0.f, 0.f};
  if (live)
    for (int s = sub; s < a.S; s += 8) mac(v, ld2(a.W, (size_t)c * a.S + s), ld2(a.Ha, (size_t)s * M + m));
  for (int o = 1; o < 8; o <<= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if (live && sub == 0) {
    const float p = py_mod(__ldg(a.phi + m), a.max_phase);
    float sn, cs;
    sincosf(p, &sn, &cs);
    c2 u = {0.f, 0.f};
    mac(u, v, c2{cs, sn});
    reinterpret_cast<float2 *>(U)[(size_t)c * M + m] = make_float2(u.x, u.y);
  }
}

// U[c, m] = (sum_s W[c, s] H_a[s, m]) e^{j phi'_m}: one thread per (m, c),
// loads of H_a coalesced over m, issued 8 at a time
__global__ void __launch_bounds__(128) k_prep(ObjArgs a, int M, float *U, unsigned *err) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  // the call's wait-timeout word starts clear (the GEMMs that can set it
  // run after this kernel)
  if (err && m == 0 && c == 0) *err = 0u;
  if (m >= M) return;
  c2 v = {0.f, 0.f};
  int s = 0;
  for (; s + 8 <= a.S; s += 8) {
    c2 h[8], w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      h[j] = ld2(a.Ha, (size_t)(s + j) * M + m);
      w[j] = ld2(a.W, (size_t)c * a.S + s + j);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) mac(v, w[j], h[j]);
  }
  for (; s < a.S; s++) mac(v, ld2(a.W, (size_t)c * a.S + s), ld2(a.Ha, (size_t)s * M + m));
  const float p = py_mod(__ldg(a.phi + m), a.max_phase);  // go.py:133
  float sn, cs;
  sincosf(p, &sn, &cs);
  c2 u = {0.f, 0.f};
  mac(u, v, c2{cs, sn});
  reinterpret_cast<float2 *>(U)[(size_t)c * M + m] = make_float2(u.x, u.y);
}

// pass 1: partial Y over a k-range; lanes = 32 columns, warps share the rows
template <int CB>
__global__ void __launch_bounds__(256) k_pass1(ObjArgs a, int M, int K, int kper, const float *U,
                                               float *Ypart) {
  __shared__ c2 sC[KCHUNK][CB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  const bool live = r < a.R;
  const int k0 = blockIdx.y * kper, k1 = min(K, k0 + kper);
  c2 y[CB];
#pragma unroll
  for (int c = 0; c < CB; c++) y[c] = {0.f, 0.f};
  for (int kc = k0; kc < k1; kc += KCHUNK) {
    const int kn = min(KCHUNK, k1 - kc);
    __syncthreads();
    for (int i = threadIdx.x; i < kn * CB; i += blockDim.x) {
      const int kk = i / CB, c = i % CB, k = kc + kk;
      c2 v = {0.f, 0.f};
      if (c < a.C) v = k < M ? ld2(U, (size_t)c * M + k) : ld2(a.W, (size_t)c * a.S + (k - M));
      sC[kk][c] = v;
    }
    __syncthreads();
    if (live) {
      int kk = warp;
      for (; kk + 24 < kn; kk += 32) {
        const c2 h0 = ld2(row_ptr(a.Hr, a.Hd, M, a.R, kc + kk), r);
        const c2 h1 = ld2(row_ptr(a.Hr, a.Hd, M, a.R, kc + kk + 8), r);
        const c2 h2 = ld2(row_ptr(a.Hr, a.Hd, M, a.R, kc + kk + 16), r);
        const c2 h3 = ld2(row_ptr(a.Hr, a.Hd, M, a.R, kc + kk + 24), r);
#pragma unroll
        for (int c = 0; c < CB; c++) {
          mac(y[c], sC[kk][c], h0);
          mac(y[c], sC[kk + 8][c], h1);
          mac(y[c], sC[kk + 16][c], h2);
          mac(y[c], sC[kk + 24][c], h3);
        }
      }
      for (; kk < kn; kk += 8) {
        const c2 h = ld2(row_ptr(a.Hr, a.Hd, M, a.R, kc + kk), r);
#pragma unroll
        for (int c = 0; c < CB; c++) mac(y[c], sC[kk][c], h);
      }
    }
  }
  // reduce the 8 warps, 8 codes at a time
  __shared__ c2 red[8][32][8];
  for (int cg = 0; cg < CB; cg += 8) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (cg + j < CB) red[warp][lane][j] = y[cg + j < CB ? cg + j : 0];
    __syncthreads();
    if (warp == 0 && live) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int c = cg + j;
        if (c >= CB || c >= a.C) continue;
        c2 t = red[0][lane][j];
        for (int w2 = 1; w2 < 8; w2++) { t.x += red[w2][lane][j].x; t.y += red[w2][lane][j].y; }
        reinterpret_cast<float2 *>(Ypart)[((size_t)blockIdx.y * a.C + c) * a.R + r] =
            make_float2(t.x, t.y);
      }
    }
  }
}

// Sum of the CTAs' (sum_max, sum_sq) pairs by every thread of the last CTA
// (FP64 adds have a long latency on this part; one thread alone would chain
// thousands of them).  Reads bypass L1: the pairs were written by other CTAs.
// The result is valid in thread 0; all threads of the block must call it.
__device__ __forceinline__ void block_sum_pairs(const double *partials, int nb, double &x,
                                                double &z) {
  __threadfence();
  double px = 0.0, pz = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    px += __ldcg(partials + 2 * b);
    pz += __ldcg(partials + 2 * b + 1);
  }
  for (int o = 16; o > 0; o >>= 1) {
    px += __shfl_xor_sync(0xffffffffu, px, o);
    pz += __shfl_xor_sync(0xffffffffu, pz, o);
  }
  __shared__ double red[2][32];
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { red[0][wid] = px; red[1][wid] = pz; }
  __syncthreads();
  x = 0.0;
  z = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) { x += red[0][i]; z += red[1][i]; }
}

// epilogue: Y from the partials, per-Rx capacity / dropout / max / mask and
// the gradient parts; the last CTA reduces the block sums into the loss.
template <int CB>
__global__ void __launch_bounds__(256) k_epilogue(ObjArgs a, int kspl, const float *Ypart,
                                                  float *G1, float *G2, double *partials,
                                                  unsigned *counter, float *scal,
                                                  const unsigned *err) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  float sum_max = 0.f, sum_sq = 0.f;  // FP32 within a warp, FP64 across warps
  if (r < a.R) {
    c2 y[CB];
    float cap[CB], amp[CB];
    int arg = 0;
    float mx = -1.f;
#pragma unroll
    for (int c = 0; c < CB; c++) {
      y[c] = {0.f, 0.f};
      if (c >= a.C) { cap[c] = 0.f; amp[c] = 0.f; continue; }
      int sp = 0;
      for (; sp + 4 <= kspl; sp += 4) {
        c2 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = ld2(Ypart, ((size_t)(sp + j) * a.C + c) * a.R + r);
#pragma unroll
        for (int j = 0; j < 4; j++) { y[c].x += v[j].x; y[c].y += v[j].y; }
      }
      for (; sp < kspl; sp++) {
        c2 v = ld2(Ypart, ((size_t)sp * a.C + c) * a.R + r);
        y[c].x += v.x;
        y[c].y += v.y;
      }
      amp[c] = sqrtf(y[c].x * y[c].x + y[c].y * y[c].y);
      const float aa = amp[c] + kEps;
      float v = log2f(1.0f + aa * aa / kN0);
      if (a.drop && a.drop[c]) v = 0.f;
      cap[c] = v;
      if (v > mx) { mx = v; arg = c; }  // first index of the maximum
      if (a.recv_amp) a.recv_amp[(size_t)c * a.R + r] = amp[c];
    }
    sum_max = mx;
#pragma unroll
    for (int c = 0; c < CB; c++) {
      if (c >= a.C) continue;
      const bool dropped = a.drop && a.drop[c];
      const float msk = (cap[c] != mx) ? cap[c] : 0.f;  // cap' * mask
      sum_sq += msk * msk;
      const float aa = amp[c] + kEps;
      const float dcap = (2.0f * aa / kN0) / (1.0f + aa * aa / kN0) * kInvLn2;
      float g1 = (c == arg) ? -a.w : 0.f, g2 = msk;
      if (dropped) { g1 = 0.f; g2 = 0.f; }
      const float sc = amp[c] > 0.f ? dcap / amp[c] : 0.f;
      reinterpret_cast<float2 *>(G1)[(size_t)c * a.R + r] =
          make_float2(g1 * sc * y[c].x, g1 * sc * y[c].y);
      if (G2)
        reinterpret_cast<float2 *>(G2)[(size_t)c * a.R + r] =
            make_float2(g2 * sc * y[c].x, g2 * sc * y[c].y);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    sum_max += __shfl_xor_sync(0xffffffffu, sum_max, o);
    sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
  }
  __shared__ double sp[2][8];
  __shared__ bool last;
  const int wid = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) { sp[0][wid] = sum_max; sp[1][wid] = sum_sq; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0, z = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) { x += sp[0][i]; z += sp[1][i]; }
    partials[2 * blockIdx.x] = x;
    partials[2 * blockIdx.x + 1] = z;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    double x, z;
    block_sum_pairs(partials, (int)gridDim.x, x, z);
    if (threadIdx.x == 0) {
      const double nrm = sqrt(z);
      if (a.loss) *a.loss = obj_failed(err) ? obj_nan() : (float)(-(double)a.w * x + nrm);
      scal[0] = nrm > 0 ? (float)(1.0 / nrm) : 0.f;
      *counter = 0u;  // ready for the next call
    }
  }
}

// epilogue for codebooks (CB >= 8): a CTA takes 32 Rx (one per lane) and
// its 8 warps split the codes (warp w: c = w, w + 8, ...), so a thread keeps
// CB / 8 codes.  The max over codes (first index on ties) is reduced across
// the warps in shared memory; then each thread writes its codes' gradient
// parts.  Loss partials and the last-CTA reduction as in k_epilogue.
template <int CB>
__global__ void __launch_bounds__(256) k_epilogue_wide(ObjArgs a, int kspl, const float *Ypart,
                                                       float *G1, float *G2, double *partials,
                                                       unsigned *counter, float *scal) {
  constexpr int CPT = CB / 8;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  const bool live = r < a.R;
  c2 y[CPT];
  float amp[CPT], cap[CPT];
  float mx = -1.f;
  int arg = 0x7fffffff;
  // all loads first (independent across codes), then the arithmetic
  const int rr = live ? r : 0;
  for (int sp = 0; sp < kspl; sp++) {
    c2 v[CPT];
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      const int c = min(wid + 8 * j, a.C - 1);
      v[j] = ld2(Ypart, ((size_t)sp * a.C + c) * a.R + rr);
    }
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      if (sp == 0) y[j] = v[j];
      else { y[j].x += v[j].x; y[j].y += v[j].y; }
    }
  }
#pragma unroll
  for (int j = 0; j < CPT; j++) {
    const int c = wid + 8 * j;
    amp[j] = 0.f;
    cap[j] = 0.f;
    if (!live || c >= a.C) continue;
    amp[j] = sqrtf(y[j].x * y[j].x + y[j].y * y[j].y);
    const float aa = amp[j] + kEps;
    float v = log2f(1.0f + aa * aa / kN0);
    if (a.drop && a.drop[c]) v = 0.f;
    cap[j] = v;
    if (v > mx) { mx = v; arg = c; }  // codes ascend within a thread
    if (a.recv_amp) a.recv_amp[(size_t)c * a.R + r] = amp[j];
  }
  __shared__ float smx[8][32];
  __shared__ int sarg[8][32];
  smx[wid][lane] = mx;
  sarg[wid][lane] = arg;
  __syncthreads();
  float M_ = smx[0][lane];
  int A_ = sarg[0][lane];
#pragma unroll
  for (int w2 = 1; w2 < 8; w2++) {
    const float v = smx[w2][lane];
    const int g = sarg[w2][lane];
    if (v > M_ || (v == M_ && g < A_)) { M_ = v; A_ = g; }
  }
  // FP32 within a warp (FP64 arithmetic is slow here), FP64 across warps
  float sum_max = (live && wid == 0) ? M_ : 0.f, sum_sq = 0.f;
#pragma unroll
  for (int j = 0; j < CPT; j++) {
    const int c = wid + 8 * j;
    if (!live || c >= a.C) continue;
    const bool dropped = a.drop && a.drop[c];
    const float msk = (cap[j] != M_) ? cap[j] : 0.f;
    sum_sq += msk * msk;
    const float aa = amp[j] + kEps;
    const float dcap = (2.0f * aa / kN0) / (1.0f + aa * aa / kN0) * kInvLn2;
    float g1 = (c == A_) ? -a.w : 0.f, g2 = msk;
    if (dropped) { g1 = 0.f; g2 = 0.f; }
    const float sc = amp[j] > 0.f ? dcap / amp[j] : 0.f;
    reinterpret_cast<float2 *>(G1)[(size_t)c * a.R + r] =
        make_float2(g1 * sc * y[j].x, g1 * sc * y[j].y);
    if (G2)
      reinterpret_cast<float2 *>(G2)[(size_t)c * a.R + r] =
          make_float2(g2 * sc * y[j].x, g2 * sc * y[j].y);
  }
  for (int o = 16; o > 0; o >>= 1) {
    sum_max += __shfl_xor_sync(0xffffffffu, sum_max, o);
    sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
  }
  __shared__ double spart[2][8];
  __shared__ bool last;
  if (lane == 0) { spart[0][wid] = sum_max; spart[1][wid] = sum_sq; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0, z = 0;
    for (int i = 0; i < 8; i++) { x += spart[0][i]; z += spart[1][i]; }
    partials[2 * blockIdx.x] = x;
    partials[2 * blockIdx.x + 1] = z;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    double x, z;
    block_sum_pairs(partials, (int)gridDim.x, x, z);
    if (threadIdx.x == 0) {
      const double nrm = sqrt(z);
      if (a.loss) *a.loss = (float)(-(double)a.w * x + nrm);
      scal[0] = nrm > 0 ? (float)(1.0 / nrm) : 0.f;
      *counter = 0u;  // ready for the next call
    }
  }
}

// Operands lie k-block by k-block: 64 values (128 bytes) of row after row, so a
// stage's tile is one contiguous piece of memory (its pieces of 128 bytes lay
// 4 KB or more apart with K contiguous in a row: 211 us against 219 for the two
// products of 60 codes, K = 1,040, R = 65,536).  In pairs of values: pair `col2` of row `row` of `rows`.
__device__ __forceinline__ size_t kb_pair(int row, int col2, int rows) {
  return ((size_t)(col2 >> 5) * rows + row) * 32 + (col2 & 31);
}

namespace tcg {
constexpr int BM = 128, BK = 64, BN_MIN = 64, BN_MAX = 160, STAGES_MAX = 6;
constexpr uint32_t A_BYTES = BM * BK * 2;  // one of the two A tiles of a stage
constexpr uint32_t stage_bytes(int bn) { return 2 * A_BYTES + 2u * bn * BK * 2; }
constexpr size_t SMEM = 225 * 1024;  // 1 KB of it for alignment
constexpr int stages(int bn) {
  const int n = (int)((SMEM - 1024) / stage_bytes(bn));
  return n < STAGES_MAX ? n : STAGES_MAX;
}
static_assert(stages(BN_MAX) >= 3 && BN_MAX % 16 == 0, "stages");
}  // namespace tcg

// Two-phase epilogue of the tensor-core path (CB >= 8), same thread layout
// as k_epilogue_wide.  Phase A: loss partials, and per Rx the max over codes
// and its first index.  Phase B: re-reads Y, forms G = G1 + G2 / ||masked||
// and writes it straight into the A operand of the adjoint GEMM (and
// grad_Y), so G1 / G2 are never stored.  Both phases evaluate the capacity
// with the same inline code, so they see bit-identical values.
template <int CPT>
__device__ __forceinline__ void epi_load_y(const ObjArgs &a, int kspl, const float *Ypart, int wid,
                                           int rr, c2 (&y)[CPT]) {
  const float2 *q = reinterpret_cast<const float2 *>(Ypart) + (size_t)wid * a.R + rr;
  const size_t step = (size_t)8 * a.R;
  for (int sp = 0; sp < kspl; sp++, q += (size_t)a.C * a.R) {
    float2 v[CPT];
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      v[j] = make_float2(0.f, 0.f);
      if (wid + 8 * j < a.C) v[j] = __ldg(q + j * step);
    }
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      if (sp == 0) y[j] = {v[j].x, v[j].y};
      else { y[j].x += v[j].x; y[j].y += v[j].y; }
    }
  }
}
// 1 / N0 = 1e9 is a float32 value, which float32(1e-9) is not exactly: the
// product is the nearer one, and a division is ten instructions
constexpr float kInvN0 = 1e9f;
__device__ __forceinline__ void epi_cap(const ObjArgs &a, int c, c2 y, float &amp, float &cap) {
  amp = sqrtf(y.x * y.x + y.y * y.y);
  const float aa = amp + kEps;
  float v = log2f(1.0f + aa * aa * kInvN0);
  if (a.drop && a.drop[c]) v = 0.f;
  cap = v;
}

// s + x with the rounding error added to e (Knuth's two-sum): a loss partial of
// many Rx is summed in FP32, where FP64 is slow, and keeps what FP64 would
__device__ __forceinline__ void add_kept(float &s, float &e, float x) {
  const float t = s + x, b = t - s;
  e += (s - (t - b)) + (x - b);
  s = t;
}
__device__ __forceinline__ double warp_sum_kept(float s, float e) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float x = __shfl_xor_sync(0xffffffffu, s, o), y = __shfl_xor_sync(0xffffffffu, e, o);
    add_kept(s, e, x);
    e += y;
  }
  return (double)s + (double)e;
}

// (Phase A takes groups of 32 Rx in turn and forms its loss partial once: with
// a CTA and an arrival per group it waited at its barriers, 28.5 us for 60 codes
// and R = 65,536 against 22.4.)
template <int CB>
__global__ void __launch_bounds__(256) k_tc_epi_a(ObjArgs a, int kspl, const float *Ypart,
                                                  float *maxr, int *argr, double *partials,
                                                  unsigned *counter, float *scal,
                                                  const unsigned *err) {
  constexpr int CPT = CB / 8;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __shared__ float smx[2][8][32];
  __shared__ int sarg[2][8][32];
  float sum_max = 0.f, sum_sq = 0.f, low_max = 0.f, low_sq = 0.f;
  const int ngroups = (a.R + 31) / 32;
  for (int grp = blockIdx.x, buf = 0; grp < ngroups; grp += gridDim.x, buf ^= 1) {
    const int r = grp * 32 + lane;
    const bool live = r < a.R;
    c2 y[CPT];
    float cap[CPT];
    epi_load_y<CPT>(a, kspl, Ypart, wid, live ? r : 0, y);
    float mx = -1.f;
    int arg = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      const int c = wid + 8 * j;
      cap[j] = 0.f;
      if (!live || c >= a.C) continue;
      float amp;
      epi_cap(a, c, y[j], amp, cap[j]);
      if (cap[j] > mx) { mx = cap[j]; arg = c; }
      if (a.recv_amp) a.recv_amp[(size_t)c * a.R + r] = amp;
    }
    // (the buffers alternate: a warp may write the next group's while others
    // still read this one's)
    smx[buf][wid][lane] = mx;
    sarg[buf][wid][lane] = arg;
    __syncthreads();
    float M_ = smx[buf][0][lane];
    int A_ = sarg[buf][0][lane];
#pragma unroll
    for (int w2 = 1; w2 < 8; w2++) {
      const float v = smx[buf][w2][lane];
      const int g = sarg[buf][w2][lane];
      if (v > M_ || (v == M_ && g < A_)) { M_ = v; A_ = g; }
    }
    if (wid == 0 && live) {
      maxr[r] = M_;
      argr[r] = A_;
      add_kept(sum_max, low_max, M_);
    }
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      const int c = wid + 8 * j;
      if (!live || c >= a.C) continue;
      const float msk = (cap[j] != M_) ? cap[j] : 0.f;
      sq += msk * msk;
    }
    add_kept(sum_sq, low_sq, sq);
  }
  const double warp_max = warp_sum_kept(sum_max, low_max), warp_sq = warp_sum_kept(sum_sq, low_sq);
  __shared__ double spart[2][8];
  __shared__ bool last;
  if (lane == 0) { spart[0][wid] = warp_max; spart[1][wid] = warp_sq; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0, z = 0;
    for (int i = 0; i < 8; i++) { x += spart[0][i]; z += spart[1][i]; }
    partials[2 * blockIdx.x] = x;
    partials[2 * blockIdx.x + 1] = z;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last) {
    double x, z;
    block_sum_pairs(partials, (int)gridDim.x, x, z);
    if (threadIdx.x == 0) {
      const double nrm = sqrt(z);
      if (a.loss) *a.loss = obj_failed(err) ? obj_nan() : (float)(-(double)a.w * x + nrm);
      scal[0] = nrm > 0 ? (float)(1.0 / nrm) : 0.f;
      *counter = 0u;  // ready for the next call
    }
  }
}

template <int CB>
__global__ void __launch_bounds__(256) k_tc_epi_b(ObjArgs a, int kspl, const float *Ypart,
                                                  const float *maxr, const int *argr,
                                                  const float *scal, int K2p, __nv_bfloat16 *hi,
                                                  __nv_bfloat16 *lo) {
  constexpr int CPT = CB / 8;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane;
  const bool live = r < a.R;
  c2 y[CPT];
  epi_load_y<CPT>(a, kspl, Ypart, wid, live ? r : 0, y);
  const float M_ = live ? maxr[r] : 0.f;
  const int A_ = live ? argr[r] : 0;
  const float inv = a.C > 1 ? scal[0] : 0.f;
#pragma unroll
  for (int j = 0; j < CPT; j++) {
    const int c = wid + 8 * j;
    if (c >= a.C) continue;
    c2 g = {0.f, 0.f};
    if (live) {
      float amp, cap;
      epi_cap(a, c, y[j], amp, cap);
      const bool dropped = a.drop && a.drop[c];
      const float msk = (cap != M_) ? cap : 0.f;
      const float aa = amp + kEps;
      const float dcap = (2.0f * aa * kInvN0) / (1.0f + aa * aa * kInvN0) * kInvLn2;
      float g1 = (c == A_) ? -a.w : 0.f, g2 = msk;
      if (dropped) { g1 = 0.f; g2 = 0.f; }
      const float sc = amp > 0.f ? dcap / amp : 0.f;
      // G1 + G2 * inv with the rounding of k_tc_make_ag: fmaf(G2, inv, G1)
      const c2 q1 = {g1 * sc * y[j].x, g1 * sc * y[j].y};
      const c2 q2 = {g2 * sc * y[j].x, g2 * sc * y[j].y};
      g.x = fmaf(q2.x, inv, q1.x);
      g.y = fmaf(q2.y, inv, q1.y);
      if (a.grad_Y) reinterpret_cast<float2 *>(a.grad_Y)[(size_t)c * a.R + r] = make_float2(g.x, g.y);
    }
    if (r < K2p / 2) {
      // rows (g.x, g.y) and (g.y, -g.x); the split of -x is that of x negated
      __nv_bfloat16 hx, lx, hy, ly;
      split_bf16(g.x, hx, lx);
      split_bf16(g.y, hy, ly);
      const size_t at = kb_pair(2 * c, r, tcg::BM);
      __nv_bfloat162 *h2 = reinterpret_cast<__nv_bfloat162 *>(hi) + at;
      __nv_bfloat162 *l2 = reinterpret_cast<__nv_bfloat162 *>(lo) + at;
      h2[0] = __halves2bfloat162(hx, hy);
      l2[0] = __halves2bfloat162(lx, ly);
      h2[32] = __halves2bfloat162(hy, __hneg(hx));
      l2[32] = __halves2bfloat162(ly, __hneg(lx));
    }
  }
}

// G_U[c, k] = sum over the splits of the partials: 32 entries a CTA, its 8 warps
// share the splits (one thread an entry and 70 splits took 6 us, latency)
__global__ void __launch_bounds__(256) k_gu_reduce(const float *GUp, int splits, long long n,
                                                   float *GU) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * 32 + lane;
  float x = 0.f, y = 0.f;
  if (i < n)
    for (int s = wid; s < splits; s += 8) {
      const float2 v = __ldg(reinterpret_cast<const float2 *>(GUp) + (size_t)s * n + i);
      x += v.x;
      y += v.y;
    }
  __shared__ float2 red[8][32];
  red[wid][lane] = make_float2(x, y);
  __syncthreads();
  if (wid == 0 && i < n) {
#pragma unroll
    for (int w = 1; w < 8; w++) { x += red[w][lane].x; y += red[w][lane].y; }
    reinterpret_cast<float2 *>(GU)[i] = make_float2(x, y);
  }
}

template <int CB>
__global__ void __launch_bounds__(256) k_pass2(ObjArgs a, int M, int K, int rper, const float *G1,
                                               const float *G2, const float *scal, float *GUp) {
  constexpr int TR = CB <= 8 ? 256 : (CB <= 32 ? 64 : 32);
  __shared__ c2 sG[CB][TR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = blockIdx.x * 8 + warp;
  const int r0 = blockIdx.y * rper, r1 = min(a.R, r0 + rper);
  const float inv = G2 ? scal[0] : 0.f;
  const float *row = k < K ? row_ptr(a.Hr, a.Hd, M, a.R, k) : nullptr;
  c2 acc[CB];
#pragma unroll
  for (int c = 0; c < CB; c++) acc[c] = {0.f, 0.f};
  for (int rc = r0; rc < r1; rc += TR) {
    const int rn = min(TR, r1 - rc);
    __syncthreads();
    for (int i = threadIdx.x; i < CB * TR; i += blockDim.x) {
      const int c = i / TR, rr = i % TR;
      c2 g = {0.f, 0.f};
      if (c < a.C && rr < rn) {
        g = ld2(G1, (size_t)c * a.R + rc + rr);
        if (G2) {
          const c2 h = ld2(G2, (size_t)c * a.R + rc + rr);
          g.x = fmaf(h.x, inv, g.x);
          g.y = fmaf(h.y, inv, g.y);
        }
      }
      sG[c][rr] = g;
    }
    __syncthreads();
    if (row) {
#pragma unroll 8
      for (int rr = lane; rr < rn; rr += 32) {
        const c2 h = ld2(row, (size_t)(rc + rr));
#pragma unroll
        for (int c = 0; c < CB; c++) macc(acc[c], sG[c][rr], h);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CB; c++) {
    float x = acc[c].x, y = acc[c].y;
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (lane == 0 && row && c < a.C)
      reinterpret_cast<float2 *>(GUp)[((size_t)blockIdx.y * a.C + c) * K + k] = make_float2(x, y);
  }
}

__device__ __forceinline__ c2 gu_sum(const float *GUp, int rspl, int C, int K, int c, int k) {
  c2 g = {0.f, 0.f};
  int sp = 0;
  for (; sp + 4 <= rspl; sp += 4) {
    c2 v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = ld2(GUp, ((size_t)(sp + j) * C + c) * K + k);
#pragma unroll
    for (int j = 0; j < 4; j++) { g.x += v[j].x; g.y += v[j].y; }
  }
  for (; sp < rspl; sp++) {
    const c2 v = ld2(GUp, ((size_t)sp * C + c) * K + k);
    g.x += v.x;
    g.y += v.y;
  }
  return g;
}

// final: each CTA owns 32 metasurface rows.  It reduces their G_U partials,
// writes dphi[m] = -sum_c Im(conj(G_U) U) and the partial sums
// sum_m G_U[c,m] e^{-j phi'_m} conj(H_a[s,m]) of dL/dW; the last CTA adds the
// CTAs' partials and the H_d rows G_U[c, M+s] into grad_W.
template <int CB>
__global__ void __launch_bounds__(256) k_final(ObjArgs a, int M, int K, int rspl, const float *U,
                                               const float *GUp, float *gw_part,
                                               unsigned *counter) {
  __shared__ c2 gu[CB][32];
  __shared__ c2 ph[32];
  __shared__ bool last;
  const int m0 = blockIdx.x * 32;
  const int t = threadIdx.x;
  const int nm = max(0, min(32, M - m0));
  for (int i = t; i < CB * 32; i += blockDim.x) {
    const int c = i / 32, j = i % 32;
    gu[c][j] = (c < a.C && j < nm) ? gu_sum(GUp, rspl, a.C, K, c, m0 + j) : c2{0.f, 0.f};
  }
  if (t < 32) {
    c2 e = {0.f, 0.f};
    if (t < nm) {
      const float p = py_mod(__ldg(a.phi + m0 + t), a.max_phase);
      sincosf(p, &e.y, &e.x);
    }
    ph[t] = e;
  }
  __syncthreads();
  if (a.grad_phi && t < nm) {
    float sacc = 0.f;
    for (int c = 0; c < a.C; c++) {
      const c2 g = gu[c][t], u = ld2(U, (size_t)c * M + m0 + t);
      sacc += g.x * u.y - g.y * u.x;  // Im(conj(g) u)
    }
    a.grad_phi[m0 + t] = -sacc;
  }
  if (!a.grad_W) return;
  for (int i = t; i < a.C * a.S; i += blockDim.x) {
    const int c = i / a.S, s2 = i % a.S;
    c2 acc = {0.f, 0.f};
    for (int j = 0; j < nm; j++) {
      const c2 g = gu[c][j], e = ph[j];
      const c2 gv = {g.x * e.x + g.y * e.y, g.y * e.x - g.x * e.y};  // g e^{-j p}
      macc(acc, gv, ld2(a.Ha, (size_t)s2 * M + m0 + j));
    }
    reinterpret_cast<float2 *>(gw_part)[(size_t)blockIdx.x * a.C * a.S + i] = make_float2(acc.x, acc.y);
  }
  __threadfence();
  __syncthreads();
  if (t == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = t; i < a.C * a.S; i += blockDim.x) {
    const int c = i / a.S, s2 = i % a.S;
    c2 acc = gu_sum(GUp, rspl, a.C, K, c, M + s2);
    const volatile float2 *pp = reinterpret_cast<const volatile float2 *>(gw_part);
    for (int b = 0; b < (int)gridDim.x; b++) {
      acc.x += pp[(size_t)b * a.C * a.S + i].x;
      acc.y += pp[(size_t)b * a.C * a.S + i].y;
    }
    reinterpret_cast<float2 *>(a.grad_W)[i] = make_float2(acc.x, acc.y);
  }
  if (t == 0) *counter = 0u;  // ready for the next call
}

// dphi[m] = -sum_c Im(conj(G_U[c, m]) U[c, m]); a CTA takes 32 elements
// (lanes) and its 8 warps split the codes
__global__ void __launch_bounds__(256) k_tc_dphi(const float *GU, const float *U, int C, int M,
                                                 int K, float *dphi, const unsigned *err) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int m = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (m < M)
    for (int c = wid; c < C; c += 8) {
      const float2 g = __ldg(reinterpret_cast<const float2 *>(GU) + (size_t)c * K + m);
      const float2 u = __ldg(reinterpret_cast<const float2 *>(U) + (size_t)c * M + m);
      acc += g.x * u.y - g.y * u.x;
    }
  __shared__ float red[8][32];
  red[wid][lane] = acc;
  __syncthreads();
  if (wid == 0 && m < M) {
    float t = 0.f;
#pragma unroll
    for (int w2 = 0; w2 < 8; w2++) t += red[w2][lane];
    dphi[m] = obj_failed(err) ? obj_nan() : -t;
  }
}

// grad_W[c, s] = G_U[c, M + s] + sum_m G_U[c, m] e^{-j phi'_m} conj(H_a[s, m]).
// k_tc_dw_part: a CTA forms 16 AP elements' sums of every code (64 at most) over
// a slice of the m range, 32 of it in shared memory at a time, and writes them
// to dwp[c][part][s]; k_tc_dw_sum adds the slices and the H_d term.  (A CTA per
// code read all of H_a and formed every e^{-j phi'_m} for each code and was
// bound by its shuffles: 18 us for M = 2,304, S = 36, 60 codes, 5 us now.)
// Slices are whole 32s, one where that makes no more than 128 of them.
int dw_parts(int M) {
  const int n = (M + 31) / 32, per = (n + 127) / 128;
  return (n + per - 1) / per;
}
__global__ void __launch_bounds__(256) k_tc_dw_part(const float *GU, const float *Ha,
                                                    const float *phi, float max_phase, int C,
                                                    int S, int M, int K, float *dwp) {
  __shared__ c2 ge[32][65], ha[32][16];
  const int part = blockIdx.x, parts = gridDim.x, s0 = blockIdx.y * 16;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int per = ((M + 31) / 32 + parts - 1) / parts * 32;
  const int m_lo = part * per, m_hi = min(M, m_lo + per);
  const int s = t & 15, cg = t >> 4;  // this thread's sums: codes cg + 16 j
  c2 acc[4];
#pragma unroll
  for (int j = 0; j < 4; j++) acc[j] = {0.f, 0.f};
  for (int m0 = m_lo; m0 < m_hi; m0 += 32) {
    const int m = m0 + lane;
    const bool in = m < m_hi;
    float sn = 0.f, cs = 0.f;
    c2 g[8], h[2];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = warp + 8 * i;
      g[i] = {0.f, 0.f};
      if (in && c < C) g[i] = ld2(GU, (size_t)c * K + m);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int q = s0 + warp + 8 * i;
      h[i] = {0.f, 0.f};
      if (in && q < S) h[i] = ld2(Ha, (size_t)q * M + m);
    }
    if (in) sincosf(py_mod(__ldg(phi + m), max_phase), &sn, &cs);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++)  // g e^{-j p}
      ge[lane][warp + 8 * i] = {g[i].x * cs + g[i].y * sn, g[i].y * cs - g[i].x * sn};
#pragma unroll
    for (int i = 0; i < 2; i++) ha[lane][warp + 8 * i] = h[i];
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < 32; k++) {
      const c2 x = ha[k][s];
#pragma unroll
      for (int j = 0; j < 4; j++) macc(acc[j], ge[k][cg + 16 * j], x);
    }
  }
  if (s0 + s < S)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c = cg + 16 * j;
      if (c < C)
        reinterpret_cast<float2 *>(dwp)[((size_t)c * parts + part) * S + s0 + s] =
            make_float2(acc[j].x, acc[j].y);
    }
}

// out[c][j] = GU[c][k0 + j], j < n (complex), NaN after a run-out wait
__global__ void k_tc_copy_rows(const float *GU, int K, int k0, int n, int C, float *out,
                               const unsigned *err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C * n) return;
  const int c = i / n, j = i % n;
  float2 v = __ldg(reinterpret_cast<const float2 *>(GU) + (size_t)c * K + k0 + j);
  if (obj_failed(err)) v = make_float2(obj_nan(), obj_nan());
  reinterpret_cast<float2 *>(out)[i] = v;
}

// 32 entries a CTA, its 8 warps share the slices
__global__ void __launch_bounds__(256) k_tc_dw_sum(const float *GU, const float *dwp, int C, int S,
                                                   int M, int K, int parts, float *grad_W,
                                                   const unsigned *err) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  const bool in = i < C * S;
  const int c = in ? i / S : 0, s2 = in ? i % S : 0;
  c2 t = {0.f, 0.f};
  if (in) {
    if (wid == 0) t = ld2(GU, (size_t)c * K + M + s2);
    for (int q = wid; q < parts; q += 8) {
      const c2 v = ld2(dwp, ((size_t)c * parts + q) * S + s2);
      t.x += v.x;
      t.y += v.y;
    }
  }
  __shared__ c2 red[8][32];
  red[wid][lane] = t;
  __syncthreads();
  if (wid == 0 && in) {
#pragma unroll
    for (int w = 1; w < 8; w++) { t.x += red[w][lane].x; t.y += red[w][lane].y; }
    if (obj_failed(err)) t = {obj_nan(), obj_nan()};
    reinterpret_cast<float2 *>(grad_W)[i] = make_float2(t.x, t.y);
  }
}

// Streaming paths, after the streaming kernel: one CTA per 32 rows k of
// [H_r; H_d] (lanes, loads coalesced over k), 32 warps.
//   G_U[c, k] = sum_b P1[b][c][k] + (sum_b P2[b][c][k]) / ||masked||, the
//     warps splitting the CTA partials b; every CTA derives 1/||masked|| from
//     the loss partials (CTA 0 also writes the loss);
//   dphi[k] = -sum_c Im(conj(G_U[c, k]) U[c, k]) for metasurface rows;
//   dwp[blk][c][s] = sum over the CTA's metasurface rows of
//     G_U[c, k] e^{-j phi'_k} conj(H_a[s, k]), warp w taking s = w, w + 32, ...
// The last CTA to finish (arrival counter) forms dL/dW: the H_d rows
// G_U[c, M + s] plus the CTAs' dwp, a warp per entry with lanes over CTAs.
template <int CB>
__global__ void __launch_bounds__(1024) k_stream_tail(ObjArgs a, int M, int nparts,
                                                      const float *Ppart, const double *lpart,
                                                      const float *U, float *GU, float *dwp,
                                                      unsigned *counter, const unsigned *err) {
  constexpr int NW = 32;
  const int K = M + a.S;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  // call inputs (not written by the streaming grid) are fetched before the
  // wait: this warp's first H_a row for the dL/dW part and phi for the phase
  const c2 ha_first = warp < a.S && k < M ? ld2(a.Ha, (size_t)warp * M + k) : c2{0.f, 0.f};
  const float phi_k = warp == 0 && k < M ? __ldg(a.phi + k) : 0.f;
  // launched early (programmatic dependent launch): wait for the streaming
  // grid to complete before reading its partials or its wait-timeout word
  cudaGridDependencySynchronize();
  // a bounded wait of the streaming kernel ran out: its partials are
  // incomplete, so every output of the call is NaN
  const bool bad = obj_failed(err);
  __shared__ float inv_s;
  __shared__ c2 r1[NW][CB][32], r2[NW][CB][32];
  __shared__ c2 gv[CB][32];
  // Every loop below issues a batch of UNR independent loads before adding
  // them (in the same order as one load per iteration would), so a warp pays
  // one memory round trip per batch rather than one per partial.
  constexpr int UNR = 8;
  if (warp == 1) {
    double x = 0.0, z = 0.0;
    for (int b0 = lane; b0 < nparts; b0 += 32 * UNR) {
      double xv[UNR], zv[UNR];
#pragma unroll
      for (int u = 0; u < UNR; u++) {
        const int b = b0 + 32 * u;
        xv[u] = b < nparts ? lpart[2 * b] : 0.0;
        zv[u] = b < nparts ? lpart[2 * b + 1] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < UNR; u++) { x += xv[u]; z += zv[u]; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    if (lane == 0) {
      const double nrm = sqrt(z);
      inv_s = nrm > 0 ? (float)(1.0 / nrm) : 0.f;
      if (blockIdx.x == 0 && a.loss) *a.loss = bad ? obj_nan() : (float)(-(double)a.w * x + nrm);
    }
  }
  const float2 *P = reinterpret_cast<const float2 *>(Ppart);
  const int kk = k < K ? k : K - 1;
  c2 s1[CB], s2[CB];
#pragma unroll
  for (int c = 0; c < CB; c++) { s1[c] = {0.f, 0.f}; s2[c] = {0.f, 0.f}; }
  constexpr int UNP = UNR / CB;  // partial loads per batch (registers)
  for (int b0 = warp; b0 < nparts; b0 += NW * UNP) {
    float2 pu[UNP][CB], pv[UNP][CB];
#pragma unroll
    for (int u = 0; u < UNP; u++) {
      const int b = b0 + NW * u;
#pragma unroll
      for (int c = 0; c < CB; c++) {
        const bool on = b < nparts && c < a.C;
        pu[u][c] = on ? __ldg(P + ((size_t)b * 2 * a.C + c) * K + kk) : make_float2(0.f, 0.f);
        if (CB > 1)
          pv[u][c] = on ? __ldg(P + ((size_t)b * 2 * a.C + a.C + c) * K + kk)
                        : make_float2(0.f, 0.f);
      }
    }
#pragma unroll
    for (int u = 0; u < UNP; u++) {
#pragma unroll
      for (int c = 0; c < CB; c++) {
        if (b0 + NW * u >= nparts || c >= a.C) continue;
        s1[c].x += pu[u][c].x;
        s1[c].y += pu[u][c].y;
        if (CB > 1) {
          s2[c].x += pv[u][c].x;
          s2[c].y += pv[u][c].y;
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CB; c++) { r1[warp][c][lane] = s1[c]; r2[warp][c][lane] = s2[c]; }
  __syncthreads();
  if (warp == 0) {
    const float inv = inv_s;
    c2 e = {1.f, 0.f};
    const bool ms_row = k < M;
    if (ms_row) {
      const float pp = py_mod(phi_k, a.max_phase);
      sincosf(pp, &e.y, &e.x);
    }
    float dph = 0.f;
#pragma unroll
    for (int c = 0; c < CB; c++) {
      c2 g = {0.f, 0.f};
      if (c < a.C && k < K) {
        c2 t1 = {0.f, 0.f}, t2 = {0.f, 0.f};
#pragma unroll 8
        for (int w = 0; w < NW; w++) {
          t1.x += r1[w][c][lane].x; t1.y += r1[w][c][lane].y;
          t2.x += r2[w][c][lane].x; t2.y += r2[w][c][lane].y;
        }
        g = {fmaf(t2.x, inv, t1.x), fmaf(t2.y, inv, t1.y)};
        reinterpret_cast<float2 *>(GU)[(size_t)c * K + k] = make_float2(g.x, g.y);
        if (ms_row) {
          const c2 u = ld2(U, (size_t)c * M + k);
          dph += g.x * u.y - g.y * u.x;  // Im(conj(g) u)
        }
      }
      // g e^{-j phi'} of metasurface rows (zero elsewhere) for the dW sums
      gv[c][lane] = ms_row && c < a.C ? c2{g.x * e.x + g.y * e.y, g.y * e.x - g.x * e.y}
                                      : c2{0.f, 0.f};
    }
    if (ms_row && a.grad_phi) a.grad_phi[k] = bad ? obj_nan() : -dph;
  }
  if (!a.grad_W) return;
  __syncthreads();
  for (int s2 = warp; s2 < a.S; s2 += NW) {
    const c2 h = s2 == warp ? ha_first : k < M ? ld2(a.Ha, (size_t)s2 * M + k) : c2{0.f, 0.f};
#pragma unroll
    for (int c = 0; c < CB; c++) {
      if (c >= a.C) continue;
      c2 d = {0.f, 0.f};
      macc(d, gv[c][lane], h);
      for (int o = 16; o > 0; o >>= 1) {
        d.x += __shfl_xor_sync(0xffffffffu, d.x, o);
        d.y += __shfl_xor_sync(0xffffffffu, d.y, o);
      }
      if (lane == 0)
        reinterpret_cast<float2 *>(dwp)[((size_t)blockIdx.x * a.C + c) * a.S + s2] =
            make_float2(d.x, d.y);
    }
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = warp; i < a.C * a.S; i += NW) {
    const int c = i / a.S, s2 = i % a.S;
    const float2 g = __ldcg(reinterpret_cast<const float2 *>(GU) + (size_t)c * K + M + s2);
    c2 acc = {0.f, 0.f};
    for (int b = lane; b < (int)gridDim.x; b += 32) {
      const float2 v = __ldcg(reinterpret_cast<const float2 *>(dwp) + (size_t)b * a.C * a.S + i);
      acc.x += v.x;
      acc.y += v.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (lane == 0) {
      reinterpret_cast<float2 *>(a.grad_W)[i] =
          bad ? make_float2(obj_nan(), obj_nan()) : make_float2(g.x + acc.x, g.y + acc.y);
    }
  }
  if (threadIdx.x == 0) *counter = 0u;  // ready for the next call
}

// grad_Y = G1 + G2 / ||masked||
__global__ void k_grad_y(const float *G1, const float *G2, const float *scal, long long n,
                         float *out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float inv = G2 ? scal[0] : 0.f;
  c2 g = ld2(G1, i);
  if (G2) {
    const c2 h = ld2(G2, i);
    g.x = fmaf(h.x, inv, g.x);
    g.y = fmaf(h.y, inv, g.y);
  }
  reinterpret_cast<float2 *>(out)[i] = make_float2(g.x, g.y);
}

int cbucket(int C) {
  int b = 1;
  while (b < C) b <<= 1;
  return b;
}

// CTAs the CUDA-core split path aims for: a work split that fills a device
// of this size (8 per SM on a 152-SM GB300) and that fixes the scratch
// layout, so it is a constant rather than a device query
constexpr int kTargetBlocks = 1216;

struct Split {
  int K, kspl, kper, rspl, rper, nb_epi;
};

Split make_split(int S, int M, int R) {
  Split sp;
  sp.K = M + S;
  const int bx = (R + 31) / 32;
  sp.kspl = std::max(1, std::min((kTargetBlocks + bx - 1) / bx, (sp.K + 63) / 64));
  sp.kper = (sp.K + sp.kspl - 1) / sp.kspl;
  sp.kspl = (sp.K + sp.kper - 1) / sp.kper;
  const int by = (sp.K + 7) / 8;
  sp.rspl = std::max(1, std::min((kTargetBlocks + by - 1) / by, (R + 255) / 256));
  sp.rper = (R + sp.rspl - 1) / sp.rspl;
  sp.rspl = (R + sp.rper - 1) / sp.rper;
  sp.nb_epi = (R + 127) / 128;
  return sp;
}

template <int CB>
cudaError_t run_cb(const ObjArgs &a, const Split &sp, int M, float *U, float *Ypart, float *G1,
                   float *G2, double *part, unsigned *counter, float *scal, float *GUp,
                   float *gw_part, cudaStream_t st) {
  if (M > 0) {
    dim3 gp((M + 127) / 128, a.C);
    k_prep<<<gp, 128, 0, st>>>(a, M, U, nullptr);
  }
  dim3 g1((a.R + 31) / 32, sp.kspl);
  k_pass1<CB><<<g1, 256, 0, st>>>(a, M, sp.K, sp.kper, U, Ypart);
  if (CB >= 8)
    k_epilogue_wide<(CB >= 8 ? CB : 8)><<<(a.R + 31) / 32, 256, 0, st>>>(a, sp.kspl, Ypart, G1,
                                                                        G2, part, counter, scal);
  else
    k_epilogue<CB><<<sp.nb_epi, 128, 0, st>>>(a, sp.kspl, Ypart, G1, G2, part, counter, scal,
                                              nullptr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (a.grad_Y) {
    const long long n = (long long)a.C * a.R;
    k_grad_y<<<(int)((n + 255) / 256), 256, 0, st>>>(G1, G2, scal, n, a.grad_Y);
  }
  if (!a.grad_W && !a.grad_phi) return cudaGetLastError();
  dim3 g2((sp.K + 7) / 8, sp.rspl);
  k_pass2<CB><<<g2, 256, 0, st>>>(a, M, sp.K, sp.rper, G1, G2, scal, GUp);
  const int nbf = std::max(1, (M + 31) / 32);
  k_final<CB><<<nbf, 256, 0, st>>>(a, M, sp.K, sp.rspl, U, GUp, gw_part, counter + 1);
  return cudaGetLastError();
}

// ------------------------------------------------------------------
// Single-pass streaming path (one HBM read of H_r and H_d).
//
// A cluster of CTAs walks column tiles of TR = 16 (or 8) Rx: the K = M + S rows
// of [H_r; H_d] are split among the cluster's CTAs, so that a row's piece of a
// tile is a whole 128-byte line (64 bytes) and a CTA's part of a tile still
// fits its shared memory several times.  TMA copies (cp.async.bulk.tensor,
// swizzled, mbarrier completion) fill a ring of stages.  For each tile a CTA
// (A) forms its rows' part of Y, which the cluster's CTAs send each other through
// distributed shared memory, then (B) evaluates the per-Rx capacity, max and
// mask and the two gradient parts, and (C) accumulates P1[c,k] += sum_col
// G1[c,col] conj(H[k,col]) (and P2 for the norm term) from the same
// shared-memory tile.  Two warps do B while the others run A of later tiles: B
// is a chain of 800 cycles for 16 columns, and done by every warp it took half
// of the kernel's instructions.  The clusters' P1 / P2 and loss partials are
// reduced by k_stream_tail.

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// bounded mbarrier wait of the tcgen05 kernels (tc_ptx.cuh): try_wait with a
// suspend-time hint, so waiting warps sleep instead of taking issue slots
// from the other CTA on the SM; false after 2 s
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity) {
  return tc::mbar_wait(bar, parity);
}
// the same for a whole warp, one answer for all lanes
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) {
  return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity));
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// store into CTA `rank` of the cluster; its mbarrier counts the 8 bytes (no fence
// and no barrier on either side: a cluster barrier with its release cost about
// 4 us a tile here).  st.async is an illegal instruction in a kernel that was
// launched without a cluster dimension.
__device__ __forceinline__ void cluster_store(uint32_t addr, uint32_t bar, int rank, c2 v) {
  uint32_t a, b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(bar), "r"(rank));
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a),
      "f"(v.x), "f"(v.y), "r"(b)
      : "memory");
}

// per-Rx capacity of one column: the gradient parts ga (max term) and gb (norm
// term, before 1 / ||masked||) of every code, the max over codes, the squares
// of the masked capacities and the amplitudes
template <int CB>
__device__ __forceinline__ void stream_column(const ObjArgs &a, const c2 (&y)[CB], c2 (&ga)[CB],
                                              c2 (&gb)[CB], float &mx, float &sq,
                                              float (&amp)[CB]) {
  float cap[CB];
  int arg = 0;
  mx = -1.f;
  sq = 0.f;
#pragma unroll
  for (int c = 0; c < CB; c++) {
    if (c >= a.C) { cap[c] = 0.f; amp[c] = 0.f; continue; }
    amp[c] = sqrtf(y[c].x * y[c].x + y[c].y * y[c].y);
    const float aa = amp[c] + kEps;
    float v = log2f(1.0f + aa * aa / kN0);
    if (a.drop && a.drop[c]) v = 0.f;
    cap[c] = v;
    if (v > mx) { mx = v; arg = c; }
  }
#pragma unroll
  for (int c = 0; c < CB; c++) {
    ga[c] = {0.f, 0.f};
    gb[c] = {0.f, 0.f};
    if (c >= a.C) continue;
    const bool dropped = a.drop && a.drop[c];
    const float msk = (cap[c] != mx) ? cap[c] : 0.f;
    sq += msk * msk;
    const float aa = amp[c] + kEps;
    const float dcap = (2.0f * aa / kN0) / (1.0f + aa * aa / kN0) * kInvLn2;
    float g1 = (c == arg) ? -a.w : 0.f, g2 = msk;
    if (dropped) { g1 = 0.f; g2 = 0.f; }
    const float sc = amp[c] > 0.f ? dcap / amp[c] : 0.f;
    ga[c] = {g1 * sc * y[c].x, g1 * sc * y[c].y};
    gb[c] = {g2 * sc * y[c].x, g2 * sc * y[c].y};
  }
}

// The split of a problem over clusters (stream_plan).
struct StreamShape {
  int M, K, S, Kc;   // rows of a CTA: virtual rows rank * Kc on
  int boxR;          // rows of an H_r box (divides Kc)
  int rows;          // rows of a stage: Kc and the room for padded H_d rows
  int CL, stages, ntiles;
};
constexpr int kHdBox = 8;   // rows of an H_d box
// Tiles between A and C of a compute warp, and epilogue warps (tile i goes to
// warp i mod kLag): the exchange and B of a tile take about two tiles' time.
constexpr int kLag = 2;
constexpr int kNC = 16;  // compute warps
constexpr int kMaxClusters = 512;  // partials the scratch holds
// Buffers of what passes between the roles.  A compute warp that works on tile i
// has read G of tile i - kLag - 1, so every CTA of the cluster had reached that
// tile's A: what is older than 2 kLag + 2 tiles has been read everywhere, what
// is older than kLag + 1 in this CTA.
constexpr int kSlots = 8, kBufs = 4;
static_assert(kSlots >= 2 * kLag + 3 && kSlots <= 8 && kBufs >= kLag + 2, "buffers");

// 16-byte chunk ch of row s in a stage, as the copy's swizzle places it
template <int TR>
__device__ __forceinline__ uint32_t tile_chunk(int s, int ch) {
  return TR == 16 ? (uint32_t)s * 128u + (uint32_t)((ch ^ (s & 7)) << 4)
                  : (uint32_t)s * 64u + (uint32_t)((ch ^ ((s >> 1) & 3)) << 4);
}

// Warps 0 .. NC - 1 compute (A and C), warps NC .. NC + kLag - 1 form G (the
// exchange and B), the last warp copies.  The roles meet on mbarriers only, all
// waits bounded; a wait that ran out ends its role, the others' waits run out
// in turn, and the CTAs of the cluster leave together.
template <int CB, int TR, int RPT>
__global__ void __launch_bounds__(32 * (kNC + kLag + 1), 1)
    k_obj_stream(const __grid_constant__ ObjArgs a, const __grid_constant__ CUtensorMap mapR,
                 const __grid_constant__ CUtensorMap mapD, const StreamShape sh, const float *U,
                 float *Ppart, double *lpart, unsigned *err) {
  constexpr int NC = kNC, NT = 32 * NC, CH = TR / 2;  // chunks of a row
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  const uint32_t stage_bytes = (uint32_t)sh.rows * (TR * 8u);
  c2 *coef = reinterpret_cast<c2 *>(base + (size_t)sh.stages * stage_bytes);  // [rows][CB]
  c2 *ybuf = coef + (size_t)sh.rows * CB;              // [kSlots][CL][CB][TR]
  __shared__ __align__(16) c2 red[kBufs][NC][CB][TR];
  __shared__ __align__(16) c2 gbuf[kBufs][2 * CB][TR];
  __shared__ __align__(8) uint64_t full[8], empty[8], redf[kBufs], gf[kBufs], got[kSlots];
  __shared__ double sums[kLag][2];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int rank = (int)blockIdx.x % sh.CL, cluster = (int)blockIdx.x / sh.CL,
            nclusters = (int)gridDim.x / sh.CL;
  // this CTA's virtual rows [k0, k1): nr rows of H_r at stage rows 0 on, nd
  // rows of H_d from d0 on at stage rows hd on
  const int k0 = rank * sh.Kc, k1 = min(sh.K, k0 + sh.Kc);
  const int nr = max(0, min(k1, sh.M) - k0), nd = max(0, k1 - max(k0, sh.M)),
            d0 = max(k0 - sh.M, 0);
  const int hd = (nr + sh.boxR - 1) / sh.boxR * sh.boxR;
  const int used = nd > 0 ? hd + nd : nr;  // stage rows that hold anything
  const int n = cluster < sh.ntiles ? (sh.ntiles - cluster + nclusters - 1) / nclusters : 0;
  if (t < 8) {
    if (t < sh.stages) { tc::mbar_init(&full[t], 1); tc::mbar_init(&empty[t], NC); }
    if (t < kBufs) { tc::mbar_init(&redf[t], NC); tc::mbar_init(&gf[t], 1); }
    if (t < kSlots) tc::mbar_init(&got[t], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // every CTA of the cluster runs, its barriers set, before anyone stores into
  // its memory.  A CTA alone is launched without a cluster and takes no cluster
  // instruction: S = 4, M = 16, R = 512 12.7 -> 11.8 us, M = 64, R = 1,024 13.0 ->
  // 12.2 (a CTA without roles per tile of 8 Rx: 11.3 and 12.0, but M = 256, R =
  // 4,096 16.4 against 14.0)
  __syncthreads();
  if (sh.CL > 1) {
    cluster_arrive();
    cluster_wait();
  }

  if (warp == NC + kLag) {
    // ---- copies
    if (lane == 0) {
      const int n_box = hd / sh.boxR, d_box = (nd + kHdBox - 1) / kHdBox;
      const uint32_t tx = (uint32_t)(hd + d_box * kHdBox) * (TR * 8u);
      int it = 0;
      bool ok = true;
      for (; it < n; it++) {
        const int stg = it % sh.stages;
        if (it >= sh.stages &&
            !mbar_wait_bounded(&empty[stg], (uint32_t)(it / sh.stages - 1) & 1u)) {
          ok = false;
          break;
        }
        unsigned char *dst = base + (size_t)stg * stage_bytes;
        const int x = (cluster + it * nclusters) * TR * 2;
        tc::mbar_expect_tx(&full[stg], tx);
        for (int i = 0; i < n_box; i++)
          tc::tma_load_2d(dst + (size_t)i * sh.boxR * (TR * 8), &mapR, x, k0 + i * sh.boxR, &full[stg]);
        for (int i = 0; i < d_box; i++)
          tc::tma_load_2d(dst + (size_t)(hd + i * kHdBox) * (TR * 8), &mapD, x, d0 + i * kHdBox,
                          &full[stg]);
      }
      if (!ok) atomicOr(err, 1u);
      // the copies issued land before the CTA exits (in a good run the compute
      // warps have seen them land; the last ones are looked at again)
      for (int i = max(0, it - sh.stages); i < it; i++)
        mbar_wait_bounded(&full[i % sh.stages], (uint32_t)(i / sh.stages) & 1u);
    }
  } else if (warp >= NC) {
    // ---- G of tiles warp - NC, warp - NC + kLag, ...
    double sum_max = 0.0, sum_sq = 0.0;
    const int col = lane & (TR - 1), cs = lane / TR;
    for (int it = warp - NC; it < n; it += kLag) {
      const int bi = it % kBufs, si = it % kSlots;
      if (!warp_wait(&redf[bi], (uint32_t)(it / kBufs) & 1u)) { atomicOr(err, 1u); break; }
      if (lane == 0 && sh.CL > 1)
        tc::mbar_expect_tx(&got[si], (uint32_t)(sh.CL * CB * TR * sizeof(c2)));
      __syncwarp();
      if (cs < CB) {  // the CTA's part of Y, to every CTA of the cluster
        c2 v[NC];  // added in pairs
#pragma unroll
        for (int w = 0; w < NC; w++) v[w] = red[bi][w][cs][col];
#pragma unroll
        for (int h = NC / 2; h > 0; h /= 2)
#pragma unroll
          for (int w = 0; w < h; w++) { v[w].x += v[w + h].x; v[w].y += v[w + h].y; }
        c2 *at = ybuf + ((size_t)(si * sh.CL + rank) * CB + cs) * TR + col;
        if (sh.CL > 1)
          for (int r = 0; r < sh.CL; r++)
            cluster_store(smem_addr(at), smem_addr(&got[si]), r, v[0]);
        else
          *at = v[0];
      }
      __syncwarp();
      if (sh.CL > 1 && !warp_wait(&got[si], (uint32_t)(it / kSlots) & 1u)) {
        atomicOr(err, 1u);
        break;
      }
      const c2 *yb = ybuf + (size_t)si * sh.CL * CB * TR;
      c2 y[CB], ga[CB], gb[CB];
#pragma unroll
      for (int c = 0; c < CB; c++) {
        y[c] = {0.f, 0.f};
        for (int r = 0; r < sh.CL; r++) {
          const c2 v = yb[(r * CB + c) * TR + col];
          y[c].x += v.x;
          y[c].y += v.y;
        }
      }
      float mx, sq, amp[CB];
      stream_column<CB>(a, y, ga, gb, mx, sq, amp);
      const int r = (cluster + it * nclusters) * TR + col;
      const bool live = r < a.R;
      if (lane < TR) {
#pragma unroll
        for (int c = 0; c < CB; c++) {
          gbuf[bi][c][col] = live ? ga[c] : c2{0.f, 0.f};
          if (CB > 1) gbuf[bi][CB + c][col] = live ? gb[c] : c2{0.f, 0.f};
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&gf[bi]);
      // (what C does not wait for: FP64 sums cost nothing here)
      if (rank == 0 && live && lane < TR) {
        sum_max += (double)mx;
        sum_sq += (double)sq;
        if (a.recv_amp)
#pragma unroll
          for (int c = 0; c < CB; c++)
            if (c < a.C) a.recv_amp[(size_t)c * a.R + r] = amp[c];
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      sum_max += __shfl_xor_sync(0xffffffffu, sum_max, o);
      sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
    }
    // (the barrier below orders the warps' sums)
    if (lane == 0) { sums[warp - NC][0] = sum_max; sums[warp - NC][1] = sum_sq; }
  }
  c2 p1[RPT][CB], p2[RPT][CB];
#pragma unroll
  for (int q = 0; q < RPT; q++)
#pragma unroll
    for (int c = 0; c < CB; c++) { p1[q][c] = {0.f, 0.f}; p2[q][c] = {0.f, 0.f}; }
  if (warp < NC) {
    // ---- compute.  The first tiles are on their way; wait for the U kernel,
    // then stage the coefficients of the stage's rows (0 for padding): U for
    // metasurface rows, W for the H_d rows
    cudaGridDependencySynchronize();
    for (int i = t; i < sh.rows * CB; i += NT) {
      const int s = i / CB, c = i % CB;
      c2 v = {0.f, 0.f};
      if (c < a.C) {
        if (s < nr) v = ld2(U, (size_t)c * sh.M + k0 + s);
        else if (s >= hd && s - hd < nd) v = ld2(a.W, (size_t)c * sh.S + d0 + s - hd);
      }
      coef[i] = v;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");  // the compute warps
    for (int it = 0; it < n + kLag; it++) {
      // (A) this CTA's part of Y for the columns: CH lanes take a row's 16-byte
      // chunks (two columns each), a warp 32 / CH rows at a time
      if (it < n) {
        const int stg = it % sh.stages;
        if (!warp_wait(&full[stg], (uint32_t)(it / sh.stages) & 1u)) {
          atomicOr(err, 1u);
          break;
        }
        const unsigned char *T = base + (size_t)stg * stage_bytes;
        c2 y0[CB], y1[CB];
#pragma unroll
        for (int c = 0; c < CB; c++) { y0[c] = {0.f, 0.f}; y1[c] = {0.f, 0.f}; }
        const int sub = lane / CH, ch = lane % CH;
#pragma unroll 4
        for (int s = 32 / CH * warp + sub; s < used; s += 32 / CH * NC) {
          const float4 h = *reinterpret_cast<const float4 *>(T + tile_chunk<TR>(s, ch));
#pragma unroll
          for (int c = 0; c < CB; c++) {
            const c2 u = coef[s * CB + c];
            mac(y0[c], u, c2{h.x, h.y});
            mac(y1[c], u, c2{h.z, h.w});
          }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < CB; c++) {
#pragma unroll
          for (int o = CH; o < 32; o <<= 1) {
            y0[c].x += __shfl_xor_sync(0xffffffffu, y0[c].x, o);
            y0[c].y += __shfl_xor_sync(0xffffffffu, y0[c].y, o);
            y1[c].x += __shfl_xor_sync(0xffffffffu, y1[c].x, o);
            y1[c].y += __shfl_xor_sync(0xffffffffu, y1[c].y, o);
          }
          if (lane < CH)
            *reinterpret_cast<float4 *>(&red[it % kBufs][warp][c][2 * ch]) =
                make_float4(y0[c].x, y0[c].y, y1[c].x, y1[c].y);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&redf[it % kBufs]);
      }
      if (it < kLag) continue;
      // (C) P += G conj(H) over the columns of the tile kLag before, a thread
      // per row.  A tile is summed by itself first: a cluster sums 1/36 of the
      // Rx, and in one FP32 chain the error of dphi came to 1.1e-6 (M = 2,304,
      // R = 65,536) against 4e-7 of 152 shorter chains
      const int ct = it - kLag, bi = ct % kBufs;
      if (!warp_wait(&gf[bi], (uint32_t)(ct / kBufs) & 1u)) {
        atomicOr(err, 1u);
        break;
      }
      const unsigned char *T = base + (size_t)(ct % sh.stages) * stage_bytes;
      // the tile's sums (of eight columns where the registers need it)
      constexpr bool kEight = CB * RPT > 2;
      c2 t1[RPT][CB], t2[RPT][CB];
#pragma unroll
      for (int hcol = 0; hcol < TR; hcol += 8) {
        c2 g1[CB][8], g2[CB][8];
#pragma unroll
        for (int c = 0; c < CB; c++)
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            const float4 u = *reinterpret_cast<const float4 *>(&gbuf[bi][c][hcol + j]);
            g1[c][j] = {u.x, u.y};
            g1[c][j + 1] = {u.z, u.w};
            if (CB > 1) {
              const float4 v = *reinterpret_cast<const float4 *>(&gbuf[bi][CB + c][hcol + j]);
              g2[c][j] = {v.x, v.y};
              g2[c][j + 1] = {v.z, v.w};
            }
          }
#pragma unroll
        for (int q = 0; q < RPT; q++) {
          const int s = t + NT * q;
          if (kEight || hcol == 0)
#pragma unroll
            for (int c = 0; c < CB; c++) { t1[q][c] = {0.f, 0.f}; t2[q][c] = {0.f, 0.f}; }
          if (s < used) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              const float4 h =
                  *reinterpret_cast<const float4 *>(T + tile_chunk<TR>(s, (hcol + j) >> 1));
#pragma unroll
              for (int c = 0; c < CB; c++) {
                macc(t1[q][c], g1[c][j], c2{h.x, h.y});
                macc(t1[q][c], g1[c][j + 1], c2{h.z, h.w});
                if (CB > 1) {
                  macc(t2[q][c], g2[c][j], c2{h.x, h.y});
                  macc(t2[q][c], g2[c][j + 1], c2{h.z, h.w});
                }
              }
            }
          }
          if (kEight || hcol == TR - 8)
#pragma unroll
            for (int c = 0; c < CB; c++) {
              p1[q][c].x += t1[q][c].x;
              p1[q][c].y += t1[q][c].y;
              if (CB > 1) { p2[q][c].x += t2[q][c].x; p2[q][c].y += t2[q][c].y; }
            }
        }
      }
      // the stage is free: this warp's generic reads before the async-proxy
      // refill
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[ct % sh.stages]);
    }
  }
  // no CTA leaves while another one may still store into its memory
  __syncwarp();
  if (sh.CL > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  // the tail kernel may launch now; its grid-dependency wait still waits for
  // this grid to complete, with every write below visible
  cudaTriggerProgrammaticLaunchCompletion();
  if (warp >= NC) {
    if (rank == 0 && t == NT) {
      double x = 0.0, z = 0.0;
      for (int e = 0; e < kLag; e++) { x += sums[e][0]; z += sums[e][1]; }
      lpart[2 * cluster] = x;
      lpart[2 * cluster + 1] = z;
    }
    return;
  }
  // partials of this cluster: P1 at [b][c][k], P2 at [b][C + c][k]
#pragma unroll
  for (int q = 0; q < RPT; q++) {
    const int s = t + NT * q;
    if (s >= used || (s >= nr && s < hd)) continue;
    const int k = s < nr ? k0 + s : sh.M + d0 + s - hd;
#pragma unroll
    for (int c = 0; c < CB; c++) {
      if (c >= a.C) continue;
      float2 *o = reinterpret_cast<float2 *>(Ppart) + ((size_t)cluster * 2 * a.C + c) * sh.K + k;
      o[0] = make_float2(p1[q][c].x, p1[q][c].y);
      if (CB > 1) o[(size_t)a.C * sh.K] = make_float2(p2[q][c].x, p2[q][c].y);
    }
  }
}

// the coefficients of the virtual rows into shared memory, coef[k][c]: U for
// metasurface rows, W for the H_d rows.  Four loads per thread are issued
// before their stores, so the staging costs one memory round trip per four
// rows instead of one per row.
template <int NTH, int CB>
__device__ __forceinline__ void stage_coef(const ObjArgs &a, int M, int K, const float *U,
                                           c2 *coef) {
  const int n = K * CB;
  for (int i0 = threadIdx.x; i0 < n; i0 += 4 * NTH) {
    c2 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = i0 + u * NTH, k = i / CB, c = i % CB;
      v[u] = {0.f, 0.f};
      if (i < n && c < a.C)
        v[u] = k < M ? ld2(U, (size_t)c * M + k) : ld2(a.W, (size_t)c * a.S + (k - M));
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * NTH < n) coef[i0 + u * NTH] = v[u];
  }
}

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                              const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                              const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn tmap_encoder() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  }
  return fn;
}

// complex [rows, R] as a float [rows, 2R] tensor; box of 2 TR floats (one
// swizzle row of 128 or 64 bytes) x box_rows
bool make_cmap(CUtensorMap *m, const float *base, int rows, int R, int TR, int box_rows) {
  EncodeFn enc = tmap_encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)2 * R, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)R * 8};
  cuuint32_t box[2] = {(cuuint32_t)(2 * TR), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             TR == 16 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct StreamPlan {
  bool ok = false;
  StreamShape sh{};
  int TR = 0, rpt = 0;  // Rx of a tile, rows of a thread
  size_t smem = 0;
};

int sm_count() { return ams_device_sms(); }

// Shared memory of a CTA (227 KB an SM can give one), and its static part.
constexpr size_t kStreamSmem = 226 * 1024;
constexpr size_t stream_static_smem(int CB, int TR) {
  return sizeof(c2) * TR * CB * kBufs * (kNC + 2) + 512;
}

// The smallest cluster whose CTAs hold their part of a tile in enough stages
// (kLag tiles between A and C, the one in A, two on their way): tiles of 16 Rx
// while a cluster of four will do (K up to 1,300), then of 8 Rx (up to 2,550,
// and to 3,200 with one on its way).
// Clusters of eight are half as many and no faster each: 250 us against 128 us
// with clusters of four at K = 1,040, R = 65,536.
StreamPlan stream_plan(int S, int M, int R, int C, bool grad_y) {
  StreamPlan p;
  const int CB = cbucket(C);
  if (grad_y || CB > 2 || R % 2 || M < 0) return p;
  const int K = M + S;
  struct { int TR, ahead; } const tiles[] = {{16, 2}, {8, 2}, {8, 1}};
  for (const auto &tl : tiles)
    for (int CL : {1, 2, 4}) {
      const int TR = tl.TR;
      StreamShape h{};
      h.M = M; h.K = K; h.S = S; h.CL = CL;
      // up to 5% more rows where that splits them into fewer boxes (a box has
      // 256 rows at most, a multiple of 8)
      int boxes = 1 << 30;
      const int least = ((K + CL - 1) / CL + 7) / 8 * 8;
      for (int Kc = least; Kc <= least + least / 20; Kc += 8) {
        int nb = 1;
        while (Kc / 8 % nb || Kc / nb > 256) nb++;
        if (nb < boxes) { boxes = nb; h.Kc = Kc; h.boxR = Kc / nb; }
      }
      h.rows = h.Kc + (M > 0 ? (std::min(S, h.Kc) + kHdBox - 1) / kHdBox * kHdBox : 0);
      const int rpt = (h.rows + 32 * kNC - 1) / (32 * kNC);
      if (rpt > 2) continue;
      const size_t dyn = 1024 + sizeof(c2) * CB * ((size_t)h.rows + (size_t)kSlots * CL * TR);
      const size_t room = kStreamSmem - stream_static_smem(CB, TR);
      const size_t stage = (size_t)h.rows * TR * 8;
      if (dyn + (kLag + 1 + tl.ahead) * stage > room) continue;
      h.stages = (int)std::min<size_t>(8, (room - dyn) / stage);
      h.ntiles = (R + TR - 1) / TR;
      p.sh = h;
      p.TR = TR;
      p.rpt = rpt;
      p.smem = dyn + h.stages * stage;
      p.ok = true;
      return p;
    }
  return p;
}

template <int CB, int TR, int RPT>
cudaError_t launch_stream_t(const ObjArgs &a, const StreamPlan &pl, const CUtensorMap &mr,
                            const CUtensorMap &md, const float *U, float *Ppart, double *lpart,
                            unsigned *err, int *clusters, cudaStream_t st) {
  auto kfn = k_obj_stream<CB, TR, RPT>;
  static size_t set_bytes[AMS_MAX_DEVICES] = {0};
  // the most dynamic shared memory of any plan (the static part beside it)
  const size_t room = kStreamSmem - stream_static_smem(CB, TR);
  cudaError_t e = ams_set_smem_atleast(set_bytes, kfn, room);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(32 * (kNC + kLag + 1));
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)pl.sh.CL;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  // clusters resident at once with the most shared memory this kernel takes,
  // looked up once per device and cluster size
  static std::atomic<int> resident[AMS_MAX_DEVICES][3];
  const int dev = ams_current_device();
  if (dev < 0) return cudaErrorInvalidDevice;
  const int ci = pl.sh.CL == 1 ? 0 : pl.sh.CL == 2 ? 1 : 2;
  int most = resident[dev][ci].load();
  if (most == 0) {
    cfg.attrs = attr + 1;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)pl.sh.CL);
    cfg.dynamicSmemBytes = room;
    if ((e = cudaOccupancyMaxActiveClusters(&most, kfn, &cfg)) != cudaSuccess) return e;
    most = std::max(1, std::min(most, kMaxClusters));
    resident[dev][ci].store(most);
  }
  *clusters = std::min(most, pl.sh.ntiles);
  cfg.attrs = attr;
  cfg.numAttrs = pl.sh.CL > 1 ? 2 : 1;
  cfg.gridDim = dim3((unsigned)(*clusters * pl.sh.CL));
  cfg.dynamicSmemBytes = pl.smem;
  return cudaLaunchKernelEx(&cfg, kfn, a, mr, md, pl.sh, U, Ppart, lpart, err);
}

template <int CB>
cudaError_t stream_tail(const ObjArgs &a, int M, int nparts, const float *U, const float *Pp,
                        const double *lp, float *GU, float *dwp, unsigned *counter,
                        const unsigned *err, cudaStream_t st);

template <int CB>
cudaError_t run_stream(const ObjArgs &a, const StreamPlan &pl, int M, float *U, float *Ppart,
                       double *lpart, float *GU, float *dwp, unsigned *err, unsigned *counter,
                       cudaStream_t st) {
  CUtensorMap mr, md;
  const float *Hr = M > 0 ? a.Hr : a.Hd;  // no metasurface: mapR is unused
  if (!make_cmap(&mr, Hr, std::max(M, 1), a.R, pl.TR, pl.sh.boxR) ||
      !make_cmap(&md, a.Hd, a.S, a.R, pl.TR, kHdBox))
    return cudaErrorInvalidValue;
  if (M > 0) {
    const long long n = (long long)M * a.C * 8;
    k_prep_wide<<<(int)((n + 255) / 256), 256, 0, st>>>(a, M, U, err);
  }
  cudaError_t e = obj_begin_call(err, M > 0, st);
  if (e != cudaSuccess) return e;
  int clusters = 0;
  if (pl.TR == 16 && pl.rpt == 1)
    e = launch_stream_t<CB, 16, 1>(a, pl, mr, md, U, Ppart, lpart, err, &clusters, st);
  else if (pl.TR == 16)
    e = launch_stream_t<CB, 16, 2>(a, pl, mr, md, U, Ppart, lpart, err, &clusters, st);
  else if (pl.rpt == 1)
    e = launch_stream_t<CB, 8, 1>(a, pl, mr, md, U, Ppart, lpart, err, &clusters, st);
  else
    e = launch_stream_t<CB, 8, 2>(a, pl, mr, md, U, Ppart, lpart, err, &clusters, st);
  if (e != cudaSuccess) return e;
  return stream_tail<CB>(a, M, clusters, U, Ppart, lpart, GU, dwp, counter, err, st);
}

// after a streaming kernel: G_U, dphi and the dL/dW parts, then dL/dW
template <int CB>
cudaError_t stream_tail(const ObjArgs &a, int M, int nparts, const float *U, const float *Pp,
                        const double *lp, float *GU, float *dwp, unsigned *counter,
                        const unsigned *err, cudaStream_t st) {
  const int K = M + a.S, nblk = (K + 31) / 32;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk);
  cfg.blockDim = dim3(1024);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_stream_tail<CB>, a, M, nparts, Pp, lp, U, GU, dwp, counter,
                            err);
}

// ------------------------------------------------------------------
// Streaming path on a plan's transposed copy HT [Rp][Kp] of [H_r; H_d]
// (row r = column r over all k), for an odd number of Rx and K beyond
// k_obj_stream's: a tile of TR Rx is one contiguous block of
// TR * Kp * 8 bytes, fetched by a single cp.async.bulk.  A CTA has all rows of
// its tile, takes the phases A, B, C one after the other and writes its own
// partials; in (A) warp w takes column w % TR and every (NW / TR)-th run of 32
// k, lanes over k.

__global__ void __launch_bounds__(256) k_make_ht(const float *Hr, const float *Hd, int M, int S,
                                                 int R, int Rp, int Kp, float *HT) {
  __shared__ float2 tl[32][33];
  const int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32, K = M + S;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int k = k0 + i, r = r0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (k < K && r < R)
      v = __ldg(reinterpret_cast<const float2 *>(k < M ? Hr + (size_t)k * R * 2
                                                        : Hd + (size_t)(k - M) * R * 2) + r);
    tl[i][threadIdx.x] = v;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, k = k0 + threadIdx.x;
    if (r < Rp && k < Kp) reinterpret_cast<float2 *>(HT)[(size_t)r * Kp + k] = tl[threadIdx.x][i];
  }
}

template <int CB, int TR, int KPT>
__global__ void __launch_bounds__(256)
    k_obj_stream_t(ObjArgs a, const float *HT, int M, int Kp, int stage_bytes, int ntiles,
                   const float *U, float *Ppart, double *lpart, unsigned *err) {
  constexpr int NTH = 256, NW = NTH / 32, NPART = NW / TR;
  const int K = M + a.S;
  const uint32_t tile_bytes = (uint32_t)TR * Kp * 8;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  c2 *coef = reinterpret_cast<c2 *>(base + 2 * (size_t)stage_bytes);  // [K][CB]
  __shared__ c2 red[NW][CB];
  __shared__ c2 g1s[CB][TR], g2s[CB][TR];
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int abort_flag;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

  auto issue = [&](int tile, int stage) {
    uint64_t *bar = &full[stage];
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(tile_bytes)
                 : "memory");
    const float *src = HT + (size_t)tile * TR * Kp * 2;
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_addr(base + (size_t)stage * stage_bytes)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(tile_bytes), "r"(smem_addr(bar))
        : "memory");
  };
  const int first = blockIdx.x;
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&full[0])), "r"(1));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&full[1])), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    if (first < ntiles) issue(first, 0);
    if (first + (int)gridDim.x < ntiles) issue(first + gridDim.x, 1);
  }
  cudaGridDependencySynchronize();
  stage_coef<NTH, CB>(a, M, K, U, coef);
  __syncthreads();

  c2 p1[KPT][CB], p2[KPT][CB];
#pragma unroll
  for (int q = 0; q < KPT; q++)
#pragma unroll
    for (int c = 0; c < CB; c++) { p1[q][c] = {0.f, 0.f}; p2[q][c] = {0.f, 0.f}; }
  float sum_max = 0.f, sum_sq = 0.f;  // FP32 within a warp, FP64 across warps
  const int acol = warp % TR, apart = warp / TR;

  int it = 0;
  for (int tile = first; tile < ntiles; tile += gridDim.x, it++) {
    const int stg = it & 1;
    if (!mbar_wait_bounded(&full[stg], (it >> 1) & 1)) {
      if (t == 0) atomicOr(err, 1u);
      abort_flag = 1;
    }
    __syncthreads();
    if (abort_flag) {
      // before the CTA exits, let the copies it issued land (bounded again):
      // this tile's and, if it was issued, the next tile's in the other stage
      if (t == 0) {
        mbar_wait_bounded(&full[stg], (it >> 1) & 1);
        if (tile + (int)gridDim.x < ntiles) mbar_wait_bounded(&full[stg ^ 1], ((it + 1) >> 1) & 1);
      }
      break;
    }
    const float2 *T = reinterpret_cast<const float2 *>(base + (size_t)stg * stage_bytes);
    // (A) Y of column acol over this warp's runs of k
    {
      c2 y[CB];
#pragma unroll
      for (int c = 0; c < CB; c++) y[c] = {0.f, 0.f};
      const float2 *row = T + (size_t)acol * Kp;
#pragma unroll 4
      for (int k = apart * 32 + lane; k < K; k += NPART * 32) {
        const float2 h = row[k];
#pragma unroll
        for (int c = 0; c < CB; c++) mac(y[c], coef[(size_t)k * CB + c], c2{h.x, h.y});
      }
#pragma unroll
      for (int c = 0; c < CB; c++)
        for (int o = 16; o > 0; o >>= 1) {
          y[c].x += __shfl_xor_sync(0xffffffffu, y[c].x, o);
          y[c].y += __shfl_xor_sync(0xffffffffu, y[c].y, o);
        }
      if (lane == 0)
#pragma unroll
        for (int c = 0; c < CB; c++) red[warp][c] = y[c];
    }
    __syncthreads();
    // (B) per-Rx capacity, max, mask, gradient parts
    if (t < TR) {
      const int r = tile * TR + t;
      c2 yy[CB];
      float cap[CB], amp[CB];
#pragma unroll
      for (int c = 0; c < CB; c++) {
        c2 acc = {0.f, 0.f};
#pragma unroll
        for (int pp = 0; pp < NPART; pp++) {
          acc.x += red[pp * TR + t][c].x;
          acc.y += red[pp * TR + t][c].y;
        }
        yy[c] = acc;
      }
      int arg = 0;
      float mx = -1.f;
#pragma unroll
      for (int c = 0; c < CB; c++) {
        if (c >= a.C) { cap[c] = 0.f; amp[c] = 0.f; continue; }
        amp[c] = sqrtf(yy[c].x * yy[c].x + yy[c].y * yy[c].y);
        const float aa = amp[c] + kEps;
        float v = log2f(1.0f + aa * aa / kN0);
        if (a.drop && a.drop[c]) v = 0.f;
        cap[c] = v;
        if (v > mx) { mx = v; arg = c; }
        if (a.recv_amp && r < a.R) a.recv_amp[(size_t)c * a.R + r] = amp[c];
      }
#pragma unroll
      for (int c = 0; c < CB; c++) {
        c2 ga = {0.f, 0.f}, gb = {0.f, 0.f};
        if (c < a.C && r < a.R) {
          const bool dropped = a.drop && a.drop[c];
          const float msk = (cap[c] != mx) ? cap[c] : 0.f;
          sum_sq += msk * msk;
          const float aa = amp[c] + kEps;
          const float dcap = (2.0f * aa / kN0) / (1.0f + aa * aa / kN0) * kInvLn2;
          float g1 = (c == arg) ? -a.w : 0.f, g2 = msk;
          if (dropped) { g1 = 0.f; g2 = 0.f; }
          const float sc = amp[c] > 0.f ? dcap / amp[c] : 0.f;
          ga = {g1 * sc * yy[c].x, g1 * sc * yy[c].y};
          gb = {g2 * sc * yy[c].x, g2 * sc * yy[c].y};
        }
        g1s[c][t] = ga;
        g2s[c][t] = gb;
      }
      if (r < a.R) sum_max += mx;
    }
    __syncthreads();
    // (C) P += G conj(H) over the tile's columns, rows k = t + NTH q
#pragma unroll
    for (int q = 0; q < KPT; q++) {
      const int k = t + NTH * q;
      if (k < K) {
#pragma unroll
        for (int cc = 0; cc < TR; cc++) {
          const float2 h = T[(size_t)cc * Kp + k];
#pragma unroll
          for (int c = 0; c < CB; c++) {
            macc(p1[q][c], g1s[c][cc], c2{h.x, h.y});
            if (CB > 1) macc(p2[q][c], g2s[c][cc], c2{h.x, h.y});
          }
        }
      }
    }
    __syncthreads();
    if (t == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (tile + 2 * (int)gridDim.x < ntiles) issue(tile + 2 * gridDim.x, stg);
    }
  }
  // the tail kernel may launch now; its grid-dependency wait still waits for
  // this grid to complete, with every write below visible
  cudaTriggerProgrammaticLaunchCompletion();
#pragma unroll
  for (int q = 0; q < KPT; q++) {
    const int k = t + NTH * q;
    if (k >= K) continue;
#pragma unroll
    for (int c = 0; c < CB; c++) {
      if (c >= a.C) continue;
      float2 *o = reinterpret_cast<float2 *>(Ppart) + ((size_t)blockIdx.x * 2 * a.C + c) * K + k;
      o[0] = make_float2(p1[q][c].x, p1[q][c].y);
      if (CB > 1) o[(size_t)a.C * K] = make_float2(p2[q][c].x, p2[q][c].y);
    }
  }
  if (t < 32) {
    for (int o = 16; o > 0; o >>= 1) {
      sum_max += __shfl_xor_sync(0xffffffffu, sum_max, o);
      sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
    }
    if (t == 0) {
      lpart[2 * blockIdx.x] = sum_max;
      lpart[2 * blockIdx.x + 1] = sum_sq;
    }
  }
}

// ------------------------------------------------------------------
// Tensor-core path (tcgen05, 3xBF16 split precision, FP32 accumulation).
//
// A complex product over k becomes one real GEMM on interleaved real views;
// output c occupies the accumulator rows 2c (real part) and 2c+1 (imaginary
// part), which adjacent lanes of one warp read back.
//   forward  Y[c, r] = sum_k coef[c, k] [H_r; H_d][k, r]       (pass 1)
//     A_y row 2c = (Re coef, -Im coef) per k, row 2c+1 = (Im coef, Re coef)
//     B_y = [H_r; H_d]^T as a real [R, 2K] matrix (row r: Re, Im of each k)
//   adjoint  G_U[c, k] = sum_r G[c, r] conj([H_r; H_d][k, r])  (pass 2)
//     A_g row 2c = (Re G, Im G) per r, row 2c+1 = (Im G, -Re G)
//     B_g = [H_r; H_d] as a real [K, 2R] matrix (its native layout)
// Each operand x is held as x_hi = bf16(x) and x_lo = bf16(x - x_hi); the
// product is A_hi B_hi + A_hi B_lo + A_lo B_hi (the dropped A_lo B_lo term is
// below 2^-16 of it).  B_y and B_g are built once per channel set (a plan);
// an evaluation rebuilds only the small A operands.



// B_y [Rp, Kp] from [H_r; H_d] [K, R] complex: 32 x 32 complex tiles turned
// through shared memory (reads coalesced over r, writes over k); entries
// beyond R or K are zero.  Block (32, 8), grid (Rp / 32, Kp / 64).
__global__ void __launch_bounds__(256) k_tc_make_by(const float *Hr, const float *Hd, int M,
                                                    int S, int R, int Rp, int Kp,
                                                    __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  __shared__ float2 t[32][33];
  const int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32, K = M + S;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int k = k0 + i, r = r0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (k < K && r < R)
      v = __ldg(reinterpret_cast<const float2 *>(k < M ? Hr + (size_t)k * R * 2
                                                        : Hd + (size_t)(k - M) * R * 2) + r);
    t[i][threadIdx.x] = v;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, k = k0 + threadIdx.x;
    if (r >= Rp || 2 * k >= Kp) continue;
    const float2 v = t[threadIdx.x][i];
    put_pair(hi, lo, kb_pair(r, k, Rp), v.x, v.y);
  }
}

// B_g [Np, K2p] = [H_r; H_d] real view, zero padded; one thread per complex
__global__ void k_tc_make_bg(const float *Hr, const float *Hd, int M, int S, int R, int Np,
                             int K2p, __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ncol = K2p / 2;
  if (i >= (long long)Np * ncol) return;
  const int k = (int)(i / ncol), r = (int)(i % ncol);
  float2 v = make_float2(0.f, 0.f);
  if (k < M + S && r < R)
    v = __ldg(reinterpret_cast<const float2 *>(k < M ? Hr + (size_t)k * R * 2
                                                      : Hd + (size_t)(k - M) * R * 2) + r);
  put_pair(hi, lo, kb_pair(k, r, Np), v.x, v.y);
}

// A_y rows 2c, 2c+1 [., Kp] from coef[c, k] = U[c, k] (k < M), W[c, k - M]
// (M <= k < M + S), zero beyond; one thread per (c, k), c < C
__global__ void k_tc_make_ay(const float *U, const float *W, int C, int M, int S, int Kp,
                             __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int kc = Kp / 2;
  if (i >= (long long)C * kc) return;
  const int c = (int)(i / kc), k = (int)(i % kc);
  float2 v = make_float2(0.f, 0.f);
  if (k < M) v = reinterpret_cast<const float2 *>(U)[(size_t)c * M + k];
  else if (k < M + S) v = __ldg(reinterpret_cast<const float2 *>(W) + (size_t)c * S + (k - M));
  put_pair(hi, lo, kb_pair(2 * c, k, tcg::BM), v.x, -v.y);
  put_pair(hi, lo, kb_pair(2 * c + 1, k, tcg::BM), v.y, v.x);
}

// A_g rows 2c, 2c+1 [., K2p] from G = G1 + G2 / ||masked||; one thread per
// (c, r), c < C
__global__ void k_tc_make_ag(const float *G1, const float *G2, const float *scal, int C, int R,
                             int K2p, __nv_bfloat16 *hi, __nv_bfloat16 *lo) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int rc = K2p / 2;
  if (i >= (long long)C * rc) return;
  const int c = (int)(i / rc), r = (int)(i % rc);
  float2 g = make_float2(0.f, 0.f);
  if (r < R) {
    g = reinterpret_cast<const float2 *>(G1)[(size_t)c * R + r];
    if (G2) {
      const float inv = scal[0];
      const float2 h = reinterpret_cast<const float2 *>(G2)[(size_t)c * R + r];
      g.x = fmaf(h.x, inv, g.x);
      g.y = fmaf(h.y, inv, g.y);
    }
  }
  put_pair(hi, lo, kb_pair(2 * c, r, tcg::BM), g.x, g.y);
  put_pair(hi, lo, kb_pair(2 * c + 1, r, tcg::BM), g.y, -g.x);
}

// D = A_hi B_hi^T + A_hi B_lo^T + A_lo B_hi^T, A [128, Kd] and B [N, Kd] bf16 k-block by
// k-block, in items of 128 x bn outputs over kper k-blocks.  Rows 2c /
// 2c+1 of D are stored as out[(z * C + c) * ldo + n] (complex) for c < C and n <
// n_valid, z the split of the k range.
//
// B is read once from HBM, and A comes along with every B tile from L2; the two
// together bound the kernel.  A CTA stays for all its items, with two
// accumulators: warps 2-5 drain one while warp 0 loads and warp 1 multiplies the
// next, and bn is chosen so that the items fill whole rounds of the chip
// (pick_split).
// 60 codes, K = 1,040, R = 65,536: Y and the adjoint 124 us each with 128 x 128
// tiles, one a CTA; 101 and 107 us now.  (Two CTAs of a cluster, each loading half
// of A into both, took 102 and 108 us.)
__global__ void __launch_bounds__(192, 1)
    k_cgemm3(const __grid_constant__ CUtensorMap tah, const __grid_constant__ CUtensorMap tal,
             const __grid_constant__ CUtensorMap tbh, const __grid_constant__ CUtensorMap tbl,
             int bn, int tiles, int nitems, int kper, int nkb, int C, int n_valid, long long ldo,
             float *out, unsigned *err) {
  using namespace tcg;
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[STAGES_MAX], empty[STAGES_MAX], accf[2], acce[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, n_issued, n_used;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = blockIdx.x, step = gridDim.x;
  const int nst = stages(bn);
  const uint32_t sbytes = stage_bytes(bn), b_bytes = (uint32_t)bn * BK * 2;
  // two accumulators of up to 256 columns, or one where each CTA has one item
  const uint32_t tcols = nitems > step ? 512u : 256u;
  if (tid == 0) {
    for (int s = 0; s < nst; s++) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    for (int i = 0; i < 2; i++) { tc::mbar_init(&accf[i], 1); tc::mbar_init(&acce[i], 4); }
    abort_flag = 0;
    n_issued = 0;
    n_used = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tc::tmem_alloc(&tmem_slot, tcols);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0 && lane == 0) {
    int it = 0;  // k-blocks issued
    bool ok = true;
    for (int i = first; ok && i < nitems; i += step) {
      const int z = i / tiles, n0 = (i - z * tiles) * bn;
      const int k0 = z * kper, nk = min(kper, nkb - k0);
      for (int kb = 0; kb < nk; kb++, it++) {
        const int s = it % nst;
        if (it >= nst && !tc::mbar_wait(&empty[s], (uint32_t)(it / nst - 1) & 1u)) {
          atomicOr(err, 1u);
          ok = false;
        }
        if (!ok || *(volatile int *)&abort_flag) { ok = false; break; }
        unsigned char *sp = smem + (size_t)s * sbytes;
        const int ya = (k0 + kb) * BM;
        tc::mbar_expect_tx(&full[s], sbytes);
        tc::tma_load_2d(sp, &tah, 0, ya, &full[s]);
        tc::tma_load_2d(sp + A_BYTES, &tal, 0, ya, &full[s]);
        tc::tma_load_3d(sp + 2 * A_BYTES, &tbh, 0, n0, k0 + kb, &full[s]);
        tc::tma_load_3d(sp + 2 * A_BYTES + b_bytes, &tbl, 0, n0, k0 + kb, &full[s]);
      }
    }
    n_issued = it;
    if (!ok) *(volatile int *)&abort_flag = 1;
    // the last releases arrive before the CTA may leave
    for (int j = max(0, it - nst); ok && j < it; j++)
      if (!tc::mbar_wait(&empty[j % nst], (uint32_t)(j / nst) & 1u)) { atomicOr(err, 1u); ok = false; }
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = tc::idesc_bf16(BM, bn);
    int it = 0, q = 0;
    bool ok = true;
    for (int i = first; ok && i < nitems; i += step, q++) {
      const int k0 = i / tiles * kper, nk = min(kper, nkb - k0);
      const uint32_t acc = tmem + (uint32_t)(q & 1) * 256u;
      // the accumulator's last item but one has been drained
      if (q >= 2 && !tc::mbar_wait(&acce[q & 1], (uint32_t)(q / 2 - 1) & 1u)) {
        atomicOr(err, 2u);
        ok = false;
        break;
      }
      tc::fence_after();
      for (int kb = 0; kb < nk; kb++, it++) {
        const int s = it % nst;
        if (!tc::mbar_wait(&full[s], (uint32_t)(it / nst) & 1u)) {
          atomicOr(err, 2u);
          ok = false;
          break;
        }
        tc::fence_after();
        const uint32_t ah = tc::smem_u32(smem + (size_t)s * sbytes), al = ah + A_BYTES;
        const uint32_t bh = ah + 2 * A_BYTES, bl = bh + b_bytes;
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) {
          const uint32_t o = kk * 32;  // 16 bf16 = 32 bytes along K
          tc::umma_bf16(acc, tc::sdesc_sw128(ah + o), tc::sdesc_sw128(bh + o), idesc,
                        (kb > 0 || kk > 0) ? 1u : 0u);
          tc::umma_bf16(acc, tc::sdesc_sw128(ah + o), tc::sdesc_sw128(bl + o), idesc, 1u);
          tc::umma_bf16(acc, tc::sdesc_sw128(al + o), tc::sdesc_sw128(bh + o), idesc, 1u);
        }
        tc::umma_commit(&empty[s]);
      }
      tc::umma_commit(&accf[q & 1]);
    }
    n_used = it;
    if (!ok) *(volatile int *)&abort_flag = 1;
  } else if (warp >= 2) {
    const int quarter = warp & 3;  // the TMEM lanes a warp can read
    const int c = quarter * 16 + (lane >> 1);
    const bool odd = (lane & 1) != 0, rows = quarter * 32 < 2 * C;
    int q = 0;
    for (int i = first; i < nitems; i += step, q++) {
      const bool have = warp_wait(&accf[q & 1], (uint32_t)(q / 2) & 1u);
      if (!have && lane == 0) { atomicOr(err, 4u); *(volatile int *)&abort_flag = 1; }
      // warp-uniform: tcgen05.ld and the shuffles below are warp-collective
      if (__any_sync(0xffffffffu, !have || *(volatile int *)&abort_flag)) break;
      tc::fence_after();
      const int z = i / tiles, n0 = (i - z * tiles) * bn;
      const int n1 = min(n0 + bn, n_valid);
      const uint32_t acc = tmem + (uint32_t)(q & 1) * 256u + ((uint32_t)(quarter * 32) << 16);
      float2 *o2 = reinterpret_cast<float2 *>(out) + ((size_t)z * C + c) * (size_t)ldo;
      if (rows)
#pragma unroll 1
        for (int c0 = 0; c0 < bn; c0 += 32) {
          uint32_t r[32];
          tc::tmem_ld32(acc + (uint32_t)c0, r);
          // the even lane of a pair writes columns 0-15 of the chunk, the odd 16-31
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const float a0 = __uint_as_float(r[j]), a1 = __uint_as_float(r[16 + j]);
            const float b0 = __shfl_xor_sync(0xffffffffu, a0, 1);
            const float b1 = __shfl_xor_sync(0xffffffffu, a1, 1);
            const int n = n0 + c0 + (odd ? 16 : 0) + j;
            if (c < C && n < n1) o2[n] = odd ? make_float2(b1, a1) : make_float2(a0, b0);
          }
        }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[q & 1]);
    }
  }
  __syncwarp();
  __syncthreads();
  // after an abort, the tiles issued but never consumed land before the CTA
  // exits (each stage holds at most one of them; bounded waits again)
  if (abort_flag && tid == 0)
    for (int j = n_used; j < n_issued; j++) tc::mbar_wait(&full[j % nst], (uint32_t)(j / nst) & 1u);
  __syncwarp();
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, tcols);
  }
}

int round_up(long long v, int m) { return (int)((v + m - 1) / m * m); }

// Items of a product of N columns and nkb k-blocks: the tile width bn and the
// split of the k range whose rounds over the chip take the least time.  In units
// of a row of B (256 bytes a k-block) an item's k-block costs its bn rows and
// about 48 for A (32, 64, 96 and 128 within 2% or slower), 144 at least (its
// latency); every split writes its partial sums, and the epilogues read them
// twice (48 bytes a sum: with 16 or 24 the splits of small products cost up to 5%
// more).  An item's sums are one FP32 chain in TMEM, and it gets no longer than
// that of 128 x 128 tiles which fill the chip once: 13 k-blocks instead of 8
// brought the error of dW from 1.9e-6 to 2.3e-6 (60 codes, K = 1,040, R = 4,096).
struct GemmSplit {
  int bn = 0, tiles = 0, ks = 1, kper = 0;
  int items() const { return tiles * ks; }
};
GemmSplit pick_split(int N, int nkb, int C, int sms) {
  GemmSplit best;
  double least = 0;
  const int slots = std::max(1, sms);
  const int least_ks = std::min(nkb, std::max(1, slots / ((N + 127) / 128)));
  const int longest = (nkb + least_ks - 1) / least_ks;
  for (int bn = tcg::BN_MIN; bn <= tcg::BN_MAX; bn += 16)
    for (int want = 1; want <= std::min(nkb, slots); want++) {
      GemmSplit g;
      g.bn = bn;
      g.tiles = (N + bn - 1) / bn;
      g.kper = (nkb + want - 1) / want;
      g.ks = (nkb + g.kper - 1) / g.kper;
      if (g.ks != want || g.kper > longest) continue;
      const int rounds = (g.items() + slots - 1) / slots;
      const double t = (double)rounds * g.kper * std::max(bn + 48, 144) + 2.0 * bn +
                       (g.ks > 1 ? (double)g.ks * N * C * 48 / (256.0 * sms) : 0.0);
      if (!best.bn || t < least) { best = g; least = t; }
    }
  return best;
}

}  // namespace

namespace {
std::atomic<int> g_inject_timeouts{0};
}  // namespace

// Start of a call on a path with bounded waits, after its first kernel: the
// wait-timeout word is cleared (by that kernel when `cleared`, else here), so
// the word reports this call only.  An injected timeout (test hook of the
// error path) then sets it, as a wait that ran out would.
cudaError_t obj_begin_call(unsigned *err, bool cleared, cudaStream_t st) {
  cudaError_t e = cleared ? cudaSuccess : cudaMemsetAsync(err, 0, 4, st);
  if (e != cudaSuccess) return e;
  int n = g_inject_timeouts.load();
  while (n > 0 && !g_inject_timeouts.compare_exchange_weak(n, n - 1)) {
  }
  if (n > 0) e = cudaMemsetAsync(err, 1, 1, st);
  return e;
}

void obj_inject_timeouts(int calls) { g_inject_timeouts.store(calls > 0 ? calls : 0); }

ObjScratchLayout obj_scratch_layout(int S, int M, int R, int C) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const Split sp = make_split(S, M, R);
  ObjScratchLayout L;
  size_t o = 0;
  L.inv = o; o += 256;                                    // control block (see header)
  L.Um = o; o += al(8 * (size_t)C * std::max(M, 1));      // U = (W H_a) e^{j phi'}
  L.gw = o;  // dL/dW partials (k_final CTAs, or the streaming tail CTAs)
  o += al(8 * (size_t)std::max((M + 31) / 32, (M + S + 31) / 32) * C * S);
  L.U = o; o += al(8 * (size_t)sp.kspl * C * R);          // Y partials
  L.G1 = o; o += al(8 * (size_t)C * R);
  L.G2 = o; o += al(8 * (size_t)C * R);
  L.part = o; o += al(16 * (size_t)std::max(sp.nb_epi, (R + 31) / 32));  // either epilogue
  L.GU = o; o += al(8 * (size_t)sp.rspl * C * sp.K);      // G_U partials
  const int nsm = kMaxClusters;                           // partials of the streaming path
  L.Pp = o; o += al(8 * (size_t)nsm * 2 * C * sp.K);
  L.lp = o; o += al(16 * (size_t)nsm);
  L.GUs = o; o += al(8 * (size_t)C * sp.K);
  L.total = o;
  return L;
}

cudaError_t obj_run(const ObjArgs &a0, char *scratch, cudaStream_t st) {
  ObjArgs a = a0;
  const bool ms = a.Ha && a.Hr;
  const int M = ms ? a.M : 0;
  if (!ms) { a.Ha = nullptr; a.Hr = nullptr; a.grad_phi = nullptr; }
  const ObjScratchLayout L = obj_scratch_layout(a.S, M, a.R, a.C);
  const Split sp = make_split(a.S, M, a.R);
  float *Ypart = reinterpret_cast<float *>(scratch + L.U);
  float *G1 = reinterpret_cast<float *>(scratch + L.G1);
  float *G2 = a.C > 1 ? reinterpret_cast<float *>(scratch + L.G2) : nullptr;
  double *part = reinterpret_cast<double *>(scratch + L.part);
  float *GUp = reinterpret_cast<float *>(scratch + L.GU);
  float *scal = reinterpret_cast<float *>(scratch + L.inv);
  unsigned *counter = reinterpret_cast<unsigned *>(scratch + L.inv + 32);
  float *Um = reinterpret_cast<float *>(scratch + L.Um);
  float *gw = reinterpret_cast<float *>(scratch + L.gw);
  const StreamPlan pl = stream_plan(a.S, M, a.R, a.C, a.grad_Y != nullptr);
  if (pl.ok &&
      !((reinterpret_cast<uintptr_t>(a.Hd) | reinterpret_cast<uintptr_t>(ms ? a.Hr : a.Hd)) & 15)) {
    float *Pp = reinterpret_cast<float *>(scratch + L.Pp);
    double *lp = reinterpret_cast<double *>(scratch + L.lp);
    unsigned *err = reinterpret_cast<unsigned *>(scratch + L.inv + 48);
    float *GUs = reinterpret_cast<float *>(scratch + L.GUs);
    if (cbucket(a.C) == 1) return run_stream<1>(a, pl, M, Um, Pp, lp, GUs, gw, err, counter + 2, st);
    return run_stream<2>(a, pl, M, Um, Pp, lp, GUs, gw, err, counter + 2, st);
  }
  switch (cbucket(a.C)) {
#define CASE(CB) case CB: return run_cb<CB>(a, sp, M, Um, Ypart, G1, G2, part, counter, scal, GUp, gw, st);
    CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32) CASE(64)
#undef CASE
    default: return cudaErrorInvalidValue;
  }
}

// ------------------------------------------------------------------ plans
struct ObjTcPlan {
  const float *Hd, *Ha, *Hr;
  // stream mode (C_max <= 2): the streaming kernels, over an FP32 copy of the
  // channels, as they are (direct) or transposed
  bool stream = false, direct = false;
  float *HT = nullptr;
  int tKp = 0, tTR = 0, tKPT = 0, tStage = 0, tTiles = 0, tGrid = 0;
  size_t tSmem = 0, oPp = 0, oLp = 0, oGwS = 0;
  int S, M, R, Cmax, K, Kp, Rp, Np, K2p, Mp;
  GemmSplit gy, gg;
  __nv_bfloat16 *by_hi, *by_lo, *bg_hi, *bg_lo, *ay_hi, *ay_lo, *ag_hi, *ag_lo;
  CUtensorMap m_byh, m_byl, m_bgh, m_bgl, m_ayh, m_ayl, m_agh, m_agl;
  char *mem;      // one allocation: operands then scratch
  size_t bytes;
  size_t oCtl, oU, oY, oG1, oG2, oPart, oGU, oGUs, oDw;  // byte offsets in mem
};

namespace {
// Stream mode over the channels as they are, where k_obj_stream takes them: an
// even number of Rx, K up to about 3,200.  A transposed copy is no faster there
// (S = 16, C = 1: R = 65,536, M = 1,024 133 against 127 us, M = 2,304 266
// against 253 us; R = 4,096, M = 1,024 23.8 against 21.6 us).  Like every other
// plan this one evaluates the H_d and H_r that it was made of, whatever is
// written into the caller's arrays later, so it keeps a copy of them.
bool plan_direct(int S, int M, int R, int Cmax) {
  for (int C = 1; C <= Cmax; C++)
    if (!stream_plan(S, M, R, C, false).ok) return false;
  return true;
}
cudaError_t plan_direct_create(ObjTcPlan *p, cudaStream_t st, ObjTcPlan **out) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const int nparts = std::min(kMaxClusters, (p->R + 7) / 8);
  const size_t n_hr = 8 * (size_t)p->M * p->R, n_hd = 8 * (size_t)p->S * p->R;
  size_t o = 0;
  const size_t ohr = o; o += al(n_hr);
  const size_t ohd = o; o += al(n_hd);
  p->oCtl = o; o += kObjControlBytes;
  p->oU = o; o += al(8 * (size_t)p->Cmax * p->M);
  p->oPp = o; o += al(8 * (size_t)nparts * 2 * p->Cmax * p->K);
  p->oLp = o; o += al(16 * (size_t)nparts);
  p->oGwS = o; o += al(8 * (size_t)p->Cmax * p->K);
  p->oDw = o; o += al(8 * (size_t)((p->K + 31) / 32) * p->Cmax * p->S);
  p->bytes = o;
  cudaError_t e = cudaMalloc(&p->mem, o);
  if (e != cudaSuccess) { delete p; return e; }
  p->stream = p->direct = true;
  e = cudaMemsetAsync(p->mem + p->oCtl, 0, kObjControlBytes, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(p->mem + ohr, p->Hr, n_hr, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(p->mem + ohd, p->Hd, n_hd, cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) { cudaFree(p->mem); delete p; return e; }
  p->Hr = reinterpret_cast<const float *>(p->mem + ohr);
  p->Hd = reinterpret_cast<const float *>(p->mem + ohd);
  *out = p;
  return cudaSuccess;
}

// Stream mode: HT [Rp][Kp] holds [H_r; H_d] transposed (FP32 complex, rows
// padded to an even length so a tile is a whole number of 16-byte units).
cudaError_t plan_stream_create(ObjTcPlan *p, cudaStream_t st, ObjTcPlan **out) {
  const int K = p->K, CB = cbucket(p->Cmax), S = p->S, M = p->M, R = p->R;
  const int kpt = (K + 255) / 256;
  p->tKPT = kpt <= 4 ? 4 : (kpt <= 8 ? 8 : (kpt <= 16 ? 16 : 0));
  if (!p->tKPT || (CB == 2 && p->tKPT > 8)) { delete p; return cudaErrorInvalidValue; }
  p->tKp = (K + 1) / 2 * 2;
  int per_sm = 2;
  for (int TR : {8, 4, 2}) {
    const size_t stage = ((size_t)TR * p->tKp * 8 + 1023) / 1024 * 1024;
    const size_t smem = 1024 + 2 * stage + (size_t)K * CB * 8;
    if (smem <= 110 * 1024) { p->tTR = TR; p->tStage = (int)stage; p->tSmem = smem; break; }
  }
  if (!p->tTR) {  // long columns: two-Rx tiles, one CTA per SM
    const size_t stage = ((size_t)2 * p->tKp * 8 + 1023) / 1024 * 1024;
    const size_t smem = 1024 + 2 * stage + (size_t)K * CB * 8;
    if (smem > 220 * 1024) { delete p; return cudaErrorInvalidValue; }
    p->tTR = 2; p->tStage = (int)stage; p->tSmem = smem;
    per_sm = 1;
  }
  const int Rp = (R + p->tTR - 1) / p->tTR * p->tTR;
  p->tTiles = Rp / p->tTR;
  p->tGrid = std::min(per_sm * sm_count(), p->tTiles);
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  size_t o = 0;
  const size_t oht = o; o += al(8 * (size_t)Rp * p->tKp);
  p->oCtl = o; o += kObjControlBytes;
  p->oU = o; o += al(8 * (size_t)p->Cmax * M);
  p->oPp = o; o += al(8 * (size_t)p->tGrid * 2 * p->Cmax * K);
  p->oLp = o; o += al(16 * (size_t)p->tGrid);
  p->oGwS = o; o += al(8 * (size_t)p->Cmax * K);           // G_U
  p->oDw = o; o += al(8 * (size_t)((K + 31) / 32) * p->Cmax * S);  // dL/dW per tail CTA
  p->bytes = o;
  cudaError_t e = cudaMalloc(&p->mem, o);
  if (e != cudaSuccess) { delete p; return e; }
  p->HT = reinterpret_cast<float *>(p->mem + oht);
  p->stream = true;
  e = cudaMemsetAsync(p->mem + p->oCtl, 0, kObjControlBytes, st);
  if (e == cudaSuccess) {
    dim3 g((Rp + 31) / 32, (p->tKp + 31) / 32), b(32, 8);
    k_make_ht<<<g, b, 0, st>>>(p->Hr, p->Hd, M, S, R, Rp, p->tKp, p->HT);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) { cudaFree(p->mem); delete p; return e; }
  *out = p;
  return cudaSuccess;
}

template <int CB, int TR, int KPT>
cudaError_t launch_stream_ht(ObjTcPlan *p, const ObjArgs &a, const float *U, float *Pp,
                             double *lp, unsigned *err, cudaStream_t st) {
  auto kfn = k_obj_stream_t<CB, TR, KPT>;
  static size_t set_bytes[AMS_MAX_DEVICES] = {0};
  {
    cudaError_t e = ams_set_smem_atleast(set_bytes, kfn, p->tSmem);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p->tGrid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = p->tSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kfn, a, (const float *)p->HT, p->M, p->tKp, p->tStage,
                            p->tTiles, U, Pp, lp, err);
}

template <int CB, int TR>
cudaError_t launch_stream_ht_k(ObjTcPlan *p, const ObjArgs &a, const float *U, float *Pp,
                               double *lp, unsigned *err, cudaStream_t st) {
  switch (p->tKPT) {
    case 4: return launch_stream_ht<CB, TR, 4>(p, a, U, Pp, lp, err, st);
    case 8: return launch_stream_ht<CB, TR, 8>(p, a, U, Pp, lp, err, st);
    case 16:
      if (CB == 1) return launch_stream_ht<1, TR, 16>(p, a, U, Pp, lp, err, st);
      return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
}

template <int CB>
cudaError_t run_plan_stream(ObjTcPlan *p, const ObjArgs &a, cudaStream_t st) {
  const int M = p->M;
  float *U = reinterpret_cast<float *>(p->mem + p->oU);
  float *Pp = reinterpret_cast<float *>(p->mem + p->oPp);
  double *lp = reinterpret_cast<double *>(p->mem + p->oLp);
  float *gw = reinterpret_cast<float *>(p->mem + p->oGwS);
  char *ctl = p->mem + p->oCtl;
  unsigned *counter = reinterpret_cast<unsigned *>(ctl + 40);
  unsigned *err = reinterpret_cast<unsigned *>(ctl + 48);
  if (p->direct)
    return run_stream<CB>(a, stream_plan(p->S, M, p->R, a.C, false), M, U, Pp, lp, gw,
                          reinterpret_cast<float *>(p->mem + p->oDw), err, counter, st);
  const long long n = (long long)M * a.C * 8;
  k_prep_wide<<<(int)((n + 255) / 256), 256, 0, st>>>(a, M, U, err);
  cudaError_t e = obj_begin_call(err, true, st);
  if (e != cudaSuccess) return e;
  switch (p->tTR) {
    case 8: e = launch_stream_ht_k<CB, 8>(p, a, U, Pp, lp, err, st); break;
    case 4: e = launch_stream_ht_k<CB, 4>(p, a, U, Pp, lp, err, st); break;
    default: e = launch_stream_ht_k<CB, 2>(p, a, U, Pp, lp, err, st); break;
  }
  if (e != cudaSuccess) return e;
  return stream_tail<CB>(a, M, p->tGrid, U, Pp, lp, gw, reinterpret_cast<float *>(p->mem + p->oDw),
                         counter, err, st);
}
}  // namespace

cudaError_t obj_tc_plan_create(const float *Hd, const float *Ha, const float *Hr, int S, int M,
                               int R, int Cmax, cudaStream_t st, ObjTcPlan **out,
                               bool force_tc) {
  *out = nullptr;
  if (S <= 0 || M <= 0 || R <= 0 || Cmax <= 0 || Cmax > 64) return cudaErrorInvalidValue;
  ObjTcPlan *p = new ObjTcPlan();
  p->Hd = Hd; p->Ha = Ha; p->Hr = Hr;
  p->S = S; p->M = M; p->R = R; p->Cmax = Cmax;
  p->K = M + S;
  p->Kp = round_up(2LL * p->K, 64);
  p->Rp = round_up(R, 32);
  p->Np = p->K;
  p->K2p = round_up(2LL * R, 64);
  p->Mp = round_up(2LL * Cmax, tcg::BM);
  const int sms = sm_count();
  // stream mode when the streaming kernel's per-thread rows cover K (16 rows
  // a thread for one code, 8 for two); otherwise the tensor-core mode
  const int kpt = (p->K + 255) / 256;
  if (!force_tc && Cmax <= 2 && plan_direct(S, M, R, Cmax))
    return plan_direct_create(p, st, out);
  if (!force_tc && Cmax <= 2 && kpt <= (Cmax == 1 ? 16 : 8)) return plan_stream_create(p, st, out);
  p->gy = pick_split(R, p->Kp / tcg::BK, Cmax, sms);
  p->gg = pick_split(p->K, p->K2p / tcg::BK, Cmax, sms);
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  size_t o = 0;
  const size_t nby = (size_t)p->Rp * p->Kp, nbg = (size_t)p->Np * p->K2p;
  const size_t nay = (size_t)p->Mp * p->Kp, nag = (size_t)p->Mp * p->K2p;
  size_t oby = o; o += al(2 * nby) * 2;
  size_t obg = o; o += al(2 * nbg) * 2;
  size_t oay = o; o += al(2 * nay) * 2;
  size_t oag = o; o += al(2 * nag) * 2;
  p->oCtl = o;
  o += kObjControlBytes;
  p->oU = o; o += al(8 * (size_t)Cmax * M);
  p->oY = o; o += al(8 * (size_t)p->gy.ks * Cmax * R);
  p->oG1 = o; o += al(8 * (size_t)Cmax * R);
  p->oG2 = o; o += al(8 * (size_t)Cmax * R);
  p->oPart = o; o += al(16 * (size_t)((R + 31) / 32));
  p->oGU = o; o += al(8 * (size_t)p->gg.ks * Cmax * p->K);
  p->oGUs = o; o += al(8 * (size_t)Cmax * p->K);
  p->oDw = o; o += al(8 * (size_t)Cmax * dw_parts(M) * S);
  p->bytes = o;
  cudaError_t e = cudaMalloc(&p->mem, o);
  if (e != cudaSuccess) { delete p; return e; }
  p->by_hi = reinterpret_cast<__nv_bfloat16 *>(p->mem + oby);
  p->by_lo = reinterpret_cast<__nv_bfloat16 *>(p->mem + oby + al(2 * nby));
  p->bg_hi = reinterpret_cast<__nv_bfloat16 *>(p->mem + obg);
  p->bg_lo = reinterpret_cast<__nv_bfloat16 *>(p->mem + obg + al(2 * nbg));
  p->ay_hi = reinterpret_cast<__nv_bfloat16 *>(p->mem + oay);
  p->ay_lo = reinterpret_cast<__nv_bfloat16 *>(p->mem + oay + al(2 * nay));
  p->ag_hi = reinterpret_cast<__nv_bfloat16 *>(p->mem + oag);
  p->ag_lo = reinterpret_cast<__nv_bfloat16 *>(p->mem + oag + al(2 * nag));
  const bool ok =
      tc::make_map_bf16_planes(&p->m_byh, p->by_hi, p->Kp / 64, p->Rp, p->gy.bn) &&
      tc::make_map_bf16_planes(&p->m_byl, p->by_lo, p->Kp / 64, p->Rp, p->gy.bn) &&
      tc::make_map_bf16_planes(&p->m_bgh, p->bg_hi, p->K2p / 64, p->Np, p->gg.bn) &&
      tc::make_map_bf16_planes(&p->m_bgl, p->bg_lo, p->K2p / 64, p->Np, p->gg.bn) &&
      tc::make_map_bf16(&p->m_ayh, p->ay_hi, (long long)p->Mp * (p->Kp / 64), 64, tcg::BM) &&
      tc::make_map_bf16(&p->m_ayl, p->ay_lo, (long long)p->Mp * (p->Kp / 64), 64, tcg::BM) &&
      tc::make_map_bf16(&p->m_agh, p->ag_hi, (long long)p->Mp * (p->K2p / 64), 64, tcg::BM) &&
      tc::make_map_bf16(&p->m_agl, p->ag_lo, (long long)p->Mp * (p->K2p / 64), 64, tcg::BM);
  if (!ok) { cudaFree(p->mem); delete p; return cudaErrorInvalidValue; }
  static size_t attr[AMS_MAX_DEVICES] = {0};
  e = ams_set_smem_atleast(attr, k_cgemm3, tcg::SMEM);
  if (e != cudaSuccess) { cudaFree(p->mem); delete p; return e; }
  // the A operands (rows beyond 2 C stay zero) and the control block
  e = cudaMemsetAsync(p->mem + oay, 0, o - oay, st);
  if (e == cudaSuccess) {
    dim3 gb(p->Rp / 32, p->Kp / 64), bb(32, 8);
    k_tc_make_by<<<gb, bb, 0, st>>>(Hr, Hd, M, S, R, p->Rp, p->Kp, p->by_hi, p->by_lo);
    const long long ng = (long long)p->Np * (p->K2p / 2);
    k_tc_make_bg<<<(unsigned)((ng + 255) / 256), 256, 0, st>>>(Hr, Hd, M, S, R, p->Np, p->K2p,
                                                               p->bg_hi, p->bg_lo);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) { cudaFree(p->mem); delete p; return e; }
  *out = p;
  return cudaSuccess;
}

const unsigned *obj_tc_plan_status_word(const ObjTcPlan *p) {
  return p ? reinterpret_cast<const unsigned *>(p->mem + p->oCtl + 48) : nullptr;
}

size_t obj_tc_plan_bytes(const ObjTcPlan *p) { return p ? p->bytes : 0; }
bool obj_tc_plan_streams(const ObjTcPlan *p) { return p && p->stream; }

void obj_tc_plan_destroy(ObjTcPlan *p) {
  if (!p) return;
  cudaFree(p->mem);
  delete p;
}

namespace {
template <int CB>
cudaError_t run_tc(ObjTcPlan *p, const ObjArgs &a, char *ctl, cudaStream_t st) {
  const int M = p->M, R = p->R, C = a.C;
  const bool given = a.U_in != nullptr;
  const float *U = given ? a.U_in : reinterpret_cast<float *>(p->mem + p->oU);
  float *Ypart = reinterpret_cast<float *>(p->mem + p->oY);
  float *G1 = reinterpret_cast<float *>(p->mem + p->oG1);
  float *G2 = C > 1 ? reinterpret_cast<float *>(p->mem + p->oG2) : nullptr;
  double *part = reinterpret_cast<double *>(p->mem + p->oPart);
  float *GUp = reinterpret_cast<float *>(p->mem + p->oGU);
  float *scal = reinterpret_cast<float *>(ctl);
  unsigned *counter = reinterpret_cast<unsigned *>(ctl + 32);
  unsigned *err = reinterpret_cast<unsigned *>(ctl + 48);
  if (!given)
    k_prep<<<dim3((M + 127) / 128, C), 128, 0, st>>>(a, M, reinterpret_cast<float *>(p->mem + p->oU), err);
  {
    cudaError_t e0 = obj_begin_call(err, !given, st);
    if (e0 != cudaSuccess) return e0;
  }
  const long long nay = (long long)C * (p->Kp / 2);
  k_tc_make_ay<<<(unsigned)((nay + 255) / 256), 256, 0, st>>>(U, a.W, C, M, p->S, p->Kp,
                                                              p->ay_hi, p->ay_lo);
  const int slots = std::max(1, sm_count());
  k_cgemm3<<<std::min(p->gy.items(), slots), 192, tcg::SMEM, st>>>(
      p->m_ayh, p->m_ayl, p->m_byh, p->m_byl, p->gy.bn, p->gy.tiles, p->gy.items(), p->gy.kper,
      p->Kp / tcg::BK, C, R, R, Ypart, err);
  const bool need_g = a.grad_W || a.grad_phi || a.grad_U;
  if (CB >= 8) {
    constexpr int CW = CB >= 8 ? CB : 8;
    float *maxr = G1;  // G1 / G2 are not needed on this branch: per-Rx max and argmax
    int *argr = reinterpret_cast<int *>(G2 ? G2 : G1 + R);
    const int nb = (R + 31) / 32;
    k_tc_epi_a<CW><<<std::min(nb, 4 * sm_count()), 256, 0, st>>>(a, p->gy.ks, Ypart, maxr, argr, part, counter, scal, err);
    if (need_g || a.grad_Y) {
      // with no gradient wanted the A operand is still written (harmless)
      const int nbb = std::max(nb, (p->K2p / 2 + 31) / 32);
      k_tc_epi_b<CW><<<nbb, 256, 0, st>>>(a, p->gy.ks, Ypart, maxr, argr, scal, p->K2p, p->ag_hi,
                                          p->ag_lo);
    }
  } else {
    k_epilogue<CB><<<(R + 127) / 128, 128, 0, st>>>(a, p->gy.ks, Ypart, G1, G2, part, counter,
                                                    scal, err);
    if (a.grad_Y) {
      const long long n = (long long)C * R;
      k_grad_y<<<(int)((n + 255) / 256), 256, 0, st>>>(G1, G2, scal, n, a.grad_Y);
    }
    if (need_g) {
      const long long nag = (long long)C * (p->K2p / 2);
      k_tc_make_ag<<<(unsigned)((nag + 255) / 256), 256, 0, st>>>(G1, G2, scal, C, R, p->K2p,
                                                                  p->ag_hi, p->ag_lo);
    }
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (!need_g) return cudaGetLastError();
  k_cgemm3<<<std::min(p->gg.items(), slots), 192, tcg::SMEM, st>>>(
      p->m_agh, p->m_agl, p->m_bgh, p->m_bgl, p->gg.bn, p->gg.tiles, p->gg.items(), p->gg.kper,
      p->K2p / tcg::BK, C, p->K, p->K, GUp, err);
  float *GU = reinterpret_cast<float *>(p->mem + p->oGUs);
  const long long ngu = (long long)C * p->K;
  k_gu_reduce<<<(unsigned)((ngu + 31) / 32), 256, 0, st>>>(GUp, p->gg.ks, ngu, GU);
  if (given) {
    // dL/dU is G_U's metasurface rows, dL/dW its H_d rows (poisoned like
    // the other outputs when a wait ran out)
    if (a.grad_U)
      k_tc_copy_rows<<<(C * M + 255) / 256, 256, 0, st>>>(GU, p->K, 0, M, C, a.grad_U, err);
    if (a.grad_W)
      k_tc_copy_rows<<<(C * p->S + 255) / 256, 256, 0, st>>>(GU, p->K, M, p->S, C, a.grad_W, err);
    return cudaGetLastError();
  }
  if (a.grad_phi) k_tc_dphi<<<(M + 31) / 32, 256, 0, st>>>(GU, U, C, M, p->K, a.grad_phi, err);
  if (a.grad_W) {
    float *dwp = reinterpret_cast<float *>(p->mem + p->oDw);
    const int parts = dw_parts(M);
    k_tc_dw_part<<<dim3(parts, (p->S + 15) / 16), 256, 0, st>>>(GU, p->Ha, a.phi, a.max_phase, C,
                                                                p->S, M, p->K, dwp);
    k_tc_dw_sum<<<(C * p->S + 31) / 32, 256, 0, st>>>(GU, dwp, C, p->S, M, p->K, parts, a.grad_W,
                                                        err);
  }
  return cudaGetLastError();
}
}  // namespace

cudaError_t obj_tc_run(ObjTcPlan *p, const ObjArgs &a0, cudaStream_t st) {
  if (!p || a0.C <= 0 || a0.C > p->Cmax) return cudaErrorInvalidValue;
  ObjArgs a = a0;
  a.Hd = p->Hd; a.Ha = p->Ha; a.Hr = p->Hr;
  a.S = p->S; a.M = p->M; a.R = p->R;
  // a coefficient-given call needs the tensor-core mode; a call that forms
  // U from W, H_a and phi needs H_a
  if (a.U_in ? p->stream : (p->Ha == nullptr)) return cudaErrorInvalidValue;
  if (p->stream) {
    if (a.grad_Y) return cudaErrorInvalidValue;  // not produced by the streaming kernels
    return cbucket(a.C) == 1 ? run_plan_stream<1>(p, a, st) : run_plan_stream<2>(p, a, st);
  }
  char *ctl = p->mem + p->oCtl;
  switch (cbucket(a.C)) {
#define CASE(CB) case CB: return run_tc<CB>(p, a, ctl, st);
    CASE(1) CASE(2) CASE(4) CASE(8) CASE(16) CASE(32) CASE(64)
#undef CASE
    default: return cudaErrorInvalidValue;
  }
}

namespace {
// draw_channel + amp_data_to_image (go.py:849-851, 944-964):
// 20 log10 |sum_s H[s,r]|, NaN -> threshold, + offset, clamp below at threshold
__global__ void k_coverage_db(const float *H, int S, int R, float threshold, float offset,
                              float *out) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  double x = 0, y = 0;
  for (int s = 0; s < S; s++) {
    float2 v = __ldg(reinterpret_cast<const float2 *>(H) + (size_t)s * R + r);
    x += v.x;
    y += v.y;
  }
  float a = (float)sqrt(x * x + y * y);
  float d = 20.0f * log10f(a);
  if (isnan(d)) d = threshold;
  d = d + offset;
  out[r] = fmaxf(d, threshold);
}
}  // namespace

namespace {
// complex GEMM, 16 x 16 output tiles through shared memory, FP32
__device__ __forceinline__ float2 cg_ld(const float2 *X, int ld, int op, int r, int c) {
  // element (r, c) of op(X): 0 X, 1 X^T, 2 X^H, 3 conj(X)
  if (op == 0) return X[(size_t)r * ld + c];
  if (op == 3) {
    const float2 v = X[(size_t)r * ld + c];
    return make_float2(v.x, -v.y);
  }
  const float2 v = X[(size_t)c * ld + r];
  return op == 1 ? v : make_float2(v.x, -v.y);
}
__global__ void __launch_bounds__(256) k_cgemm_small(int m, int n, int k, const float2 *A, int lda,
                                                     int opA, const float2 *B, int ldb, int opB,
                                                     float2 *C, int ldc, int accumulate) {
  __shared__ float2 As[16][17], Bs[16][17];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int row = blockIdx.y * 16 + ty, col = blockIdx.x * 16 + tx;
  float2 acc = make_float2(0.f, 0.f);
  for (int k0 = 0; k0 < k; k0 += 16) {
    As[ty][tx] = (row < m && k0 + tx < k) ? cg_ld(A, lda, opA, row, k0 + tx) : make_float2(0.f, 0.f);
    Bs[ty][tx] = (k0 + ty < k && col < n) ? cg_ld(B, ldb, opB, k0 + ty, col) : make_float2(0.f, 0.f);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const float2 a = As[ty][q], b = Bs[q][tx];
      acc.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x));
      acc.y = fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y));
    }
    __syncthreads();
  }
  if (row < m && col < n) {
    float2 *o = C + (size_t)row * ldc + col;
    if (accumulate) { acc.x += o->x; acc.y += o->y; }
    *o = acc;
  }
}
}  // namespace

// ------------------------------------------------------------------
// Paths over several metasurfaces (go.py:107-157).  With V^l_m the sum, over the
// paths of l hops that end on metasurface m, of the path products,
//   V^1_m = (W H_a^m) o e_m,  V^(l+1)_m = (sum_{m' != m} V^l_m' H^(m'm)) o e_m,
//   U_m = sum_l V^l_m,  e = exp(j phi'),
// and of the adjoint, with G_U from the stacked evaluation,
//   D^hops_m = G_U,m,  D^l_m = G_U,m + sum_{m' != m} (D^(l+1)_m' o conj e_m') H^(mm')^H,
//   dphi_m = -sum_l Im(conj(D^l_m) o V^l_m) over the codes,
//   dW = G_W + sum_m (D^1_m o conj e_m) (H_a^m)^H.
// (H^(m'm) = H^(mm')^T: only m < m' is stored.)  A level is one launch: a CTA
// forms 32 codes x 16 elements of one metasurface from all its sources.  Path
// by path, the step took a product per path and hop and eight elementwise
// launches beside each, all issued from Python, and that bound it: a step with
// its backward pass, two hops, C = 30, S = 36: M = 576 + 256, R = 2,116 2,390 ->
// 790 us; M = 2,304 + 1,024 2,375 -> 1,087 us; three hops over 3 x 1,024, C = 64,
// R = 1,000 11.5 -> 1.6 ms.  The products are FP32 FMAs (what is stored is read
// once per 32 codes); the kernel is bound by its shared-memory reads.
namespace {
struct MhSrc {
  const float2 *A;  // [C, k], lda
  const float2 *e;  // A's columns are multiplied by conj(e[k]) (NULL: not)
  const float2 *B;  // op(B) [k, n]
  int lda, ldb, op, k;
};
struct MhDst {
  float2 *out;        // [C, n], ldo
  const float2 *add;  // added (ld ldo), or NULL
  const float2 *e;    // out's columns multiplied by e[n], or NULL
  float2 *sum;        // out also goes here (ld ldo): stored, or added with sum_add
  int ldo, n, nsrc, tile0, sum_add;
  MhSrc src[kMhMax];
};
struct MhLevel {
  int C, ndst;
  MhDst dst[kMhMax];
};
constexpr int kMhK = 64;  // inner dimension staged at a time

__global__ void __launch_bounds__(256) k_mh_gemm(const __grid_constant__ MhLevel lv) {
  __shared__ float2 As[kMhK][33];
  __shared__ __align__(16) float2 Bs[kMhK][16];
  int di = 0;
  while (di + 1 < lv.ndst && (int)blockIdx.x >= lv.dst[di + 1].tile0) di++;
  const MhDst &d = lv.dst[di];
  const int n0 = ((int)blockIdx.x - d.tile0) * 16, c0 = blockIdx.y * 32;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  c2 acc0 = {0.f, 0.f}, acc1 = {0.f, 0.f};  // columns 2 warp, 2 warp + 1 of row lane
  for (int si = 0; si < d.nsrc; si++) {
    const MhSrc &s = d.src[si];
    const bool trans = s.op == 1 || s.op == 2;
    const float conj_b = s.op >= 2 ? -1.f : 1.f;
    float2 ra[8], rb[4];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int i = 0; i < 8; i++) {  // thread t: column t % 64 of rows t / 64 + 4 i
        const int k = k0 + (t & 63), r = c0 + (t >> 6) + 4 * i;
        ra[i] = make_float2(0.f, 0.f);
        if (k < s.k && r < lv.C) {
          ra[i] = __ldg(s.A + (size_t)r * s.lda + k);
          if (s.e) {
            const float2 e = __ldg(s.e + k), x = ra[i];
            ra[i] = make_float2(x.x * e.x + x.y * e.y, x.y * e.x - x.x * e.y);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int q = t + 256 * i;
        const int kk = trans ? q % kMhK : q / 16, col = trans ? q / kMhK : q % 16;
        const int k = k0 + kk, n = n0 + col;
        rb[i] = make_float2(0.f, 0.f);
        if (k < s.k && n < d.n) {
          rb[i] = __ldg(s.B + (trans ? (size_t)n * s.ldb + k : (size_t)k * s.ldb + n));
          rb[i].y *= conj_b;
        }
      }
    };
    fetch(0);
    for (int k0 = 0; k0 < s.k; k0 += kMhK) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; i++) As[t & 63][(t >> 6) + 4 * i] = ra[i];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int q = t + 256 * i;
        const int kk = trans ? q % kMhK : q / 16, col = trans ? q / kMhK : q % 16;
        Bs[kk][col] = rb[i];
      }
      __syncthreads();
      if (k0 + kMhK < s.k) fetch(k0 + kMhK);  // in flight during the products
      // what is staged is summed by itself first: one chain over all sources is
      // longer than a path's product was
      c2 t0 = {0.f, 0.f}, t1 = {0.f, 0.f};
#pragma unroll 8
      for (int k = 0; k < kMhK; k++) {
        const float2 x = As[k][lane];
        const float4 b = *reinterpret_cast<const float4 *>(&Bs[k][2 * warp]);
        mac(t0, c2{x.x, x.y}, c2{b.x, b.y});
        mac(t1, c2{x.x, x.y}, c2{b.z, b.w});
      }
      acc0.x += t0.x; acc0.y += t0.y;
      acc1.x += t1.x; acc1.y += t1.y;
    }
  }
  const int c = c0 + lane;
  if (c >= lv.C) return;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int n = n0 + 2 * warp + j;
    if (n >= d.n) continue;
    c2 v = j ? acc1 : acc0;
    const size_t o = (size_t)c * d.ldo + n;
    if (d.add) { const float2 x = __ldg(d.add + o); v.x += x.x; v.y += x.y; }
    if (d.e) {
      const float2 e = __ldg(d.e + n);
      v = {v.x * e.x - v.y * e.y, v.x * e.y + v.y * e.x};
    }
    d.out[o] = make_float2(v.x, v.y);
    if (d.sum) {
      const float2 x = d.sum_add ? d.sum[o] : make_float2(0.f, 0.f);
      d.sum[o] = make_float2(x.x + v.x, x.y + v.y);
    }
  }
}

// e[m] = exp(j (phi[m] mod max_phase of its metasurface))
struct MhSizes { int n; int first[kMhMax + 1]; float max_phase[kMhMax]; };
__global__ void __launch_bounds__(256) k_mh_phase(const float *phi, MhSizes z, float2 *e) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= z.first[z.n]) return;
  int i = 0;
  while (m >= z.first[i + 1]) i++;
  float sn, cs;
  sincosf(py_mod(__ldg(phi + m), z.max_phase[i]), &sn, &cs);
  e[m] = make_float2(cs, sn);
}

// dphi[m] = -sum over levels and codes of Im(conj(D) V); a CTA takes 32
// elements (lanes), its 8 warps split the levels' codes.  D of the last level is
// G_U (gu); the others lie behind each other in D, all V in V ([hops][C][M]).
__global__ void __launch_bounds__(256) k_mh_dphi(const float2 *V, const float2 *D, const float2 *gu,
                                                 int hops, int C, int M, float *dphi) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int m = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (m < M)
    for (int q = wid; q < hops * C; q += 8) {
      const int l = q / C, c = q - l * C;
      const float2 v = __ldg(V + (size_t)q * M + m);
      const float2 g = __ldg((l == hops - 1 ? gu + (size_t)c * M : D + (size_t)q * M) + m);
      acc += g.x * v.y - g.y * v.x;  // Im(conj(g) v)
    }
  __shared__ float red[8][32];
  red[wid][lane] = acc;
  __syncthreads();
  if (wid == 0 && m < M) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) t += red[w][lane];
    dphi[m] = -t;
  }
}

cudaError_t mh_launch(MhLevel &lv, cudaStream_t st) {
  int tiles = 0;
  for (int i = 0; i < lv.ndst; i++) {
    lv.dst[i].tile0 = tiles;
    tiles += (lv.dst[i].n + 15) / 16;
  }
  k_mh_gemm<<<dim3(tiles, (lv.C + 31) / 32), 256, 0, st>>>(lv);
  return cudaGetLastError();
}
}  // namespace

size_t mh_scratch_bytes(int M, int C, int S, int hops) {
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t cm = 8 * (size_t)C * M;
  return al(8 * (size_t)M) + al(cm * hops) + al(cm * std::max(hops - 1, 0)) + 2 * al(cm) +
         al(8 * (size_t)C * S);
}

cudaError_t mh_run(ObjTcPlan *p, const MhArgs &m, const ObjArgs &a0, char *scratch,
                   cudaStream_t st) {
  if (m.n < 1 || m.n > kMhMax || m.hops < 1) return cudaErrorInvalidValue;
  const int M = p->M, C = a0.C, S = p->S, n = m.n;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t cm = (size_t)C * M;
  char *at = scratch;
  auto take = [&](size_t bytes) { float2 *r = reinterpret_cast<float2 *>(at); at += al(bytes); return r; };
  float2 *e = take(8 * (size_t)M), *V = take(8 * cm * m.hops),
         *D = take(8 * cm * std::max(m.hops - 1, 0)), *U = take(8 * cm), *gU = take(8 * cm),
         *gW = take(8 * (size_t)C * S);
  MhSizes z{};
  z.n = n;
  for (int i = 0; i < n; i++) {
    z.first[i + 1] = z.first[i] + m.size[i];
    z.max_phase[i] = m.max_phase[i];
  }
  if (z.first[n] != M) return cudaErrorInvalidValue;
  k_mh_phase<<<(M + 255) / 256, 256, 0, st>>>(m.phi, z, e);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  // H between metasurfaces a -> b as op(B) of what is stored
  auto between = [&](int a, int b, bool adjoint, MhSrc &s) {
    const int lo = std::min(a, b), hi = std::max(a, b);
    s.B = reinterpret_cast<const float2 *>(m.Hmm[lo * n + hi]);
    s.ldb = m.size[hi];
    const bool trans = (a > b) != adjoint;  // stored as [lo, hi]
    s.op = (trans ? 1 : 0);
    if (adjoint) s.op = trans ? 2 : 3;
  };
  // paths forward
  for (int l = 0; l < m.hops; l++) {
    MhLevel lv{};
    lv.C = C;
    lv.ndst = n;
    for (int i = 0; i < n; i++) {
      MhDst &d = lv.dst[i];
      d.out = V + cm * l + z.first[i];
      d.ldo = M;
      d.n = m.size[i];
      d.e = e + z.first[i];
      d.sum = U + z.first[i];
      d.sum_add = l > 0;
      if (l == 0) {
        d.nsrc = 1;
        MhSrc &s = d.src[0];
        s.A = reinterpret_cast<const float2 *>(a0.W);
        s.lda = S;
        s.k = S;
        s.B = reinterpret_cast<const float2 *>(m.Ha[i]);
        s.ldb = m.size[i];
      } else {
        for (int j = 0; j < n; j++) {
          if (j == i) continue;
          MhSrc &s = d.src[d.nsrc++];
          s.A = V + cm * (l - 1) + z.first[j];
          s.lda = M;
          s.k = m.size[j];
          between(j, i, false, s);
        }
      }
    }
    if ((err = mh_launch(lv, st)) != cudaSuccess) return err;
  }
  ObjArgs a = a0;
  a.U_in = reinterpret_cast<const float *>(U);
  a.grad_U = reinterpret_cast<float *>(gU);
  a.grad_W = reinterpret_cast<float *>(gW);
  a.grad_phi = nullptr;
  if ((err = obj_tc_run(p, a, st)) != cudaSuccess) return err;
  // adjoint: D^(l + 1) is G_U for the last level, else at D + cm l
  for (int l = m.hops - 2; l >= 0; l--) {
    const float2 *next = l + 1 == m.hops - 1 ? gU : D + cm * (l + 1);
    MhLevel lv{};
    lv.C = C;
    lv.ndst = n;
    for (int i = 0; i < n; i++) {
      MhDst &d = lv.dst[i];
      d.out = D + cm * l + z.first[i];
      d.add = gU + z.first[i];
      d.ldo = M;
      d.n = m.size[i];
      for (int j = 0; j < n; j++) {
        if (j == i) continue;
        MhSrc &s = d.src[d.nsrc++];
        s.A = next + z.first[j];
        s.lda = M;
        s.k = m.size[j];
        s.e = e + z.first[j];
        between(i, j, true, s);  // (H^(ij))^H [M_j, M_i]
      }
    }
    if ((err = mh_launch(lv, st)) != cudaSuccess) return err;
  }
  const float2 *D1 = m.hops == 1 ? gU : D;
  if (a0.grad_W) {
    MhLevel lv{};
    lv.C = C;
    lv.ndst = 1;
    MhDst &d = lv.dst[0];
    d.out = reinterpret_cast<float2 *>(a0.grad_W);
    d.add = gW;
    d.ldo = S;
    d.n = S;
    d.nsrc = n;
    for (int i = 0; i < n; i++) {
      MhSrc &s = d.src[i];
      s.A = D1 + z.first[i];
      s.lda = M;
      s.k = m.size[i];
      s.e = e + z.first[i];
      s.B = reinterpret_cast<const float2 *>(m.Ha[i]);
      s.ldb = m.size[i];
      s.op = 2;
    }
    if ((err = mh_launch(lv, st)) != cudaSuccess) return err;
  }
  if (m.grad_phi) {
    k_mh_dphi<<<(M + 31) / 32, 256, 0, st>>>(V, D, gU, m.hops, C, M, m.grad_phi);
    err = cudaGetLastError();
  }
  return err;
}

cudaError_t cgemm_run(int m, int n, int k, const float *A, int lda, int opA, const float *B,
                      int ldb, int opB, float *C, int ldc, bool accumulate, cudaStream_t st) {
  if (m <= 0 || n <= 0 || k <= 0 || opA < 0 || opA > 3 || opB < 0 || opB > 3)
    return cudaErrorInvalidValue;
  dim3 grid((n + 15) / 16, (m + 15) / 16), block(16, 16);
  if (grid.y > 65535u) return cudaErrorInvalidValue;
  k_cgemm_small<<<grid, block, 0, st>>>(m, n, k, reinterpret_cast<const float2 *>(A), lda, opA,
                                        reinterpret_cast<const float2 *>(B), ldb, opB,
                                        reinterpret_cast<float2 *>(C), ldc, accumulate ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t coverage_db_run(const float *H, int S, int R, float threshold, float offset,
                            float *out, cudaStream_t st) {
  k_coverage_db<<<(R + 255) / 256, 256, 0, st>>>(H, S, R, threshold, offset, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------
// Fixed scratch for callers that cannot allocate device memory.  The array
// is part of the module image: every device that loads the library holds
// AMS_OBJECTIVE_NOALLOC_MAX_SCRATCH bytes of it until the process exits.
// Host code must not use the symbol itself as a device address; the address
// is looked up per device with cudaGetSymbolAddress.
static __device__ __align__(256) char g_noalloc_scratch[AMS_OBJECTIVE_NOALLOC_MAX_SCRATCH];

cudaError_t obj_noalloc_scratch(char **out) {
  static std::mutex mu;
  static std::vector<char *> per_device;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  if ((int)per_device.size() <= dev) per_device.resize(dev + 1, nullptr);
  if (!per_device[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);  // with `dev` current
    if (e != cudaSuccess) return e;
    per_device[dev] = static_cast<char *>(p);
  }
  *out = per_device[dev];
  return cudaSuccess;
}
