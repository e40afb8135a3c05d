// Train-step kernels around the rasterizer: the L1 + D-SSIM photometric loss with its image
// gradient, and the Adam step of the Gaussian parameters fused with their activations.
//
// Loss (include/loss_utils.h:30-131, as used at src/gaussian_mapper.cpp:384-409):
//   L = (1 - lambda) mean|img - gt| + lambda (1 - mean SSIM(img, gt)),
// SSIM with the 11x11 Gaussian window (sigma 1.5, zero padding 5, per channel), C1 = 0.01^2,
// C2 = 0.03^2.  The window is separable, so every 2D convolution runs as a horizontal 11-tap pass over a
// shared row and a vertical one as running sums in registers.  The gradient follows from
//   dSSIM/dimg(p) = 1/N [ (w * A)(p) + 2 img(p) (w * B)(p) + gt(p) (w * Cm)(p) ]
// with per-pixel A = dS/dmu1, B = dS/d(w * img^2), Cm = dS/d(w * img gt) (the window is
// symmetric, so the adjoint convolution is the same convolution).  One kernel walks the image down
// column strips and does all of it in registers and two shared rows: it computes the local
// statistics, S and A, B, Cm of a row, convolves them back ten rows behind its input and writes
// dL/dimg, with per-block FP64 sums; a second kernel writes the three loss values.
//
// Adam (torch::optim::Adam as configured at src/gaussian_model.cpp:485-518: per-group learning
// rates, betas (0.9, 0.999), eps 1e-15, no weight decay) of the raw parameters xyz, f_dc, f_rest,
// opacity (pre-sigmoid), scaling (log) and rotation (unnormalised), given the rasterizer's
// gradients with respect to the activated values (gaussian_model.cpp:54-77): the activation
// backward (exp, sigmoid, L2 normalisation, SH split) is fused into the step, and the kernel
// writes the activated values for the next forward (SH as FP32 or BF16).  The step counter and
// learning rates are read from device memory, so a captured CUDA graph replays across steps.
#include <algorithm>
#include <cmath>
#include <cuda_bf16.h>

#include "../../include/omnigs_b200.h"
#include "capi_internal.h"
#include "device_util.cuh"

namespace omnigs {
namespace {

constexpr int kWin = 11, kHalf = 5;
constexpr double kC1 = 0.01 * 0.01, kC2 = 0.03 * 0.03;

struct LossParams {
  const float* img;   // [C][H][W]
  const float* gt;
  float* dimg;        // [C][H][W] gradient; rows >= `rows` are set to 0
  double* sums;       // [2 * blocks]: per-block sum |img - gt|, sum S
  int C, H, W, rows;
  int chunk;          // output rows of a block
  float lambda;
  float w[kWin];
};

// A block owns kLossCols output columns of `chunk` rows of one channel; a thread owns one column of
// the kLossThreads statistics columns these need.
constexpr int kLossThreads = 128;
constexpr int kLossCols = kLossThreads - 2 * kHalf;
constexpr int kLossInCols = kLossThreads + 2 * kHalf;
constexpr int kLossMinChunk = 4;
constexpr int kLossBlocksPerSm = 3;  // (168 registers; four measured 171 us against 137)

// Block sums of (a, b) into partials[2 * block] (no contended atomics; loss_finalize adds them).
__device__ __forceinline__ void block_sum2(double a, double b, double* partials) {
  __shared__ double s_red[2][kLossThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFullMask, a, o);
    b += __shfl_xor_sync(kFullMask, b, o);
  }
  if (lane == 0) {
    s_red[0][warp] = a;
    s_red[1][warp] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (int k = 0; k < kLossThreads / 32; ++k) {
      ta += s_red[0][k];
      tb += s_red[1][k];
    }
    const size_t blk = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    partials[2 * blk] = ta;
    partials[2 * blk + 1] = tb;
  }
}

// acc[j] holds the window sum of the row that is complete in j + 1 more rows; a row's value v enters
// all eleven windows that contain it, and the one that it completes comes back.
__device__ __forceinline__ float window_step(float (&acc)[kWin - 1], const float* w, float v) {
  const float done = fmaf(w[kWin - 1], v, acc[0]);
#pragma unroll
  for (int j = 0; j < kWin - 2; ++j) acc[j] = fmaf(w[kWin - 2 - j], v, acc[j + 1]);
  acc[kWin - 2] = w[0] * v;
  return done;
}
// The same for two quantities in packed arithmetic (each lane rounded as the scalar form).
__device__ __forceinline__ float2 window_step(float2 (&acc)[kWin - 1], const float2* w2, float2 v) {
  const float2 done = __ffma2_rn(w2[kWin - 1], v, acc[0]);
#pragma unroll
  for (int j = 0; j < kWin - 2; ++j) acc[j] = __ffma2_rn(w2[kWin - 2 - j], v, acc[j + 1]);
  acc[kWin - 2] = __fmul2_rn(w2[0], v);
  return done;
}

// Loss and gradient in one walk down a strip.  Row y of the inputs is in shared memory; a thread
// filters it horizontally at its column (img, gt and their three products), the vertical windows are
// running sums in registers, and they complete the statistics of row y - 5.  Their A, B, Cm go through
// a second shared row and a second set of windows, which a row later complete the gradient of row
// y - 11.  Both shared rows are double buffered, so a row costs one barrier; the inputs are loaded three
// rows ahead.  Every sum runs over its taps in the order of a direct 11-tap pass, rounded tap by tap.
//
// The pass is bound by instruction issue and the latency of its FMA chains (363 instructions a row and
// warp, three warps a scheduler, 64 % issue active), not by memory: 75 MB at 2048x1024x3.  Measured
// there on a B200, against two kernels through a 75 MB workspace, each with its horizontal and
// vertical pass in shared memory: 213 -> 137 us (157 us with the pairs in scalar arithmetic, 140 us
// with the two horizontal passes on either side of the barrier).  Strips recompute ten columns a side
// and chunks ten rows at each end (loss_chunk).
__global__ void __launch_bounds__(kLossThreads, kLossBlocksPerSm) ssim_loss_kernel(const __grid_constant__ LossParams p) {
  __shared__ float2 s_in[2][kLossInCols];          // (img, gt) of the current and next input row
  __shared__ float2 s_ab[2][kLossInCols];          // (A, B) of a statistics row, from column xs - 5 of thread 0
  __shared__ float s_c[2][kLossInCols];            // Cm
  const int t = threadIdx.x;
  const int x0 = blockIdx.x * kLossCols;           // first output column
  const int xs = x0 - kHalf + t;                   // this thread's column
  const int ya = blockIdx.y * p.chunk, yb = min(ya + p.chunk, p.rows);
  const size_t plane = (size_t)p.H * p.W;
  const float* img = p.img + blockIdx.z * plane;
  const float* gt = p.gt + blockIdx.z * plane;
  float* d = p.dimg + blockIdx.z * plane;
  const bool in_x = xs >= 0 && xs < p.W;
  const bool owner = in_x && t >= kHalf && t < kLossThreads - kHalf;
  const float invN = (float)(1.0 / ((double)p.C * p.rows * p.W));
  const float k_l1 = (1.f - p.lambda) * invN, k_ssim = -p.lambda * invN;
  const float* w = p.w;

  // input columns x0 - 10 + c, c = t and (the first ten threads) c = kLossThreads + t; offsets within a
  // plane fit 32 bits (at most 2^28 pixels)
  const int xi = x0 - 2 * kHalf + t, xe = xi + kLossThreads;
  const bool in_i = xi >= 0 && xi < p.W, in_e = t < 2 * kHalf && xe < p.W;
  const bool extra = t < 2 * kHalf;
  auto load = [&](bool ok, int y, int x) {
    float2 v = make_float2(0.f, 0.f);
    if (ok && (unsigned)y < (unsigned)p.rows) {
      const int o = y * p.W + x;
      v = make_float2(__ldg(img + o), __ldg(gt + o));
    }
    return v;
  };
  float2 n1, n2, n3, e1 = {}, e2 = {}, e3 = {};
  const int y_first = ya - 2 * kHalf;
  s_in[y_first & 1][t] = load(in_i, y_first, xi);
  n1 = load(in_i, y_first + 1, xi);
  n2 = load(in_i, y_first + 2, xi);
  if (extra) {
    s_in[y_first & 1][kLossThreads + t] = load(in_e, y_first, xe);
    e1 = load(in_e, y_first + 1, xe);
    e2 = load(in_e, y_first + 2, xe);
  }
  // (img, gt), (img^2, gt^2) and (A, B) run as packed pairs
  float2 w2[kWin];
#pragma unroll
  for (int k = 0; k < kWin; ++k) w2[k] = make_float2(w[k < kHalf ? k : kWin - 1 - k], w[k < kHalf ? k : kWin - 1 - k]);
  float2 acc_m[kWin - 1] = {}, acc_s[kWin - 1] = {}, acc_ab[kWin - 1] = {};
  float acc_x[kWin - 1] = {}, acc_c[kWin - 1] = {};
  double l1 = 0.0, ssum = 0.0;
  for (int i = t; i < kLossInCols; i += kLossThreads)  // (the margins are read by threads that own nothing)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      s_ab[q][i] = make_float2(0.f, 0.f);
      s_c[q][i] = 0.f;
    }
  __syncthreads();

  float2 uo = make_float2(0.f, 0.f), uo_next = uo;  // (img, gt) at the gradient's row and the next one's
#pragma unroll 1
  for (int y = y_first; y <= yb + 2 * kHalf; ++y) {
    const int cur = y & 1;
    n3 = load(in_i, y + 3, xi);
    if (extra) e3 = load(in_e, y + 3, xe);
    const int yo = y - 1 - 2 * kHalf;  // the gradient row that the previous statistics row completes
    uo = uo_next;
    if (yo + 1 >= ya) uo_next = load(owner, yo + 1, xs);
    // the input row and the previous statistics row, filtered horizontally
    float2 hm = make_float2(0.f, 0.f), hs = hm, hab = hm;
    float hx = 0.f, hc = 0.f;
    const float2* in = &s_in[cur][t];
    const float2* ab = &s_ab[cur ^ 1][t];
    const float* cm = &s_c[cur ^ 1][t];
#pragma unroll
    for (int k = 0; k < kWin; ++k) {
      const float2 v = in[k];
      hm = __ffma2_rn(w2[k], v, hm);
      hs = __ffma2_rn(w2[k], __fmul2_rn(v, v), hs);
      hx = fmaf(w[k], __fmul_rn(v.x, v.y), hx);
      hab = __ffma2_rn(w2[k], ab[k], hab);
      hc = fmaf(w[k], cm[k], hc);
    }
    const float2 mu = window_step(acc_m, w2, hm), m2 = window_step(acc_s, w2, hs);
    const float mu1 = mu.x, mu2 = mu.y, m11 = m2.x, m22 = m2.y;
    const float m12 = window_step(acc_x, w, hx);
    const float2 cab = window_step(acc_ab, w2, hab);
    const float ca = cab.x, cb = cab.y, cc = window_step(acc_c, w, hc);
    if (owner && yo >= ya) {
      const float u = uo.x, g = uo.y, diff = u - g;
      const float sgn = diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f);
      const float dssim = ca + 2.f * u * cb + g * cc;
      d[yo * p.W + xs] = k_l1 * sgn + k_ssim * dssim;
    }
    // statistics of row y - 5 (0 outside the image, where there is no S, and before the first full window)
    const int ys = y - kHalf;
    float A = 0.f, B = 0.f, Cm = 0.f;
    if (y >= ya && in_x && (unsigned)ys < (unsigned)p.rows) {
      const float mu1_sq = mu1 * mu1, mu2_sq = mu2 * mu2, mu1_mu2 = mu1 * mu2;
      const float s1 = m11 - mu1_sq, s2 = m22 - mu2_sq, s12 = m12 - mu1_mu2;
      const float a1 = 2.f * mu1_mu2 + (float)kC1, a2 = 2.f * s12 + (float)kC2;
      const float b1 = mu1_sq + mu2_sq + (float)kC1, b2 = s1 + s2 + (float)kC2;
      const float inv = 1.f / (b1 * b2);
      const float S = a1 * a2 * inv;
      // dS/dmu1, dS/d(w * img^2), dS/d(w * img gt) with mu2 and the gt moments fixed
      A = 2.f * mu2 * (a2 - a1) * inv - 2.f * mu1 * S * (1.f / b1 - 1.f / b2);
      B = -S / b2;
      Cm = 2.f * a1 * inv;
      if (owner && ys >= ya && ys < yb) ssum += (double)S;
    }
    if (owner && y >= ya && y < yb) {
      const float2 v = in[kHalf];
      l1 += (double)fabsf(v.x - v.y);
    }
    s_ab[cur][kHalf + t] = make_float2(A, B);
    s_c[cur][kHalf + t] = Cm;
    s_in[cur ^ 1][t] = n1;
    if (extra) s_in[cur ^ 1][kLossThreads + t] = e1;
    __syncthreads();
    n1 = n2;
    n2 = n3;
    e1 = e2;
    e2 = e3;
  }
  // rows below `rows` are not part of the loss
  if (blockIdx.y == gridDim.y - 1 && owner)
    for (int y = p.rows; y < p.H; ++y) d[y * p.W + xs] = 0.f;
  block_sum2(l1, ssum, p.sums);
}

__global__ void __launch_bounds__(1024) loss_finalize_kernel(const double* partials, int blocks, float* loss,
                                                              double invN, float lambda) {
  __shared__ double s_red[2][32];
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
    a += partials[2 * i];
    b += partials[2 * i + 1];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFullMask, a, o);
    b += __shfl_xor_sync(kFullMask, b, o);
  }
  if (lane == 0) {
    s_red[0][warp] = a;
    s_red[1][warp] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (int k = 0; k < (int)(blockDim.x / 32); ++k) {
      ta += s_red[0][k];
      tb += s_red[1][k];
    }
    const double l1 = ta * invN, ssim = tb * invN;
    loss[0] = (float)((1.0 - lambda) * l1 + lambda * (1.0 - ssim));
    loss[1] = (float)l1;
    loss[2] = (float)ssim;
  }
}

// ---------------------------------------------------------------- Adam ------------------------
struct AdamParams {
  OmnigsGaussianParams prm;
  OmnigsAdamState st;
  OmnigsActivated act;
  const float* dL_dmeans3D;
  const float* dL_dsh;
  const float* dL_dopacity;
  const float* dL_dscales;
  const float* dL_drotations;
  const OmnigsAdamHyper* hyper;  // device
  bool aligned;                  // every array starts on 16 bytes
  int sh_tile;                   // Gaussians per SH tile (adam_sh_gaussians)
  unsigned first_chunk[4];       // first block of the xyz, scaling, rotation and opacity chunks
};

struct AdamScalars {
  float step_size, bc2_sqrt, beta1, one_minus_beta1, beta2, one_minus_beta2, eps;
};

// x^n by repeated squaring: at most two multiplications per bit of n, in every block, where pow()'s
// latency measured 30 us of a step over 1M Gaussians.  Its error, some 2 log2(n) units in the last place
// of a double, is far below the rounding to float that follows.
__device__ __forceinline__ double power_int(double x, long long n) {
  double r = 1.0;
  for (long long k = n < 0 ? -n : n; k > 0; k >>= 1, x *= x)
    if (k & 1) r *= x;
  return n < 0 ? 1.0 / r : r;
}

// The float coefficients torch::optim::Adam applies to a group (its double options rounded once);
// bc: 1 - beta^t.
__device__ __forceinline__ AdamScalars adam_scalars(const OmnigsAdamHyper& h, int group, const double bc[2]) {
  AdamScalars s;
  s.step_size = (float)(h.lr[group] / bc[0]);
  s.bc2_sqrt = (float)sqrt(bc[1]);
  s.beta1 = (float)h.beta1;
  s.one_minus_beta1 = (float)(1.0 - h.beta1);
  s.beta2 = (float)h.beta2;
  s.one_minus_beta2 = (float)(1.0 - h.beta2);
  s.eps = (float)h.eps;
  return s;
}
// Those of groups ga and gb, with the two powers evaluated by two threads of the block (all call it).
__device__ __forceinline__ void adam_scalars2(const OmnigsAdamHyper& h, int ga, int gb, AdamScalars& a, AdamScalars& b) {
  __shared__ AdamScalars s_sc[2];
  __shared__ double s_bc[2];
  if (threadIdx.x < 2) s_bc[threadIdx.x] = 1.0 - power_int(threadIdx.x ? h.beta2 : h.beta1, h.step);
  __syncthreads();
  if (threadIdx.x < 2) s_sc[threadIdx.x] = adam_scalars(h, threadIdx.x ? gb : ga, s_bc);
  __syncthreads();
  a = s_sc[0];
  b = s_sc[1];
}

// One Adam update of one parameter value (torch::optim::Adam: exp_avg = b1 m + (1 - b1) g,
// exp_avg_sq = b2 v + (1 - b2) g^2, p -= step_size m / (sqrt(v) / sqrt(bc2) + eps)).
__device__ __forceinline__ float adam_update(float& p, float& m, float& v, float g, const AdamScalars& s) {
  m = __fmaf_rn(s.one_minus_beta1, g, __fmul_rn(m, s.beta1));
  v = __fmaf_rn(__fmul_rn(s.one_minus_beta2, g), g, __fmul_rn(v, s.beta2));
  const float denom = __fadd_rn(__fdiv_rn(sqrtf(v), s.bc2_sqrt), s.eps);
  p = __fsub_rn(p, __fmul_rn(s.step_size, __fdiv_rn(m, denom)));
  return p;
}

// Every block updates a contiguous piece of one part of the model, so that all loads and stores are
// coalesced and a block has few arrays open: the first blocks take the SH coefficients (f_dc, f_rest) of
// a tile of Gaussians each, the others kAdamChunk elements of xyz, scaling, opacity or rotation.  A thread
// loads its elements of p, m, v (16 bytes each when the piece is whole and the arrays are aligned) before
// it updates any.
//
// The pass is bound by HBM: 1.88 GB per step over 1M Gaussians (16 SH coefficients).  Measured there on a
// B200: a loop over the Gaussians with a thread each (accesses of stride 3 and 4 floats) and one over the
// f_rest elements 596 us; blocks that take all groups of 64 Gaussians, with 30 arrays open at once,
// 405-425 us whatever the tile, occupancy or work per thread; this split 326 us, 89 % of the copy rate.
// A tile is at most two vectors a thread: with 16 coefficients 32 Gaussians and 192 threads measured
// fastest (318 us over one model's buffers; 256 threads 334 us, 128 threads 351 us; tiles of 64 with 256 or 384
// threads 349 and 332 us).
// Fewer coefficients take more Gaussians (with one, tiles of 32 left 7 of 8 threads idle: 168 us per step
// over 1.1M Gaussians, 96 with tiles of 512).
constexpr int kAdamThreads = 192;
constexpr int kAdamVecs = 2;  // 16-byte vectors per thread and SH tile
inline int adam_sh_gaussians(int M) { return kAdamVecs * kAdamThreads * 4 / (3 * M) & ~3; }
constexpr int kAdamChunk = 2 * 4 * kAdamThreads;
constexpr int kAdamBlocksPerSm = 5;

template <int kW>
struct AdamVec {
  float v[kW];
};
template <int kW>
__device__ __forceinline__ AdamVec<kW> adam_load(const float* p, int64_t i) {
  AdamVec<kW> r;
  if (kW == 4) {
    const float4 f = reinterpret_cast<const float4*>(p)[i];
    r.v[0] = f.x, r.v[1 % kW] = f.y, r.v[2 % kW] = f.z, r.v[3 % kW] = f.w;
  } else {
    r.v[0] = p[i];
  }
  return r;
}
template <int kW>
__device__ __forceinline__ void adam_store(float* p, int64_t i, const AdamVec<kW>& r) {
  if (kW == 4)
    reinterpret_cast<float4*>(p)[i] = make_float4(r.v[0], r.v[1 % kW], r.v[2 % kW], r.v[3 % kW]);
  else
    p[i] = r.v[0];
}

// One vector of one parameter group: p, m, v loaded by the caller, gradients g.
template <int kW>
__device__ __forceinline__ void adam_vec(float* prm, float* m, float* v, int64_t i, AdamVec<kW>& pv, AdamVec<kW>& mv,
                                         AdamVec<kW>& vv, const AdamVec<kW>& g, const AdamScalars& s) {
#pragma unroll
  for (int k = 0; k < kW; ++k) adam_update(pv.v[k], mv.v[k], vv.v[k], g.v[k], s);
  adam_store<kW>(prm, i, pv);
  adam_store<kW>(m, i, mv);
  adam_store<kW>(v, i, vv);
}

// Vectors [first, end) of a group by the block's threads: grad(i) and put(i, new values) take the index of a vector.  A
// thread loads 16 bytes of p, m and v, also where they come one by one (one after the other, unaligned gradients of 100,000
// Gaussians took 64 us instead of 50).
template <int kW, class Grad, class Put>
__device__ __forceinline__ void adam_span(float* prm, float* m, float* v, int64_t first, int64_t end, const AdamScalars& s,
                                          Grad grad, Put put) {
  constexpr int kSteps = 4 / kW;
  for (int64_t i0 = first + threadIdx.x; i0 < end; i0 += kSteps * kAdamThreads) {
    AdamVec<kW> pv[kSteps], mv[kSteps], vv[kSteps], g[kSteps];
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
      const int64_t i = i0 + u * kAdamThreads;
      if (i < end) pv[u] = adam_load<kW>(prm, i), mv[u] = adam_load<kW>(m, i), vv[u] = adam_load<kW>(v, i), g[u] = grad(i);
    }
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
      const int64_t i = i0 + u * kAdamThreads;
      if (i >= end) break;
      adam_vec<kW>(prm, m, v, i, pv[u], mv[u], vv[u], g[u], s);
      put(i, pv[u]);
    }
  }
}
// Elements [first, first + kAdamChunk) of a group of n elements.
template <int kW, class Grad, class Put>
__device__ __forceinline__ void adam_group(float* prm, float* m, float* v, int64_t first, int64_t n,
                                           const AdamScalars& s, Grad grad, Put put) {
  adam_span<kW>(prm, m, v, first / kW, min(n, first + kAdamChunk) / kW, s, grad, put);
}

// One chunk of xyz (group 0), scaling (4), opacity (3) or rotation (5).
template <int kW>
__device__ __forceinline__ void adam_chunk(const AdamParams& p, int group, int64_t first) {
  const int64_t P = p.prm.P;
  AdamScalars s, unused;
  adam_scalars2(*p.hyper, group, group, s, unused);
  if (group == 0) {  // the activated mean is the parameter itself
    adam_group<kW>(p.prm.xyz, p.st.m_xyz, p.st.v_xyz, first, 3 * P, s,
                   [&](int64_t i) { return adam_load<kW>(p.dL_dmeans3D, i); },
                   [&](int64_t i, const AdamVec<kW>& x) { if (p.act.means3D != p.prm.xyz) adam_store<kW>(p.act.means3D, i, x); });
  } else if (group == 4) {  // exp
    adam_group<kW>(p.prm.scaling, p.st.m_scaling, p.st.v_scaling, first, 3 * P, s,
                   [&](int64_t i) {
                     AdamVec<kW> x = adam_load<kW>(p.dL_dscales, i);
                     const AdamVec<kW> e = adam_load<kW>(p.act.scales, i);  // exp of the current parameter
#pragma unroll
                     for (int k = 0; k < kW; ++k) x.v[k] = x.v[k] * e.v[k];
                     return x;
                   },
                   [&](int64_t i, AdamVec<kW> x) {
#pragma unroll
                     for (int k = 0; k < kW; ++k) x.v[k] = expf(x.v[k]);
                     adam_store<kW>(p.act.scales, i, x);
                   });
  } else if (group == 3) {  // sigmoid
    adam_group<kW>(p.prm.opacity, p.st.m_opacity, p.st.v_opacity, first, P, s,
                   [&](int64_t i) {
                     AdamVec<kW> x = adam_load<kW>(p.dL_dopacity, i);
                     const AdamVec<kW> o = adam_load<kW>(p.act.opacities, i);  // sigmoid of the current parameter
#pragma unroll
                     for (int k = 0; k < kW; ++k) x.v[k] = x.v[k] * o.v[k] * (1.f - o.v[k]);
                     return x;
                   },
                   [&](int64_t i, AdamVec<kW> x) {
#pragma unroll
                     for (int k = 0; k < kW; ++k) x.v[k] = 1.f / (1.f + expf(-x.v[k]));
                     adam_store<kW>(p.act.opacities, i, x);
                   });
  } else {  // rotation: a quaternion per thread, L2 normalisation (F.normalize, eps 1e-12)
    for (int64_t g = first / 4 + threadIdx.x; g < min(P, (first + kAdamChunk) / 4); g += kAdamThreads) {
      auto quat = [&](const float* a) {
        if (kW == 4) return adam_load<4>(a, g);
        return AdamVec<4>{{a[4 * g], a[4 * g + 1], a[4 * g + 2], a[4 * g + 3]}};
      };
      auto put = [&](float* a, const AdamVec<4>& x) {
        if (kW == 4)
          adam_store<4>(a, g, x);
        else
          for (int k = 0; k < 4; ++k) a[4 * g + k] = x.v[k];
      };
      AdamVec<4> r = quat(p.prm.rotation), gr = quat(p.dL_drotations), m = quat(p.st.m_rotation), v = quat(p.st.v_rotation);
      const float n = fmaxf(sqrtf(r.v[0] * r.v[0] + r.v[1] * r.v[1] + r.v[2] * r.v[2] + r.v[3] * r.v[3]), 1e-12f);
      const float inv = 1.f / n;
      const float yg = (r.v[0] * gr.v[0] + r.v[1] * gr.v[1] + r.v[2] * gr.v[2] + r.v[3] * gr.v[3]) * inv;  // y . g
#pragma unroll
      for (int k = 0; k < 4; ++k) adam_update(r.v[k], m.v[k], v.v[k], (gr.v[k] - r.v[k] * inv * yg) * inv, s);
      const float n2 = fmaxf(sqrtf(r.v[0] * r.v[0] + r.v[1] * r.v[1] + r.v[2] * r.v[2] + r.v[3] * r.v[3]), 1e-12f);
      AdamVec<4> y;
#pragma unroll
      for (int k = 0; k < 4; ++k) y.v[k] = r.v[k] / n2;
      put(p.prm.rotation, r);
      put(p.st.m_rotation, m);
      put(p.st.v_rotation, v);
      put(p.act.rotations, y);
    }
  }
}

// The SH coefficients of Gaussians [g0, g0 + ng): the gradients and the new values, whose rows interleave
// f_dc (group 1) and f_rest (group 2), pass through shared memory.
template <int kW>
__device__ __forceinline__ void adam_sh_tile(const AdamParams& p, float* s_sh, int g0, int ng) {
  const int M = p.prm.M, per = (M - 1) * 3, row = M * 3, t = threadIdx.x;
  const float* dsh = p.dL_dsh + (size_t)g0 * row;
#pragma unroll 4
  for (int i = t; i < ng * row / kW; i += kAdamThreads) {
    if (kW == 4) {
      cp_async16(s_sh + 4 * i, dsh + 4 * i);
    } else {
      s_sh[i] = dsh[i];
    }
  }
  // element e of the tile's f_dc and f_rest in shared memory; e / per as a multiply-high by
  // ceil(2^32 / per), exact for e < 2^16
  const uint32_t magic = per > 0 ? (uint32_t)((0x100000000ull + per - 1) / per) : 0u;
  auto rest_at = [&](int e) -> float& { return s_sh[e + 3 * (int)__umulhi((uint32_t)e, magic) + 3]; };
  auto dc_at = [&](int e) -> float& { const int g = e / 3; return s_sh[g * row + (e - 3 * g)]; };
  float* dc_p = p.prm.features_dc + (size_t)3 * g0;
  float* dc_m = p.st.m_dc + (size_t)3 * g0;
  float* dc_v = p.st.v_dc + (size_t)3 * g0;
  float* rest_p = per > 0 ? p.prm.features_rest + (size_t)g0 * per : nullptr;
  float* rest_m = per > 0 ? p.st.m_rest + (size_t)g0 * per : nullptr;
  float* rest_v = per > 0 ? p.st.v_rest + (size_t)g0 * per : nullptr;
  const int dc_n = 3 * ng / kW, rest_n = ng * per / kW;
  AdamScalars s_dc, s_rest;
  if (kW == 4) {  // a whole tile: everything is loaded before the gradients have arrived
    AdamVec<4> pv[kAdamVecs], mv[kAdamVecs], vv[kAdamVecs];
    auto at = [&](int u, float*& prm, float*& m, float*& v) {  // the thread's vector u: f_rest's, then f_dc's
      const int i = t + u * kAdamThreads;
      const bool rest = i < rest_n;
      prm = rest ? rest_p : dc_p, m = rest ? rest_m : dc_m, v = rest ? rest_v : dc_v;
      return rest ? i : i < rest_n + dc_n ? i - rest_n : -1;
    };
#pragma unroll
    for (int u = 0; u < kAdamVecs; ++u) {
      float *prm, *m, *v;
      const int j = at(u, prm, m, v);
      if (j >= 0) pv[u] = adam_load<4>(prm, j), mv[u] = adam_load<4>(m, j), vv[u] = adam_load<4>(v, j);
    }
    adam_scalars2(*p.hyper, 1, 2, s_dc, s_rest);
    cp_async_wait_all();
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kAdamVecs; ++u) {
      float *prm, *m, *v;
      const int j = at(u, prm, m, v);
      if (j < 0) continue;
      // element e of f_rest lies at e + 3 (e / per) + 3 of the tile's rows, of f_dc at e + (row - 3) (e / 3)
      const bool rest = t + u * kAdamThreads < rest_n;
      const uint32_t by = rest ? magic : 0x55555556u;
      const int skip = rest ? 3 : row - 3, off = rest ? 3 : 0;
      AdamScalars s = s_dc;
      s.step_size = rest ? s_rest.step_size : s_dc.step_size;  // (all that differs by group)
      int pos[4];
      AdamVec<4> g;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        pos[k] = 4 * j + k + skip * (int)__umulhi((uint32_t)(4 * j + k), by) + off;
        g.v[k] = s_sh[pos[k]];
      }
      adam_vec<4>(prm, m, v, j, pv[u], mv[u], vv[u], g, s);
#pragma unroll
      for (int k = 0; k < 4; ++k) s_sh[pos[k]] = pv[u].v[k];
    }
  } else {
    adam_scalars2(*p.hyper, 1, 2, s_dc, s_rest);
    __syncthreads();
    auto span = [&](float* prm, float* m, float* v, int n, const AdamScalars& sc, auto at) {
      adam_span<1>(prm, m, v, 0, n, sc, [&](int64_t i) { return AdamVec<1>{{at((int)i)}}; },
                   [&](int64_t i, const AdamVec<1>& x) { at((int)i) = x.v[0]; });
    };
    span(rest_p, rest_m, rest_v, rest_n, s_rest, rest_at);
    span(dc_p, dc_m, dc_v, dc_n, s_dc, dc_at);
  }
  __syncthreads();
  if (p.act.shs_bf16) {
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.act.shs) + (size_t)g0 * row;
    if (kW == 4) {
      for (int i = t; i < ng * row / 4; i += kAdamThreads) {
        const AdamVec<4> f = adam_load<4>(s_sh, i);
        const __nv_bfloat162 lo = __floats2bfloat162_rn(f.v[0], f.v[1]), hi = __floats2bfloat162_rn(f.v[2], f.v[3]);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&lo);
        u.y = *reinterpret_cast<const uint32_t*>(&hi);
        reinterpret_cast<uint2*>(out)[i] = u;
      }
    } else {
      for (int i = t; i < ng * row; i += kAdamThreads) out[i] = __float2bfloat16_rn(s_sh[i]);
    }
  } else {
    float* out = static_cast<float*>(p.act.shs) + (size_t)g0 * row;
    for (int i = t; i < ng * row / kW; i += kAdamThreads) adam_store<kW>(out, i, adam_load<kW>(s_sh, i));
  }
}

__global__ void __launch_bounds__(kAdamThreads, kAdamBlocksPerSm) adam_gaussian_kernel(const __grid_constant__ AdamParams p) {
  extern __shared__ float4 s_sh4[];  // [sh_tile][M][3]
  // SH tiles first; 16-byte accesses need whole pieces (which then start on 16 bytes if the arrays do)
  if (blockIdx.x < p.first_chunk[0]) {
    const int g0 = blockIdx.x * p.sh_tile, ng = min(p.sh_tile, p.prm.P - g0);
    if (p.aligned && ng == p.sh_tile)
      adam_sh_tile<4>(p, reinterpret_cast<float*>(s_sh4), g0, ng);
    else
      adam_sh_tile<1>(p, reinterpret_cast<float*>(s_sh4), g0, ng);
    return;
  }
  // then the chunks of xyz, scaling, rotation and opacity
  const int part = (blockIdx.x >= p.first_chunk[1]) + (blockIdx.x >= p.first_chunk[2]) + (blockIdx.x >= p.first_chunk[3]);
  const int group = part == 0 ? 0 : part == 1 ? 4 : part == 2 ? 5 : 3;
  const int per = part < 2 ? 3 : part == 2 ? 4 : 1;
  const int64_t first = (int64_t)(blockIdx.x - p.first_chunk[part]) * kAdamChunk;
  if (p.aligned && first + kAdamChunk <= (int64_t)p.prm.P * per)
    adam_chunk<4>(p, group, first);
  else
    adam_chunk<1>(p, group, first);
}

// Activated values from the raw parameters (the first forward of a training run).
__global__ void __launch_bounds__(256) activate_kernel(const OmnigsGaussianParams prm, const OmnigsActivated act) {
  const int P = prm.P, M = prm.M;
  const int64_t rest_n = (int64_t)P * (M - 1) * 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto put_sh = [&](size_t idx, float v) {
    if (act.shs_bf16)
      reinterpret_cast<__nv_bfloat16*>(act.shs)[idx] = __float2bfloat16_rn(v);
    else
      static_cast<float*>(act.shs)[idx] = v;
  };
  if (i < P) {
    const int g = (int)i;
    for (int k = 0; k < 3; ++k) {
      if (act.means3D != prm.xyz) act.means3D[3 * g + k] = prm.xyz[3 * g + k];
      put_sh((size_t)g * M * 3 + k, prm.features_dc[3 * g + k]);
      act.scales[3 * g + k] = expf(prm.scaling[3 * g + k]);
    }
    act.opacities[g] = 1.f / (1.f + expf(-prm.opacity[g]));
    float r[4];
    for (int k = 0; k < 4; ++k) r[k] = prm.rotation[4 * g + k];
    const float n = fmaxf(sqrtf(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]), 1e-12f);
    for (int k = 0; k < 4; ++k) act.rotations[4 * g + k] = r[k] / n;
  } else if (i - P < rest_n) {
    const uint32_t e = (uint32_t)(i - P);
    const uint32_t per = (uint32_t)(M - 1) * 3u;
    const uint32_t g = e / per, r = e - g * per;
    put_sh((size_t)g * M * 3 + 3 + r, prm.features_rest[e]);
  }
}

int validate_params(const OmnigsGaussianParams* prm, const OmnigsActivated* act) {
  if (prm == nullptr || act == nullptr) return fail(OMNIGS_ERR_INVALID_ARGUMENT, "parameters are NULL");
  if (prm->P < 0 || prm->M < 1 || prm->M > 16)
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "P must be >= 0 and M (SH coefficients) in [1, 16]");
  if ((int64_t)prm->P * (prm->M - 1) * 3 >= (int64_t(1) << 32))
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "P * (M - 1) * 3 must be below 2^32");
  if (prm->P == 0) return OMNIGS_OK;
  if (!prm->xyz || !prm->features_dc || (prm->M > 1 && !prm->features_rest) || !prm->opacity || !prm->scaling ||
      !prm->rotation || !act->means3D || !act->shs || !act->opacities || !act->scales || !act->rotations)
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "a parameter or activated-value array is NULL");
  return OMNIGS_OK;
}

// Workspace part of the loss kernel's block sums, the first; the last holds the gradient when that goes over one of the
// images.  Two doubles a block, whose strips are wider than 32 columns; blocks of less than 16 rows also use what lies
// between, two floats a pixel.
size_t loss_sums_bytes(int C, int H, int W) {
  const size_t blocks = (size_t)C * ((W + 31) / 32) * ((H + 15) / 16);
  return align_up(sizeof(double) * 2 * blocks);
}

// Rows of a block: as many as one wave of blocks takes (a chunk recomputes 20 rows), but at least 16 where such chunks give
// every SM a block, and at least kLossMinChunk where they do not.  Measured on a B200, three channels, 16 rows / fewer: 16x16
// 25 / 19 us, 128x256 28 / 22, 512x100 28 / 23; where they do, 256x512 32 / 33-38.
int loss_chunk(int C, int rows, int W, int sms) {
  const int64_t columns = (int64_t)((W + kLossCols - 1) / kLossCols) * C;
  const bool small = columns * ((rows + 15) / 16) < sms;
  const int chunks = (int)std::max<int64_t>(1, (int64_t)sms * (small ? 1 : kLossBlocksPerSm) / columns);
  return std::max(small ? kLossMinChunk : 16, (rows + chunks - 1) / chunks);
}

}  // namespace
}  // namespace omnigs

using namespace omnigs;

extern "C" {

size_t omnigs_l1_dssim_workspace_bytes(int C, int H, int W) {
  if (C <= 0 || H <= 0 || W <= 0) return 0;
  return loss_sums_bytes(C, H, W) + sizeof(float) * 3 * (size_t)C * H * W;
}

int omnigs_l1_dssim(const float* image, const float* gt, int C, int H, int W, int rows, float lambda_dssim,
                    float* dL_dimage, float* loss, void* workspace, size_t workspace_bytes, omnigs_stream_t stream) {
  g_last_error.clear();
  if (image == nullptr || gt == nullptr || dL_dimage == nullptr || loss == nullptr || workspace == nullptr)
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "image, gt, dL_dimage, loss and workspace are required");
  if (C <= 0 || H <= 0 || W <= 0 || rows <= 0 || rows > H || (int64_t)H * W > (int64_t(1) << 28))
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "image size must be positive with 0 < rows <= H");
  if (!(lambda_dssim >= 0.f && lambda_dssim <= 1.f))
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "lambda_dssim must be in [0, 1]");
  if (workspace_bytes < omnigs_l1_dssim_workspace_bytes(C, H, W))
    return fail(OMNIGS_ERR_BUFFER_TOO_SMALL, "workspace smaller than omnigs_l1_dssim_workspace_bytes()");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  LossParams p{};
  p.img = image;
  p.gt = gt;
  p.sums = static_cast<double*>(workspace);
  // The kernel reads pixels around those it has written: a gradient that goes over one of the images
  // is written to the workspace first.
  const size_t bytes = sizeof(float) * (size_t)C * H * W;
  auto overlaps = [&](const float* in) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(in), y = reinterpret_cast<uintptr_t>(dL_dimage);
    return x < y + bytes && y < x + bytes;
  };
  const bool in_place = overlaps(image) || overlaps(gt);
  p.dimg = in_place ? reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + loss_sums_bytes(C, H, W) + 2 * bytes) : dL_dimage;
  p.C = C;
  p.H = H;
  p.W = W;
  p.rows = rows;
  p.lambda = lambda_dssim;
  // the reference's window: exp(-x^2 / (2 sigma^2)) in float, normalised (loss_utils.h:54-68)
  float sum = 0.f;
  for (int k = 0; k < kWin; ++k) {
    const int t = k - kWin / 2;
    p.w[k] = std::exp(-(float)(t * t) / (2.0f * 1.5f * 1.5f));
    sum += p.w[k];
  }
  for (int k = 0; k < kWin; ++k) p.w[k] /= sum;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int strips = (W + kLossCols - 1) / kLossCols;
  p.chunk = loss_chunk(C, rows, W, sms);
  const dim3 grid(strips, (rows + p.chunk - 1) / p.chunk, C);
  const int blocks = (int)(grid.x * grid.y * grid.z);
  staged(OMNIGS_STAGE_OTHER, 2, s, [&] {
    ssim_loss_kernel<<<grid, kLossThreads, 0, s>>>(p);
    loss_finalize_kernel<<<1, 1024, 0, s>>>(p.sums, blocks, loss, 1.0 / ((double)C * rows * W), lambda_dssim);
  });
  if (in_place && cudaMemcpyAsync(dL_dimage, p.dimg, bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return check_launch("copy image gradient");
  return check_launch("l1 + d-ssim");
}

int omnigs_activate(const OmnigsGaussianParams* prm, const OmnigsActivated* act, omnigs_stream_t stream) {
  g_last_error.clear();
  if (int rc = validate_params(prm, act)) return rc;
  if (prm->P == 0) return OMNIGS_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int64_t n = (int64_t)prm->P + (int64_t)prm->P * (prm->M - 1) * 3;
  staged(OMNIGS_STAGE_OTHER, 1, s,
         [&] { activate_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(*prm, *act); });
  return check_launch("activate");
}

int omnigs_adam_step(const OmnigsGaussianParams* prm, const OmnigsAdamState* st, const OmnigsActivated* act,
                     const float* dL_dmeans3D, const float* dL_dsh, const float* dL_dopacity, const float* dL_dscales,
                     const float* dL_drotations, const OmnigsAdamHyper* hyper, omnigs_stream_t stream) {
  g_last_error.clear();
  if (int rc = validate_params(prm, act)) return rc;
  if (st == nullptr || hyper == nullptr) return fail(OMNIGS_ERR_INVALID_ARGUMENT, "Adam state and hyper are required");
  if (prm->P == 0) return OMNIGS_OK;
  if (!dL_dmeans3D || !dL_dsh || !dL_dopacity || !dL_dscales || !dL_drotations || !st->m_xyz || !st->v_xyz ||
      !st->m_dc || !st->v_dc || (prm->M > 1 && (!st->m_rest || !st->v_rest)) || !st->m_opacity || !st->v_opacity ||
      !st->m_scaling || !st->v_scaling || !st->m_rotation || !st->v_rotation)
    return fail(OMNIGS_ERR_INVALID_ARGUMENT, "a gradient or Adam moment array is NULL");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  AdamParams p{};
  p.prm = *prm;
  p.st = *st;
  p.act = *act;
  p.dL_dmeans3D = dL_dmeans3D;
  p.dL_dsh = dL_dsh;
  p.dL_dopacity = dL_dopacity;
  p.dL_dscales = dL_dscales;
  p.dL_drotations = dL_drotations;
  p.hyper = hyper;
  const void* arrays[] = {prm->xyz, prm->features_dc, prm->features_rest, prm->opacity, prm->scaling, prm->rotation,
                          st->m_opacity, st->v_opacity, act->opacities, dL_dopacity, st->m_xyz,
                          st->v_xyz, st->m_dc, st->v_dc, st->m_rest, st->v_rest, st->m_scaling, st->v_scaling,
                          st->m_rotation, st->v_rotation, act->means3D, act->shs, act->scales, act->rotations,
                          dL_dmeans3D, dL_dsh, dL_dscales, dL_drotations};
  p.aligned = true;
  for (const void* q : arrays) p.aligned = p.aligned && (reinterpret_cast<uintptr_t>(q) & 15) == 0;
  // blocks: SH tiles, then chunks of xyz, scaling, rotation and opacity
  const int64_t P = prm->P;
  auto chunks = [&](int64_t per) { return (unsigned)((P * per + kAdamChunk - 1) / kAdamChunk); };
  p.sh_tile = adam_sh_gaussians(prm->M);
  p.first_chunk[0] = (unsigned)((P + p.sh_tile - 1) / p.sh_tile);
  p.first_chunk[1] = p.first_chunk[0] + chunks(3);
  p.first_chunk[2] = p.first_chunk[1] + chunks(3);
  p.first_chunk[3] = p.first_chunk[2] + chunks(4);
  const unsigned blocks = p.first_chunk[3] + chunks(1);
  const size_t smem = sizeof(float) * p.sh_tile * 3 * (size_t)prm->M;
  staged(OMNIGS_STAGE_OTHER, 1, s, [&] { adam_gaussian_kernel<<<blocks, kAdamThreads, smem, s>>>(p); });
  return check_launch("adam step");
}

}  // extern "C"
