// Backward back-to-front blend of one 16x16 tile per block (backward.cu:672-843).
//
// Per pixel this replays the reference's recurrence: start from the stored final transmittance
// and last-contributor index, walk the tile's instances from the back, undo T /= (1 - alpha) and
// accumulate the colour behind each splat (the reference defers that update to the next splat it
// meets; here it is applied right after the splat, the same sums).  A thread's two pixels share
// their column, so their arithmetic runs in packed f32x2 instructions, lane x for the upper pixel
// and lane y for the lower: one issue slot for both pixels' FMAs.  One approximate reciprocal of
// 1 - alpha serves both of the reference's divisions by it (relative error ~1e-7 per step, far
// inside the gradients' 1e-3 tolerance).  The per-(pixel, splat) gradients (2 screen-space mean,
// 3 conic, 1 opacity, 3 colour) are not pushed with 9 global atomics per pixel as in the
// reference: a thread sums them over its two pixels and writes six sums to its warp's shared buffer;
// after every fifth contributing splat the warp that owns the 8 x 8 patch reduces the buffer transposed
// and adds the accumulator records with one atomic per value (flush_reduction).  The mean terms are
// summed as w dx and w dy with w = G dL/dalpha, without the opacity and the conic, the conic terms
// without the opacity, all without their constant factors -W/2, -H/2, -1/2: the backward preprocess
// applies those per Gaussian.  A warp walks only the splats that can reach alpha >= 1/255 in its patch
// and do not lie behind all of its pixels' last contributors (blend_common.cuh), and the block starts at
// the batch holding its largest last contributor instead of at the end of the range.
//
// Bound by instruction issue (78 % of the slots on a 400k-Gaussian view).  Measured on a B200
// (300k / 1M-Gaussian 2048x1024 view / 16-view batch): 315 / 760 / 9710 us with the warps scanning ballots
// of their own tests, every sum in a row of its own (nine, two splats a flush) and the clamp and sign
// tests for every splat; 272 / 673 / 8430 us now.  The same sums on the tensor cores (mma.m16n8k8, TF32
// operands split in two) took 319 / 812 / 10600: fewer instructions, but the fragments' registers and
// shared memory leave six blocks per SM.
#include "blend_common.cuh"

namespace omnigs {
namespace {

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---- the reduction of a splat's gradients over the warp's 64 pixels ----
// A lane keeps six sums over its two pixels (w = G dL/dalpha, d = alpha T): w, w dy, w dy^2 and d times the
// three components of dL/dpix.  The other three, w dx, w dx^2 and w dx dy, need no rows of their own: dx is
// the same for all pixels of a column, so the lane that adds up a row's eight columns multiplies the column
// sums by dx.  Row 6 h + q of a warp's buffer holds sum q of buffered splat h for the 32 lanes; five splats
// make 30 rows, one lane each.  The row stride of 36 floats puts the 16-byte reads of 8 consecutive rows
// (one quarter-warp) on distinct banks; the lanes' writes of one row are consecutive words.
constexpr int kRedSplats = 5;
constexpr int kRedRows = 6;
constexpr int kRedStride = 36;

template <int kBatch>
struct BackwardSmem {
  BlendStage<kBatch> stage;
  __align__(16) float red[kBlendWarps][kRedSplats * kRedRows][kRedStride];
  float2 info[kBlendWarps][kRedSplats];  // {x of the splat less the patch's first column, its record}
  uint32_t last[kBlendWarps];
};

// Adds the first n buffered splats' sums to their accumulator records {w dx, w dy, w dx^2, w dx dy}
// {w dy^2, w, r, g}{b, 0, 0, 0}, one atomic per value.
template <int kBatch>
__device__ __forceinline__ void flush_reduction(BackwardSmem<kBatch>& sm, int n, float* grad_acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncwarp();
  if (lane < n * kRedRows) {
    const int h = lane / kRedRows, q = lane - kRedRows * h;
    const float4* row = reinterpret_cast<const float4*>(sm.red[warp][lane]);
    float2 c[4];  // sums of the columns 2 i and 2 i + 1
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 lo = row[2 * i], hi = row[2 * i + 1];
      const float2 v[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y), make_float2(hi.z, hi.w)};
#pragma unroll
      for (int j = 0; j < 4; ++j) c[j] = i ? add2(c[j], v[j]) : v[j];
    }
    const float2 info = sm.info[warp][h];
    const float2 dx0 = make_float2(info.x, info.x - 1.f);
    float2 m1 = mul2(c[0], dx0), m2 = mul2(m1, dx0);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
      const float2 dx = add2(dx0, f2(-2.f * j)), t = mul2(c[j], dx);
      m1 = add2(m1, t);
      m2 = fma2(t, dx, m2);
    }
    const float2 m0 = add2(add2(c[0], c[1]), add2(c[2], c[3]));
    float* acc = grad_acc + 12 * (size_t)__float_as_uint(info.y);
    atomicAdd(acc + ((0x876415u >> (4 * q)) & 15u), m0.x + m0.y);  // w, w dy, w dy^2, r, g, b
    if (q < 2) atomicAdd(acc + 3 * q, m1.x + m1.y);                // w dx, w dx dy
    if (q == 0) atomicAdd(acc + 2, m2.x + m2.y);                   // w dx^2
  }
  __syncwarp();  // the rows are rewritten next
}

// Seven resident blocks per SM (at most 72 registers).  Measured on a B200 (1M-Gaussian view / 16-view
// batch): six 678 / 8610 us, seven 673 / 8430, eight (64 registers, spilling with the seam) 696 / 8840.
constexpr int kBlendBwdMinBlocks = 7;

// kRecompute (transmittance checkpointing): the forward stored no per-pixel state; each pixel's
// final transmittance and last contributor are recomputed first by the forward's own front-to-back
// pass without colour (forward_pass), which yields the values the forward would have stored.
template <int kBatch, bool kWrap, bool kRecompute>
__device__ __forceinline__ void blend_backward_tile(const TileJob& job, const BlendSource& src, float* grad_acc) {
  static_assert(kBlendPx == 2, "a thread owns two pixels of one column");
  __shared__ BackwardSmem<kBatch> sm;
  const BlendPatch patch = BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = job.range.y - job.range.x;
  if (n == 0) return;

  // Per-pixel state of the thread's two pixels (rows py0 and py0 + 4).
  const int64_t HW = (int64_t)job.H * job.W;
  float Tf[2], dp[3][2];
  uint32_t lc[2];
  if (kRecompute) {
    float C[2][3];
    forward_pass<kBatch, kWrap, false>(job, src, patch, sm.stage, Tf, lc, C);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (!patch.inside(i, job.W, job.H)) Tf[i] = 0.f;
      lc[i] = min(lc[i], n);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool in = patch.inside(i, job.W, job.H);
    const int64_t pix = in ? patch.pixel(i, job.W) : 0;
    if (!kRecompute) {
      Tf[i] = in ? job.final_T[pix] : 0.f;
      lc[i] = in ? min(job.n_contrib[pix], n) : 0u;
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) dp[ch][i] = in ? job.dL_dpix[ch * HW + pix] : 0.f;
  }
  float2 T = make_float2(Tf[0], Tf[1]);
  const float2 dp0 = make_float2(dp[0][0], dp[0][1]);
  const float2 dp1 = make_float2(dp[1][0], dp[1][1]);
  const float2 dp2 = make_float2(dp[2][0], dp[2][1]);
  float2 bgdot = make_float2(0.f, 0.f);
  bgdot = fma2(f2(job.bg[0]), dp0, bgdot);
  bgdot = fma2(f2(job.bg[1]), dp1, bgdot);
  bgdot = fma2(f2(job.bg[2]), dp2, bgdot);
  const float2 neg_T_bg = mul2(make_float2(-Tf[0], -Tf[1]), bgdot);
  // the colour of everything behind the current splat, accumulated back to front, enters the
  // gradients only through its dot product with dL/dpix: that product is accumulated instead
  float2 acc_dp = make_float2(0.f, 0.f);
  const float pyf[2] = {patch.pyf(0), patch.pyf(1)};

  const uint32_t warp_last = __reduce_max_sync(kFullMask, max(lc[0], lc[1]));
  if (lane == 0) sm.last[warp] = warp_last;
  init_stage(sm.stage, job);
  __syncthreads();
  uint32_t block_last = 0;
#pragma unroll
  for (int w = 0; w < kBlendWarps; ++w) block_last = max(block_last, sm.last[w]);

  const char* slots = reinterpret_cast<const char*>(&sm.stage.d[0][0]);
  const uint32_t* list = sm.stage.list[warp];
  int nred = 0;  // buffered splats (warp-uniform)
  auto blend = [&](uint32_t off, auto plain) {
    // No per-lane branches: a pixel behind its last contributor, or that this splat does not reach, is
    // inactive, and the masked G = 0 makes alpha, w and d exactly 0 and 1 / (1 - alpha) exactly 1: sm_100's
    // approximate reciprocal of 1 is 1, which its documented error bound does not say (a test holds the gradients
    // of a pixel under 700 such splats to the bit; selecting 1 instead takes two more issue slots a splat).
    constexpr bool kPlain = decltype(plain)::value;
    const float4* slot = reinterpret_cast<const float4*>(slots + off);
    const float4 v0 = slot[0], v1 = slot[1], v2 = slot[2];
    const float x = kWrap ? patch.template center_x<true>(v0.x) : v0.x;
    const float dx = x - patch.pxf;
    const float hx = __fmul_rn(v0.z, dx), bx = __fmul_rn(v0.w, dx);
    const uint32_t at = __float_as_uint(v2.y);
    const float2 dy = make_float2(v0.y - pyf[0], v0.y - pyf[1]);
    const float2 q2 = mul2(make_float2(__fmul_rn(v1.x, dy.x), __fmul_rn(v1.x, dy.y)), dy);
    const float2 power = add2(make_float2(__fmaf_rn(hx, dx, q2.x), __fmaf_rn(hx, dx, q2.y)),
                              make_float2(__fmul_rn(bx, dy.x), __fmul_rn(bx, dy.y)));
    float2 G = make_float2(expf(power.x), expf(power.y));
    const float2 oG = make_float2(__fmul_rn(v1.y, G.x), __fmul_rn(v1.y, G.y));
    bool act0 = lc[0] >= at && !(oG.x < 1.0f / 255.0f), act1 = lc[1] >= at && !(oG.y < 1.0f / 255.0f);
    if (!kPlain) {
      act0 = act0 && !(power.x > 0.0f);
      act1 = act1 && !(power.y > 0.0f);
    }
    // a warp-uniform skip of the gradient arithmetic when no pixel of the warp blends this splat
    if (!__any_sync(kFullMask, act0 || act1)) return;
    G = make_float2(act0 ? G.x : 0.f, act1 ? G.y : 0.f);
    float2 alpha = make_float2(__fmul_rn(v1.y, G.x), __fmul_rn(v1.y, G.y));
    if (!kPlain) alpha = make_float2(act0 ? fminf(0.99f, alpha.x) : 0.f, act1 ? fminf(0.99f, alpha.y) : 0.f);
    const float2 onem = fma2(alpha, f2(-1.f), f2(1.f));
    const float2 inv = make_float2(rcp_approx(onem.x), rcp_approx(onem.y));
    T = mul2(T, inv);  // transmittance in front of this splat
    const float2 d = mul2(alpha, T);
    // (this splat's colour minus the colour behind it) . dL/dpix; the colour behind becomes
    // alpha c + (1 - alpha) acc, so its product with dL/dpix grows by alpha times this
    float2 dLda;
    dLda.x = fmaf(v2.x, dp2.x, fmaf(v1.w, dp1.x, __fmul_rn(v1.z, dp0.x)));
    dLda.y = fmaf(v2.x, dp2.y, fmaf(v1.w, dp1.y, __fmul_rn(v1.z, dp0.y)));
    dLda = fma2(acc_dp, f2(-1.f), dLda);
    acc_dp = fma2(alpha, dLda, acc_dp);
    dLda = mul2(dLda, T);
    dLda = fma2(neg_T_bg, inv, dLda);  // the background term -T_final / (1 - alpha) bg.dL/dpix
    // With q = G dL/dG = o G dL/dalpha and the conic (a, b, c):
    //   dL/d(delta x) = -q (a dx + b dy), dL/d(delta y) = -q (c dy + b dx),
    //   dL/d(conic) = -q (dx^2, dx dy, dy^2) / 2.
    // The sums keep only w, w dx, w dy, w dx^2, ... with w = q / o = G dL/dalpha: the opacity and the
    // conic (constant over the Gaussian's pixels) and the constant factors are applied once per Gaussian
    // by the backward preprocess.
    const float2 w = mul2(G, dLda), wy = mul2(w, dy);
    float(*red)[kRedStride] = sm.red[warp] + kRedRows * nred;
    red[0][lane] = w.x + w.y;
    red[1][lane] = wy.x + wy.y;
    red[2][lane] = fmaf(wy.x, dy.x, wy.y * dy.y);
    red[3][lane] = fmaf(d.x, dp0.x, d.y * dp0.y);
    red[4][lane] = fmaf(d.x, dp1.x, d.y * dp1.y);
    red[5][lane] = fmaf(d.x, dp2.x, d.y * dp2.y);
    if (lane == 0) sm.info[warp][nred] = make_float2(x - patch.wx0, v2.z);
    if (++nred == kRedSplats) {
      flush_reduction(sm, nred, grad_acc);
      nred = 0;
    }
  };
  auto blend_list = [&](int cnt, auto plain) {
    int i = 0;
#pragma unroll 1
    for (; i + 2 <= cnt; i += 2) {
      const uint2 o = *reinterpret_cast<const uint2*>(list + i);
      blend(o.x, plain);
      blend(o.y, plain);
    }
    if (i < cnt) blend(list[i], plain);
  };
  for (int hi = (int)block_last; hi > 0; hi -= kBatch) {
    __syncthreads();
    const int staged = min(kBatch, hi);
    stage_splats<kBatch, kWrap, true, /*kReverse=*/true>(sm.stage, src, job, job.range.x, hi, staged);
    __syncthreads();
    const int first = max(0, hi - (int)warp_last);  // slots before it lie behind every last contributor
#pragma unroll 1
    for (int from = 0; from < staged; from += BlendStage<kBatch>::kListSplats) {
      if (first >= from + BlendStage<kBatch>::kListSplats) continue;
      bool special;
      const int cnt = list_candidates(sm.stage, from, first, staged, special);
      if (special)
        blend_list(cnt, std::false_type{});
      else
        blend_list(cnt, std::true_type{});
    }
  }
  if (nred) flush_reduction(sm, nred, grad_acc);
}

// One view: a block back-propagates one tile (block_tile).
template <int kBatch, bool kRecompute>
__global__ void __launch_bounds__(kBlendThreads, kBlendBwdMinBlocks) render_backward_kernel(RenderParams p) {
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.y * p.gx + blockIdx.x, blockIdx.y << 16 | blockIdx.x);
  const TileJob job = tile_job(p, tile_view(p, tile.z), tile.z, make_uint2(tile.x, tile.y));
  blend_backward_tile<kBatch, false, kRecompute>(job, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P, p.capacity},
                                                 p.grad_acc);
}

// All views of a batch in one launch: a block back-propagates one of the views' tiles.
template <int kBatch, bool kWrap>
__global__ void __launch_bounds__(kBlendThreads, kBlendBwdMinBlocks) batch_render_backward_kernel(const __grid_constant__ BatchRenderParams p) {
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.x, blockIdx.x);
  if (tile.z >= p.total_tiles) return;  // (never, after a binning)
  const TileJob job = tile_job(p, tile_view(p, tile.z), tile.z, make_uint2(tile.x, tile.y));
  blend_backward_tile<kBatch, kWrap, false>(job, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P * (uint32_t)p.V, p.capacity},
                                            p.grad_acc);
}

template <bool kWrap>
void launch_batch_blend(const BatchRenderParams& p, cudaStream_t s) {
  switch (blend_batch_size(true)) {
    case 128: batch_render_backward_kernel<128, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
    case 512: batch_render_backward_kernel<512, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
    default: batch_render_backward_kernel<256, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
  }
}

template <bool kRecompute>
void launch_single_view_backward(const RenderParams& p, const dim3 grid, cudaStream_t s) {
  switch (blend_batch_size(true)) {
    case 128: render_backward_kernel<128, kRecompute><<<grid, kBlendThreads, 0, s>>>(p); break;
    case 512: render_backward_kernel<512, kRecompute><<<grid, kBlendThreads, 0, s>>>(p); break;
    default: render_backward_kernel<256, kRecompute><<<grid, kBlendThreads, 0, s>>>(p); break;
  }
}

}  // namespace

void launch_render_backward(const RenderParams& p, cudaStream_t s) {
  if (p.gx <= 0 || p.gy <= 0) return;
  const dim3 grid(p.gx, p.gy);
  if (p.final_T == nullptr)  // transmittance checkpointing: recompute the per-pixel state
    launch_single_view_backward<true>(p, grid, s);
  else
    launch_single_view_backward<false>(p, grid, s);
}

void launch_batch_render_backward(const BatchRenderParams& p, cudaStream_t s) {
  if (p.total_tiles == 0) return;
  if (p.seam_wrap)
    launch_batch_blend<true>(p, s);
  else
    launch_batch_blend<false>(p, s);
}

}  // namespace omnigs
