// Forward front-to-back alpha blend of one 16x16 tile per block (forward.cu:346-467).
//
// Every pixel evaluates exactly the reference's per-pair arithmetic and control flow (power,
// alpha = min(0.99, o exp(power)), the 1/255 skip, the T < 1e-4 stop), so the image, final
// transmittance and last-contributor index are identical for the same sorted instance list.
// What changes is the work around it:
//  * a thread owns two pixels of one column (rows 4 apart), a warp an 8 x 8 patch; the per-splat
//    shared-memory reads and loop control are paid once per thread, not once per pixel, and the
//    pixels' arithmetic runs in packed f32x2 instructions where that saves any (each lane rounded
//    exactly as the scalar operation, so results are unchanged);
//  * the thread that stages a splat tests whether it can reach alpha >= 1/255 somewhere in each of
//    the block's patches (the exact minimum of the splat's quadratic form over the patch against a
//    threshold computed in the preprocess); a warp iterates only over its patch's list, so pairs that
//    the reference rejects pixel by pixel are skipped a warp at a time;
//  * a warp stops once all of its pixels saturated (a vote every eighth candidate; a saturated pixel's
//    updates are predicated off), and the block stops when every warp has (block vote), as in the
//    reference;
//  * splat geometry and colour are staged together (48 bytes per instance) so the inner loop
//    reads only shared memory.
#include "blend_common.cuh"

namespace omnigs {
namespace {

// Resident blocks per SM (at most 64 registers).  Measured on a B200, seven / eight / nine / ten: 1M-Gaussian 2048x1024
// view 408 / 397 / 412 / 408 us, 16-view batch 5.21 / 5.09 / 5.30 / 5.11 ms, views at the poles 304 / 291 / 294 / 298 us.
// Short lists hide their loads behind other blocks: twelve (40 registers) / ten 12,000 Gaussians at 4096x2048 64 / 70 us.
constexpr int kBlendMinBlocks = 8, kShortMinBlocks = 12;

// Whether lists are short on the average: at most kShortList instances a tile, which the list's capacity bounds, or few
// Gaussians where the capacity is loose.  Measured on a B200, forward blend by lists / with the short kernel: 12,000
// Gaussians at 4096x2048 (9 a tile) 85 / 64 us, 20,000 at 2048x1024 (21) 33 / 30, 4000 in 32 views at 512x256 (20) 62 / 56,
// 40,000 at 2048x1024 (38) 46 / 46, 70,000 at 4096x2048 (47) 178 / 181, 150,000 there (100) 326 / 355.
constexpr int64_t kShortList = 44, kShortRecords = 2;
bool short_lists(int64_t capacity, int64_t records, int64_t tiles) {
  return capacity <= kShortList * tiles || records <= kShortRecords * tiles;
}

// Writes the thread's two pixels; T may be negative (forward_pass).
__device__ __forceinline__ void store_tile(const TileJob& job, const float T[2], const uint32_t lc[2], const float C[2][3]) {
  const BlendPatch patch = BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w);
  const int64_t HW = (int64_t)job.H * job.W;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (!patch.inside(i, job.W, job.H)) continue;
    const int64_t pix = patch.pixel(i, job.W);
    const float t = fabsf(T[i]);
    if (job.final_T != nullptr) {  // stored unless the backward recomputes it
      job.final_T[pix] = t;
      job.n_contrib[pix] = lc[i];
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) job.out_color[ch * HW + pix] = __fmaf_rn(t, job.bg[ch], C[i][ch]);
  }
}

// Blends a block's tile (block_tile).  The job is made again for the stores: its pointers would hold a dozen of the
// loop's registers; its view is kept (looked up again, 32 views of few Gaussians took 5 % longer).
template <int kBatch, bool kWrap, class Params>
__device__ __forceinline__ void blend_forward_tile(const Params& p, uint3 tile, const BlendSource& src) {
  __shared__ __align__(16) BlendStage<kBatch> stage;
  float T[2], C[2][3];
  uint32_t lc[2];
  {
    const uint32_t view = tile_view(p, tile.z);
    const TileJob job = tile_job(p, view, tile.z, make_uint2(tile.x, tile.y));
    if ((threadIdx.x & 31) == 0) stage.tile = tile.z, stage.view = view;  // (as init_stage)
    forward_pass<kBatch, kWrap, true>(job, src, BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w), stage, T, lc, C);
  }
  store_tile(tile_job(p, stage.view, stage.tile, make_uint2(0u, 0u)), T, lc, C);
}

// The same for short lists: a few splats a tile, staged as they are, and every warp tests them itself, so that a block
// has little to do before and after its few candidates and needs few registers.
constexpr int kShortBatch = 128;

template <bool kWrap, class Params>
__device__ __forceinline__ void blend_forward_short(const Params& p, uint3 tile, const BlendSource& src) {
  __shared__ float4 s_splat[kShortBatch][3];
  const uint32_t view = tile_view(p, tile.z);
  const int lane = threadIdx.x & 31;
  float T[2], C[2][3] = {};
  uint32_t lc[2] = {0u, 0u};
  {
    const TileJob job = tile_job(p, view, tile.z, make_uint2(tile.x, tile.y));
    const BlendPatch patch = BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w);
#pragma unroll
    for (int i = 0; i < 2; ++i) T[i] = patch.inside(i, job.W, job.H) ? 1.0f : -1.0f;
    const float pyf[2] = {patch.pyf(0), patch.pyf(1)};
    const uint32_t first = job.range.x, n = job.range.y - job.range.x;
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += kShortBatch) {
      if (base > 0 && __syncthreads_and(T[0] < 0.f && T[1] < 0.f)) break;
      const uint32_t cnt = min((uint32_t)kShortBatch, n - base);
      for (uint32_t t = threadIdx.x; t < cnt; t += kBlendThreads) {
        const uint32_t g = min(src.point_list[first + base + t], src.num_records - 1u);  // (below, for a consistent list)
        s_splat[t][0] = src.splat[2 * (size_t)g];
        s_splat[t][1] = src.splat[2 * (size_t)g + 1];
        s_splat[t][2] = src.color[g];
      }
      __syncthreads();
#pragma unroll 1
      for (uint32_t k = 0; k < cnt; k += 32) {
        unsigned m = __ballot_sync(kFullMask, k + lane < cnt && patch.template hit<kWrap>(s_splat[k + lane][0], s_splat[k + lane][1]));
#pragma unroll 1
        for (; m; m &= m - 1) {
          const uint32_t j = k + (uint32_t)__ffs(m) - 1u;
          const float4 a = s_splat[j][0], b = s_splat[j][1], c = s_splat[j][2];
          // (the arithmetic of forward_pass)
          const float dx = patch.template center_x<kWrap>(a.x) - patch.pxf;
          const float hx = __fmul_rn(-0.5f * a.z, dx), bx = __fmul_rn(-a.w, dx), hc = -0.5f * b.x;
          const float2 dy = make_float2(a.y - pyf[0], a.y - pyf[1]);
          const float2 q2 = mul2(make_float2(__fmul_rn(hc, dy.x), __fmul_rn(hc, dy.y)), dy);
          const float2 power = add2(make_float2(__fmaf_rn(hx, dx, q2.x), __fmaf_rn(hx, dx, q2.y)),
                                    make_float2(__fmul_rn(bx, dy.x), __fmul_rn(bx, dy.y)));
          const float2 alpha = make_float2(fminf(0.99f, __fmul_rn(b.y, expf(power.x))), fminf(0.99f, __fmul_rn(b.y, expf(power.y))));
          const float2 test_T = mul2(make_float2(T[0], T[1]), fma2(alpha, f2(-1.0f), f2(1.0f)));
          const uint32_t at = base + j + 1u;
          forward_pixel<false, true>(alpha.x, power.x, test_T.x, c.x, c.y, c.z, at, T[0], lc[0], C[0][0], C[0][1], C[0][2]);
          forward_pixel<false, true>(alpha.y, power.y, test_T.y, c.x, c.y, c.z, at, T[1], lc[1], C[1][0], C[1][1], C[1][2]);
        }
        if (__all_sync(kFullMask, T[0] < 0.f && T[1] < 0.f)) break;
      }
    }
  }
  store_tile(tile_job(p, view, tile.z, make_uint2(0u, 0u)), T, lc, C);
}

// One view: a block blends one tile (block_tile).
template <int kBatch>
__global__ void __launch_bounds__(kBlendThreads, kBlendMinBlocks) render_forward_kernel(RenderParams p) {
  chain_begin();
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.y * p.gx + blockIdx.x, blockIdx.y << 16 | blockIdx.x);
  blend_forward_tile<kBatch, false>(p, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P, p.capacity});
}

__global__ void __launch_bounds__(kBlendThreads, kShortMinBlocks) render_forward_short_kernel(RenderParams p) {
  chain_begin();
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.y * p.gx + blockIdx.x, blockIdx.y << 16 | blockIdx.x);
  blend_forward_short<false>(p, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P, p.capacity});
}

template <bool kWrap>
__global__ void __launch_bounds__(kBlendThreads, kShortMinBlocks) batch_render_forward_short_kernel(const __grid_constant__ BatchRenderParams p) {
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.x, blockIdx.x);
  if (tile.z >= p.total_tiles) return;  // (never, after a binning)
  blend_forward_short<kWrap>(p, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P * (uint32_t)p.V, p.capacity});
}

// All views of a batch in one launch: a block blends one of the views' tiles.
template <int kBatch, bool kWrap>
__global__ void __launch_bounds__(kBlendThreads, kBlendMinBlocks) batch_render_forward_kernel(const __grid_constant__ BatchRenderParams p) {
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.x, blockIdx.x);
  if (tile.z >= p.total_tiles) return;  // (never, after a binning)
  blend_forward_tile<kBatch, kWrap>(p, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P * (uint32_t)p.V, p.capacity});
}

template <bool kWrap>
void launch_batch_blend(const BatchRenderParams& p, cudaStream_t s) {
  switch (blend_batch_size(false)) {
    case 128: batch_render_forward_kernel<128, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
    case 512: batch_render_forward_kernel<512, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
    default: batch_render_forward_kernel<256, kWrap><<<p.total_tiles, kBlendThreads, 0, s>>>(p); break;
  }
}

}  // namespace

void launch_render_forward(const RenderParams& p, cudaStream_t s) {
  if (p.gx <= 0 || p.gy <= 0) return;
  const dim3 grid(p.gx, p.gy);
  if (short_lists(p.capacity, p.P, (int64_t)p.gx * p.gy)) {
    launch_chained(p.chained, render_forward_short_kernel, grid, kBlendThreads, 0, s, p);
    return;
  }
  switch (blend_batch_size(false)) {
    case 128: launch_chained(p.chained, render_forward_kernel<128>, grid, kBlendThreads, 0, s, p); break;
    case 512: launch_chained(p.chained, render_forward_kernel<512>, grid, kBlendThreads, 0, s, p); break;
    default: launch_chained(p.chained, render_forward_kernel<256>, grid, kBlendThreads, 0, s, p); break;
  }
}

void launch_batch_render_forward(const BatchRenderParams& p, cudaStream_t s) {
  if (p.total_tiles == 0) return;
  if (short_lists(p.capacity, (int64_t)p.P * p.V, p.total_tiles)) {
    if (p.seam_wrap)
      batch_render_forward_short_kernel<true><<<p.total_tiles, kBlendThreads, 0, s>>>(p);
    else
      batch_render_forward_short_kernel<false><<<p.total_tiles, kBlendThreads, 0, s>>>(p);
    return;
  }
  if (p.seam_wrap)
    launch_batch_blend<true>(p, s);
  else
    launch_batch_blend<false>(p, s);
}

}  // namespace omnigs
