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

// Resident blocks per SM, one view / a batch (at most 72 / 64 registers).  Measured on a B200: 1M-Gaussian
// 2048x1024 view, six / seven / eight / ten: 415 / 406 / 415 / 420 us, 3M Gaussians 1006 / 985 / 1001 / 1019;
// 16-view batch 5.44 / 5.35 / 5.16 / 5.25 ms, views at the poles 325 / 314 / 302 / 318 us.
constexpr int kBlendFwdMinBlocks = 7, kBatchFwdMinBlocks = 8;

// Blends the tile that make_job(tile, range) describes.  The job is made again for the stores: its pointers
// would hold a dozen of the loop's registers.
template <int kBatch, bool kWrap, class MakeJob>
__device__ __forceinline__ void blend_forward_tile(const MakeJob& make_job, uint3 tile, const BlendSource& src) {
  __shared__ __align__(16) BlendStage<kBatch> stage;
  float T[2], C[2][3];
  uint32_t lc[2];
  {
    const TileJob job = make_job(tile.z, make_uint2(tile.x, tile.y));
    if (threadIdx.x == 0) stage.tile = tile.z;
    forward_pass<kBatch, kWrap, true>(job, src, BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w), stage, T, lc, C);
  }
  const TileJob job = make_job(stage.tile, make_uint2(0u, 0u));
  const BlendPatch patch = BlendPatch::make(job.tile_x, job.tile_y, job.wrap_w);
  const int64_t HW = (int64_t)job.H * job.W;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (!patch.inside(i, job.W, job.H)) continue;
    const int64_t pix = patch.pixel(i, job.W);
    if (job.final_T != nullptr) {  // stored unless the backward recomputes it
      job.final_T[pix] = T[i];
      job.n_contrib[pix] = lc[i];
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) job.out_color[ch * HW + pix] = __fmaf_rn(T[i], job.bg[ch], C[i][ch]);
  }
}

// One view: a block blends one tile (block_tile).
template <int kBatch>
__global__ void __launch_bounds__(kBlendThreads, kBlendFwdMinBlocks) render_forward_kernel(RenderParams p) {
  chain_begin();
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.y * p.gx + blockIdx.x, blockIdx.y << 16 | blockIdx.x);
  auto make_job = [&](uint32_t t, uint2 range) { return tile_job(p, t, range); };
  blend_forward_tile<kBatch, false>(make_job, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P, p.capacity});
}

// All views of a batch in one launch: a block blends one of the views' tiles.
template <int kBatch, bool kWrap>
__global__ void __launch_bounds__(kBlendThreads, kBatchFwdMinBlocks) batch_render_forward_kernel(const __grid_constant__ BatchRenderParams p) {
  const uint3 tile = block_tile(p.block_tiles, p.ranges, blockIdx.x, blockIdx.x);
  if (tile.z >= p.total_tiles) return;  // (never, after a binning)
  auto make_job = [&](uint32_t t, uint2 range) { return tile_job(p, t, range); };
  blend_forward_tile<kBatch, kWrap>(make_job, tile, BlendSource{p.point_list, p.splat, p.color, (uint32_t)p.P * (uint32_t)p.V, p.capacity});
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
  switch (blend_batch_size(false)) {
    case 128: launch_chained(p.chained, render_forward_kernel<128>, grid, kBlendThreads, 0, s, p); break;
    case 512: launch_chained(p.chained, render_forward_kernel<512>, grid, kBlendThreads, 0, s, p); break;
    default: launch_chained(p.chained, render_forward_kernel<256>, grid, kBlendThreads, 0, s, p); break;
  }
}

void launch_batch_render_forward(const BatchRenderParams& p, cudaStream_t s) {
  if (p.total_tiles == 0) return;
  if (p.seam_wrap)
    launch_batch_blend<true>(p, s);
  else
    launch_batch_blend<false>(p, s);
}

}  // namespace omnigs
