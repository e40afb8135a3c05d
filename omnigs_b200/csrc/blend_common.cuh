// Shared pieces of the forward and backward tile blends: the pixel patch a warp owns, the
// alpha-support test of a splat against it, and the staging of a batch of splats into shared memory.
#pragma once

#include <type_traits>

#include "device_util.cuh"
#include "kernels.h"

namespace omnigs {

// Pixels per thread: a thread owns kBlendPx pixels of one column, 4 rows apart, so a warp (8
// columns x 4 rows of threads) owns an 8 x (4 kBlendPx) patch and a block of kBlendThreads
// threads one 16x16 tile.
#ifndef OMNIGS_BLEND_PX
#define OMNIGS_BLEND_PX 2
#endif
constexpr int kBlendPx = OMNIGS_BLEND_PX;
static_assert(kBlendPx == 1 || kBlendPx == 2 || kBlendPx == 4, "a 16x16 tile splits into 8/kBlendPx warps");
constexpr int kBlendThreads = 256 / kBlendPx;
constexpr int kBlendWarps = kBlendThreads / 32;

// One 16x16 tile of one view, as a blend block sees it.  The per-pixel pointers are the view's.
struct TileJob {
  int tile_x, tile_y;
  int W, H;
  uint2 range;              // [begin, end) of the tile's instances in the sorted list
  const float* bg;          // [3]
  float* out_color;         // [3,H,W]
  float* final_T;           // [H*W]
  uint32_t* n_contrib;      // [H*W]
  const float* dL_dpix;     // [3,H,W] (backward)
  float wrap_w;             // image width when blending across the longitude seam, else 0
};

// The range and tile (TileListParams::block_tiles) that a block blends.  A list that gives both costs a block
// no more dependent loads than its range alone.
__device__ __forceinline__ uint3 block_tile(const uint4* block_tiles, const uint2* ranges, uint32_t block, uint32_t own) {
  if (block_tiles != nullptr) {
    const uint4 w = block_tiles[block];
    return make_uint3(w.x, w.y, w.z);
  }
  const uint2 r = ranges[block];
  return make_uint3(r.x, r.y, own);
}

// The sorted instance list and the per-record splat data it points into.
struct BlendSource {
  const uint32_t* point_list;  // record index per instance
  const float4* splat;         // [records][2]
  const float4* color;         // [records]
  uint32_t num_records;
  int64_t capacity;            // instances the list can hold; larger range bounds are rejected
};

// A tile's range, emptied if inconsistent with the list's capacity.
__device__ __forceinline__ uint2 checked_range(uint2 range, int64_t capacity) {
  if (range.y > (uint64_t)capacity || range.x > range.y) range = make_uint2(0, 0);
  return range;
}

// Rows of the patch a warp owns (8 columns wide).
constexpr int kPatchRows = 4 * kBlendPx;

struct BlendPatch {
  int px, py0;       // this thread's column and first row
  float pxf;         // column as float
  float wx0, wy0;    // first column and row of the warp's patch
  float wcx;         // centre column of the warp's patch
  float wrap_w;      // image width in seam-wrapping mode, else 0

  // x of the splat's copy (shifted by a multiple of the image width) nearest this patch; the
  // splat's own x unless the seam wraps (kWrap, a template flag so that the non-wrapping kernels
  // carry no trace of it).
  template <bool kWrap>
  __device__ __forceinline__ float center_x(float ax) const {
    return kWrap ? ax - wrap_w * rintf((ax - wcx) / wrap_w) : ax;
  }

  // The bounds of a warp's patch in the tile whose first pixel is `origin`.
  static __device__ __forceinline__ BlendPatch bounds(float2 origin, int warp, float wrap_w) {
    BlendPatch b{};
    b.wx0 = origin.x + (float)((warp & 1) * 8);
    b.wy0 = origin.y + (float)((warp >> 1) * kPatchRows);
    b.wcx = b.wx0 + 3.5f;
    b.wrap_w = wrap_w;
    return b;
  }
  static __device__ __forceinline__ BlendPatch make(int tile_x, int tile_y, float wrap_w = 0.f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wx0 = tile_x * 16 + (warp & 1) * 8;
    const int wy0 = tile_y * 16 + (warp >> 1) * kPatchRows;
    BlendPatch b;
    b.px = wx0 + (lane & 7);
    b.py0 = wy0 + (lane >> 3);
    b.pxf = (float)b.px;
    b.wx0 = (float)wx0;
    b.wy0 = (float)wy0;
    b.wcx = (float)wx0 + 3.5f;
    b.wrap_w = wrap_w;
    return b;
  }
  __device__ __forceinline__ int py(int i) const { return py0 + 4 * i; }
  __device__ __forceinline__ float pyf(int i) const { return (float)(py0 + 4 * i); }
  __device__ __forceinline__ bool inside(int i, int W, int H) const { return px < W && py(i) < H; }
  __device__ __forceinline__ int64_t pixel(int i, int W) const { return (int64_t)py(i) * W + px; }

  // Whether the splat (a = {x, y, conic a, conic b}, b = {conic c, opacity, thr, det}) can reach
  // alpha >= 1/255 at some pixel centre of the patch: the minimum of its quadratic form
  // q(d) = a dx^2 + 2 b dx dy + c dy^2 over the patch's offsets d = centre - pixel, a rectangle
  // [dxl, dxh] x [dyl, dyh], against thr.  A convex form's minimum over a rectangle that does not
  // contain its centre lies on a side facing the centre (KKT), so two candidate sides suffice: the
  // column side at dxn (the x offset nearest 0) minimised over dy, and the row side at dyn minimised
  // over dx.  Scaled by c (resp. a) each is a clamp and a sum of squares without division:
  //   c q(dxn, dy) = (c dy + b dxn)^2 + det dxn^2, minimised at c dy = clamp(-b dxn, c dyl, c dyh).
  // When the centre lies inside the patch both offsets are 0 and the value is 0.  Any other side
  // value is q at a point of the patch, so it never claims a miss wrongly.  Written as a negated
  // "misses" test so that NaN (det of a non-positive-definite conic, non-finite inputs) hits: the
  // per-pixel test decides.
  template <bool kWrap>
  __device__ __forceinline__ bool hit(const float4& a, const float4& b) const {
    const float dxh = center_x<kWrap>(a.x) - wx0, dxl = dxh - 7.0f;
    const float dyh = a.y - wy0, dyl = dyh - (float)(kPatchRows - 1);
    const float dxn = fminf(fmaxf(dxl, 0.0f), dxh), dyn = fminf(fmaxf(dyl, 0.0f), dyh);
    const float bx = a.w * dxn, by = a.w * dyn;
    const float sx = fminf(fmaxf(-bx, b.x * dyl), b.x * dyh) + bx;
    const float sy = fminf(fmaxf(-by, a.z * dxl), a.z * dxh) + by;
    const float vx = fmaf(sx, sx, b.w * dxn * dxn);
    const float vy = fmaf(sy, sy, b.w * dyn * dyn);
    return !(vx > b.x * b.z && vy > a.z * b.z);
  }
};

// Packed f32x2 arithmetic (one instruction for both lanes, each rounded as its scalar form).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Whether the blends can leave the positive-exponent test and the 0.99 clamp out for this splat
// (a = {x, y, conic a, conic b}, b = {conic c, opacity, thr, det}):
//  * power <= 0 at every offset: with S = a dx^2 + c dy^2 the cross term is at most
//    sqrt(1 - det / (a c)) S / 2 in size, and the float evaluation of power is off by less than
//    6 * 2^-24 S / 2, so det > 1e-5 a c keeps it negative (a NaN or non-positive-definite conic,
//    det = NaN, fails the test);
//  * opacity times an exponential of a non-positive number stays below the clamp;
//  * with the conic below 1e9 nothing overflows, so alpha is a finite number.
__device__ __forceinline__ bool plain_splat(const float4& a, const float4& b) {
  return b.y < 0.98999f && b.w > 1e-5f * a.z * b.x && a.z + b.x < 1e9f;
}

// A batch of staged splats, as the blends' inner loops read it.  The loops are bound by instruction
// issue, so the staging thread does once per splat what every warp or candidate would repeat:
//  * it tests its splat against the block's four patches (from registers; a ballot per patch), and
//    every warp turns its masks into a list of its candidates' offsets, so the loop over them has no
//    bit scanning or address arithmetic;
//  * a slot (48 bytes) holds {x, y, -a/2, -b}{-c/2, o, r, g}{b, 1 + position, record, -}.
// The exponent at offset d = centre - pixel (forward.cu:416, backward.cu:763) is
//   power = -0.5 (a dx^2 + c dy^2) - b dx dy,
// whose rounding the reference leaves to the compiler's FMA contraction.  Both blends write it with
// explicit roundings in the one fusion that reproduces the reference's compiled results bit for bit
// (checked on the 1M-Gaussian 2048x1024 scene: identical transmittance, last contributors and image):
// a dx dx fused into the sum with the rounded c dy dy, the b dx dy term rounded on its own.  The slot's
// factors -1/2 and signs are exact, so applying them before the roundings changes nothing.  Forward and
// backward agree on every 1/255 and saturation decision.
constexpr uint32_t kSlotBytes = 48;

template <int kBatch>
struct BlendStage {
  static constexpr int kListSplats = kBatch < 256 ? kBatch : 256;
  float4 d[kBatch][kSlotBytes / 16];
  uint32_t list[kBlendWarps][kListSplats];      // byte offsets of a warp's candidates
  uint32_t mask[kBatch / 32][kBlendWarps];      // candidates of a group of 32 by warp
  uint32_t special[kBatch / 32];                // the group's splats that are not plain (plain_splat)
  float2 origin;                                // the tile's first pixel
  uint32_t first;                               // its range's begin
  uint32_t tile, view;                          // block_tile's and its view (the forward's; these four are here
                                                // because registers are scarce: 1-3 % of the blends)
};

// Every warp writes what it reads (the same values), so no barrier is needed.
template <int kBatch>
__device__ __forceinline__ void init_stage(BlendStage<kBatch>& st, const TileJob& job) {
  if ((threadIdx.x & 31) == 0) {
    st.origin = make_float2((float)(job.tile_x * 16), (float)(job.tile_y * 16));
    st.first = job.range.x;
  }
  __syncwarp();
}

// Stages instances [base, base + cnt) of the tile's list, which begins at `first` (from the back when kReverse: slot t holds
// position base - 1 - t, with base the exclusive upper end) with their patch masks; the colour only
// with kColor.
template <int kBatch, bool kWrap, bool kColor, bool kReverse>
__device__ __forceinline__ void stage_splats(BlendStage<kBatch>& st, const BlendSource& src, const TileJob& job,
                                             uint32_t first, int base, int cnt) {
  const int lane = threadIdx.x & 31;
  const float2 origin = st.origin;
#pragma unroll 1
  for (int t = threadIdx.x; t - lane < cnt; t += kBlendThreads) {  // (whole groups of 32)
    bool hits[kBlendWarps] = {}, special = false;
    if (t < cnt) {
      const uint32_t pos = kReverse ? (uint32_t)(base - 1 - t) : (uint32_t)(base + t);
      const uint32_t g = src.point_list[first + pos];
      if (g < src.num_records) {  // (always, for a consistent instance list)
        const float4 a = src.splat[2 * (size_t)g], b = src.splat[2 * (size_t)g + 1];
        const float4 c = kColor ? src.color[g] : make_float4(0.f, 0.f, 0.f, 0.f);
        st.d[t][0] = make_float4(a.x, a.y, -0.5f * a.z, -a.w);
        st.d[t][1] = make_float4(-0.5f * b.x, b.y, c.x, c.y);
        st.d[t][2] = make_float4(c.z, __uint_as_float(pos + 1u), __uint_as_float(g), 0.f);
        special = !plain_splat(a, b);
#pragma unroll
        for (int w = 0; w < kBlendWarps; ++w)
          hits[w] = BlendPatch::bounds(origin, w, job.wrap_w).template hit<kWrap>(a, b);
      }
    }
    const unsigned ms = __ballot_sync(kFullMask, special);
    if (lane == 0) st.special[t >> 5] = ms;
#pragma unroll
    for (int w = 0; w < kBlendWarps; ++w) {
      const unsigned m = __ballot_sync(kFullMask, hits[w]);
      if (lane == 0) st.mask[t >> 5][w] = m;
    }
  }
}

// The warp's candidates among slots [max(from, first), min(from + kListSplats, cnt)) of the staged batch of cnt, in slot
// order: writes their offsets to its list, returns their number and whether any is special.  (Short lists are a large
// part of the blends' time in sparse views, so groups past cnt are not looked at, and nothing is padded.)
template <int kBatch>
__device__ __forceinline__ int list_candidates(BlendStage<kBatch>& st, int from, int first, int cnt, bool& special) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* list = st.list[warp];
  const unsigned lt = (1u << lane) - 1u;
  int n = 0;
  unsigned sp = 0;
  __syncwarp();  // the warp has read its previous list
  auto group = [&](int k) {
    unsigned m = st.mask[k][warp];
    if (first > k * 32) m = first - k * 32 >= 32 ? 0u : m & (kFullMask << (first - k * 32));
    sp |= m & st.special[k];
    if ((m >> lane) & 1u) list[n + __popc(m & lt)] = (uint32_t)(k * 32 + lane) * kSlotBytes;
    n += __popc(m);
  };
  constexpr int kGroups = BlendStage<kBatch>::kListSplats / 32;
  if (cnt > from + (kGroups - 1) * 32) {
#pragma unroll
    for (int i = 0; i < kGroups; ++i) group(from / 32 + i);
  } else {
#pragma unroll 1
    for (int k = from / 32; k * 32 < cnt; ++k) group(k);
  }
  __syncwarp();
  special = sp != 0;
  return n;
}

// One splat at one pixel of the forward's pass: alpha is the splat's, test_T = T (1 - alpha) with T
// the pixel's transmittance, negated once the pixel has stopped.  Where the splat reaches the pixel
// (alpha >= 1/255, and the exponent is not positive) and test_T stays at or above 1e-4, the colour
// c alpha T is added (rounded as the reference's compiled blend: fused add), T becomes test_T and lc
// the splat's position; where test_T falls below (always so for a stopped pixel, whose T is negative)
// the pixel stops, T = -|T|.  One comparison gives both outcomes (setp's two predicates), and
// everything else is predicated: no branches, no selects.
template <bool kPlain, bool kColor>
__device__ __forceinline__ void forward_pixel(float alpha, float power, float test_T, float r, float g, float b,
                                              uint32_t at, float& T, uint32_t& lc, float& C0, float& C1, float& C2) {
// operands: %0 T, %1 lc, %2-%4 C, %5 alpha, %6 test_T, %7 position, %8 power, %9-%11 colour
#define OMNIGS_PIXEL_TEST                                                                       \
  "setp.geu.f32 p, %5, 0f3B808081;\n\t" /* !(alpha < 1/255) */
#define OMNIGS_PIXEL_TEST_ANY                                                                   \
  "setp.leu.and.f32 p, %8, 0f00000000, p;\n\t" /* !(power > 0) */                               \
  "setp.geu.and.f32 p, %0, 0f00000000, p;\n\t" /* a NaN alpha revives no stopped pixel */
#define OMNIGS_PIXEL_STATE                                                                      \
  "setp.lt.and.f32 stop|act, %6, 0f38D1B717, p;\n\t" /* test_T < 1e-4, or not */
#define OMNIGS_PIXEL_COLOR                                                                      \
  "mul.rn.f32 c0, %9, %5;\n\tmul.rn.f32 c1, %10, %5;\n\tmul.rn.f32 c2, %11, %5;\n\t"          \
  "@act fma.rn.f32 %2, c0, %0, %2;\n\t@act fma.rn.f32 %3, c1, %0, %3;\n\t@act fma.rn.f32 %4, c2, %0, %4;\n\t"
#define OMNIGS_PIXEL_UPDATE                                                                     \
  "@act mov.f32 %0, %6;\n\t@stop or.b32 %0, %0, 0x80000000;\n\t@act mov.b32 %1, %7;\n\t"
#define OMNIGS_PIXEL(body)                                                                      \
  asm("{\n\t.reg .pred p, act, stop;\n\t.reg .f32 c0, c1, c2;\n\t" body "}"                   \
      : "+f"(T), "+r"(lc), "+f"(C0), "+f"(C1), "+f"(C2)                                          \
      : "f"(alpha), "f"(test_T), "r"(at), "f"(power), "f"(r), "f"(g), "f"(b))
  if (kPlain && kColor)
    OMNIGS_PIXEL(OMNIGS_PIXEL_TEST OMNIGS_PIXEL_STATE OMNIGS_PIXEL_COLOR OMNIGS_PIXEL_UPDATE);
  else if (kPlain)
    OMNIGS_PIXEL(OMNIGS_PIXEL_TEST OMNIGS_PIXEL_STATE OMNIGS_PIXEL_UPDATE);
  else if (kColor)
    OMNIGS_PIXEL(OMNIGS_PIXEL_TEST OMNIGS_PIXEL_TEST_ANY OMNIGS_PIXEL_STATE OMNIGS_PIXEL_COLOR OMNIGS_PIXEL_UPDATE);
  else
    OMNIGS_PIXEL(OMNIGS_PIXEL_TEST OMNIGS_PIXEL_TEST_ANY OMNIGS_PIXEL_STATE OMNIGS_PIXEL_UPDATE);
#undef OMNIGS_PIXEL_TEST
#undef OMNIGS_PIXEL_TEST_ANY
#undef OMNIGS_PIXEL_STATE
#undef OMNIGS_PIXEL_COLOR
#undef OMNIGS_PIXEL_UPDATE
#undef OMNIGS_PIXEL
}

// The forward's front-to-back pass over a tile's instances (forward.cu:394-456) for the thread's two
// pixels (rows py0 and py0 + 4): transmittance T and last contributor lc, and with kColor the blended
// colour C.  Every pixel evaluates the reference's per-pair arithmetic and control flow (power,
// alpha = min(0.99, o exp(power)), the 1/255 skip, the T < 1e-4 stop), so T and lc are the same whether
// or not colour is blended: the forward kernel runs it with colour, the backward runs it without to
// recompute the state it did not store.
//
// The loop over a warp's candidates has two bodies: where all of them are plain (plain_splat) the
// exponent's sign test and the clamp are left out.  The two pixels' arithmetic is packed (f32x2, one
// issue slot) where both factors differ by pixel, and scalar where one is the splat's: broadcasting that
// into a register pair costs the moves that packing saves.  Bound by instruction issue.  Measured on a
// B200 (1M-Gaussian 2048x1024 view / 16-view batch) against a warp testing every staged splat itself and
// walking the ballots' bits: 424 -> 397 us / 5.20 -> 5.02 ms (short lists aside: blend_forward_short).
template <int kBatch, bool kWrap, bool kColor>
__device__ __forceinline__ void forward_pass(const TileJob& job, const BlendSource& src, const BlendPatch& patch,
                                             BlendStage<kBatch>& st, float T[2], uint32_t lc[2], float C[2][3]) {
  static_assert(kBlendPx == 2, "a thread owns two pixels of one column");
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    T[i] = patch.inside(i, job.W, job.H) ? 1.0f : -1.0f;  // a pixel outside the image starts stopped
    lc[i] = 0;
    C[i][0] = C[i][1] = C[i][2] = 0.f;
  }
  const float pyf[2] = {patch.pyf(0), patch.pyf(1)};
  const int n = (int)(job.range.y - job.range.x);
  const char* slots = reinterpret_cast<const char*>(&st.d[0][0]);
  const uint32_t* list = st.list[threadIdx.x >> 5];
  init_stage(st, job);

  auto blend = [&](uint32_t off, auto plain) {
    constexpr bool kPlain = decltype(plain)::value;
    const float4* slot = reinterpret_cast<const float4*>(slots + off);
    const float4 v0 = slot[0], v1 = slot[1];
    const float2 v2 = *reinterpret_cast<const float2*>(slot + 2);
    const float dx = (kWrap ? patch.template center_x<true>(v0.x) : v0.x) - patch.pxf;
    const float hx = __fmul_rn(v0.z, dx), bx = __fmul_rn(v0.w, dx);
    const float2 dy = make_float2(v0.y - pyf[0], v0.y - pyf[1]);
    const float2 q2 = mul2(make_float2(__fmul_rn(v1.x, dy.x), __fmul_rn(v1.x, dy.y)), dy);
    const float2 power = add2(make_float2(__fmaf_rn(hx, dx, q2.x), __fmaf_rn(hx, dx, q2.y)),
                              make_float2(__fmul_rn(bx, dy.x), __fmul_rn(bx, dy.y)));
    float2 alpha = make_float2(__fmul_rn(v1.y, expf(power.x)), __fmul_rn(v1.y, expf(power.y)));
    if (!kPlain) alpha = make_float2(fminf(0.99f, alpha.x), fminf(0.99f, alpha.y));
    const float2 test_T = mul2(make_float2(T[0], T[1]), fma2(alpha, f2(-1.0f), f2(1.0f)));
    const uint32_t at = __float_as_uint(v2.y);
    forward_pixel<kPlain, kColor>(alpha.x, power.x, test_T.x, v1.z, v1.w, v2.x, at, T[0], lc[0], C[0][0], C[0][1], C[0][2]);
    forward_pixel<kPlain, kColor>(alpha.y, power.y, test_T.y, v1.z, v1.w, v2.x, at, T[1], lc[1], C[1][0], C[1][1], C[1][2]);
  };
  auto blend_list = [&](int cnt, auto plain) {
    int i = 0;
#pragma unroll 1
    for (; i + 4 <= cnt; i += 4) {
      const uint4 o = *reinterpret_cast<const uint4*>(list + i);
      blend(o.x, plain);
      blend(o.y, plain);
      blend(o.z, plain);
      blend(o.w, plain);
      if ((i & 4) && __all_sync(kFullMask, T[0] < 0.f && T[1] < 0.f)) return;
    }
#pragma unroll 1
    for (; i < cnt; ++i) blend(list[i], plain);
  };
  for (int base = 0; base < n; base += kBatch) {
    if (base > 0 && __syncthreads_and(T[0] < 0.f && T[1] < 0.f)) break;
    const int staged = min(kBatch, n - base);
    stage_splats<kBatch, kWrap, kColor, /*kReverse=*/false>(st, src, job, st.first, base, staged);
    __syncthreads();
#pragma unroll 1
    for (int from = 0; from < staged; from += BlendStage<kBatch>::kListSplats) {
      if (__all_sync(kFullMask, T[0] < 0.f && T[1] < 0.f)) break;
      bool special;
      const int cnt = list_candidates(st, from, 0, staged, special);
      if (special)
        blend_list(cnt, std::false_type{});
      else
        blend_list(cnt, std::true_type{});
    }
  }
  T[0] = fabsf(T[0]);
  T[1] = fabsf(T[1]);
}

// The view of a block's tile, and that tile: of one view, whose tiles are y << 16 | x.
__device__ __forceinline__ uint32_t tile_view(const RenderParams&, uint32_t) { return 0u; }
__device__ __forceinline__ TileJob tile_job(const RenderParams& p, uint32_t, uint32_t tile, uint2 range) {
  TileJob job;
  job.tile_x = (int)(tile & 0xffffu);
  job.tile_y = (int)(tile >> 16);
  job.W = p.W;
  job.H = p.H;
  job.range = checked_range(range, p.capacity);
  job.bg = p.bg;
  job.out_color = p.out_color;
  job.final_T = p.final_T;
  job.n_contrib = p.n_contrib;
  job.dL_dpix = p.dL_dpix;
  job.wrap_w = 0.f;
  return job;
}

// Of a batch, whose tiles are numbered over the views in the order of tile_base (the host lays the views out
// heaviest tiles first).
__device__ __forceinline__ uint32_t tile_view(const BatchRenderParams& p, uint32_t block) {
  // the largest first tile not beyond the block, a lane per view (one by one, 32 views took a tenth of the
  // forward blend of few Gaussians)
  static_assert(kMaxBatchViews == 32, "a lane per view");
  const int lane = threadIdx.x & 31;
  uint32_t base = lane < p.V ? p.views[lane].tile_base : 0xffffffffu;
  base = base <= block ? base + 1u : 0u;
  return (uint32_t)__ffs(__ballot_sync(kFullMask, base == __reduce_max_sync(kFullMask, base))) - 1u;
}
__device__ __forceinline__ TileJob tile_job(const BatchRenderParams& p, uint32_t v, uint32_t block, uint2 range) {
  const BatchView& bv = p.views[v];
  const uint32_t local = block - bv.tile_base;
  TileJob job;
  job.tile_y = (int)(local / (uint32_t)bv.gx);
  job.tile_x = (int)(local - (uint32_t)job.tile_y * (uint32_t)bv.gx);
  job.W = bv.W;
  job.H = bv.H;
  job.range = checked_range(range, p.capacity);
  job.bg = p.backgrounds + 3 * v;
  job.out_color = bv.out_color;
  job.final_T = p.final_T + bv.pixel_base;
  job.n_contrib = p.n_contrib + bv.pixel_base;
  job.dL_dpix = bv.dL_dpix;
  job.wrap_w = p.seam_wrap ? (float)bv.W : 0.f;
  return job;
}

}  // namespace omnigs
