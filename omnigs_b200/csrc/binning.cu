// Binning: the reference's sorted instance list and tile ranges (rasterizer_impl.cu:94-167,
// 622-679) from a depth sort of the Gaussians, a coarse list per bin of 8x4 tiles and, out of it, a
// compaction per tile.
//
// The reference emits one (tile << 32 | depth_bits) key per (Gaussian, tile) pair in Gaussian
// order and sorts them with a stable LSD radix sort over bits [0, 32 + getHigherMsb(tiles)).  The
// result is fully determined: instances ordered by tile, then by depth bits, then -- a Gaussian
// appears at most once per tile and the list starts in Gaussian order -- by Gaussian index.  The
// same order is produced here without sorting the instances at all:
//  1. depth sort: a stable LSD radix sort (4 onesweep passes of 8 bits) of the P Gaussians by the
//     bits of their depth, i.e. the order (depth bits, index);
//  2. coarse lists: a scan of the Gaussians' bin counts in that order (decoupled look-back), a
//     load-balanced emission of the (bin, depth-order position) pairs in that order, and a stable
//     LSD radix sort of the pairs by bin (one onesweep pass up to 256 bins): every bin's Gaussians
//     in depth order.  A splat covers far fewer bins than tiles;
//  3. tile lists: warps count the tiles' instances of a piece of the sorted pairs each (the pairs' tiles are
//     bit masks), a scan of the counts in tile order gives the ranges, and the warps append their pieces
//     to the tiles' lists, in order.
// Few Gaussians (counts_order) are ordered by counting, which costs less than the five launches of the
// depth sort: a Gaussian's position is the number of smaller depths.  Where Gaussians times bins are
// few (kWholeMaxPairs) there are no coarse lists: every bin reads its view's whole order.
// Counts live on the device: every kernel reads num_rendered from the geometry header and does no
// work if it exceeds the binning capacity.  Waits on other blocks are bounded.
//
// Measured on a B200 against emitting every instance and sorting the list by tile id in two or three
// passes, all stages of the binning: 1M Gaussians at 2048x1024 (8.6M instances) 353 -> 238 us, 3M at
// 4096x2048 (72M) 1895 -> 813 us, 16 views over 1M Gaussians (112M) 3.49 -> 2.14 ms, 10,000 at 512x256
// 115 -> 49 us.  The sort passes over the instances were what it cost (80 us each over 8.2M), and the
// pairs are a fifth of them.
#include <algorithm>

#include "device_util.cuh"
#include "kernels.h"
#include "lonlat_math.cuh"

namespace omnigs {
namespace {

constexpr uint32_t kLbAggregate = 1u << 30;
constexpr uint32_t kLbPrefix = 2u << 30;
constexpr uint32_t kLbValue = (1u << 30) - 1;
constexpr unsigned long long kScanAggregate = 1ull << 62;
constexpr unsigned long long kScanPrefix = 2ull << 62;
constexpr unsigned long long kScanValue = (1ull << 62) - 1;
// Predecessors a look-back reads per round.  Measured on a B200, the sorts of a 1M-Gaussian view /
// 16-view batch: 4 / 8 / 16 / 32 a round 118 / 118 / 128 / 136 and 1106 / 1123 / 1296 / 1276 us, so the walk
// is not bound by its round trips.  Nor is the pass bound by its look-back: a
// reduce-then-scan in its place (a kernel counting every tile's digits and scanning the counts
// over the tiles, then the pass without waits) made the sort slower, 0.294 -> 0.366 ms per view:
// the count kernels took 12-27 us each and the passes got only 4-10 us faster.
constexpr int kLookbackBatch = 4;

__device__ __forceinline__ bool instances_fit(const GeomHeader* hdr, int64_t capacity) {
  return (hdr->status & kStatusOverflow) == 0 && hdr->num_rendered64 <= (unsigned long long)capacity;
}

// Number of (Gaussian, bin) pairs, at most one per instance (0 if the instances do not fit the
// capacity, which the scan has flagged).
__device__ __forceinline__ uint32_t pair_count(const GeomHeader* hdr, int64_t capacity) {
  return instances_fit(hdr, capacity) ? (uint32_t)min((long long)hdr->num_pairs, (long long)capacity) : 0u;
}

// ---------------------------------------------------------------- digit histograms ------------
// Adds the warp's digits (lanes in `live`, a prefix of the warp) to a shared histogram.  Keys of a
// sort are either spread over many digits (per-lane atomics rarely collide) or nearly constant
// within a warp (the top digit of depth bits): when every live lane holds lane 0's digit, lane 0
// adds the whole count with one atomic.
__device__ __forceinline__ void count_digit(uint32_t* hist, uint32_t digit, bool valid, unsigned live, int lane) {
  const uint32_t d0 = __shfl_sync(kFullMask, digit, 0);
  if (__all_sync(kFullMask, !valid || digit == d0)) {
    if (lane == 0 && live) atomicAdd(&hist[d0], (uint32_t)__popc(live));
  } else if (valid) {
    atomicAdd(&hist[digit], 1u);
  }
}

constexpr int kHistUnroll = 4;  // keys per thread loaded before any of them is counted

__global__ void __launch_bounds__(256) histogram_kernel(const __grid_constant__ HistParams p) {
  chain_begin();
  __shared__ uint32_t s_hist[kDepthPasses][kRadix];
  for (int i = threadIdx.x; i < kDepthPasses * kRadix; i += blockDim.x) (&s_hist[0][0])[i] = 0;
  __syncthreads();
  const uint32_t n = p.seg_len;
  const size_t seg_base = (size_t)blockIdx.y * n;  // gridDim.y segments
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  // Whole warps iterate together (the counting votes over the warp); each thread first loads
  // kHistUnroll keys (independent loads in flight), then counts them.
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride * kHistUnroll) {
    uint32_t key[kHistUnroll];
    bool valid[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u) {
      const uint32_t i = base + u * stride + lane;
      valid[u] = i < n;
      key[u] = valid[u] ? p.keys[seg_base + i] : 0u;
    }
    unsigned live[kHistUnroll];
#pragma unroll
    for (int u = 0; u < kHistUnroll; ++u) live[u] = __ballot_sync(kFullMask, valid[u]);
#pragma unroll
    for (int q = 0; q < kDepthPasses; ++q) {
      if (q >= p.passes) break;
#pragma unroll
      for (int u = 0; u < kHistUnroll; ++u)
        count_digit(s_hist[q], (key[u] >> p.shift[q]) & p.mask[q], valid[u], live[u], lane);
    }
  }
  __syncthreads();
  uint32_t* hist = p.hist + (size_t)blockIdx.y * p.passes * kRadix;
  for (int i = threadIdx.x; i < p.passes * kRadix; i += blockDim.x) {
    const uint32_t v = (&s_hist[0][0])[i];
    if (v) atomicAdd(&hist[i], v);
  }
}

// ---------------------------------------------------------------- onesweep pass ---------------
template <int kTile>
struct SortSmem {
  uint32_t warp_hist[kSortThreads / 32][kRadix];
  uint32_t block_excl[kRadix];
  uint32_t global_base[kRadix];
  uint32_t scan_tmp[kSortThreads / 32];
  uint32_t tile;
  uint32_t pad[3];
  uint32_t keys[kTile];
  uint32_t vals[kTile];
};

// Exclusive scan of one value per thread across the block (kSortThreads == kRadix == 256).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* scan_tmp, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(kFullMask, x, o);
    if (lane >= o) x += n;
  }
  if (lane == 31) scan_tmp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = (lane < kSortThreads / 32) ? scan_tmp[lane] : 0u;
#pragma unroll
    for (int o = 1; o < kSortThreads / 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(kFullMask, w, o);
      if (lane >= o) w += n;
    }
    if (lane < kSortThreads / 32) scan_tmp[lane] = w;
  }
  __syncthreads();
  total = scan_tmp[kSortThreads / 32 - 1];
  const uint32_t r = x - v + (warp > 0 ? scan_tmp[warp - 1] : 0u);
  __syncthreads();
  return r;
}

// One stable LSD pass over (u32 key, u32 value) pairs on the digit (key >> shift) & mask.  A block
// ranks a 4096-item tile in shared memory (warp multi-split from per-bit ballots: equal digits keep
// their input order), publishes its per-digit counts, resolves its global digit offsets by
// decoupled look-back (tiles are taken in launch order from an atomic counter, so a block only
// waits on blocks that are already running) and writes runs of equal digits coalesced.  In a
// segmented sort every segment is an independent sort whose look-back chain starts at the
// segment's first tile; a value-less first pass numbers items by their global index.
// Bound by a tile's own work: ranking, scans, scatter.  The tile is reordered before the look-back and its
// values are loaded after the ranking, so that registers hold 24 words of a thread's 16 items at a time, not
// 48.  Measured on a B200, the sorts of a 1M / 3M-Gaussian view / 16-view batch: 125 / 447 / 1202 us with
// everything held to the end, 117 / 382 / 1020 now.
// Launches of this pass measured ~2 us slower each on a B200 with a 136-byte parameter block than
// with a 128-byte one.
static_assert(sizeof(OnesweepParams) <= 128, "keep the onesweep parameter block at 128 bytes or less");

// Tiles of kSortTile keys, 16 per thread.  Measured on a B200: 1024-key tiles (4 per thread, five
// blocks per SM) made the depth passes over 1M Gaussians slower, 22 -> 30 us each (4x the blocks,
// look-back chains and per-tile scans), so passes over many keys use the 4096-key tiles; passes that
// 1024-key tiles spread over at most kSmallSortTiles blocks are bound by a tile's own latency and use
// those: 282 -> 276 us for the whole forward of 150,000 Gaussians (147 tiles), nothing at 300,000 (293).
template <int kItems, int kMinBlocks, int kLookback>
__global__ void __launch_bounds__(kSortThreads, kMinBlocks) onesweep_kernel(OnesweepParams p) {
  chain_begin();
  constexpr int kTile = kSortThreads * kItems;
  __shared__ SortSmem<kTile> sm;
  const uint32_t n = p.seg_len ? p.seg_len : pair_count(p.hdr, p.capacity);
  const uint32_t tiles_per_seg = (n + kTile - 1) / kTile;
  const uint32_t ntiles = tiles_per_seg * (p.seg_len ? p.num_segs : 1u);
  if (threadIdx.x == 0) sm.tile = atomicAdd(p.tile_counter, 1u);
  for (int i = threadIdx.x; i < (kSortThreads / 32) * kRadix; i += kSortThreads) (&sm.warp_hist[0][0])[i] = 0;
  __syncthreads();
  const uint32_t ticket = sm.tile;
  if (ticket >= ntiles) return;
  const uint32_t seg = ticket / tiles_per_seg;
  const uint32_t tile = ticket - seg * tiles_per_seg;  // tile index within the segment
  const size_t seg_base = (size_t)seg * n;
  const uint32_t* keys_in = p.keys_in + seg_base;
  const uint32_t* vals_in = p.vals_in ? p.vals_in + seg_base : nullptr;
  uint32_t* keys_out = p.keys_out + seg_base;
  uint32_t* vals_out = p.vals_out + seg_base;
  const uint32_t* hist = p.hist + (size_t)seg * p.hist_seg_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const uint32_t mask = p.mask;
  const int shift = p.shift;

  // load the tile's keys first (independent loads in flight), then rank
  uint32_t key[kItems];
  const uint32_t tile_base = tile * kTile + warp * (kItems * 32) + lane;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const uint32_t idx = tile_base + k * 32;
    key[k] = idx < n ? keys_in[idx] : 0xffffffffu;
  }
  // where each digit starts in the whole output
  uint32_t unused;
  sm.global_base[threadIdx.x] = block_exclusive_scan(hist[threadIdx.x], sm.scan_tmp, unused);

  uint32_t ranks[kItems / 2] = {};  // two a register: a warp's running count stays below 2^16
  auto rank = [&](int k) { return k & 1 ? ranks[k / 2] >> 16 : ranks[k / 2] & 0xffffu; };
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const bool valid = tile_base + k * 32 < n;
    const uint32_t digit = (key[k] >> shift) & mask;
    // the valid lanes holding the same digit: one ballot per digit bit (measured faster on a B200
    // than match.any: depth passes 21 -> 18 us, tile passes 86-96 -> 80 us at 1M Gaussians)
    unsigned peers = __ballot_sync(kFullMask, valid);
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {
      const bool bit = (digit >> b) & 1u;
      const unsigned bal = __ballot_sync(kFullMask, bit);
      peers &= bit ? bal : ~bal;
    }
    if (!valid) peers = 1u << lane;
    const int leader = __ffs(peers) - 1;
    // every lane reads its digit's running count; the digit's first lane then advances it
    const uint32_t old = valid ? sm.warp_hist[warp][digit] : 0u;
    __syncwarp();
    if (valid && lane == leader) sm.warp_hist[warp][digit] = old + __popc(peers);
    __syncwarp();
    const uint32_t r = old + __popc(peers & lt_mask);
    ranks[k / 2] = k & 1 ? ranks[k / 2] | r << 16 : r;
  }
  // the values, in flight while the counts are summed (loaded with the keys they cost registers: spills)
  uint32_t val[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const uint32_t idx = tile_base + k * 32;
    val[k] = idx < n ? (vals_in ? vals_in[idx] : (uint32_t)(seg_base + idx)) : 0u;
  }
  __syncthreads();

  // per digit: exclusive offsets of each warp, block count, block-local digit start
  const int d = threadIdx.x;
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kSortThreads / 32; ++w) {
    const uint32_t t = sm.warp_hist[w][d];
    sm.warp_hist[w][d] = run;
    run += t;
  }
  const uint32_t count = run;
  uint32_t tile_items;
  sm.block_excl[d] = block_exclusive_scan(count, sm.scan_tmp, tile_items);
  __syncthreads();  // every digit's block-local start is read by other threads below

  // digit d's count for the later tiles (digits above the mask are empty everywhere)
  uint32_t* lb = p.lookback + (size_t)(ticket - tile) * kRadix;  // this segment's chain
  const bool first = tile == 0 || (uint32_t)d > mask;
  st_relaxed_u32(&lb[(size_t)tile * kRadix + d], (first ? kLbPrefix : kLbAggregate) | count);

  // reorder the tile in shared memory by digit
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (tile_base + k * 32 < n) {
      const uint32_t digit = (key[k] >> shift) & mask;
      const uint32_t pos = sm.block_excl[digit] + sm.warp_hist[warp][digit] + rank(k);
      if (pos < (uint32_t)kTile) {  // always true: ranks are consistent within the block
        sm.keys[pos] = key[k];
        sm.vals[pos] = val[k];
      }
    }
  }

  // decoupled look-back for digit d
  if (!first) {
    uint32_t prev = 0;
    int64_t j = (int64_t)tile - 1;
    bool gave_up = false, found = false;
    while (!found) {
      uint32_t w[kLookback];
#pragma unroll
      for (int b = 0; b < kLookback; ++b)
        w[b] = (j - b >= 0) ? ld_relaxed_u32(&lb[(size_t)(j - b) * kRadix + d]) : kLbPrefix;
#pragma unroll
      for (int b = 0; b < kLookback; ++b) {
        uint32_t x = w[b];
        if (!found && (x >> 30) == 0) {
          int spins = 0;
          do {
            if (++spins > kMaxSpins) {
              gave_up = true;
              x = kLbPrefix;
              break;
            }
            __nanosleep(32);
            x = ld_relaxed_u32(&lb[(size_t)(j - b) * kRadix + d]);
          } while ((x >> 30) == 0);
        }
        if (!found) {
          prev += x & kLbValue;
          found = (x >> 30) == 2;
        }
      }
      j -= kLookback;
    }
    if (gave_up) atomicOr(&p.hdr->status, kStatusLookback);
    st_relaxed_u32(&lb[(size_t)tile * kRadix + d], kLbPrefix | ((prev + count) & kLbValue));
    sm.global_base[d] += prev;
  }

  __syncthreads();
  for (uint32_t i = threadIdx.x; i < tile_items; i += kSortThreads) {
    const uint32_t k32 = sm.keys[i];
    const uint32_t digit = (k32 >> shift) & mask;
    const uint32_t out = sm.global_base[digit] + (i - sm.block_excl[digit]);
    if (out < n) {  // always true unless a look-back gave up (the status word then says so)
      keys_out[out] = k32;
      vals_out[out] = sm.vals[i];
    }
  }
}

// ---------------------------------------------------------------- start of a pass -------------
// Clears the pass's counters, histograms and look-back words in one launch (four memsets and a kernel
// took five).
__global__ void __launch_bounds__(256) begin_binning_kernel(const __grid_constant__ BeginParams p) {
  chain_begin();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    GeomHeader* hdr = p.hdr;
    const unsigned long long total = hdr->num_rendered64;
    uint32_t status = hdr->status & ~(kStatusCapacity | kStatusInconsistent);
    if (total > (unsigned long long)kMaxInstances) status |= kStatusOverflow;
    hdr->status = status;
    hdr->num_rendered = (uint32_t)(total > 0xffffffffull ? 0xffffffffull : total);
    hdr->dup_tile_counter = 0;
    hdr->num_pairs = 0;
    for (int i = 0; i < kMaxSortPasses; ++i) hdr->sort_tile_counter[i] = 0;
  }
  const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
#pragma unroll
  for (int r = 0; r < BeginParams::kRegions; ++r)
    for (size_t i = first; i < p.bytes[r] / 16; i += stride) p.region[r][i] = make_uint4(0u, 0u, 0u, 0u);
}

// ---------------------------------------------------------------- coarse lists ----------------
// duplicateWithKeys (rasterizer_impl.cu:94-140) by bins of kBinW x kBinH tiles instead of tiles, over the
// depth-sorted Gaussians, in two kernels:
//  1. pair_scan_kernel: the inclusive scan of the Gaussians' bin counts in depth order (block b takes
//     sorted positions [1024 b, 1024 b + 1024), four per thread: block scan plus a decoupled look-back
//     over the preceding blocks), written to p.incl with the tile rects; every Gaussian whose pairs
//     hold the first or last pair of an emit block (kEmitBlock pairs) records its position there
//     (p.emit_first / p.emit_last);
//  2. pair_emit_kernel: block b writes pairs [2048 b, 2048 b + 2048) of the list: every block does the
//     same amount of work however the pairs are spread over the Gaussians (the nearest splats, first
//     in depth order, cover most bins).  It stages the offsets and bin rects of its Gaussians in
//     shared memory; each thread writes 8 consecutive pairs (one binary search for the first one's
//     Gaussian, then a walk through the rect and on to the next Gaussians, two 16-byte stores per
//     array) and counts the digit histograms of the bin sort that follows.

__device__ __forceinline__ uint32_t record_view(const TileGrid& g, uint32_t i) {
  return (g.V == 1) ? 0u : i / (uint32_t)g.P;  // the depth order keeps records in their view
}

// Tile rect of record `rec` as the kernels keep it: first column | end << 16 (the first column may be
// negative and the end past gx when the seam wraps) and first row | end << 16; empty: 0, 0.
__device__ __forceinline__ uint2 record_rect(const TileGrid& grid, const int* radii, const float4* splat, uint32_t rec,
                                             uint32_t view) {
  uint2 r = make_uint2(0u, 0u);
  const int radius = (rec - view * (uint32_t)grid.P < (uint32_t)grid.P) ? radii[rec] : 0;
  if (radius > 0) {
    const float4 a = splat[2 * (size_t)rec];
    int2 rmin, rmax;
    if (grid.seam_wrap)
      tile_rect_cyclic(make_float2(a.x, a.y), radius, grid.gx[view], grid.gy[view], rmin, rmax);
    else
      tile_rect(make_float2(a.x, a.y), radius, grid.gx[view], grid.gy[view], rmin, rmax);
    if (rmax.x > rmin.x && rmax.y > rmin.y)
      r = make_uint2(((uint32_t)rmin.x & 0xffffu) | ((uint32_t)rmax.x << 16), (uint32_t)rmin.y | ((uint32_t)rmax.y << 16));
  }
  return r;
}

// The bins of a tile rect: first column (the columns run on modulo the view's bx when the seam wraps),
// columns, first row, rows.
struct BinRect {
  uint32_t col, cols, row, rows;
};
__device__ __forceinline__ BinRect bin_rect(uint2 r, int gx, int bx) {
  BinRect b{0u, 0u, 0u, 0u};
  int x0 = (int)(int16_t)(r.x & 0xffffu), x1 = (int)(r.x >> 16);
  const uint32_t y0 = r.y & 0xffffu, y1 = r.y >> 16;
  if (y1 <= y0) return b;
  if (x0 < 0) {  // columns [x0 + gx, gx) and [0, x1): the rect is at most gx wide
    x0 += gx;
    x1 += gx;
  }
  if (x0 >= gx) {
    x0 -= gx;
    x1 -= gx;
  }
  b.col = (uint32_t)x0 / kBinW;
  if (x1 <= gx)
    b.cols = (uint32_t)(x1 - 1) / kBinW + 1u - b.col;
  else
    b.cols = min((uint32_t)bx, (uint32_t)bx - b.col + (uint32_t)(x1 - gx - 1) / kBinW + 1u);
  b.row = y0 / kBinH;
  b.rows = (y1 - 1u) / kBinH + 1u - b.row;
  return b;
}

// A pair's word: the bin's tiles that the rect covers (bits [0, 8) its columns, bits [8, 12) its rows), and
// above them the bin (at most 2^20 of them: 32 views of 2^28 pixels).  It is the key that the pairs are
// sorted by, so the fine stage reads everything it needs in order, without a gather.
static_assert(kBinW * kBinH == 32, "a lane per tile of a bin");

__device__ __forceinline__ uint32_t tile_mask(int tx0, int ty0, int gx, bool wrap, uint2 rect) {
  const int x0 = (int)(int16_t)(rect.x & 0xffffu) - tx0, x1 = (int)(rect.x >> 16) - tx0;
  const int y0 = (int)(rect.y & 0xffffu) - ty0, y1 = (int)(rect.y >> 16) - ty0;
  auto span = [](int lo, int hi, int width) {  // bits [lo, hi) of `width`
    const int l = min(max(lo, 0), width), h = min(max(hi, 0), width);
    return h > l ? ((1u << h) - 1u) & ~((1u << l) - 1u) : 0u;
  };
  uint32_t cols = span(x0, x1, kBinW);
  if (wrap) cols = (cols | span(x0 + gx, x1 + gx, kBinW) | span(x0 - gx, x1 - gx, kBinW)) & span(0, gx - tx0, kBinW);
  return cols | (span(y0, y1, kBinH) << kBinW);
}

constexpr int kScanItems = kScanTile / kScanBlock;  // Gaussians per scan thread

__global__ void __launch_bounds__(kScanBlock) pair_scan_kernel(const __grid_constant__ DuplicateParams p) {
  chain_begin();
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[kScanBlock / 32];
  __shared__ unsigned long long s_excl;
  if (!instances_fit(p.hdr, p.capacity)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&p.hdr->status, kStatusCapacity);
    return;
  }
  if (threadIdx.x == 0) s_tile = atomicAdd(&p.hdr->dup_tile_counter, 1u) + p.skip_tiles;
  __syncthreads();
  const uint32_t tile = s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t items = (uint32_t)p.grid.P * (uint32_t)p.grid.V;
  const uint32_t i0 = tile * (uint32_t)kScanTile + threadIdx.x * (uint32_t)kScanItems;
  uint32_t cnt[kScanItems];
#pragma unroll
  for (int u = 0; u < kScanItems; ++u) {
    const uint32_t i = i0 + u;
    cnt[u] = 0;
    if (i < items) {
      const uint32_t view = record_view(p.grid, i);
      const uint2 r = record_rect(p.grid, p.radii, p.splat, p.order[i], view);
      const BinRect b = bin_rect(r, p.grid.gx[view], bins_x(p.grid.gx[view]));
      cnt[u] = b.cols * b.rows;
      p.rect_x[i] = r.x;
      p.rect_y[i] = r.y;
    }
  }
  uint32_t thread_total = 0;
#pragma unroll
  for (int u = 0; u < kScanItems; ++u) thread_total += cnt[u];
  // block inclusive scan of the thread totals
  uint32_t v = thread_total;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(kFullMask, v, o);
    if (lane >= o) v += n;
  }
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = (lane < kScanBlock / 32) ? s_warp[lane] : 0u;
#pragma unroll
    for (int o = 1; o < kScanBlock / 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(kFullMask, w, o);
      if (lane >= o) w += n;
    }
    if (lane < kScanBlock / 32) s_warp[lane] = w;
  }
  __syncthreads();
  const uint32_t thread_excl = v - thread_total + (warp > 0 ? s_warp[warp - 1] : 0u);
  const unsigned long long block_total = s_warp[kScanBlock / 32 - 1];
  // decoupled look-back across blocks (warp 0)
  if (warp == 0) {
    if (tile == 0) {
      if (lane == 0) {
        st_relaxed_u64(&p.scan_state[0], kScanPrefix | block_total);
        s_excl = 0;
      }
    } else {
      if (lane == 0) st_relaxed_u64(&p.scan_state[tile], kScanAggregate | block_total);
      unsigned long long excl = 0;
      long long base = (long long)tile - 1;
      bool gave_up = false;
      const int max_spins = p.max_spins > 0 ? p.max_spins : kMaxSpins;
      for (;;) {
        const long long j = base - lane;
        unsigned long long w = kScanPrefix;  // virtual zero prefix before the first block
        if (j >= 0) {
          w = ld_relaxed_u64(&p.scan_state[j]);
          int spins = 0;
          while ((w >> 62) == 0) {
            if (++spins > max_spins) {
              gave_up = true;
              w = kScanPrefix;
              break;
            }
            __nanosleep(64);
            w = ld_relaxed_u64(&p.scan_state[j]);
          }
        }
        const unsigned prefix_lanes = __ballot_sync(kFullMask, (w >> 62) == 2);
        const int stop = prefix_lanes ? (__ffs(prefix_lanes) - 1) : 31;
        unsigned long long c = (lane <= stop) ? (w & kScanValue) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFullMask, c, o);
        excl += c;
        if (prefix_lanes) break;
        base -= 32;
      }
      if (__any_sync(kFullMask, gave_up) && lane == 0) atomicOr(&p.hdr->status, kStatusLookback);
      if (lane == 0) {
        st_relaxed_u64(&p.scan_state[tile], kScanPrefix | ((excl + block_total) & kScanValue));
        s_excl = excl;
      }
    }
  }
  __syncthreads();
  // (past the capacity only when the scan is inconsistent: at most one pair per instance)
  const unsigned long long max_blocks = ((unsigned long long)p.capacity + kEmitBlock - 1) / kEmitBlock;
  unsigned long long incl = s_excl + thread_excl;
#pragma unroll
  for (int u = 0; u < kScanItems; ++u) {
    const uint32_t i = i0 + u;
    const unsigned long long start = incl;
    incl += cnt[u];
    if (i >= items) continue;
    p.incl[i] = (uint32_t)min(incl, 0xffffffffull);
    if (cnt[u] == 0) continue;
    // the emit blocks whose first pair (b * kEmitBlock) lies in [start, incl)
    for (unsigned long long b = (start + kEmitBlock - 1) / kEmitBlock; b * kEmitBlock < incl && b < max_blocks; ++b)
      p.emit_first[b] = i;
    // ... and those whose last pair does, the last block (whose end the emission finds) aside
    for (unsigned long long b = start / kEmitBlock; b < max_blocks && (b + 1) * kEmitBlock <= incl; ++b)
      p.emit_last[b] = i;
  }
  const uint32_t last_tile = (items + kScanTile - 1) / kScanTile - 1u;
  if (tile == last_tile && threadIdx.x == kScanBlock - 1)
    p.hdr->num_pairs = (uint32_t)min(s_excl + block_total, (unsigned long long)p.capacity);
}

constexpr int kEmitPerThread = kEmitBlock / kScanBlock;
// Gaussians of a block staged in shared memory: as many as it can have pairs, and one.  Measured on a B200, stages of 1025 /
// 2049: the 16-view batch 540 / 528 us, 3M Gaussians 159 / 156 (at some 1.4 pairs a Gaussian most blocks have more than 1025;
// none staged: 545 and 161, but 150,000 Gaussians 31 / 27).
constexpr int kEmitStage = kEmitBlock + 1;

__device__ __forceinline__ float rcp_approx_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__global__ void __launch_bounds__(kScanBlock) pair_emit_kernel(const __grid_constant__ DuplicateParams p) {
  chain_begin();
  __shared__ uint32_t s_hist[kTilePasses * kRadix];  // digit counts of the bin sort
  // the block's Gaussians: inclusive offset, record, tile rect
  __shared__ uint32_t s_incl[kEmitStage], s_rec[kEmitStage];
  __shared__ uint2 s_rect[kEmitStage];
  __shared__ uint32_t s_last;
  const uint32_t R = pair_count(p.hdr, p.capacity);  // (0 when the scan kernel has flagged an overflow)
#pragma unroll 1
  for (uint32_t block = blockIdx.x; block < (R + kEmitBlock - 1u) / kEmitBlock; block += gridDim.x) {
    const uint32_t o_lo = block * (uint32_t)kEmitBlock;
    const uint32_t o_hi = min(R, o_lo + (uint32_t)kEmitBlock);  // exclusive (R <= capacity)
    const int lane = threadIdx.x & 31;
    const uint32_t items = (uint32_t)p.grid.P * (uint32_t)p.grid.V;
    for (int k = threadIdx.x; k < kTilePasses * kRadix; k += kScanBlock) s_hist[k] = 0;
    // (both clamped: after an inconsistent scan, which the status word reports, the entries may be
    // stale; the reads stay in range)
    const uint32_t g_first = min(p.emit_first[block], items - 1u);
    if (threadIdx.x == 0) {
      uint32_t last = items - 1u;
      if (o_hi - o_lo == (uint32_t)kEmitBlock) {
        last = min(p.emit_last[block], items - 1u);
      } else {  // the list's end: the first Gaussian whose inclusive offset reaches it
        uint32_t lo = g_first;
        while (lo < last) {
          const uint32_t mid = (lo + last) >> 1;
          if (p.incl[mid] >= R)
            last = mid;
          else
            lo = mid + 1u;
        }
      }
      s_last = last;
    }
    __syncthreads();
    const uint32_t g_last = s_last;
    const uint32_t n = g_last >= g_first ? g_last - g_first + 1u : 1u;
    // Gaussians between g_first and g_last with no pairs (culled views' records) can make the range longer
    // than the block's pairs: then offsets and rects are read from global memory
    const bool staged = n <= (uint32_t)kEmitStage;
    if (staged)
      for (uint32_t t = threadIdx.x; t < n; t += kScanBlock) {
        s_incl[t] = p.incl[g_first + t];
        s_rec[t] = p.order[g_first + t];
        s_rect[t] = make_uint2(p.rect_x[g_first + t], p.rect_y[g_first + t]);
      }
    __syncthreads();
    const uint32_t* incl = staged ? s_incl : p.incl + g_first;
    const uint32_t excl0 = g_first > 0 ? p.incl[g_first - 1] : 0u;
    // Thread t writes the kEmitPerThread consecutive pairs from o0: one binary search finds the Gaussian
    // of the first, the others step through the rect (or on to the next Gaussians with pairs, whose
    // first pair they then are) without a search or a division.
    const uint32_t o0 = o_lo + (uint32_t)threadIdx.x * (uint32_t)kEmitPerThread;
    uint32_t j = 0;  // the first of the block's Gaussians whose inclusive offset exceeds o0
    {
      uint32_t hi = n - 1u;
      while (j < hi) {
        const uint32_t mid = (j + hi) >> 1;
        if (incl[mid] > o0)
          hi = mid;
        else
          j = mid + 1u;
      }
    }
    uint32_t end_j = incl[j];
    uint32_t rec = 0, view = 0, width = 1;
    int gx = 1, bx = 1;
    uint2 rect = make_uint2(0u, 0u);
    BinRect bins{0u, 1u, 0u, 1u};
    auto load_rect = [&](uint32_t jj) {
      const uint32_t i = g_first + jj;
      view = record_view(p.grid, i);
      rec = staged ? s_rec[jj] : p.order[i];
      rect = staged ? s_rect[jj] : make_uint2(p.rect_x[i], p.rect_y[i]);
      gx = p.grid.gx[view];
      bx = bins_x(gx);
      bins = bin_rect(rect, gx, bx);
      width = max(bins.cols, 1u);
    };
    load_rect(j);
    // row and column of o0 in the rect: local / width from an approximate reciprocal (local < 2^21, a rect
    // holds at most every bin of a view, so the truncated estimate is within one of the quotient; one
    // step fixes it)
    const uint32_t local = o0 - (j > 0 ? incl[j - 1] : excl0);
    uint32_t ry = (uint32_t)((float)local * rcp_approx_f((float)width));
    int rem = (int)(local - ry * width);
    if (rem < 0) {
      ry -= 1u;
      rem += (int)width;
    } else if (rem >= (int)width) {
      ry += 1u;
      rem -= (int)width;
    }
    uint32_t keys[kEmitPerThread], vals[kEmitPerThread];
  #pragma unroll
    for (int k = 0; k < kEmitPerThread; ++k) {
      const uint32_t o = o0 + (uint32_t)k;
      const bool ok = o < o_hi;
      if (k > 0 && ok) {
        // past Gaussian j: on to the next one that has pairs, whose first pair o is (j stays below n even
        // after an inconsistent scan, which the status word reports)
        if (o >= end_j && j + 1u < n) {
          do {
            ++j;
            end_j = incl[j];
          } while (end_j <= o && j + 1u < n);
          load_rect(j);
          ry = 0;
          rem = 0;
        } else if (++rem == (int)width) {
          rem = 0;
          ++ry;
        }
      }
      uint32_t col = bins.col + (uint32_t)rem;
      if (col >= (uint32_t)bx) col -= (uint32_t)bx;  // the seam wraps
      const uint32_t row = bins.row + ry;
      const uint32_t key = ((p.grid.bin_base[view] + row * (uint32_t)bx + col) << kPairBinShift) |
                           tile_mask((int)col * kBinW, (int)row * kBinH, gx, p.grid.seam_wrap != 0, rect);
      keys[k] = key;
      vals[k] = rec;
      // digit histograms of the bin sort (the pass that would otherwise re-read every key)
      const unsigned live = __ballot_sync(kFullMask, ok);
  #pragma unroll
      for (int q = 0; q < kTilePasses; ++q)
        if (q < p.hist_passes)
          count_digit(s_hist, q * kRadix + ((key >> p.hist_shift[q]) & p.hist_mask[q]), ok, live, lane);
    }
    // the thread's run of the list: 16-byte stores when it is whole (o0 is a multiple of 8, the
    // lists start 256-byte aligned)
    static_assert(kEmitPerThread == 8, "two 16-byte stores per array");
    if (o0 + (uint32_t)kEmitPerThread <= o_hi) {
      uint4* kd = reinterpret_cast<uint4*>(p.keys + o0);
      uint4* vd = reinterpret_cast<uint4*>(p.vals + o0);
      kd[0] = make_uint4(keys[0], keys[1], keys[2], keys[3]);
      kd[1] = make_uint4(keys[4], keys[5], keys[6], keys[7]);
      vd[0] = make_uint4(vals[0], vals[1], vals[2], vals[3]);
      vd[1] = make_uint4(vals[4], vals[5], vals[6], vals[7]);
    } else {
  #pragma unroll
      for (int k = 0; k < kEmitPerThread; ++k)
        if (o0 + (uint32_t)k < o_hi) {
          p.keys[o0 + k] = keys[k];
          p.vals[o0 + k] = vals[k];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kTilePasses * kRadix; k += kScanBlock) {
      const uint32_t c = s_hist[k];
      if (c) atomicAdd(&p.hist[k], c);
    }
    __syncthreads();  // (the next pairs' stage and histograms)
  }
}

// ---------------------------------------------------------------- depth order by counting -----
// A Gaussian's place in the (depth bits, index) order is the number of Gaussians before it.  A block has
// kRankItems of them; its threads share the view's keys, and each compares its keys with all of the
// block's, so a key is loaded once per block and nothing is staged.  Keys at lower indices count when
// they are <= a Gaussian's, that is when the float below them is <; keys at higher ones when they are <.
//
// Bound by issue: V P^2 comparisons.  An integer comparison and a predicated add both go to the ALU's 16
// lanes (22 us for 10,000 Gaussians); here a comparison is sat(2^40 own - 2^40 key) and an add, both on
// the FMA pipes: a key >= 2^-3 (depths are beyond the near cull at 0.2) differs from another by at least
// 2^-26, so the difference is 0 or beyond 1 and the saturated value exactly 0 or 1, whatever its
// rounding; culled Gaussians' infinite keys become 2^70, beyond any finite distance (at most 2^64).
constexpr int kRankThreads = 256;
constexpr int kRankItems = 16;
static_assert(kRankItems * kRankItems == kRankThreads, "a thread per pair of the block's own Gaussians");
static_assert(kRankMaxP < (1 << 24), "the counts are exact in float");

__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float r;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__global__ void __launch_bounds__(kRankThreads) rank_kernel(const __grid_constant__ RankParams p) {
  chain_begin();
  __shared__ uint32_t s_rank[kRankItems];
  const uint32_t P = (uint32_t)p.grid.P, view = blockIdx.y;
  const uint32_t* keys = p.keys + (size_t)view * P;
  const uint32_t j0 = blockIdx.x * (uint32_t)kRankItems;
  if (threadIdx.x < kRankItems) s_rank[threadIdx.x] = 0;
  const float far = 0x1p70f, scale = 0x1p40f;
  float own[kRankItems], rank[kRankItems];
#pragma unroll
  for (int q = 0; q < kRankItems; ++q) {
    own[q] = j0 + q < P ? fminf(__uint_as_float(keys[j0 + q]), far) : 0.f;
    rank[q] = 0.f;
  }
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < P; i += kRankThreads) {
    const uint32_t bits = __float_as_uint(fminf(__uint_as_float(keys[i]), far));
    float neg = -scale * __uint_as_float(bits - (i < j0 ? 1u : 0u));
    if (i - j0 < (uint32_t)kRankItems) neg = -0x1p126f;  // (the block's own: below)
#pragma unroll
    for (int q = 0; q < kRankItems; ++q) rank[q] += fma_sat(own[q], scale, neg);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kRankItems; ++q) {
    const uint32_t sum = __reduce_add_sync(kFullMask, (uint32_t)rank[q]);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&s_rank[q], sum);
  }
  {
    const uint32_t a = j0 + threadIdx.x / kRankItems, c = j0 + threadIdx.x % kRankItems;
    if (a < P && c < P) {
      const uint32_t ka = keys[a], kc = keys[c];
      if (kc < ka || (kc == ka && c < a)) atomicAdd(&s_rank[threadIdx.x / kRankItems], 1u);
    }
  }
  __syncthreads();
  const uint32_t j = j0 + threadIdx.x;
  if (threadIdx.x < kRankItems && j < P) {
    const uint32_t rec = view * P + j, at = view * P + s_rank[threadIdx.x];
    const uint2 r = record_rect(p.grid, p.radii, p.splat, rec, view);
    p.order[at] = rec;
    p.rect_x[at] = r.x;
    p.rect_y[at] = r.y;
  }
}

// Tile rects in depth order, where the depth order comes from the sort and no scan needs them.
__global__ void __launch_bounds__(256) rect_kernel(const __grid_constant__ RankParams p) {
  chain_begin();
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= (uint32_t)p.grid.P * (uint32_t)p.grid.V) return;
  const uint2 r = record_rect(p.grid, p.radii, p.splat, p.order[i], record_view(p.grid, i));
  p.rect_x[i] = r.x;
  p.rect_y[i] = r.y;
}

// ---------------------------------------------------------------- tile lists ------------------
// The fine stage works a warp at a time: a warp counts its pairs by tile, and later, with the places that the
// scan and the earlier warps' counts give it, appends them to the tiles' lists.  No warp waits for another.
//  * From coarse lists, a warp has a piece of consecutive pairs of the sorted list, whatever bins they are
//    in: all warps do the same work however the Gaussians are spread over the image (tile_count / tile_fill).
//    Only a bin that runs on into the next piece needs a piece's counts there, so a slot per piece holds them
//    (those of the piece's last bin), and a sum of its slots per block shortens the walk back to a bin's begin.
//  * Without coarse lists, every bin reads its view's whole order, split into TileGrid::parts, eight to a block
//    (whole_count / whole_fill).
// Measured on a B200, all of the fine stage, with every bin split into as many parts as an even spread asks for /
// pieces: 1M Gaussians at 2048x1024 within 0.1 rad 608 / 106 us, 3M at 4096x2048 within 0.02 rad 2930 / 490; evenly
// spread 1M 71 / 71, 3M 264 / 279, 16 views over 1M 588 / 577, 71,000 at 2132x1093 39 / 36.
constexpr int kListThreads = 32 * kListWarps;
constexpr uint32_t kNoBin = 0xffffffffu >> kPairBinShift;

static_assert(kMaxBatchViews == 32, "a lane per view");

// A bin's place: its first tile column and row in its view.
struct BinTiles {
  int tx0, ty0;
  int gx, gy;
  uint32_t tile0;  // the view's first tile
};
__device__ __forceinline__ BinTiles bin_tiles(const TileGrid& g, uint32_t view, uint32_t local) {
  const uint32_t bx = (uint32_t)bins_x(g.gx[view]);
  return {(int)(local % bx) * kBinW, (int)(local / bx) * kBinH, g.gx[view], g.gy[view], g.tile_base[view]};
}
// The views' first bins in shared memory, for bin_tiles by a warp (a lane per view); a block barrier follows.
__device__ __forceinline__ void load_bases(const TileGrid& g, uint32_t (&bases)[kMaxBatchViews]) {
  if ((int)threadIdx.x < kMaxBatchViews) bases[threadIdx.x] = (int)threadIdx.x < g.V ? g.bin_base[threadIdx.x] : kNoBin;
}
__device__ __forceinline__ BinTiles bin_tiles(const TileGrid& g, const uint32_t (&bases)[kMaxBatchViews], uint32_t bin) {
  const uint32_t view = (uint32_t)__popc(__ballot_sync(kFullMask, bases[threadIdx.x & 31] <= bin)) - 1u;
  return bin_tiles(g, view, bin - bases[view]);
}
// Whether the lane's tile (lane / 8, lane % 8) of the bin lies in the image, and its index.
__device__ __forceinline__ bool lane_tile(const BinTiles& b, uint32_t& tile) {
  const int lane = threadIdx.x & 31, tx = b.tx0 + lane % kBinW, ty = b.ty0 + lane / kBinW;
  tile = b.tile0 + (uint32_t)(ty * b.gx + tx);
  return tx < b.gx && ty < b.gy;
}

// First index of the sorted words with a bin >= bin, by a warp (32 probes a step).
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t* words, uint32_t n, uint32_t bin) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t lo = 0, len = n;  // the answer lies in [lo, lo + len]
  while (len > 0) {
    const uint32_t step = (len + 31u) / 32u;
    const bool below = lane * step < len && (words[lo + lane * step] >> kPairBinShift) < bin;
    const uint32_t c = (uint32_t)__popc(__ballot_sync(kFullMask, below));  // probes 0 .. c - 1 are below
    if (c == 0) return lo;
    const uint32_t end = lo + len;
    lo += (c - 1u) * step + 1u;
    len = min(step - 1u, end - lo);
  }
  return lo;
}

// The bits of a nibble as the low bits of four bytes (bit k in byte k): with a tile row's eight columns in
// two such words, a warp counts and ranks all eight tiles with additions.
__device__ __forceinline__ uint32_t spread4(uint32_t nibble) { return (nibble * 0x00204081u) & 0x01010101u; }

// Counts of a bin's tiles: every lane keeps the 32 tiles' counts as bytes in eight words, which the warp then
// adds.  (A ballot and a popcount per tile and 32 pairs took 38 us of the 1M-Gaussian view instead of 15.)
struct TileCounts {
  uint32_t acc[kBinH][2] = {};
  __device__ __forceinline__ void add(uint32_t mask) {
    const uint32_t lo = spread4(mask & 15u), hi = spread4((mask >> 4) & 15u);
#pragma unroll
    for (int r = 0; r < kBinH; ++r) {
      const uint32_t on = (mask >> (kBinW + r)) & 1u;
      acc[r][0] += lo * on;
      acc[r][1] += hi * on;
    }
  }
  // The sum over the warp of the lane's tile (lane / 8, lane % 8), after at most 255 pairs a lane; starts again at zero.
  __device__ __forceinline__ uint32_t sum() {
    const int lane = threadIdx.x & 31;
    uint32_t mine = 0;
#pragma unroll
    for (int r = 0; r < kBinH; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // tile 8 r + 4 h + k is byte k of acc[r][h]
        const uint32_t even = __reduce_add_sync(kFullMask, acc[r][h] & 0x00ff00ffu);        // bytes 0 and 2
        const uint32_t odd = __reduce_add_sync(kFullMask, (acc[r][h] >> 8) & 0x00ff00ffu);  // bytes 1 and 3
        if (lane >> 2 == 2 * r + h) {
          const uint32_t w = lane & 1 ? odd : even;
          mine = lane & 2 ? w >> 16 : w & 0xffffu;
        }
        acc[r][h] = 0u;
      }
    return mine;
  }
};

// ---- from coarse lists: pieces of the sorted pairs
// A piece's pairs: as many as give kPieceTarget warps (about two waves of blocks), within limits.  Measured on a B200:
// at least 32 / 64, 20,000 Gaussians at 2132x1093 36 / 42 us of the fine stage; at most 160 / 192 / 256 / 384 / 512, the
// 16-view batch 650 / 617 / 578 / 583 / 576 us, 3M Gaussians at 4096x2048 279 / 278 / 280 / 317 / 339; targets of
// 5920 / 8192 / 11,000, 1M Gaussians 73 / 71 / 73.
constexpr uint32_t kMinPiece = 32, kMaxPiece = 256, kPieceTarget = 8192;
struct Pieces {
  uint32_t n;       // pairs
  uint32_t len;     // of a piece, whole groups of 32
  uint32_t count;   // pieces
  uint32_t blocks;  // of kListWarps pieces
  uint32_t* sums;   // [blocks][32]: counts of the pieces' last bins, by block ...
  uint16_t* slots;  // [count][32]: ... and by piece
  __device__ __forceinline__ Pieces(const TileListParams& p) : n(pair_count(p.hdr, p.capacity)) {
    len = min(max((n / kPieceTarget + 31u) & ~31u, kMinPiece), kMaxPiece);
    count = (n + len - 1u) / len;
    blocks = (count + kListWarps - 1u) / kListWarps;
    sums = p.counts;
    slots = reinterpret_cast<uint16_t*>(p.counts + 32 * (size_t)blocks);
  }
  __device__ __forceinline__ uint32_t first(uint32_t piece) const { return min(piece * len, n); }
};
// The counts take 16 words a piece and 32 a block, 5/8 n + 52 at most: room of as many words as there are pairs, in
// whole 64, holds them (with fewer than 128 pairs, of one to four pieces, too).
static_assert(kMinPiece >= 32 && kListWarps >= 8 && kAlign >= 64 * sizeof(uint32_t), "the counts fit");
static_assert(kMaxPiece <= 255 * 32, "a lane's counts fit in bytes");

// The warp's counts of a bin, added to its tiles' totals.
__device__ __forceinline__ void add_total(const TileListParams& p, const uint32_t (&bases)[kMaxBatchViews], uint32_t bin,
                                          uint32_t count) {
  uint32_t t;
  if (lane_tile(bin_tiles(p.grid, bases, bin), t) && count) atomicAdd(p.totals ? &p.totals[t] : &p.ranges[t].x, count);
}

// Walks a piece by a warp: use(bin, in, word, begins, ends, at_end) for every run of a bin within a group of 32 of its
// pairs: `in` the lanes of the run, whether the bin begins with it (in this piece) and whether it or the piece ends with
// it, at_end for the piece.  next_group(e0, after) gives the group's words, and in `after` those of the group behind.
template <class Next, class Use>
__device__ __forceinline__ void walk_piece(uint32_t begin, uint32_t end, Next next_group, Use use) {
  const int lane = threadIdx.x & 31;
  uint32_t bin = kNoBin;
#pragma unroll 1
  for (uint32_t e0 = begin; e0 < end; e0 += 32) {
    uint32_t after;  // the first word of the group behind
    const uint32_t w = next_group(e0, after);
    unsigned left = __ballot_sync(kFullMask, e0 + lane < end);
    const uint32_t follows = e0 + 32 < end ? __shfl_sync(kFullMask, after, 0) >> kPairBinShift : kNoBin;
    do {  // (once, unless a bin ends within the group)
      const uint32_t b = __shfl_sync(kFullMask, w, __ffs(left) - 1) >> kPairBinShift;
      const bool in = ((left >> lane) & 1u) && (w >> kPairBinShift) == b;
      left &= ~__ballot_sync(kFullMask, in);
      use(b, in, w, b != bin, left != 0 || b != follows, left == 0 && follows == kNoBin);
      bin = b;
    } while (left);
  }
}

__global__ void __launch_bounds__(kListThreads) tile_count_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  __shared__ uint32_t s_own[kListWarps][32], s_bin[kListWarps], s_bases[kMaxBatchViews];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pieces all(p);
  load_bases(p.grid, s_bases);
  __syncthreads();
  for (uint32_t block = blockIdx.x; block < all.blocks; block += gridDim.x) {
    const uint32_t piece = block * kListWarps + (uint32_t)warp, begin = all.first(piece), end = all.first(piece + 1);
    auto load = [&](uint32_t e) { return e < end ? p.words[e] : 0u; };
    uint32_t w0 = load(begin + lane), w1 = load(begin + 32 + lane), own = 0, last = kNoBin;
    TileCounts c;
    walk_piece(begin, end, [&](uint32_t e0, uint32_t& after) {
      const uint32_t w = w0;
      after = w0 = w1;
      w1 = load(e0 + 64 + lane);
      return w;
    }, [&](uint32_t bin, bool in, uint32_t w, bool, bool ends, bool at_end) {
      c.add(in ? w : 0u);
      if (!ends) return;
      own = c.sum();
      last = bin;
      if (!at_end) add_total(p, s_bases, bin, own);
    });
    s_own[warp][lane] = own;
    if (lane == 0) s_bin[warp] = last;
    if (piece < all.count) all.slots[32 * (size_t)piece + lane] = (uint16_t)own;
    __syncthreads();
    // the pieces' last bins' totals, one addition a bin, and the block's sum
    if (last != kNoBin && (warp == kListWarps - 1 || s_bin[warp + 1] != last)) {
      uint32_t run = 0;
#pragma unroll
      for (int k = 0; k < kListWarps; ++k) run += s_bin[k] == last ? s_own[k][lane] : 0u;
      add_total(p, s_bases, last, run);
    }
    if (warp == 0) {
      uint32_t sum = 0;
#pragma unroll
      for (int k = 0; k < kListWarps; ++k) sum += s_own[k][lane];
      all.sums[32 * (size_t)block + lane] = sum;
    }
    __syncthreads();
  }
}

// ---- without: parts of the whole order per bin
// A warp's part: the bin's tiles, and entries [first, end) of its view's depth order.
struct BinPart {
  BinTiles bin;
  uint32_t tiles;   // the view's tiles
  uint32_t counts0; // the view's counts: [parts][tiles]
  uint32_t part;    // parts or more: none
  uint32_t parts;
  uint32_t first, end;
};

__device__ __forceinline__ BinPart bin_part(const TileListParams& p, uint32_t grid_block) {
  const TileGrid& g = p.grid;
  uint32_t view = 0;
#pragma unroll 1
  for (int v = 1; v < g.V; ++v)
    if (g.block_base[v] <= grid_block) view = (uint32_t)v;
  BinPart b;
  b.tiles = (uint32_t)(g.gx[view] * g.gy[view]);
  b.counts0 = g.count_base[view];
  b.parts = g.parts[view];
  const uint32_t per_bin = (b.parts + kListWarps - 1u) / kListWarps;  // blocks
  const uint32_t block = grid_block - g.block_base[view], local = block / per_bin;
  b.part = (block - local * per_bin) * kListWarps + (threadIdx.x >> 5);
  b.bin = bin_tiles(g, view, local);
  const uint32_t first = view * (uint32_t)g.P, end = first + (uint32_t)g.P;
  // (parts of whole groups of 32)
  const uint32_t len = ((end - first + b.parts - 1u) / b.parts + 31u) & ~31u;
  b.first = (uint32_t)min((unsigned long long)end, first + (unsigned long long)b.part * len);
  b.end = min(end, b.first + len);
  return b;
}

// The tiles of the bin that entry e of the order covers.
__device__ __forceinline__ uint32_t entry_tiles(const TileListParams& p, const BinTiles& b, uint32_t e) {
  return tile_mask(b.tx0, b.ty0, b.gx, p.grid.seam_wrap != 0, make_uint2(p.rect_x[e], p.rect_y[e]));
}

// Whether a word's tiles are any of the bin's: a row and a column.
__device__ __forceinline__ bool covers(uint32_t mask) { return (mask & 255u) != 0 && ((mask >> kBinW) & 15u) != 0; }

// Every tile of the grid is written (0 when the instances do not fit).
__global__ void __launch_bounds__(kListThreads) whole_count_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  const int lane = threadIdx.x & 31;
  const bool fit = instances_fit(p.hdr, p.capacity);
  if (!fit && blockIdx.x == 0 && threadIdx.x == 0)
    atomicOr(&p.hdr->status, kStatusCapacity);  // (the scan flags it where there is one)
  BinPart b = bin_part(p, blockIdx.x);
  if (b.part >= b.parts) return;
  if (!fit) b.end = b.first;
  TileCounts c;
  uint32_t mine = 0;  // instances of the lane's tile
  int steps = 0;
  for (uint32_t e0 = b.first; e0 < b.end; e0 += 128) {
    uint32_t mask[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) mask[u] = e0 + 32 * u + lane < b.end ? entry_tiles(p, b.bin, e0 + 32 * u + lane) : 0u;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (__any_sync(kFullMask, covers(mask[u]))) c.add(mask[u]);  // (few groups, where the bins are many)
    steps += 4;
    if (steps > 255 - 4) {
      mine += c.sum();
      steps = 0;
    }
  }
  if (steps) mine += c.sum();
  uint32_t t;
  if (lane_tile(b.bin, t)) {
    if (p.counts == nullptr) {
      p.ranges[t].x = mine;
    } else {
      p.counts[b.counts0 + (size_t)b.part * b.tiles + (t - b.bin.tile0)] = mine;
      if (mine) atomicAdd(&p.totals[t], mine);
    }
  }
}

// Tile ranges from the totals, in tile order, kTileScanBlock tiles a block: a block first sums the
// totals before its own (without them, a single block walks all tiles and replaces the counts in the
// ranges).  An empty tile's range is (0, 0), as the reference leaves it.
constexpr int kTileScanThreads = 1024;
constexpr int kTileScanItems = 8;
constexpr uint32_t kTileScanBlock = kTileScanThreads * kTileScanItems;

__global__ void __launch_bounds__(kTileScanThreads) tile_scan_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_before;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = p.grid.num_tiles;
  const uint32_t* totals = p.totals;
  const uint32_t begin = blockIdx.x * kTileScanBlock;
  if (threadIdx.x == 0) s_before = 0;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < begin; i += kTileScanThreads) before += totals[i];
  before = __reduce_add_sync(kFullMask, before);
  if (lane == 0 && before) atomicAdd(&s_before, before);
  __syncthreads();
  uint32_t carry = s_before;
  for (uint32_t base = begin; base < n; base += kTileScanBlock) {
    const uint32_t t0 = base + threadIdx.x * kTileScanItems;
    uint32_t c[kTileScanItems], sum = 0;
#pragma unroll
    for (int u = 0; u < kTileScanItems; ++u) c[u] = t0 + u < n ? (totals ? totals[t0 + u] : p.ranges[t0 + u].x) : 0u;
#pragma unroll
    for (int u = 0; u < kTileScanItems; ++u) sum += c[u];
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFullMask, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, w, o);
        if (lane >= o) w += y;
      }
      s_warp[lane] = w;
    }
    __syncthreads();
    uint32_t at = carry + x - sum + (warp > 0 ? s_warp[warp - 1] : 0u);
#pragma unroll
    for (int u = 0; u < kTileScanItems; ++u)
      if (t0 + u < n) {
        p.ranges[t0 + u] = c[u] ? make_uint2(at, at + c[u]) : make_uint2(0u, 0u);
        at += c[u];
      }
    carry += s_warp[31];
    if (totals) break;  // (the next tiles are another block's)
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0 && instances_fit(p.hdr, p.capacity) && carry != p.hdr->num_rendered)
    atomicOr(&p.hdr->status, kStatusInconsistent);
}

// The order in which the blends take the tiles (block_tiles): heaviest first within each kOrderTiles tiles,
// in eight classes of list length relative to their mean, in tile order inside a class (neighbours share
// splats, and lists near the mean stay together).  Poles and dense regions hold lists many times the mean,
// and one that starts last leaves the chip idle.  Without a list of twice the mean the segment keeps tile
// order: the blends gain nothing there (1M and 3M evenly spread Gaussians: 0 and 0.3 % slower ordered), and
// the order in which the backward's sums reach a Gaussian stays that of its tiles.  A segment is one block of the fill's launch, ahead of
// the others and hidden behind them.  Measured on a B200, blends of a batch of views of a scene at the
// poles, in tile order / ordered: 366 + 520 / 300 + 449 us.
// (Rows from both ends inwards, without lengths: the same at the poles, but 4 % slower on even lists;
// ordered by the scan's one block: 5 us of every view.)
constexpr int kLoadClasses = 8;
constexpr uint32_t kOrderTiles = 8192;
constexpr uint32_t kOrderItems = kOrderTiles / kListThreads;  // per thread
static_assert(kOrderTiles < 65536, "a class of one segment fits in 16 bits");

__device__ __forceinline__ int load_class(uint32_t count, float mean) {
  const float x = (float)count;
  return (x < 4.f * mean) + (x < 2.83f * mean) + (x < 2.f * mean) + (x < 1.41f * mean) + (x < mean) +
         (x < 0.71f * mean) + (x < 0.35f * mean);
}

// Tiles per class, as 16-bit fields.
struct ClassCounts {
  unsigned long long lo, hi;
  __device__ __forceinline__ void add(int c, uint32_t n) {
    const unsigned long long x = (unsigned long long)n << (16 * (c & 3));
    lo += c < 4 ? x : 0ull;
    hi += c < 4 ? 0ull : x;
  }
  __device__ __forceinline__ uint32_t at(int c) const { return (uint32_t)((c < 4 ? lo : hi) >> (16 * (c & 3))) & 0xffffu; }
  __device__ __forceinline__ ClassCounts operator+(const ClassCounts& o) const { return {lo + o.lo, hi + o.hi}; }
  __device__ __forceinline__ ClassCounts operator-(const ClassCounts& o) const { return {lo - o.lo, hi - o.hi}; }
};

__device__ __forceinline__ void order_tiles(const TileListParams& p, uint32_t segment) {
  __shared__ uint32_t s_sum[kListWarps];
  __shared__ ClassCounts s_class[kListWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t base = segment * kOrderTiles, n = min(p.grid.num_tiles - base, kOrderTiles);
  const uint32_t t0 = base + threadIdx.x * kOrderItems, t1 = min(t0 + kOrderItems, base + n);
  auto count = [&](uint32_t t) {
    const uint2 r = p.ranges[t];
    return r.y - r.x;
  };
  uint32_t sum = 0;
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) sum += count(t);
  sum = __reduce_add_sync(kFullMask, sum);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int w = 0; w < kListWarps; ++w) sum += s_sum[w];
  const float mean = (float)sum / (float)n;
  ClassCounts own{0, 0};
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) own.add(load_class(count(t), mean), 1u);
  ClassCounts at = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long lo = __shfl_up_sync(kFullMask, at.lo, o), hi = __shfl_up_sync(kFullMask, at.hi, o);
    if (lane >= o) at = at + ClassCounts{lo, hi};
  }
  if (lane == 31) s_class[warp] = at;
  __syncthreads();
  at = at - own;
  ClassCounts all{0, 0};
#pragma unroll
  for (int w = 0; w < kListWarps; ++w) {
    const ClassCounts c = s_class[w];
    if (w < warp) at = at + c;
    all = all + c;
  }
  // no list of twice the mean: tile order
  const bool even = all.at(0) + all.at(1) + all.at(2) == 0;
  uint32_t heavier = 0;  // each class begins behind the heavier ones
#pragma unroll
  for (int k = 0; k < kLoadClasses; ++k) {
    at.add(k, heavier);
    heavier += all.at(k);
  }
  const uint32_t w = (uint32_t)p.tile_width;
  uint32_t y = w ? t0 / w : 0u, x = t0 - y * w;
#pragma unroll 4
  for (uint32_t t = t0; t < t1; ++t) {
    const uint2 r = p.ranges[t];
    const int k = load_class(r.y - r.x, mean);
    p.block_tiles[even ? t : base + at.at(k)] = make_uint4(r.x, r.y, y << 16 | x, 0u);
    at.add(k, 1u);
    if (++x == w) x = 0, ++y;
  }
}

// Appends pairs of a bin to the lists of its 32 tiles.  A warp queues its pairs by the bin's four
// tile rows (a pair covers one or two of them on average, so a walk per row would waste most lanes) and
// appends 32 of a row at a time to its eight lists: a pair's place is the list's next one plus the
// queued pairs before it that cover the tile, from a warp scan of the eight columns as bytes.  Bound by
// issue (56 % of the slots) and shared memory (41 %).  Measured on a B200 (1M-Gaussian view / 16-view batch): a block per tile row, walking all of the
// bin's pairs with ballots and popcounts per tile, 88 / 1262 us; byte scans there 75 / 967; this
// 37 / 392 us.
struct FillQueue {
  uint32_t cols[kBinH][64], rec[kBinH][64];  // queued pairs of a row: columns, record
  __align__(16) uint32_t next[32];           // next free place of every tile's list
};

struct ListFill {
  FillQueue& q;
  uint32_t* out;
  uint32_t queued[kBinH] = {};  // pairs queued by row (warp-uniform)

  __device__ __forceinline__ ListFill(FillQueue& queue, uint32_t* out_vals) : q(queue), out(out_vals) {}
  // Begins a bin: the lane's tile's next place.
  __device__ __forceinline__ void begin(uint32_t next) {
    __syncwarp();
    q.next[threadIdx.x & 31] = next;
  }
  // Queues 32 pairs: the tiles m that the lane's one covers (0: none), its record r.  Appends rows that have 32, or
  // with `ends` what there is.  (One place for both: with the rest appended by code of its own, short lists took
  // longer by the time to fetch it.)
  __device__ __forceinline__ void add(uint32_t m, uint32_t r, bool ends) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t least = ends ? 1u : 32u;
#pragma unroll
    for (int row = 0; row < kBinH; ++row) {
      const bool in = (m >> (kBinW + row)) & 1u && (m & 255u);
      const unsigned bal = __ballot_sync(kFullMask, in);
      if (in) {
        const uint32_t at = queued[row] + (uint32_t)__popc(bal & lt);
        q.cols[row][at] = m & 255u;
        q.rec[row][at] = r;
      }
      queued[row] += (uint32_t)__popc(bal);
#pragma unroll 1
      while (queued[row] >= least) {
        append(row, queued[row]);
        queued[row] -= min(queued[row], 32u);
        __syncwarp();
        const uint32_t c = q.cols[row][32 + lane], x = q.rec[row][32 + lane];  // the rest moves to the front
        __syncwarp();
        if ((uint32_t)lane < queued[row]) {
          q.cols[row][lane] = c;
          q.rec[row][lane] = x;
        }
      }
    }
  }
  // Appends the first min(n, 32) pairs queued for a row.
  __device__ __forceinline__ void append(int row, uint32_t n) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const uint32_t m = (uint32_t)lane < n ? q.cols[row][lane] : 0u, rec = q.rec[row][lane];
    uint32_t lo = spread4(m & 15u), hi = spread4(m >> 4);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(kFullMask, lo, o), y = __shfl_up_sync(kFullMask, hi, o);
      if (lane >= o) {
        lo += x;
        hi += y;
      }
    }
    const uint4 n0 = *reinterpret_cast<const uint4*>(&q.next[row * kBinW]);
    const uint4 n1 = *reinterpret_cast<const uint4*>(&q.next[row * kBinW + 4]);
    const uint32_t next[kBinW] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
    const uint32_t all_lo = __shfl_sync(kFullMask, lo, 31), all_hi = __shfl_sync(kFullMask, hi, 31);
    __syncwarp();
    if (lane < kBinW) q.next[row * kBinW + lane] += ((lane < 4 ? all_lo : all_hi) >> (8 * (lane & 3))) & 255u;
#pragma unroll
    for (int k = 0; k < kBinW; ++k)
      if ((m >> k) & 1u) out[next[k] + (((k < 4 ? lo : hi) >> (8 * (k & 3))) & 255u) - 1u] = rec;
  }
};

// Blocks of a fill's launch that order the tiles instead, ahead of the others.
__device__ __forceinline__ uint32_t order_segments(const TileListParams& p) {
  return p.block_tiles ? (p.grid.num_tiles + kOrderTiles - 1) / kOrderTiles : 0u;
}

// The piece that the bin that runs on into piece `at` begins in, by a warp: the piece behind the nearest piece
// boundary before `at` that the bin does not lie across; a search where that is more than 32 pieces back.
__device__ __forceinline__ uint32_t begin_piece(const TileListParams& p, const Pieces& all, uint32_t at, uint32_t bin) {
  const int lane = threadIdx.x & 31;
  const uint32_t j = at - 1u - (uint32_t)lane;  // (wraps below 0: past every piece)
  const bool across = j < at && j > 0 && p.words[all.first(j) - 1u] >> kPairBinShift == bin;
  const unsigned not_across = ~__ballot_sync(kFullMask, across);
  if (not_across) return at - (uint32_t)__ffs(not_across);
  return warp_lower_bound(p.words, all.first(at), bin) / all.len;
}

// Four resident blocks an SM (64 registers).  Measured on a B200, 1M-Gaussian view / 16-view batch: three 77 / 638 us of
// the fine stage, four 71 / 578, five (48 registers, spills) 76 / 595, six 86 / 656.
__global__ void __launch_bounds__(kListThreads, 4) tile_fill_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  __shared__ FillQueue s_queue[kListWarps];
  __shared__ uint32_t s_sum[kListWarps][32], s_own[kListWarps][32], s_bin[kListWarps], s_bases[kMaxBatchViews];
  const uint32_t segments = order_segments(p);
  if (blockIdx.x < segments) return order_tiles(p, blockIdx.x);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pieces all(p);
  load_bases(p.grid, s_bases);
  for (uint32_t block = blockIdx.x - segments; block < all.blocks; block += gridDim.x - segments) {
    const uint32_t piece = block * kListWarps + (uint32_t)warp, begin = all.first(piece), end = all.first(piece + 1);
    auto load = [&](uint32_t e, uint32_t& w, uint32_t& r) {
      w = r = 0;
      if (e < end) {
        w = p.words[e];
        r = p.recs[e];
      }
    };
    uint32_t w0, r0, w1, r1;
    load(begin + lane, w0, r0);
    load(begin + 32 + lane, w1, r1);
    // A bin that runs on into the block: its counts in the pieces before, whole blocks by their sums.
    const uint32_t at = block * kListWarps;
    const uint32_t before = block > 0 ? p.words[all.first(at) - 1u] >> kPairBinShift : kNoBin;
    uint32_t sum = 0;
    if (before == p.words[all.first(at)] >> kPairBinShift) {
      const uint32_t from = begin_piece(p, all, at, before);
      const uint32_t whole = (from + kListWarps - 1u) / kListWarps;  // the first whole block
      if (from + warp < whole * kListWarps) sum = all.slots[32 * (size_t)(from + warp) + lane];
#pragma unroll 4
      for (uint32_t i = whole + warp; i < block; i += kListWarps) sum += all.sums[32 * (size_t)i + lane];
    }
    s_sum[warp][lane] = sum;
    s_own[warp][lane] = piece < all.count ? all.slots[32 * (size_t)piece + lane] : 0u;
    if (lane == 0) s_bin[warp] = begin < end ? p.words[end - 1] >> kPairBinShift : kNoBin;
    __syncthreads();
    ListFill fill(s_queue[warp], p.out_vals);
    bool first = true, safe = false;
    uint32_t rec = 0;
    walk_piece(begin, end, [&](uint32_t e0, uint32_t& after) {
      const uint32_t w = w0;
      rec = r0;
      after = w0 = w1, r0 = r1;
      load(e0 + 64 + lane, w1, r1);
      return w;
    }, [&](uint32_t bin, bool in, uint32_t w, bool begins, bool ends, bool) {
      if (begins) {
        uint32_t t, place = 0, last = 0;
        if (lane_tile(bin_tiles(p.grid, s_bases, bin), t)) {
          const uint2 range = p.ranges[t];
          place = range.x, last = range.y;
        }
        if (first)  // the piece's first bin may have begun in an earlier one
#pragma unroll
          for (int k = 0; k < kListWarps; ++k)
            place += (bin == before ? s_sum[k][lane] : 0u) + (k < warp && s_bin[k] == bin ? s_own[k][lane] : 0u);
        // (always, after a sort whose waits ended; a piece's writes then end in the list, or in the arrays behind it)
        safe = __all_sync(kFullMask, place <= last && last <= (uint64_t)p.capacity);
        first = false;
        fill.begin(place);
      }
      if (safe) fill.add(in ? w : 0u, rec, ends);
    });
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kListThreads) whole_fill_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  __shared__ FillQueue s_queue[kListWarps];
  __shared__ uint32_t s_sum[kListWarps][32], s_own[kListWarps][32];
  const uint32_t segments = order_segments(p);
  if (blockIdx.x < segments) return order_tiles(p, blockIdx.x);
  if (!instances_fit(p.hdr, p.capacity)) return;
  const BinPart b = bin_part(p, blockIdx.x - segments);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the lists' next places: the range's start and the earlier parts' counts, which the warps share
  uint32_t t, next = 0, sum = 0, own = 0;
  bool safe = true;
  if (lane_tile(b.bin, t)) {
    const uint2 range = p.ranges[t];
    next = range.x;
    safe = range.y <= (uint64_t)p.capacity;  // (always, after a consistent scan)
    if (b.parts > 1) {
      const uint32_t* c = p.counts + b.counts0 + (t - b.bin.tile0);
      const uint32_t block = b.part - (uint32_t)warp;  // the block's first part
#pragma unroll 4
      for (uint32_t i = (uint32_t)warp; i < block; i += kListWarps) sum += c[(size_t)i * b.tiles];
      if (b.part < b.parts) own = c[(size_t)b.part * b.tiles];
    }
  }
  s_sum[warp][lane] = sum;
  s_own[warp][lane] = own;
  __syncthreads();
  if (b.part >= b.parts || b.first >= b.end || !__all_sync(kFullMask, safe)) return;
#pragma unroll
  for (int w = 0; w < kListWarps; ++w) next += s_sum[w][lane] + (w < warp ? s_own[w][lane] : 0u);
  ListFill fill(s_queue[warp], p.out_vals);
  fill.begin(next);
  uint32_t mask = 0, rec = 0;
  auto load = [&](uint32_t e) {
    mask = 0;
    if (e < b.end) {
      mask = entry_tiles(p, b.bin, e);
      rec = p.order[e];
    }
  };
  load(b.first + lane);
  uint32_t mask1 = mask, rec1 = rec;  // two groups ahead
  load(b.first + 32 + lane);
  for (uint32_t e0 = b.first; e0 < b.end; e0 += 32) {
    const uint32_t m = mask1, r = rec1;
    mask1 = mask, rec1 = rec;
    load(e0 + 64 + lane);
    const bool last = e0 + 32 >= b.end;
    if (last || __any_sync(kFullMask, covers(m))) fill.add(m, r, last);
  }
}

// The sorted tile ids, which only the inspection of a pass reads: a warp per tile writes its range.
__global__ void __launch_bounds__(256) tile_keys_kernel(const __grid_constant__ TileListParams p) {
  chain_begin();
  const uint32_t tile = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (tile >= p.grid.num_tiles || !instances_fit(p.hdr, p.capacity)) return;
  const uint2 r = p.ranges[tile];
  if (r.y > (uint64_t)p.capacity) return;
  for (uint32_t i = r.x + (threadIdx.x & 31); i < r.y; i += 32) p.out_keys[i] = tile;
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

void launch_histogram(const HistParams& p, bool chained, cudaStream_t s) {
  const unsigned segs = std::max(1u, p.num_segs);
  const int64_t blocks = std::max<int64_t>(
      1, std::min<int64_t>(((int64_t)p.seg_len + 256 * kHistUnroll - 1) / (256 * kHistUnroll),
                           std::max<int64_t>(1, sm_count() * 4 / segs)));
  launch_chained(chained, histogram_kernel, dim3((unsigned)blocks, segs), 256, 0, s, p);
}

void launch_onesweep(const OnesweepParams& p, int64_t max_items, int64_t expected, bool chained, cudaStream_t s) {
  if (p.seg_len && small_sort(p.seg_len, p.num_segs)) {  // (the depth sort: its look-back words have room)
    launch_chained(chained, onesweep_kernel<kSmallSortItems, 5, 16>, (unsigned)sort_blocks(p.seg_len, p.num_segs), kSortThreads, 0, s, p);
    return;
  }
  const int64_t blocks = p.seg_len ? sort_tiles(p.seg_len) * (int64_t)p.num_segs : sort_tiles(max_items);
  if (blocks <= 0) return;
  // The blocks an SM holds: three have all the registers that the ranking wants, five spill.  Tiles that fit one
  // wave of more blocks are better off so; beyond that four measured fastest.  On a B200, the sorts of a
  // 300k / 1M / 3M-Gaussian view / 16-view batch with three, four and five: 89 / 117 / 417 / 1088,
  // 92 / 118 / 408 / 1026 and 104 / 129 / 372 / 1035 us; by this rule 90 / 117 / 382 / 1025.  Five against four within
  // their window: 2.45M Gaussians 212 / 205, 2.7M 358 / 372, 3M at 1024x512 212 / 238, eight views of 350,000 199 / 210.
  // The pairs' number is only known on the device: one and a half a Gaussian are expected.
  const int64_t tiles = p.seg_len ? blocks : sort_tiles(expected), sms = sm_count();
  if (tiles <= 3 * sms)
    launch_chained(chained, onesweep_kernel<kSortItems, 3, kLookbackBatch>, (unsigned)blocks, kSortThreads, 0, s, p);
  else if (tiles > 4 * sms && tiles <= 5 * sms)
    launch_chained(chained, onesweep_kernel<kSortItems, 5, kLookbackBatch>, (unsigned)blocks, kSortThreads, 0, s, p);
  else
    launch_chained(chained, onesweep_kernel<kSortItems, 4, kLookbackBatch>, (unsigned)blocks, kSortThreads, 0, s, p);
}

void launch_rects(const RankParams& p, cudaStream_t s) {
  const int64_t items = (int64_t)p.grid.P * p.grid.V;
  if (items <= 0) return;
  launch_chained(p.chained, rect_kernel, (unsigned)((items + 255) / 256), 256, 0, s, p);
}

void launch_begin_binning(const BeginParams& p, cudaStream_t s) {
  size_t total = 0;
  for (size_t b : p.bytes) total += b / 16;
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((int64_t)(total + 1023) / 1024, (int64_t)sm_count() * 8));
  launch_chained(p.chained, begin_binning_kernel, (unsigned)blocks, 256, 0, s, p);
}

void launch_rank(const RankParams& p, cudaStream_t s) {
  if (p.grid.P <= 0) return;
  const dim3 grid((unsigned)(p.grid.P + kRankItems - 1) / kRankItems, (unsigned)p.grid.V);
  launch_chained(p.chained, rank_kernel, grid, kRankThreads, 0, s, p);
}

void launch_duplicate(const DuplicateParams& p, int64_t expected_pairs, bool chained, cudaStream_t s) {
  const int64_t items = (int64_t)p.grid.P * p.grid.V;
  if (items <= 0) return;
  const int64_t tiles = (items + kScanTile - 1) / kScanTile;
  if (tiles <= (int64_t)p.skip_tiles) return;
  // scan: one block per scan tile that is taken (block k takes tile skip_tiles + k)
  launch_chained(chained, pair_scan_kernel, (unsigned)(tiles - p.skip_tiles), kScanBlock, 0, s, p);
  // emit: a block per kEmitBlock pairs of which there may be three a Gaussian, further ones in turn (with a block per
  // kEmitBlock pairs that the binning buffer can hold, 3M Gaussians' duplicate stage took 187 us instead of 157; with
  // blocks for half as many pairs, 150,000 Gaussians' 40 instead of 31); a probe pass stops after the scan
  if (p.skip_tiles != 0 || p.capacity <= 0) return;
  const int64_t eblocks = emit_blocks(std::min<int64_t>(p.capacity, expected_pairs)) + 1;
  launch_chained(chained, pair_emit_kernel, (unsigned)eblocks, kScanBlock, 0, s, p);
}

void launch_tile_lists(const TileListParams& p, int64_t expected_pairs, cudaStream_t s) {
  const TileGrid& g = p.grid;
  if (g.num_tiles == 0) return;
  const bool whole = p.words == nullptr;
  // The pairs' number is only known on the device: as many blocks as the expected ones fill (three a Gaussian, rather too
  // many: those without a piece end at once), which take further pieces in turn.
  const int64_t pairs = std::min(expected_pairs, p.capacity);
  const int64_t piece = std::min<int64_t>(std::max<int64_t>(pairs / kPieceTarget, kMinPiece), kMaxPiece);
  const unsigned blocks = whole ? g.num_blocks : (unsigned)(pairs / (piece * kListWarps) + 1);
  launch_chained(p.chained, whole ? whole_count_kernel : tile_count_kernel, blocks, kListThreads, 0, s, p);
  const unsigned scan = p.totals ? (g.num_tiles + kTileScanBlock - 1) / kTileScanBlock : 1u;
  launch_chained(p.chained, tile_scan_kernel, scan, kTileScanThreads, 0, s, p);
  const unsigned order = p.block_tiles ? (g.num_tiles + kOrderTiles - 1) / kOrderTiles : 0u;
  launch_chained(p.chained, whole ? whole_fill_kernel : tile_fill_kernel, blocks + order, kListThreads, 0, s, p);
  launch_chained(p.chained, tile_keys_kernel, (g.num_tiles + 7) / 8, 256, 0, s, p);
}

}  // namespace omnigs
