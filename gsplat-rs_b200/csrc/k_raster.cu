// K4: per-tile raster. Built with --fmad=false; every fused multiply-add is
// an explicit fmaf, so a C++ restatement reproduces each pixel bit for bit.
//
// One block per tile; one thread per pixel, or two pixels of one column per
// thread for FP32 on 16x16 tiles (GSR_RASTER_PX, default 2). The tile's
// splat list (reference back-to-front order restricted to the tile, found in
// its bin's list) is staged into shared memory in chunks of records with cp.async (16-byte
// async copies, the record gather is random so tiled TMA does not apply),
// double-buffered so the next chunk's gather overlaps the current chunk's
// blending.
//
// Per pixel, the fragment rule of the reference shader
// (crates/gsplat-render-wgpu/shaders/splat_surface_direct.wgsl:336-369):
// local = inverse axis matrix * (pixel - centre); discard unless
// |local.x|, |local.y| <= s (the quad), r^2 = |local|^2 <= 1, and
// w = alpha * exp(-4.5 r^2) > 1/256; the source is (premult rgb * g, w).
//   FP32 mode: front to back (walks the list from its end); coverage is
//     r^2 <= s^2 and r^2 below the bound where w = 1/256 (in exact arithmetic
//     the same set as the quad clip, r^2 <= 1 and the alpha threshold);
//     C += rgb * (w T), T -= w T;
//     a pixel finishes once T < 1e-4, a warp when all its pixels have, the
//     block stops loading once all are done.
//   UNORM8 mode: back to front, dst = src + dst * (1 - w) rounded to UNORM8
//     after every splat (the reference's Rgba8Unorm premultiplied blend).

#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "bins.cuh"
#include "device_common.cuh"
#include "kernels.h"

#ifndef GSR_RASTER_PX
#define GSR_RASTER_PX 2
#endif
// Paired FP32 arithmetic for the two pixels of a thread (f32x2).
#ifndef GSR_RASTER_F32X2
#define GSR_RASTER_F32X2 1
#endif
namespace gsr {
namespace {

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Block 0 folds the frame's error and overflow bits into the sticky word
// that gsplat_context_sync reports for enqueued frames, and writes the run's
// counters, all final before the raster, to pinned host memory: beside the
// raster instead of two copies behind it (a synchronous frame of 279 k splats
// at 1920x1080 305 -> 284 us; with the phases timed by the kernels' own clock
// readings instead of seven events 238).
__device__ __forceinline__ void publish_counters(const RasterArgs &a) {
  if (blockIdx.x != 0) return;
  static_assert(sizeof(FrameCounters) % 4 == 0 && sizeof(ViewCounters) % 4 == 0, "word copies");
  constexpr uint32_t kSticky = offsetof(FrameCounters, sticky) / 4;
  constexpr uint32_t kEnd = offsetof(FrameCounters, phase_ns[6]) / 4;
  if (threadIdx.x == 0) a.counters->phase_ns[5] = global_ns();
  __syncthreads();
  const uint32_t *from = reinterpret_cast<const uint32_t *>(a.counters);
  uint32_t *to = reinterpret_cast<uint32_t *>(a.host_counters);
  for (uint32_t i = threadIdx.x; i < sizeof(FrameCounters) / 4; i += blockDim.x)
    if (i != kSticky && i / 2 != kEnd / 2) to[i] = from[i];
  from = reinterpret_cast<const uint32_t *>(a.view_counters);
  to = reinterpret_cast<uint32_t *>(a.host_views);
  for (uint32_t i = threadIdx.x; i < a.num_views * (sizeof(ViewCounters) / 4); i += blockDim.x)
    to[i] = from[i];
  if (threadIdx.x == 0) {
    uint32_t sticky = *a.sticky;
    const uint32_t bits = a.counters->error | (a.counters->overflow ? 0x80000000u : 0u);
    if (bits) {
      sticky |= bits;
      *a.sticky = sticky;
    }
    a.host_counters->sticky = sticky;
  }
}

// The last block to come here notes the raster's end for the host. (Not where
// nothing reports it: the counter's answer keeps a block a little longer, 48
// mixed views 6,198 -> 6,229 us.)
__device__ __forceinline__ void note_end(const RasterArgs &a) {
  if (a.end_ns && threadIdx.x == 0 && atomicAdd(&a.counters->raster_done, 1u) + 1 == gridDim.x)
    *a.end_ns = global_ns();
}

// The coverage bound of an entry: w > 1/256 exactly when r2 < (log2 alpha +
// 8) / (4.5 log2 e), so a pixel is covered when r2 is at most the largest
// float below that bound, capped at s^2 (nothing is covered when the bound is
// not positive).
__device__ __forceinline__ float coverage_bound(float log2_alpha, float s) {
  const float s2 = s * s;
  const float wlim = __fdiv_rn(log2_alpha + 8.0f, 6.49212768f);
  return wlim > 0.0f ? fminf(s2, __int_as_float(__float_as_int(wlim) - 1)) : -1.0f;
}

// Which warp blocks (8 columns, kRows rows) of a kTile x kTile tile the
// ellipse |local|^2 <= thr reaches (bit band * kTile/8 + column block): for
// each band of kRows rows, the x-interval the ellipse spans within the band,
// plus half a pixel on every side, tested against the 8-column blocks. q(dx, dy) =
// A dx^2 + 2B dx dy + C dy^2 is |local|^2 in pixel units; (cxl, cyl) is the
// centre relative to the tile's first pixel. The mask only culls: hardware
// reciprocal/rsqrt (a few ulp) plus an inflation of the extents far above
// their error keeps it conservative.
template <int kTile, int kRows>
__device__ __forceinline__ uint32_t ellipse_block_mask(float4 ra, float4 rb, float thr, float cxl,
                                                       float cyl) {
  constexpr int kBlocksX = kTile / 8;
  constexpr int kWarps = kTile * kTile / (8 * kRows);
  const float qa = fmaf(ra.z, ra.z, rb.x * rb.x);
  const float qb = fmaf(ra.z, ra.w, rb.x * rb.y);
  const float qc = fmaf(ra.w, ra.w, rb.y * rb.y);
  const float det = fmaf(qa, qc, -qb * qb);
  const float inv_a = __fdividef(1.0f, qa);
  const float inv_det = __fdividef(1.0f, det);
  const float hx2 = thr * qc * inv_det, hy2 = thr * qa * inv_det;
  const float hx_raw = hx2 * rsqrtf(fmaxf(hx2, 1e-30f));
  const float hx = fmaf(hx_raw, 1.0001f, 1e-3f);
  const float hy = fmaf(hy2 * rsqrtf(fmaxf(hy2, 1e-30f)), 1.0001f, 1e-3f);
  // dy of the leftmost point (rightmost at -dy_left), from the unpadded extent
  const float dy_left = qb * hx_raw * __fdividef(1.0f, qc);
  const float s2a = thr * qa;
  constexpr float kPad = 0.5f + 1.0f / 64.0f;
  uint32_t mask = 0;
#pragma unroll
  for (int band = 0; band < kTile / kRows; ++band) {
    const float lo = fmaxf((float)(kRows * band) - 0.5f - cyl, -hy);
    const float hi = fminf((float)(kRows * band + kRows) - 0.5f - cyl, hy);
    if (!(lo <= hi)) continue;
    const float qlo = fmaxf(s2a - det * lo * lo, 0.0f), qhi = fmaxf(s2a - det * hi * hi, 0.0f);
    const float r_lo = fmaf(qlo * rsqrtf(fmaxf(qlo, 1e-30f)), 1.0001f, 1e-3f);
    const float r_hi = fmaf(qhi * rsqrtf(fmaxf(qhi, 1e-30f)), 1.0001f, 1e-3f);
    float xmin = fminf((-qb * lo - r_lo) * inv_a, (-qb * hi - r_hi) * inv_a);
    float xmax = fmaxf((-qb * lo + r_lo) * inv_a, (-qb * hi + r_hi) * inv_a);
    if (dy_left >= lo && dy_left <= hi) xmin = -hx;
    if (-dy_left >= lo && -dy_left <= hi) xmax = hx;
    const float bx0f = cxl + xmin - kPad, bx1f = cxl + xmax + kPad;
#pragma unroll
    for (int colb = 0; colb < kBlocksX; ++colb)
      if (bx1f >= (float)(8 * colb) && bx0f <= (float)(8 * colb + 7))
        mask |= 1u << (band * kBlocksX + colb);
  }
  // A degenerate conic (never expected: axes are clamped to an anisotropy of
  // 64) falls back to every block.
  if (!(det > 0.0f) || !(hx < 3.0e38f) || !(hy < 3.0e38f)) mask = (1u << kWarps) - 1u;
  if (!(thr >= 0.0f)) mask = 0;
  return mask;
}

// The chunk entries each warp's block reaches, one bit per entry (word v:
// entries 32 v .. 32 v + 31): kBlocks ballots by the warp that prepared them.
template <int kBlocks, int kWords>
__device__ __forceinline__ void share_mask(uint32_t mask, uint32_t word,
                                           uint32_t (&bits)[kBlocks][kWords]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (uint32_t blk = 0; blk < (uint32_t)kBlocks; ++blk) {
    const uint32_t bal = __ballot_sync(0xffffffffu, (mask >> blk) & 1u);
    if (lane == blk) bits[blk][word] = bal;
  }
}

// Ordered list of a warp's entries, as base + 16 k for entry k (a float4
// array's byte offsets); returns their count.
template <int kWords>
__device__ __forceinline__ uint32_t list_entries(const uint32_t (&bits)[kWords], uint32_t base,
                                                 uint32_t *list) {
  const uint32_t lane = threadIdx.x & 31, lt = lanemask_lt();
  uint32_t n = 0;
#pragma unroll
  for (uint32_t v = 0; v < (uint32_t)kWords; ++v) {
    const uint32_t w = bits[v];
    if ((w >> lane) & 1u) list[n + __popc(w & lt)] = base + 16 * (32 * v + lane);
    n += __popc(w);
  }
  __syncwarp();
  return n;
}

// The view of global tile `tile` (every thread of the block calls it).
__device__ __forceinline__ uint32_t block_view(const RasterArgs &a, uint32_t tile,
                                               uint32_t &shared) {
  if (a.num_views == 1) return 0;
  if (threadIdx.x == 0)
    shared = find_view(a.num_views, tile, [&](uint32_t v) { return a.views[v].tile_base; });
  __syncthreads();
  return shared;
}

// Position of the n-th set bit (n from 0) of a word that has more than n.
__device__ __forceinline__ uint32_t nth_bit(uint32_t word, uint32_t n) {
  uint32_t at = 0;
#pragma unroll
  for (uint32_t width = 16; width >= 1; width >>= 1) {
    const uint32_t low = __popc((word >> at) & ((1u << width) - 1u));
    if (n >= low) {
      n -= low;
      at += width;
    }
  }
  return at;
}

// A tile's walk of its bin's list (bins.cuh): gathers the next kChunk entries
// that have the tile, in list order (from the end when kFromEnd). The range
// build has left one word per tile and 32 list positions (bit i: position
// 32 w + i has the tile). Every warp reads the same 32 words (1,024
// positions), one per lane, and scans their bit counts; a thread then finds
// the word and the bit of its own slots. No warp waits for another: a version
// that split the words over the warps took two block barriers a step.
template <int kThreads, int kChunk, bool kFromEnd>
struct BinScan {
  struct Smem {};
  uint32_t in_bin;      // the tile within its bin; bit 31: the sort's result is in buffer 0
  uint32_t begin, end;  // the list positions left

  // (tx, ty): the tile within its view
  __device__ __forceinline__ BinScan(const RasterArgs &a, uint32_t bin_base, uint32_t tx,
                                     uint32_t ty, uint32_t tiles_x) {
    const uint32_t bin = bin_base + (ty / kBinEdge) * bins_along(tiles_x) + tx / kBinEdge;
    const uint2 range = a.ranges[bin];
    in_bin = (ty % kBinEdge) * kBinEdge + tx % kBinEdge;
    if (a.plan->final_buffer == 0) in_bin |= 1u << 31;
    begin = range.x;
    end = range.y;
  }

  __device__ __forceinline__ void prime(const RasterArgs &, Smem &) {}

  // Starts the gather of the next chunk's records into raw (16-byte async copies,
  // entry s in slot s) and calls each(gid, record) for them; returns their
  // number (0: the list is done). Every thread of the block calls it.
  template <typename F>
  __device__ __forceinline__ uint32_t next(const RasterArgs &a, Smem &, float4 (&raw)[3][kChunk],
                                           F each) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t filled = 0;
    while (filled < (uint32_t)kChunk && begin < end) {
      const uint32_t first = begin >> 5, last = (end - 1) >> 5;
      const uint32_t w0 = kFromEnd ? last : first, w = kFromEnd ? w0 - lane : w0 + lane;
      uint32_t bits = 0;
      if (lane <= last - first) {
        const uint32_t *words = in_bin >> 31 ? a.keys1 : a.keys0;
        bits = __ldg(&words[tile_word(w, in_bin & 15u)]);
        if (w == first) bits &= ~0u << (begin & 31u);
        if (w == last) bits &= ~0u >> (31u - ((end - 1) & 31u));
        if (kFromEnd) bits = __brev(bits);  // bit i: position 32 w + 31 - i
      }
      const uint32_t mine = __popc(bits);
      uint32_t inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
      // list position of the step's n-th entry (n < total); all lanes call it
      auto position = [&](uint32_t n) {
        uint32_t c = 0;  // the first lane whose inclusive count exceeds n
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1)
          if (__shfl_sync(0xffffffffu, inc, c + step - 1) <= n) c += step;
        const uint32_t word = __shfl_sync(0xffffffffu, bits, c);
        const uint32_t before = __shfl_sync(0xffffffffu, inc - mine, c);
        const uint32_t bit = nth_bit(word, n - before);
        return kFromEnd ? 32 * (w0 - c) + 31 - bit : 32 * (w0 + c) + bit;
      };
      const uint32_t room = (uint32_t)kChunk - filled, taken = min(total, room);
#pragma unroll
      for (uint32_t t0 = 0; t0 < (uint32_t)kChunk; t0 += kThreads) {
        // this thread's slot, if the step fills any of the warp's
        const uint32_t slot = t0 + threadIdx.x, n = slot - filled;
        const bool in = slot >= filled && n < taken;
        if (!__any_sync(0xffffffffu, in)) continue;
        const uint32_t pos = position(in ? n : 0u);
        if (in) {
          const uint32_t gid = __ldg(&(in_bin >> 31 ? a.ids0 : a.ids1)[pos]);
          const Record *r = &a.records[gid];
          cp_async16(&raw[0][slot], &r->a);
          cp_async16(&raw[1][slot], &r->b);
          cp_async16(&raw[2][slot], &r->c);
          each(gid, r);
        }
      }
      // behind the last entry taken, or behind the step's words
      if (total > room) {
        const uint32_t pos = position(room);
        if (kFromEnd) end = pos + 1;
        else begin = pos;
      } else if (last - first < 32u) {
        begin = end;
      } else if (kFromEnd) {
        end = 32 * (last - 31);
      } else {
        begin = 32 * (first + 32);
      }
      filled += taken;
    }
    return filled;
  }
};

// The same walk with its chain of loads, words -> ids -> records, spread over
// three chunks: locate() starts the copies of the ids of the chunk after next
// and of the words behind them, next() those of the records whose ids have
// arrived. A window is 128 words, four to a lane. It costs more instructions
// than BinScan and gathers ids that an early end does not need, so it pays
// where a tile's own latency sets the time and not the throughput of many
// (2 M splats on 475 tiles 72 -> 55 us at equal registers; 186 M pairs at 3840x2160
// 397 -> 463).
template <int kThreads, int kChunk, bool kFromEnd>
struct BinScanAhead {
  static constexpr uint32_t kNone = 0x80000000u;  // no window has this number
  struct Smem {
    uint4 window[4][32];  // window W's words in slot W % 4
    uint32_t ids[kChunk];
  };
  uint32_t in_bin;      // the tile within its bin; bit 31: the sort's result is in buffer 0
  uint32_t begin, end;  // the list
  uint32_t window;      // the next entry's window, kNone when the list is done
  uint32_t used;        // entries of the window already taken
  uint32_t staged;      // this window and the next are in shared memory, or kNone
  uint32_t located;     // entries of the next chunk

  // (tx, ty): the tile within its view
  __device__ __forceinline__ BinScanAhead(const RasterArgs &a, uint32_t bin_base, uint32_t tx,
                                          uint32_t ty, uint32_t tiles_x) {
    const uint32_t bin = bin_base + (ty / kBinEdge) * bins_along(tiles_x) + tx / kBinEdge;
    const uint2 range = a.ranges[bin];
    in_bin = (ty % kBinEdge) * kBinEdge + tx % kBinEdge;
    if (a.plan->final_buffer == 0) in_bin |= 1u << 31;
    begin = range.x;
    end = range.y;
    used = 0;
    window = begin < end ? (kFromEnd ? end - 1 : begin) >> 12 : kNone;
    staged = kNone;
  }

  __device__ __forceinline__ const uint4 *words(const RasterArgs &a, uint32_t w) const {
    return reinterpret_cast<const uint4 *>(
        &(in_bin >> 31 ? a.keys1 : a.keys0)[tile_word(w, in_bin & 15u)]);
  }
  // Whether any of the positions of words w .. w + 3 is in the list.
  __device__ __forceinline__ bool in_list(uint32_t w) const {
    return w >= (begin >> 7 << 2) && 32 * w < end;
  }

  // Starts the copies of the next chunk's ids (slot s's by the thread that
  // gathers it) and returns their number (0: the list is done). Every thread
  // of the block calls it, with a block barrier between two calls.
  __device__ __forceinline__ uint32_t locate(const RasterArgs &a, Smem &sm) {
    if (window == kNone) return 0;
    const uint32_t lane = threadIdx.x & 31, quad = kFromEnd ? 31 - lane : lane;
    const uint32_t was = staged;
    uint32_t filled = 0;
    while (filled < (uint32_t)kChunk && window != kNone) {
      const uint32_t w = 128 * window + 4 * quad;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (in_list(w)) {
        const uint32_t ahead = kFromEnd ? was - window : window - was;
        v = was != kNone && ahead < 2 ? sm.window[window & 3][quad] : __ldg(words(a, w));
      }
      uint32_t bits[4] = {v.x, v.y, v.z, v.w};
      if (4096 * window < begin || end - 4096 * window < 4096) {  // an end of the list
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          const uint32_t p = 32 * (w + q);
          if (p < begin) bits[q] &= begin - p >= 32 ? 0u : ~0u << (begin - p);
          if (p >= end) bits[q] = 0u;
          else if (end - p < 32) bits[q] &= (1u << (end - p)) - 1u;
        }
      }
      if (kFromEnd) {  // bit i of word q: position 32 (w + 3 - q) + 31 - i
        const uint32_t b0 = __brev(bits[0]), b1 = __brev(bits[1]);
        bits[0] = __brev(bits[3]), bits[1] = __brev(bits[2]);
        bits[2] = b1, bits[3] = b0;
      }
      // counts of the words before words 1, 2, 3 and of all four, one per byte
      uint32_t pre = __popc(bits[0]);
      pre |= (pre + __popc(bits[1])) << 8;
      pre |= ((pre >> 8) + __popc(bits[2])) << 16;
      pre |= ((pre >> 16) + __popc(bits[3])) << 24;
      uint32_t inc = pre >> 24;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
      const uint32_t taken = min(total - used, (uint32_t)kChunk - filled);
#pragma unroll
      for (uint32_t t0 = 0; t0 < (uint32_t)kChunk; t0 += kThreads) {
        // this thread's slot, if the window fills any of the warp's
        const uint32_t slot = t0 + threadIdx.x;
        const bool in = slot >= filled && slot - filled < taken;
        if (!__any_sync(0xffffffffu, in)) continue;
        const uint32_t n = in ? slot - filled + used : 0u;
        uint32_t c = 0;  // the first lane whose inclusive count exceeds n
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1)
          if (__shfl_sync(0xffffffffu, inc, c + step - 1) <= n) c += step;
        const uint32_t cp = __shfl_sync(0xffffffffu, pre, c);
        uint32_t r = n + (cp >> 24) - __shfl_sync(0xffffffffu, inc, c);
        uint32_t word = __shfl_sync(0xffffffffu, bits[0], c);
        uint32_t q = 0, before = 0;
#pragma unroll
        for (uint32_t k = 1; k < 4; ++k) {
          const uint32_t wk = __shfl_sync(0xffffffffu, bits[k], c);
          const uint32_t pk = (cp >> (8 * (k - 1))) & 255u;
          if (r >= pk) q = k, word = wk, before = pk;
        }
        if (in) {
          const uint32_t at = 32 * q + nth_bit(word, r - before);
          const uint32_t pos =
              4096 * window + (kFromEnd ? 4095 - (128 * c + at) : 128 * c + at);
          cp_async4(&sm.ids[slot], &(in_bin >> 31 ? a.ids0 : a.ids1)[pos]);
        }
      }
      filled += taken;
      used += taken;
      if (used == total) {
        used = 0;
        const bool last = kFromEnd ? window == begin >> 12 : window == (end - 1) >> 12;
        window = last ? kNone : kFromEnd ? window - 1 : window + 1;
      }
    }
    // The cursor's window and the one behind it go to shared memory for the
    // next call. Other warps may still read the two that were there: two
    // windows further at most, the four slots keep them apart.
    if (window != kNone) {
      const uint32_t ahead = kFromEnd ? was - window : window - was;
      if (was != kNone && ahead > 2) {
        staged = kNone;
      } else {
        staged = window;
        const uint32_t have = was == kNone || ahead == 2 ? 0 : 2 - ahead;
        if (threadIdx.x < 32)
          for (uint32_t k = have; k < 2; ++k) {
            const uint32_t win = kFromEnd ? window - k : window + k;
            const uint32_t w = 128 * win + 4 * lane;
            if (win < kNone && in_list(w)) cp_async16(&sm.window[win & 3][lane], words(a, w));
          }
      }
    }
    return filled;
  }

  // The first chunk's ids, which the first next() gathers by.
  __device__ __forceinline__ void prime(const RasterArgs &a, Smem &sm) {
    located = locate(a, sm);
    cp_async_wait_all();
    __syncthreads();
  }

  // As BinScan's. Between two calls every thread waits for its copies and
  // then for the block.
  template <typename F>
  __device__ __forceinline__ uint32_t next(const RasterArgs &a, Smem &sm,
                                           float4 (&raw)[3][kChunk], F each) {
    const uint32_t n = located;
#pragma unroll
    for (uint32_t t0 = 0; t0 < (uint32_t)kChunk; t0 += kThreads) {
      const uint32_t slot = t0 + threadIdx.x;
      if (slot < n) {
        const uint32_t gid = sm.ids[slot];
        const Record *r = &a.records[gid];
        cp_async16(&raw[0][slot], &r->a);
        cp_async16(&raw[1][slot], &r->b);
        cp_async16(&raw[2][slot], &r->c);
        each(gid, r);
      }
    }
    located = locate(a, sm);
    return n;
  }
};

// UNORM8 parity mode: back to front over the tile list (forwards), the
// reference fragment rule with the quad clip, and the premultiplied OVER
// blend rounded to UNORM8 after every splat, exactly as the oracle's
// reference image model evaluates it. The blend has no early exit (a pixel's
// final value depends on every splat behind it), so the work it saves is
// culling: threads map to 8x4-pixel warp blocks as in the FP32 mode, one
// thread per chunk entry forms the entry's premultiplied colour (rgb * alpha,
// the vertex stage's product) and a conservative mask of the warp blocks the
// ellipse reaches (r^2 <= s^2, widened by a relative 1e-5 and an absolute
// 1e-6: alpha e^(-4.5 r^2) > 1/256 holds only below s^2 up to rounding), and
// each warp walks only the entries whose mask has its bit. A channel keeps
// its stored byte t as f = RN(t / 255), the float the next blend reads.
template <int kTile, bool kAhead>
struct U8Smem {
  static constexpr int kThreads = kTile * kTile;
  static constexpr int kWarps = kThreads / 32;
  static constexpr int kChunk = kTile == 16 || kAhead ? 256 : 128;
  using Scan = std::conditional_t<kAhead, BinScanAhead<kThreads, kChunk, false>,
                                  BinScan<kThreads, kChunk, false>>;
  float4 raw[2][3][kChunk];  // (cx, cy, ax, ay), (bx, by, s, alpha), premultiplied rgb
  typename Scan::Smem scan;
  alignas(16) uint32_t list[kWarps][kChunk];  // read by pairs
  uint32_t bits[kWarps][kChunk / 32];
  uint32_t view;
};

// RN(t / 255) for integer t in [0, 255] as t * 2^-8 + t * (1/255 - 2^-8)
// in one fma: exact for every such t (the first product is exact and the
// second's rounding never moves the sum across a rounding boundary), in two
// instructions instead of a division.
constexpr float kInv255Lo = 0x1.010102p-16f;  // RN(1/255 - 2^-8)

// Paired FP32 arithmetic, one instruction for two values, each component
// rounded as the scalar operation. Products and sums go through the fused
// form with a neutral third operand (x * y + -0 and x * 1 + y round once, to
// the product and the sum), so nothing is left to contract.
__device__ __forceinline__ float2 pair(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 mul2(float2 x, float2 y) {
  return __ffma2_rn(x, y, pair(-0.0f));
}
__device__ __forceinline__ float2 add2(float2 x, float2 y) {
  return __ffma2_rn(x, pair(1.0f), y);
}

// Two channels' blend step, dst = to_unorm8(fma(dst / 255, 1 - w, src)):
// saturate, scale by 255 and round to the nearest integer t (ties to even) by
// the 1.5 * 2^23 addition, then f = RN(t / 255), the float the next step
// reads. The kernel is bound by the FMA pipes (63% busy at 89% of the issue
// slots with scalar arithmetic throughout, 70% at 76% with pairs throughout):
// a pair takes both pipes, so it saves issue slots and no pipe time, and the
// fastest mix leaves the saturating step (a scalar modifier, two minima
// otherwise) and the coverage scalar. 1920x1080, 279 k splats: the raster takes
// 505 us with scalar steps and 480 as here; paired throughout it was 4% slower
// than this mix.
__device__ __forceinline__ float2 unorm8_step(float2 f, float om, float2 src) {
  const float2 v = make_float2(__saturatef(__fmaf_rn(f.x, om, src.x)),
                               __saturatef(__fmaf_rn(f.y, om, src.y)));
  const float2 t = add2(add2(mul2(v, pair(255.0f)), pair(kRoundMagic)), pair(-kRoundMagic));
  return __ffma2_rn(t, pair(0x1p-8f), mul2(t, pair(kInv255Lo)));
}

// 16x16 tiles: compiled for 4 resident blocks per SM (up to 64 registers a
// thread), which measured 2% faster than 5 blocks at 48 registers; weights of
// two entries are in flight a step (four at 3 or 2 blocks: 514 -> 516 us,
// 1920x1080 with 1.70 M pairs). 8x8 tiles keep four in flight at 12 blocks
// (279 k splats at 1280x720: 349 -> 317 us). kAhead: few tiles (up to 4 of
// 16x16 a SM), where the tile with the longest list sets the time and a warp of it is
// bound by its own chain of latencies: four entries in flight at half the
// blocks, chunks of 256 and a list walked ahead (144 tiles of 187 k splats
// 670 -> 594 us, 608 tiles of 8x8 and 258 k splats 807 -> 583).
template <int kTile, bool kAhead>
__global__ void __launch_bounds__(kTile *kTile, kTile == 16 ? (kAhead ? 2 : 4) : (kAhead ? 8 : 12))
    raster_unorm8_kernel(RasterArgs a) {
  using Smem = U8Smem<kTile, kAhead>;
  constexpr int kN = Smem::kChunk;
  constexpr int kThreads = Smem::kThreads;
  constexpr int kBlocksX = kTile / 8;
  __shared__ Smem sm;
  publish_counters(a);
  const uint32_t tile = blockIdx.x;
  const uint32_t view = block_view(a, tile, sm.view);
  const uint32_t width = a.views[view].p.width, height = a.views[view].p.height;
  const uint32_t tiles_x = a.views[view].p.tiles_x;
  uint32_t *__restrict__ image = a.images + a.views[view].image_base;
  const uint32_t local_tile = tile - a.views[view].tile_base;
  const uint32_t tx = local_tile % tiles_x, ty = local_tile / tiles_x;
  const uint32_t x0 = tx * kTile, y0 = ty * kTile;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t px = x0 + (warp % kBlocksX) * 8 + (lane & 7);
  const uint32_t py = y0 + (warp / kBlocksX) * 4 + (lane >> 3);
  const bool inside = px < width && py < height;
  const float fpx = (float)px, fpy = (float)py;
  const float ftx = (float)x0, fty = (float)y0;
  typename Smem::Scan scan(a, a.views[view].bin_base, tx, ty, tiles_x);
  auto fill = [&](int buf) {
    return scan.next(a, sm.scan, sm.raw[buf], [](uint32_t, const Record *) {});
  };
  // j is the entry's byte offset in raw, its first float4
  auto at = [&](uint32_t j, uint32_t q) {
    return *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(sm.raw) + j +
                                             q * (uint32_t)(16 * kN));
  };
  // Coverage and weight of entry j at this pixel (the reference fragment
  // rule), branch-free: a discarded fragment gets g = 0 and w = 0, a step that
  // leaves the stored value bit for bit as it is (rint(f * 255) = t and
  // RN(t / 255) = f for every stored t).
  auto weight = [&](uint32_t j, float &g, float &w) {
    const float4 d0 = at(j, 0);
    const float4 d1 = at(j, 1);
    const float dpx = __fsub_rn(fpx, d0.x), dpy = __fsub_rn(fpy, d0.y);
    const float lx = __fmaf_rn(d0.z, dpx, __fmul_rn(d0.w, dpy));
    const float ly = __fmaf_rn(d1.x, dpx, __fmul_rn(d1.y, dpy));
    const float r2 = __fmaf_rn(lx, lx, __fmul_rn(ly, ly));
    // the exponential's argument stays in its domain [-4.5, 0]
    const float gg = exp_neg(__fmul_rn(-4.5f, fminf(r2, 1.0f)));
    const float ww = __fmul_rn(d1.w, gg);
    const bool cov = fabsf(lx) <= d1.z && fabsf(ly) <= d1.z && r2 <= 1.0f && ww > 1.0f / 256.0f;
    g = cov ? gg : 0.0f;
    w = cov ? ww : 0.0f;
  };
  float2 rg = pair(0.0f), ba = pair(0.0f);
  auto blend = [&](uint32_t j, float g, float w) {
    const float4 pc = at(j, 2);
    const float om = __fsub_rn(1.0f, w);
    rg = unorm8_step(rg, om, mul2(make_float2(pc.x, pc.y), pair(g)));
    ba = unorm8_step(ba, om, make_float2(__fmul_rn(pc.z, g), w));
  };
  scan.prime(a, sm.scan);
  uint32_t n_in = fill(0);
  for (int buf = 0; n_in; buf ^= 1) {
    // every thread's records have landed, and the chunk before is blended
    cp_async_wait_all();
    __syncthreads();
    const uint32_t n_next = fill(buf ^ 1);
#pragma unroll
    for (uint32_t e = tid; e < (uint32_t)kN; e += kThreads) {
      uint32_t mask = 0;
      if (e < n_in) {
        const float4 ra = sm.raw[buf][0][e], rb = sm.raw[buf][1][e], rc = sm.raw[buf][2][e];
        sm.raw[buf][2][e] = make_float4(__fmul_rn(rc.x, rb.w), __fmul_rn(rc.y, rb.w),
                                        __fmul_rn(rc.z, rb.w), 0.0f);
        const float thr = __fmaf_rn(__fmul_rn(rb.z, rb.z), 1.00001f, 1e-6f);
        mask = ellipse_block_mask<kTile, 4>(ra, rb, thr, ra.x - ftx, ra.y - fty);
      }
      share_mask(mask, e / 32, sm.bits);
    }
    __syncthreads();
    uint32_t *list = sm.list[warp];
    const uint32_t n_w = list_entries(sm.bits[warp], buf * (uint32_t)sizeof(sm.raw[0]), list);
    if (inside) {
      uint32_t i = 0;
      // several entries per step: the later ones' coverage and weight do not
      // wait for the first's blend
      constexpr int kStep = kAhead || kTile == 8 ? 4 : 2;
      for (; i + (kStep - 1) < n_w; i += kStep) {
        uint32_t jj[kStep];
        float g[kStep], w[kStep];
#pragma unroll
        for (int k = 0; k < kStep; k += 2) {
          const uint2 two = *reinterpret_cast<const uint2 *>(&list[i + k]);
          jj[k] = two.x, jj[k + 1] = two.y;
        }
#pragma unroll
        for (int k = 0; k < kStep; ++k) weight(jj[k], g[k], w[k]);
#pragma unroll
        for (int k = 0; k < kStep; ++k) blend(jj[k], g[k], w[k]);
      }
      auto one = [&]() {
        float g, w;
        weight(list[i], g, w);
        blend(list[i], g, w);
      };
      if constexpr (kStep == 2) {
        if (i < n_w) one();
      } else {
        for (; i < n_w; ++i) one();
      }
    }
    n_in = n_next;
  }
  // f = RN(t / 255) of a byte t gives t back
  if (inside)
    image[(size_t)py * width + px] = to_unorm8(rg.x) | (to_unorm8(rg.y) << 8) |
                                     (to_unorm8(ba.x) << 16) | (to_unorm8(ba.y) << 24);
  note_end(a);
}

// Resident blocks per SM the FP32 kernel is compiled for with more tiles than
// are resident: 8 blocks of 4 warps fit 64 registers a thread; 6 or 7 without
// spills run slower (1.70 M pairs at 1920x1080: 122.9 and 118.8 us against
// 114.8), and so do 10 or 12, which spill (122.8, 122.9). 8x8 tiles: 16
// blocks of 2 warps (279 k splats at 1280x720: 111 us with the 9 that 97
// registers allow, 92 here).
template <int kTile>
constexpr int kManyBlocks = kTile == 16 ? 8 : 16;

// FP32 front-to-back mode. kPx = 1: threads map to 8x4-pixel warp blocks
// (lane l of warp w covers column (w % (kTile/8))*8 + (l & 7), row
// (w / (kTile/8))*4 + (l >> 3)). kPx = 2 (16x16 tiles): warp w covers the
// 8x8 block at column block w & 1, row block w >> 1, lane l the pixels of
// column l & 7 in its rows l >> 3 and 4 + (l >> 3): the entry's three shared
// loads serve two pixels, and each pixel still evaluates the same expressions
// as with kPx = 1. 8x8 blocks cull better than the 16x4 bands of two pixels
// in a row (11% fewer pixel evaluations for small splats) and need one mask
// bit for every two of 8x4. Per chunk of kChunk list entries:
//   1. raw records arrive by cp.async (double-buffered, next chunk in flight);
//   2. one thread per entry derives, for this tile, the local offsets ox, oy
//      (local = (ax*lx + ay*ly + ox, bx*lx + by*ly + oy) for pixel coordinates
//      relative to the 16-pixel grid corner), the coverage bound, and a bit
//      mask of the warps' blocks the ellipse |local|^2 <= bound reaches (band
//      intervals plus half a pixel), shared as one word of ballots per warp
//      block and 32 entries;
//   3. each warp lists the entries of its words (in list order) and blends
//      only those; a pixel stops at
//      T < 1e-4, a warp when all its pixels have, the block when all pixels
//      have.
// Culling is conservative, so results equal the unculled per-pixel walk, and
// neither the chunk size, the pixels per thread nor the tile order changes
// any pixel.
template <int kTile, int kChunk, int kPx, bool kAhead>
struct Fp32Smem {
  static_assert(kPx == 1 || (kPx == 2 && kTile == 16), "two pixels per thread on 16x16 tiles");
  static constexpr int kThreads = kTile * kTile / kPx;
  static constexpr int kWarps = kThreads / 32;
  // Chunk records as they arrive (a, b, c), overwritten in place by the
  // per-tile entry data: [0] = ax, ay, ox, thr (coverage bound on r^2);
  // [1] = bx, by, oy, -; [2] = r, g, b, log2 alpha (the record's c).
  using Scan = std::conditional_t<kAhead, BinScanAhead<kThreads, kChunk, true>,
                                  BinScan<kThreads, kChunk, true>>;
  float4 raw[2][3][kChunk];
  typename Scan::Smem scan;
  alignas(16) uint32_t list[kWarps][kChunk];
  uint32_t bits[kWarps][kChunk / 32];
  uint32_t view;
  uint32_t next;
};

template <int kTile, int kChunk, int kPx, bool kAhead>
__device__ __forceinline__ void raster_fp32_tile(const RasterArgs &a, uint32_t tile,
                                                 Fp32Smem<kTile, kChunk, kPx, kAhead> &sm) {
  constexpr int kBlocksX = kTile / 8;
  using Smem = Fp32Smem<kTile, kChunk, kPx, kAhead>;
  constexpr int kThreads = Smem::kThreads;
  constexpr int kRows = 4 * kPx;  // rows of a warp's block
  const uint32_t view = block_view(a, tile, sm.view);
  const uint32_t width = a.views[view].p.width, height = a.views[view].p.height;
  const uint32_t tiles_x = a.views[view].p.tiles_x;
  uint32_t *__restrict__ image = a.images + a.views[view].image_base;
  const uint32_t local_tile = tile - a.views[view].tile_base;
  const uint32_t tx = local_tile % tiles_x, ty = local_tile / tiles_x;
  const uint32_t x0 = tx * kTile, y0 = ty * kTile;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this warp's block of 8 columns and kRows rows
  const uint32_t lxp = (warp % kBlocksX) * 8 + (lane & 7);
  const uint32_t lyp = (warp / kBlocksX) * kRows + (lane >> 3);
  const uint32_t px = x0 + lxp, py = y0 + lyp;
  // Local coordinates are taken from the 16-pixel grid corner at or before
  // the tile, so 8x8 and 16x16 tiles evaluate every pixel identically.
  const uint32_t ax0 = x0 & ~15u, ay0 = y0 & ~15u;
  const float fx = (float)(px - ax0);
  float fy[kPx];
  bool inside[kPx];
#pragma unroll
  for (int p = 0; p < kPx; ++p) {
    fy[p] = (float)(py + 4 * p - ay0);
    inside[p] = px < width && py + 4 * p < height;
  }
  const float fax = (float)ax0, fay = (float)ay0;
  const float ftx = (float)x0, fty = (float)y0;
  typename Smem::Scan scan(a, a.views[view].bin_base, tx, ty, tiles_x);
  auto fill = [&](int buf) {
    return scan.next(a, sm.scan, sm.raw[buf], [&](uint32_t gid, const Record *r) {
      // debug tap: the inputs and the bound this kernel blends with (every
      // tile of a splat writes the same pair)
      if (a.debug_cov) {
        const float log2a = r->c.w;
        a.debug_cov[gid] = make_float2(log2a, coverage_bound(log2a, r->b.z));
      }
    });
  };

  float T[kPx], c0[kPx], c1[kPx], c2[kPx];
  bool done[kPx];
#pragma unroll
  for (int p = 0; p < kPx; ++p) {
    T[p] = 1.0f;
    c0[p] = c1[p] = c2[p] = 0.0f;
    done[p] = !inside[p];
  }
  auto all_done = [&]() {
    bool d = true;
#pragma unroll
    for (int p = 0; p < kPx; ++p) d = d && done[p];
    return d;
  };
  scan.prime(a, sm.scan);
  uint32_t n_in = fill(0);
  cp_async_wait_all();
  __syncthreads();
  for (int buf = 0; n_in; buf ^= 1) {
    // every thread's records of this chunk have landed
    const uint32_t n_next = fill(buf ^ 1);
#pragma unroll
    for (uint32_t t0 = 0; t0 < (uint32_t)kChunk; t0 += kThreads) {
      const uint32_t t = t0 + tid;
      if (kChunk < kThreads && t / 32 >= (uint32_t)kChunk / 32) break;  // whole warps
      uint32_t mask = 0;
      if (t < n_in) {
        const float4 ra = sm.raw[buf][0][t], rb = sm.raw[buf][1][t], col = sm.raw[buf][2][t];
        float cxa = ra.x - fax, cya = ra.y - fay;
        float ox = -fmaf(ra.z, cxa, ra.w * cya);
        float oy = -fmaf(rb.x, cxa, rb.y * cya);
        float cxl = ra.x - ftx, cyl = ra.y - fty;
        const float thr = coverage_bound(col.w, rb.z);
        sm.raw[buf][0][t] = make_float4(ra.z, ra.w, ox, thr);
        sm.raw[buf][1][t] = make_float4(rb.x, rb.y, oy, rb.w);
        mask = ellipse_block_mask<kTile, kRows>(ra, rb, thr, cxl, cyl);
      }
      share_mask(mask, t / 32, sm.bits);
    }
    __syncthreads();
    // This warp's entries, in order, as byte offsets in raw.
    uint32_t *list = sm.list[warp];
    const uint32_t n_w = list_entries(sm.bits[warp], buf * (uint32_t)sizeof(sm.raw[0]), list);
    // Eight list entries per step (one early-out vote, two index loads); each
    // pixel still takes them strictly in list order.
    // w = alpha e^(-4.5 r2) = 2^(log2 alpha - 4.5 log2(e) r2) (the entry's
    // log2 alpha in its colour's w), so the colour takes rgb * (w T) and the
    // transmittance loses w T.
    auto at = [&](uint32_t j, uint32_t q) {
      return *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(sm.raw) + j +
                                               q * (uint32_t)(16 * kChunk));
    };
    // Branch-free: a pixel that does not take the entry (finished, or not
    // covered) blends with wT = 0, which leaves C and T bit for bit as they
    // are (fma(x, 0, c) = c and T - 0 = T for finite x).
    auto entry = [&](uint32_t j) {
      const float4 d0 = at(j, 0);
      const float4 d1 = at(j, 1);
      const float4 col = at(j, 2);
      if constexpr (kPx == 2 && GSR_RASTER_F32X2) {
        // The two pixels' arithmetic as paired FP32 instructions (sm_100
        // f32x2, documented to round each component as the scalar operation;
        // T - wT is fma(wT, -1, T), the same single rounding). The images
        // equal the scalar build's byte for byte on the test workloads; the
        // FP32 mode is held to its tolerance, not to bit equality.
        const float2 fxp = make_float2(fx, fx), fyp = make_float2(fy[0], fy[1]);
        const float2 rx = __ffma2_rn(make_float2(d0.y, d0.y), fyp, make_float2(d0.z, d0.z));
        const float2 ry = __ffma2_rn(make_float2(d1.y, d1.y), fyp, make_float2(d1.z, d1.z));
        const float2 lx = __ffma2_rn(make_float2(d0.x, d0.x), fxp, rx);
        const float2 ly = __ffma2_rn(make_float2(d1.x, d1.x), fxp, ry);
        const float2 r2 = __ffma2_rn(lx, lx, __fmul2_rn(ly, ly));
        const float2 arg =
            __ffma2_rn(r2, make_float2(-6.49212768f, -6.49212768f), make_float2(col.w, col.w));
        const float2 wt = __fmul2_rn(make_float2(ex2_approx(arg.x), ex2_approx(arg.y)),
                                     make_float2(T[0], T[1]));
        const bool take0 = !done[0] && r2.x <= d0.w, take1 = !done[1] && r2.y <= d0.w;
        const float2 wT = make_float2(take0 ? wt.x : 0.0f, take1 ? wt.y : 0.0f);
        const float2 n0 = __ffma2_rn(make_float2(col.x, col.x), wT, make_float2(c0[0], c0[1]));
        const float2 n1 = __ffma2_rn(make_float2(col.y, col.y), wT, make_float2(c1[0], c1[1]));
        const float2 n2 = __ffma2_rn(make_float2(col.z, col.z), wT, make_float2(c2[0], c2[1]));
        const float2 nt = __ffma2_rn(wT, make_float2(-1.0f, -1.0f), make_float2(T[0], T[1]));
        c0[0] = n0.x, c0[1] = n0.y;
        c1[0] = n1.x, c1[1] = n1.y;
        c2[0] = n2.x, c2[1] = n2.y;
        T[0] = nt.x, T[1] = nt.y;
        done[0] = done[0] || T[0] < 1e-4f;
        done[1] = done[1] || T[1] < 1e-4f;
      } else {
#pragma unroll
        for (int p = 0; p < kPx; ++p) {
          const float lx = fmaf(d0.x, fx, fmaf(d0.y, fy[p], d0.z));
          const float ly = fmaf(d1.x, fx, fmaf(d1.y, fy[p], d1.z));
          const float r2 = fmaf(lx, lx, ly * ly);
          const bool take = !done[p] && r2 <= d0.w;
          const float w = blend_weight(r2, col.w);
          const float wT = take ? w * T[p] : 0.0f;
          c0[p] = fmaf(col.x, wT, c0[p]);
          c1[p] = fmaf(col.y, wT, c1[p]);
          c2[p] = fmaf(col.z, wT, c2[p]);
          T[p] = T[p] - wT;
          done[p] = done[p] || T[p] < 1e-4f;
        }
      }
    };
    uint32_t i = 0;
    for (; i + 7 < n_w; i += 8) {
      if (__all_sync(0xffffffffu, all_done())) break;
      const uint4 jj = *reinterpret_cast<const uint4 *>(&list[i]);
      const uint4 kk = *reinterpret_cast<const uint4 *>(&list[i + 4]);
      entry(jj.x);
      entry(jj.y);
      entry(jj.z);
      entry(jj.w);
      entry(kk.x);
      entry(kk.y);
      entry(kk.z);
      entry(kk.w);
    }
    for (; i + 3 < n_w; i += 4) {
      if (__all_sync(0xffffffffu, all_done())) break;
      const uint4 jj = *reinterpret_cast<const uint4 *>(&list[i]);
      entry(jj.x);
      entry(jj.y);
      entry(jj.z);
      entry(jj.w);
    }
    for (; i < n_w; ++i) {
      if (__all_sync(0xffffffffu, all_done())) break;
      entry(list[i]);
    }
    cp_async_wait_all();
    if (__syncthreads_count(all_done()) == kThreads) break;
    n_in = n_next;
  }
#pragma unroll
  for (int p = 0; p < kPx; ++p)
    if (inside[p])
      image[(size_t)(py + 4 * p) * width + px] =
          to_unorm8(c0[p]) | (to_unorm8(c1[p]) << 8) | (to_unorm8(c2[p]) << 16) |
          (to_unorm8(1.0f - T[p]) << 24);
}

// One block per tile (kPersistent false), or a fixed grid of blocks that take
// tiles from a global queue (an atomic ticket over the batch's tiles) until
// it is empty.
template <int kTile, int kChunk, int kPx, int kBlocks, bool kPersistent>
__global__ void __launch_bounds__(kTile *kTile / kPx, kBlocks)
    raster_fp32_kernel(RasterArgs a) {
  constexpr bool kAhead = kBlocks < kManyBlocks<kTile>;
  __shared__ Fp32Smem<kTile, kChunk, kPx, kAhead> sm;
  publish_counters(a);
  if constexpr (!kPersistent) {
    raster_fp32_tile<kTile, kChunk, kPx, kAhead>(a, blockIdx.x, sm);
  } else {
    for (;;) {
      if (threadIdx.x == 0) sm.next = atomicAdd(&a.counters->raster_ticket, 1u);
      __syncthreads();
      const uint32_t tile = sm.next;
      if (tile >= a.total_tiles) break;
      raster_fp32_tile<kTile, kChunk, kPx, kAhead>(a, tile, sm);
      __syncthreads();  // shared memory is reused by the next tile
    }
  }
  note_end(a);
}

}  // namespace

// With few tiles the one with the longest list sets the time, and a warp of
// it is bound by its own latencies: the registers that no further block
// would use go to it (4 or 7 blocks a SM instead of 8, 8 of 8x8 tiles
// instead of 16), its list is walked ahead, and the steps are longer (us, 8
// blocks and a direct walk -> as here: 256 tiles of 27 k pairs 32.8 -> 28.7,
// 190 tiles, 62 k splats 110.6 -> 84.0, 475 tiles, 2 M splats 71.7 -> 49.2;
// 750 tiles of 100 k splats 59.4 -> 55.3 at 7 blocks). A chunk is the most a
// step stages: with more tiles than blocks are resident half of 256 is
// better, since a tile that fills up early has then gathered fewer records
// it does not need and 8 blocks fit (1.70 M pairs at 1920x1080 116.9 ->
// 112.6 us, 186 M at 3840x2160 500 -> 397). UNORM8: at most 4 tiles a SM (16
// of 8x8 pixels), see raster_unorm8_kernel.
RasterShape raster_shape(uint32_t total_tiles, uint32_t tile, uint32_t blend_mode,
                         const RasterConfig &cfg, uint32_t sm_count) {
  if (blend_mode == 1) {
    const bool ahead = total_tiles <= (tile == 16 ? 4 : 16) * sm_count;
    const uint32_t chunk = tile == 16   ? (ahead ? U8Smem<16, true>::kChunk : U8Smem<16, false>::kChunk)
                           : ahead      ? U8Smem<8, true>::kChunk
                                        : U8Smem<8, false>::kChunk;
    return {tile, blend_mode, chunk, ahead, 0};
  }
  const uint32_t per_sm = (total_tiles + sm_count - 1) / sm_count;
  uint32_t chunk = cfg.chunk, blocks = tile == 16 ? kManyBlocks<16> : kManyBlocks<8>;
  if (tile == 16 && chunk == 256) {
    if (per_sm > 7) chunk = 128;
    else blocks = per_sm > 4 ? 7 : 4;
  } else if (tile == 8 && chunk == 64 && per_sm <= 16) {
    chunk = 128;
    blocks = 8;
  }
  return {tile, blend_mode, chunk, blocks, cfg.blocks_per_sm};
}

void launch_raster(const RasterArgs &a, uint32_t tile, uint32_t blend_mode,
                   const RasterConfig &cfg, uint32_t sm_count, cudaStream_t stream) {
  if (a.total_tiles == 0) return;
  const RasterShape s = raster_shape(a.total_tiles, tile, blend_mode, cfg, sm_count);
  if (blend_mode == 1) {
#define GSR_U8(T, A) raster_unorm8_kernel<T, A><<<a.total_tiles, T * T, 0, stream>>>(a)
    if (tile == 16) {
      if (s.blocks) GSR_U8(16, true);
      else GSR_U8(16, false);
    } else {
      if (s.blocks) GSR_U8(8, true);
      else GSR_U8(8, false);
    }
#undef GSR_U8
    return;
  }
  const bool persistent = s.blocks_per_sm > 0;
  const uint32_t grid =
      persistent ? std::min<uint32_t>(a.total_tiles, s.blocks_per_sm * sm_count) : a.total_tiles;
#define GSR_FP32(T, C, P, B)                                                     \
  do {                                                                           \
    if (persistent)                                                              \
      raster_fp32_kernel<T, C, P, B, true><<<grid, T * T / P, 0, stream>>>(a);   \
    else                                                                         \
      raster_fp32_kernel<T, C, P, B, false><<<grid, T * T / P, 0, stream>>>(a);  \
  } while (0)
  if (tile == 16) {
    if (s.chunk == 64) GSR_FP32(16, 64, GSR_RASTER_PX, kManyBlocks<16>);
    else if (s.chunk == 128) GSR_FP32(16, 128, GSR_RASTER_PX, kManyBlocks<16>);
    else if (s.blocks == 7) GSR_FP32(16, 256, GSR_RASTER_PX, 7);
    else GSR_FP32(16, 256, GSR_RASTER_PX, 4);
  } else {
    if (s.chunk == 32) GSR_FP32(8, 32, 1, kManyBlocks<8>);
    else if (s.chunk == 64) GSR_FP32(8, 64, 1, kManyBlocks<8>);
    else GSR_FP32(8, 128, 1, 8);
  }
#undef GSR_FP32
}

RasterConfig raster_config_at(uint32_t tile, RasterConfig cfg) {
  if (cfg.chosen && raster_config_valid(tile, cfg)) return cfg;
  return {tile * tile, cfg.blocks_per_sm, false};
}

bool raster_config_valid(uint32_t tile, const RasterConfig &cfg) {
  const bool chunk_ok = tile == 16 ? (cfg.chunk == 64 || cfg.chunk == 128 || cfg.chunk == 256)
                                   : (cfg.chunk == 32 || cfg.chunk == 64);
  return chunk_ok && cfg.blocks_per_sm <= 32;
}

}  // namespace gsr
