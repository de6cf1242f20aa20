// K2: (bin, splat) pair emission, and the bin-range build (bins.cuh: a bin is
// 4x4 raster tiles). Bin ids are global over the views of a batch:
// views[v].bin_base + local bin.
//
// Emission walks the depth-sorted visible ids. Each block takes the next
// kEmitThreads * kEmitIpt sorted positions from an atomic ticket. A splat
// covers, per row of its tile rect, only the span of columns its ellipse
// reaches (tile_span.cuh). Its unit of work is a bin row, up to four tile
// rows: a lane computes their spans, and with them the bin columns they reach
// and the tile pairs they stand for. Each warp walks the units of its own
// items 32 at a time (a lane finds its item by a 5-step shuffle search over
// the items' inclusive unit counts) and keeps the spans in shared memory.
// The block's pair total then gets its global offset from a decoupled
// look-back, so pairs land in exactly the order a sequential walk would write
// them: depth order, then bin rows, then bin columns. Each warp then walks
// the same unit windows again and writes the window's pairs 32 at a time (a
// lane finds its unit by a second search over the units' inclusive widths and
// codes the tiles from the unit's spans), so a splat covering hundreds of
// bins is spread over the lanes. The digit histograms the bin sort needs are
// accumulated while the pairs are written.

#include <algorithm>

#include "bins.cuh"
#include "device_common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "tile_span.cuh"

namespace gsr {
namespace {

constexpr int kEmitThreads = 256;
constexpr int kEmitWarps = kEmitThreads / 32;
// Sorted ids per thread: 2 below kEmitLargeIds ids, 4 from there on, where
// blocks of 1,024 ids fill the GPU (4 resident per SM): fewer blocks, each with
// its barriers, look-back and view table (1.0 M ids of 64 thumbnail views 81 ->
// 71 us, 21 M ids of a mixed batch 1,852 -> 1,457 us). A frame's emission with
// 2 against 4, us: 279k ids 1280x720 25 / 29, 1920x1080 26 / 33; 350k 38 / 32
// and 41 / 37; 420k 41 / 34 and 43 / 38; 500k 42 / 39 and 44 / 46; 560k 45 / 40
// and 47 / 46; 650k 59 / 58 and 61 / 65; 900k 69 / 68 and 71 / 79; 1.1 M 85 / 73
// and 90 / 84. The steps are the waves of resident blocks, 303k ids with 2 and
// 606k with 4: up to 303k and, at 1920x1080, between 606k and 1.0 M 2 is faster,
// from 303k to about 500k and beyond 1.1 M 4 is. The line was set by the ends
// (279k and 1.0 M).
constexpr uint64_t kEmitLargeIds = 600'000;
// Units whose spans each warp keeps between its two walks (16 bytes each);
// units past them are computed again in the second walk.
template <int kEmitIpt>
constexpr uint32_t kUnitSlots = kEmitIpt == 2 ? 256 : 192;

inline uint32_t emit_ipt(uint64_t ids) { return ids < kEmitLargeIds ? 2u : 4u; }

// Index of the first lane whose inclusive end exceeds x (31 when none does),
// by a 5-step shuffle search over the warp's ascending inclusive ends.
__device__ __forceinline__ uint32_t lane_search(uint32_t incl, uint32_t x) {
  uint32_t c = 0;
#pragma unroll
  for (uint32_t step = 16; step >= 1; step >>= 1) {
    const uint32_t v = __shfl_sync(0xffffffffu, incl, c + step - 1);
    if (v <= x) c += step;
  }
  return c;
}

// One window of a warp's unit walk: units r .. round_end-1 of the items from
// `it` on, one per lane. Both walks take the same windows.
struct UnitWindow {
  uint32_t inc_w;      // inclusive unit end of item it + lane (clamped to the warp's last)
  uint32_t round_end;  // one past the window's last unit
  uint32_t item;       // the lane's item (valid when r + lane < round_end)
  uint32_t row;        // the lane's bin row within its item
};

__device__ __forceinline__ UnitWindow unit_window(const uint32_t *s_rinc, uint32_t ib, uint32_t il,
                                                  uint32_t it, uint32_t r, uint32_t lane) {
  UnitWindow w;
  w.inc_w = s_rinc[min(it + lane, il)];
  const uint32_t win_start = it > ib ? s_rinc[it - 1] : 0u;
  const uint32_t win_end = __shfl_sync(0xffffffffu, w.inc_w, 31);
  w.round_end = min(r + 32u, win_end);
  const uint32_t my = r + lane;
  const uint32_t c = lane_search(w.inc_w, my);
  const uint32_t prev = __shfl_sync(0xffffffffu, w.inc_w, c ? c - 1 : 0);
  w.item = it + c;
  w.row = my - (c ? prev : win_start);
  return w;
}

// A unit's spans in shared memory, by tile row of the bin (0: none), with the
// bin columns [x, y) they reach and their tiles.
struct UnitSpans {
  uint2 cols;
  uint32_t tiles;
};

// The spans of bin row `br` of splat `id` with tile rect rc, into out[4].
__device__ __forceinline__ UnitSpans unit_spans(const EmitBuffers &b, uint32_t id, uint2 rc,
                                                uint32_t br, float inv_tile, uint32_t *out) {
  const Record *rec = &b.records[id];
  const float4 ra = rec->a, rb = rec->b;
  const uint32_t first = max(kBinEdge * br, rc.x >> 16);
  const uint32_t end = min(kBinEdge * br + kBinEdge, rc.y >> 16);
  *reinterpret_cast<uint4 *>(out) = make_uint4(0u, 0u, 0u, 0u);
  RowSpans spans(ra.x, ra.y, span_pre(ra, rb), b.tile, inv_tile, rc.x & 0xffffu,
                 rc.y & 0xffffu, first);
  uint32_t c0 = 0xffffu, c1 = 0, tiles = 0;
  for (uint32_t ty = first; ty < end; ++ty) {
    const uint2 sp = spans.next();
    if (sp.x == sp.y) continue;
    out[ty % kBinEdge] = sp.x | (sp.y << 16);
    c0 = min(c0, sp.x);
    c1 = max(c1, sp.y);
    tiles += sp.y - sp.x;
  }
  return {c1 ? make_uint2(c0 / kBinEdge, (c1 + kBinEdge - 1) / kBinEdge) : make_uint2(0u, 0u),
          tiles};
}

// The bin columns [x, y) that kept spans reach.
__device__ __forceinline__ uint2 unit_columns(uint4 sp) {
  const uint32_t rows[kBinEdge] = {sp.x, sp.y, sp.z, sp.w};
  uint32_t c0 = 0xffffu, c1 = 0;
#pragma unroll
  for (uint32_t j = 0; j < kBinEdge; ++j) {
    c0 = min(c0, rows[j] ? rows[j] & 0xffffu : 0xffffu);
    c1 = max(c1, rows[j] >> 16);
  }
  return c1 ? make_uint2(c0 / kBinEdge, (c1 + kBinEdge - 1) / kBinEdge) : make_uint2(0u, 0u);
}

template <int kEmitIpt>
__global__ void __launch_bounds__(kEmitThreads) emit_kernel(EmitBuffers b) {
  constexpr int kEmitItems = kEmitThreads * kEmitIpt;
  constexpr int kWarpItems = kEmitItems / kEmitWarps;
  constexpr uint32_t kSlots = kUnitSlots<kEmitIpt>;
  __shared__ uint4 s_span[kEmitWarps][kSlots];  // per warp unit: four rows' first | end << 16
  __shared__ uint32_t s_rinc[kEmitItems];  // inclusive unit counts within the warp's items
  __shared__ uint32_t s_id[kEmitItems];
  __shared__ uint2 s_rect[kEmitItems];
  __shared__ uint16_t s_vi[kEmitItems];
  __shared__ uint32_t s_wsum[kEmitWarps];
  __shared__ uint32_t s_hist[4 * 256];  // [passes][256], or one wide pass's
  __shared__ uint32_t s_block;
  __shared__ unsigned long long s_prefix;
  // View table columns: splat base, bin base, bins per row; tile pairs of the
  // block per view.
  extern __shared__ uint32_t s_views[];
  uint32_t *s_vsb = s_views, *s_vbb = s_views + b.num_views, *s_vbx = s_views + 2 * b.num_views;
  uint32_t *s_vpairs = s_views + 3 * b.num_views;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t hist_words = b.wide_bits ? 1u << b.wide_bits : b.bin_passes * 256;
  const uint32_t low_mask = b.wide_bits ? hist_words - 1u : 255u;
  if (blockIdx.x == 0 && tid == 0) b.counters->phase_ns[2] = global_ns();
  for (uint32_t k = tid; k < hist_words; k += kEmitThreads) s_hist[k] = 0;
  for (uint32_t v = tid; v < b.num_views; v += kEmitThreads) {
    s_vsb[v] = b.views[v].splat_base;
    s_vbb[v] = b.views[v].bin_base;
    s_vbx[v] = bins_along(b.views[v].p.tiles_x);
    s_vpairs[v] = 0;
  }
  // The sorted visible ids: this frame's, or the order reused from the last
  // sort (the plan keeps its count).
  const uint32_t V = b.depth_plan->n;
  const uint32_t *ids = b.depth_plan->final_buffer == 0 ? b.ids0 : b.ids1;
  const float inv_tile = __fdiv_rn(1.0f, (float)b.tile);
  const uint32_t ib = warp * kWarpItems, il = ib + kWarpItems - 1;
  if (tid == 0) s_block = atomicAdd(&b.counters->emit_ticket, 1u);
  __syncthreads();
  const uint32_t block = s_block;
  const uint32_t start = block * kEmitItems;
  if (start >= V) return;

  uint32_t rows[kEmitIpt];
  uint32_t local_rows = 0;
#pragma unroll
  for (int k = 0; k < kEmitIpt; ++k) {
    const uint32_t slot = tid * kEmitIpt + k;
    const uint32_t j = start + slot;
    uint32_t id = 0, h = 0, vi = 0;
    uint2 r = make_uint2(0u, 0u);
    if (j < V) {
      id = ids[j];
      r = b.rects[id];
      if ((r.y & 0xffffu) > (r.x & 0xffffu) && (r.y >> 16) > (r.x >> 16)) {
        h = bins_along(r.y >> 16) - (r.x >> 16) / kBinEdge;
        vi = find_view(b.num_views, id, [&](uint32_t v) { return s_vsb[v]; });
      }
    }
    s_id[slot] = id;
    s_rect[slot] = r;
    s_vi[slot] = (uint16_t)vi;
    rows[k] = h;
    local_rows += h;
  }
  uint32_t rinc = local_rows;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, rinc, o);
    if (lane >= (uint32_t)o) rinc += t;
  }
  uint32_t rrun = rinc - local_rows;
#pragma unroll
  for (int k = 0; k < kEmitIpt; ++k) {
    rrun += rows[k];
    s_rinc[tid * kEmitIpt + k] = rrun;
  }
  __syncwarp();

  const uint32_t rows_total = s_rinc[il];
  // First walk: every unit's spans, kept for the second walk; their pairs.
  // Units past the slots go through the last window's.
  uint32_t local = 0;
  unsigned long long tiles_sum = 0;
  for (uint32_t r = 0, it = ib; r < rows_total;) {
    const UnitWindow w = unit_window(s_rinc, ib, il, it, r, lane);
    const uint32_t my = r + lane;
    if (my < w.round_end) {
      const uint2 rc = s_rect[w.item];
      const UnitSpans u =
          unit_spans(b, s_id[w.item], rc, (rc.x >> 16) / kBinEdge + w.row, inv_tile,
                     reinterpret_cast<uint32_t *>(
                         &s_span[warp][r + 32 <= kSlots ? my : kSlots - 32 + lane]));
      local += u.cols.y - u.cols.x;
      tiles_sum += u.tiles;
      if (b.num_views > 1 && u.tiles) atomicAdd(&s_vpairs[s_vi[w.item]], u.tiles);
    }
    it += __popc(__ballot_sync(0xffffffffu, w.inc_w <= w.round_end));
    r = w.round_end;
  }
  local = warp_sum(local);
  tiles_sum = warp_sum(tiles_sum);
  if (lane == 0) {
    s_wsum[warp] = local;
    if (tiles_sum) {
      atomicAdd(&b.counters->keys, tiles_sum);
      if (b.num_views == 1) atomicAdd(&b.view_counters[0].pairs, (uint32_t)tiles_sum);
    }
  }
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kEmitWarps; ++w) {
    const uint32_t c = s_wsum[w];
    before += (w < (int)warp) ? c : 0u;
    total += c;
  }
  if (warp == 0) {
    const unsigned long long ex = lookback_warp(b.status, block, total, &b.counters->error);
    if (lane == 0) s_prefix = ex;
  }
  __syncthreads();
  const unsigned long long prefix = s_prefix;
  if (tid == 0 && block == (V - 1) / kEmitItems) {
    const unsigned long long all = prefix + total;
    b.counters->pairs = (uint32_t)(all < b.capacity ? all : b.capacity);
    if (all > b.capacity) b.counters->overflow = 1u;
  }

  // Second walk: the pairs of each unit window, 32 per round. A window that
  // reaches past the slots went through the last 32 of them, so windows with
  // units there are computed again.
  const uint32_t kept_end = rows_total <= kSlots - 32 ? kSlots : kSlots - 32;
  unsigned long long kpos = prefix + before;  // position of the warp's next pair
  for (uint32_t r = 0, it = ib; r < rows_total;) {
    const UnitWindow w = unit_window(s_rinc, ib, il, it, r, lane);
    const bool kept = r + 32 <= kept_end;
    const uint4 *spans = &s_span[warp][kept ? r : kSlots - 32];
    uint32_t bin = 0, id = 0;
    uint2 cols = make_uint2(0u, 0u);
    __syncwarp();
    if (r + lane < w.round_end) {
      const uint2 rc = s_rect[w.item];
      const uint32_t br = (rc.x >> 16) / kBinEdge + w.row;
      id = s_id[w.item];
      if (kept)
        cols = unit_columns(spans[lane]);
      else
        cols = unit_spans(b, id, rc, br, inv_tile,
                          reinterpret_cast<uint32_t *>(&s_span[warp][kSlots - 32 + lane]))
                   .cols;
      const uint32_t vi = s_vi[w.item];
      bin = s_vbb[vi] + br * s_vbx[vi];  // global id of the bin row's first bin
    }
    __syncwarp();
    uint32_t winc = cols.y - cols.x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= (uint32_t)o) winc += t;
    }
    const uint32_t W = __shfl_sync(0xffffffffu, winc, 31);
    for (uint32_t q = 0; q < W; q += 32) {
      const uint32_t myp = q + lane;
      const uint32_t j = lane_search(winc, myp);
      const uint32_t pj = __shfl_sync(0xffffffffu, winc, j ? j - 1 : 0);
      const uint32_t cj = __shfl_sync(0xffffffffu, cols.x, j);
      const uint32_t bj = __shfl_sync(0xffffffffu, bin, j);
      const uint32_t idj = __shfl_sync(0xffffffffu, id, j);
      const unsigned long long g = kpos + myp;
      if (myp < W && g < b.capacity) {
        const uint32_t bc = cj + myp - (j ? pj : 0u);
        const uint4 sp = spans[j];
        const uint32_t rows4[kBinEdge] = {sp.x, sp.y, sp.z, sp.w};
        const uint32_t t = bj + bc;
        b.pair_keys[g] = (t << kBinCodeBits) | bin_code(rows4, bc);
        b.pair_vals[g] = idj;
        atomicAdd(&s_hist[t & low_mask], 1u);
        // The higher digits of a round's bins are mostly equal: one add per
        // distinct digit instead of up to 32 colliding ones.
        const uint32_t act = __activemask();
        const uint32_t lt = lanemask_lt();
        if (b.bin_passes > 1) {
          const uint32_t d1 = (t >> 8) & 255u;
          const uint32_t peers = __match_any_sync(act, d1);
          if ((peers & lt) == 0) atomicAdd(&s_hist[256 + d1], __popc(peers));
        }
        if (b.bin_passes > 2) {
          const uint32_t d2 = (t >> 16) & 255u;
          const uint32_t peers = __match_any_sync(act, d2);
          if ((peers & lt) == 0) atomicAdd(&s_hist[512 + d2], __popc(peers));
        }
      }
    }
    kpos += W;
    it += __popc(__ballot_sync(0xffffffffu, w.inc_w <= w.round_end));
    r = w.round_end;
  }
  __syncthreads();
  if (b.num_views > 1)
    for (uint32_t v = tid; v < b.num_views; v += kEmitThreads)
      if (const uint32_t n = s_vpairs[v]) atomicAdd(&b.view_counters[v].pairs, n);
  for (uint32_t q = tid; q < hist_words; q += kEmitThreads) {
    const uint32_t n = s_hist[q];
    if (n) atomicAdd(&b.bin_hist[q], n);
  }
}

// Transpose of the warp's 32x32 bit matrix (lane l holds row l): lane l gets
// bit l of every lane.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
  uint32_t low = 0x0000ffffu;
#pragma unroll
  for (uint32_t j = 16; j >= 1; j >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((y >> j) & low) | (x & ~low) : (x & low) | ((y << j) & ~low);
    low ^= low << (j / 2);
  }
  return x;
}

// Bin boundaries of the sorted keys, and their codes as one word per tile of
// the bin and 32 keys (tile_word in bins.cuh), the form a tile's raster walks.
// A warp takes 256 keys. A lane's 16 tile bits of two keys, 32 apart, make one
// word, and the transpose of the warp's 32 words (five exchanges) gives lane t
// tile t's word of the first 32 keys and lane 16 + t that of the second; eight
// words a tile are written as one 32-byte sector. One ballot per tile instead
// took 1,100 instructions per 256 keys (113 us for 18 M pairs). The words go
// to the key buffer the sort has left free (half a word per key). The frame
// overflows when the tile pairs the keys stand for exceed the capacity.
__global__ void __launch_bounds__(256) ranges_kernel(const SortPlan *__restrict__ plan,
                                                     uint32_t *k0, uint32_t *k1,
                                                     FrameCounters *__restrict__ counters,
                                                     uint64_t capacity,
                                                     uint2 *__restrict__ ranges) {
  const uint32_t K = counters->pairs;
  const bool first = plan->final_buffer == 0;
  const uint32_t *keys = first ? k0 : k1;
  uint32_t *words = first ? k1 : k0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters->phase_ns[4] = global_ns();
    if (counters->keys > capacity) counters->overflow = 1u;
  }
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * blockDim.x / 32, groups = (K + 255) / 256;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) / 32; g < groups; g += warps) {
    uint32_t key[kWordGroup];
#pragma unroll
    for (uint32_t q = 0; q < kWordGroup; ++q) {
      const uint32_t i = 256 * g + 32 * q + lane;
      key[q] = i < K ? keys[i] : 0u;
    }
    // the neighbours of the group's keys (out of the list: an id no bin has)
    uint32_t before = ~0u, after = ~0u;
    if (lane == 0 && g > 0) before = keys[256 * g - 1] >> kBinCodeBits;
    if (lane == 31 && 256 * g + 256 < K) after = keys[256 * g + 256] >> kBinCodeBits;
#pragma unroll
    for (uint32_t q = 0; q < kWordGroup; ++q) {
      const uint32_t i = 256 * g + 32 * q + lane;
      const uint32_t bin = key[q] >> kBinCodeBits;
      uint32_t prev = __shfl_up_sync(0xffffffffu, bin, 1);
      uint32_t next = __shfl_down_sync(0xffffffffu, bin, 1);
      const uint32_t last_before =
          q > 0 ? __shfl_sync(0xffffffffu, key[q > 0 ? q - 1 : 0], 31) >> kBinCodeBits : before;
      const uint32_t first_after =
          q + 1 < kWordGroup
              ? __shfl_sync(0xffffffffu, key[q + 1 < kWordGroup ? q + 1 : q], 0) >> kBinCodeBits
              : after;
      if (lane == 0) prev = last_before;
      if (lane == 31) next = first_after;
      if (i < K) {
        if (prev != bin) ranges[bin].x = i;
        if (i + 1 == K || next != bin) ranges[bin].y = i + 1;
      }
    }
    uint32_t mine[kWordGroup / 2];
#pragma unroll
    for (uint32_t q = 0; q < kWordGroup / 2; ++q)
      mine[q] = transpose32(bin_code_tiles(key[2 * q]) | bin_code_tiles(key[2 * q + 1]) << 16,
                            lane);
    // lane t: words 0, 2, 4, 6 of tile t; lane 16 + t: words 1, 3, 5, 7
    uint32_t other[kWordGroup / 2];
#pragma unroll
    for (uint32_t q = 0; q < kWordGroup / 2; ++q)
      other[q] = __shfl_xor_sync(0xffffffffu, mine[q], 16);
    const bool odd = lane >= 16;
    uint4 *out = reinterpret_cast<uint4 *>(&words[tile_word(kWordGroup * g, lane & 15u)]);
    out[odd] = odd ? make_uint4(other[2], mine[2], other[3], mine[3])
                   : make_uint4(mine[0], other[0], mine[1], other[1]);
  }
}

__global__ void run_init_kernel(RunInit a) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && a.inline_views) {
    static_assert(sizeof(ViewSetDev) % 4 == 0 && sizeof(ViewDev) % 4 == 0, "word copies");
    const uint32_t sw = a.inline_sets * (uint32_t)(sizeof(ViewSetDev) / 4);
    const uint32_t vw = a.inline_views * (uint32_t)(sizeof(ViewDev) / 4);
    const uint32_t *ss = reinterpret_cast<const uint32_t *>(a.sets);
    const uint32_t *vs = reinterpret_cast<const uint32_t *>(a.views);
    uint32_t *sd = reinterpret_cast<uint32_t *>(a.sets_dst);
    uint32_t *vd = reinterpret_cast<uint32_t *>(a.views_dst);
    for (uint32_t i = threadIdx.x; i < sw; i += blockDim.x) sd[i] = ss[i];
    for (uint32_t i = threadIdx.x; i < vw; i += blockDim.x) vd[i] = vs[i];
  }
#pragma unroll
  for (int r = 0; r < kRunZeroRegions; ++r)
    for (uint64_t i = t; i < a.zero_words[r]; i += stride) a.zero[r][i] = 0u;
  if (t == 0) {
    const unsigned long long now = global_ns();
    for (int k = 0; k < 6; ++k) a.phase_ns[k] = now;
  }
}

__global__ void fill_kernel(uint32_t *dst, uint32_t value, uint64_t count) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = value;
}

}  // namespace

uint64_t emit_blocks(uint64_t ids) {
  const uint64_t items = kEmitThreads * emit_ipt(ids);
  return (ids + items - 1) / items;
}

uint64_t emit_status_words(uint64_t capacity) {
  return std::max(emit_blocks(std::min(capacity, kEmitLargeIds - 1)), emit_blocks(capacity));
}

void launch_emit(const EmitBuffers &b, cudaStream_t stream) {
  const uint32_t blocks = (uint32_t)emit_blocks(b.n);
  if (blocks == 0 || b.num_views == 0) return;
  const size_t smem = 4 * 4 * b.num_views;
  // The static arrays and the largest view table together pass 48 KB.
  constexpr int kMost = (int)(4 * 4 * kMaxViewsPerLaunch);
  if (emit_ipt(b.n) == 2) {
    allow_shared_memory<emit_kernel<2>>(kMost);
    emit_kernel<2><<<blocks, kEmitThreads, smem, stream>>>(b);
  } else {
    allow_shared_memory<emit_kernel<4>>(kMost);
    emit_kernel<4><<<blocks, kEmitThreads, smem, stream>>>(b);
  }
}

void launch_ranges(const SortPlan *bin_plan, uint32_t *keys0, uint32_t *keys1,
                   FrameCounters *counters, uint32_t capacity, uint2 *ranges,
                   cudaStream_t stream) {
  uint32_t blocks = (capacity + 2047) / 2048;
  const uint32_t cap = 8 * device_sm_count();
  blocks = blocks < cap ? (blocks ? blocks : 1) : cap;
  ranges_kernel<<<blocks, 256, 0, stream>>>(bin_plan, keys0, keys1, counters, capacity, ranges);
}

const void *run_init_kernel_entry() { return reinterpret_cast<const void *>(&run_init_kernel); }

void launch_run_init(const RunInit &a, cudaStream_t stream) {
  uint64_t words = 0;
  for (int r = 0; r < kRunZeroRegions; ++r) words = std::max(words, a.zero_words[r]);
  const uint64_t blocks = std::min<uint64_t>(std::max<uint64_t>((words + 255) / 256, 1), 8ull * device_sm_count());
  run_init_kernel<<<(uint32_t)blocks, 256, 0, stream>>>(a);
}

void launch_fill_u32(uint32_t *dst, uint32_t value, uint64_t count, cudaStream_t stream) {
  if (count == 0) return;
  uint64_t blocks = (count + 255) / 256;
  if (blocks > 16ull * device_sm_count()) blocks = 16ull * device_sm_count();
  fill_kernel<<<(uint32_t)blocks, 256, 0, stream>>>(dst, value, count);
}

}  // namespace gsr
