// Host orchestration of the frame pipeline over a list of views (no device
// code in this file).

#include <algorithm>
#include <chrono>
#include <cstddef>
#include <cstring>
#include <string>

#include "bins.cuh"
#include "kernels.h"
#include "cuda_check.h"
#include "pipeline.h"

namespace gsr {

namespace {
inline uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }
constexpr uint64_t kMaxSortItems = (1u << 30) - 1;
constexpr uint64_t kInitialPairsPerSplat = 16;
// The pair capacity counts tile pairs; a run of that many has about this many
// times fewer (bin, splat) pairs: 3.3 at 279k splats and 1920x1080 (whose
// capacity is 2.6 times its tile pairs), 9 at 3M and 3840x2160.
constexpr uint64_t kPairsPerBinPair = 8;
}  // namespace

DeviceBuffer::~DeviceBuffer() { release(); }

void DeviceBuffer::release() {
  if (ptr_) {
    if (ordered_) cudaFreeAsync(ptr_, stream_);
    else cudaFree(ptr_);
  }
  ptr_ = nullptr;
  bytes_ = 0;
  ordered_ = false;
  stream_ = nullptr;
}

void DeviceBuffer::reset(uint64_t bytes, cudaStream_t stream) {
  release();
  if (bytes == 0) return;
  cudaError_t e = cudaMallocAsync(&ptr_, bytes, stream);
  if (e != cudaSuccess) {
    ptr_ = nullptr;
    cudaGetLastError();
    throw Error(Code::Internal, "device allocation of " + std::to_string(bytes) +
                                    " bytes failed: " + cudaGetErrorString(e));
  }
  bytes_ = bytes;
  stream_ = stream;
  ordered_ = true;
}

void DeviceBuffer::reset(uint64_t bytes) {
  release();
  if (bytes == 0) return;
  cudaError_t e = cudaMalloc(&ptr_, bytes);
  if (e != cudaSuccess) {
    ptr_ = nullptr;
    cudaGetLastError();
    throw Error(Code::Internal, "device allocation of " + std::to_string(bytes) +
                                    " bytes failed: " + cudaGetErrorString(e));
  }
  bytes_ = bytes;
}

namespace {
uint32_t bits_below(uint32_t values) {  // bits that hold 0 .. values-1
  uint32_t bits = 0;
  while (bits < 32 && (1ull << bits) < values) ++bits;
  return bits;
}
// The bin sort: one pass of up to 10 bits, else 8-bit passes.
uint32_t bin_wide_bits(uint32_t num_bins) {
  const uint32_t bits = bits_below(num_bins);
  return bits == 9 || bits == 10 ? bits : 0u;
}
uint32_t bin_sort_passes(uint32_t num_bins) {
  if (bin_wide_bits(num_bins)) return 1;
  return std::max(1u, (bits_below(num_bins) + 7) / 8);
}
}  // namespace

uint64_t scene_device_bytes(uint64_t splats, uint32_t sh_degree) {
  const uint64_t n = std::max<uint64_t>(splats, 1);
  return 3 * align256(16 * n) + align256(16 * n * color_planes(sh_degree));
}

uint64_t scene_device_bytes(const HostScene &s) { return scene_device_bytes(s.size(), s.sh_degree); }

std::unique_ptr<DeviceScene> alloc_scene(uint64_t n, uint32_t sh_degree) {
  if (n > kMaxSortItems)
    throw Error(Code::Unsupported, "scene has more splats than the renderer supports (2^30 - 1)");
  auto sc = std::make_unique<DeviceScene>();
  sc->n = (uint32_t)n;
  sc->sh_degree = sh_degree;
  const uint32_t planes = color_planes(sh_degree);
  // Three geometry planes, then the colour planes as one tight region so
  // that plane p of splat i sits at color[p * n + i].
  const uint64_t plane = align256(16 * std::max<uint64_t>(n, 1));
  sc->mem.reset(scene_device_bytes(n, sh_degree));
  char *base = sc->mem.as<char>();
  sc->dev.pos_alpha = reinterpret_cast<const float4 *>(base);
  sc->dev.cov_a = reinterpret_cast<const float4 *>(base + plane);
  sc->dev.cov_b = reinterpret_cast<const float4 *>(base + 2 * plane);
  sc->dev.color = reinterpret_cast<const float4 *>(base + 3 * plane);
  sc->dev.n = (uint32_t)n;
  sc->dev.planes = planes;
  return sc;
}

std::unique_ptr<DeviceScene> upload_scene(const HostScene &s, cudaStream_t stream) {
  const uint64_t n = s.size();
  auto sc = alloc_scene(n, s.sh_degree);
  ScenePacked packed;
  pack_scene(s, packed);
  sc->positions = s.positions;
  if (n) {
    const SceneDev &d = sc->dev;
    GSR_CUDA(cudaMemcpyAsync((void *)d.pos_alpha, packed.pos_alpha.data(), 16 * n,
                             cudaMemcpyHostToDevice, stream));
    GSR_CUDA(cudaMemcpyAsync((void *)d.cov_a, packed.cov_a.data(), 16 * n, cudaMemcpyHostToDevice,
                             stream));
    GSR_CUDA(cudaMemcpyAsync((void *)d.cov_b, packed.cov_b.data(), 16 * n, cudaMemcpyHostToDevice,
                             stream));
    GSR_CUDA(cudaMemcpyAsync((void *)d.color, packed.color.data(), 16 * n * packed.planes,
                             cudaMemcpyHostToDevice, stream));
  }
  GSR_CUDA(cudaStreamSynchronize(stream));
  return sc;
}

Pipeline::Pipeline(int device, cudaStream_t stream) : device_(device), stream_(stream) {
  int sms = 0;
  GSR_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_));
  sm_count_ = (uint32_t)sms;
  for (auto &ev : slot_ev_) GSR_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
  int least = 0, greatest = 0;
  GSR_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  GSR_CUDA(cudaStreamCreateWithPriority(&side_stream_, cudaStreamNonBlocking, greatest));
  side_priority_ = greatest;
  GSR_CUDA(cudaEventCreateWithFlags(&fork_ev_, cudaEventDisableTiming));
  GSR_CUDA(cudaEventCreateWithFlags(&join_ev_, cudaEventDisableTiming));
  GSR_CUDA(cudaMallocHost(&counters_host_, sizeof(FrameCounters)));
  std::memset(counters_host_, 0, sizeof(FrameCounters));
  // fixed scratch: [counters | key hist | tile hist] zeroed per run, then
  // plans and the sticky word.
  uint64_t off = 0;
  const uint64_t o_counters = off; off += align256(sizeof(FrameCounters));
  const uint64_t o_khist = off; off += align256(4 * 4 * 256);
  const uint64_t o_thist = off; off += align256(4 * 4 * 256);
  const uint64_t zero_end = off;
  const uint64_t o_dplan = off; off += align256(sizeof(SortPlan));
  const uint64_t o_tplan = off; off += align256(sizeof(SortPlan));
  const uint64_t o_sticky = off; off += 256;
  fixed_.reset(off);
  GSR_CUDA(cudaMemset(fixed_.get(), 0, off));
  counters_ = fixed_.as<FrameCounters>(o_counters);
  key_hist_ = fixed_.as<uint32_t>(o_khist);
  bin_hist_ = fixed_.as<uint32_t>(o_thist);
  depth_plan_ = fixed_.as<SortPlan>(o_dplan);
  bin_plan_ = fixed_.as<SortPlan>(o_tplan);
  sticky_ = fixed_.as<uint32_t>(o_sticky);
  (void)zero_end;
}

Pipeline::~Pipeline() {
  cudaSetDevice(device_);
  cudaStreamSynchronize(stream_);  // and with it the side stream, joined in every run
  drop_graph();
  if (side_stream_) cudaStreamDestroy(side_stream_);
  if (fork_ev_) cudaEventDestroy(fork_ev_);
  if (join_ev_) cudaEventDestroy(join_ev_);
  for (auto &ev : slot_ev_)
    if (ev) cudaEventDestroy(ev);

  if (counters_host_) cudaFreeHost(counters_host_);
  if (view_counters_pinned_) cudaFreeHost(view_counters_pinned_);
  if (table_pinned_) cudaFreeHost(table_pinned_);
  if (batch_stage_) cudaFreeHost(batch_stage_);
  if (batch_ev_) cudaEventDestroy(batch_ev_);
}

void Pipeline::set_tile(uint32_t tile) {
  tile_ = tile;
  raster_cfg_ = raster_config_at(tile_, raster_cfg_);
}

void Pipeline::set_raster_config(const RasterConfig &c) {
  if (!raster_config_valid(tile_, c))
    throw Error(Code::InvalidArgument, "raster chunk " + std::to_string(c.chunk) +
                                           " or blocks per SM " + std::to_string(c.blocks_per_sm) +
                                           " not valid for tile size " + std::to_string(tile_));
  raster_cfg_ = c;
}

void Pipeline::drop_graph() {
  for (auto &g : graphs_) {
    cudaGraphExecDestroy(g.exec);
    cudaGraphDestroy(g.graph);
  }
  graphs_.clear();
  seen_keys_.clear();
  drop_batch_graphs();
}

void Pipeline::drop_batch_graphs() {
  for (auto &g : batch_graphs_) {
    cudaGraphExecDestroy(g.exec);
    cudaGraphDestroy(g.graph);
  }
  batch_graphs_.clear();
  batch_seen_.clear();
}

Pipeline::Layout Pipeline::plan_views(const ViewSpec *views, uint32_t count,
                                      const uint64_t *image_bases) {
  if (count == 0) throw Error(Code::InvalidArgument, "no views to render");
  if (count > kMaxViewsPerLaunch)
    throw Error(Code::Unsupported, "more than 1024 views in one pipeline run");
  Layout l;
  l.views = count;
  views_host_.resize(count);
  sets_host_.clear();
  uint64_t splats = 0, blocks = 0, keys = 0, tiles = 0, bins = 0;
  for (uint32_t v = 0; v < count; ++v) {
    const ViewSpec &vs = views[v];
    if (!camera_valid(vs.camera)) throw Error(Code::InvalidArgument, "invalid camera");
    if (vs.width == 0 || vs.height == 0)
      throw Error(Code::InvalidArgument, "invalid renderer configuration");
    ViewDev &d = views_host_[v];
    std::memset(&d, 0, sizeof(d));
    d.p = make_frame_params(vs.camera, vs.width, vs.height, tile_, vs.scene->sh_degree,
                            vs.scene->n);
    d.sc = vs.scene->dev;
    d.splat_base = (uint32_t)splats;
    d.tile_base = (uint32_t)tiles;
    d.bin_base = (uint32_t)bins;
    d.image_base = image_bases[v];
    // Consecutive views of one scene form a view set (one scene read in K1).
    if (sets_host_.empty() || views[v - 1].scene != vs.scene ||
        sets_host_.back().count == kMaxSetViews) {
      sets_host_.push_back(ViewSetDev{v, 0, (uint32_t)blocks, (uint32_t)keys});
      blocks += preprocess_blocks(vs.scene->n);
      keys += key_blocks(vs.scene->n);
    }
    sets_host_.back().count++;
    d.set = (uint32_t)sets_host_.size() - 1;
    splats += vs.scene->n;
    tiles += d.p.num_tiles;
    bins += (uint64_t)bins_along(d.p.tiles_x) * bins_along(d.p.tiles_y);
    l.max_planes = std::max(l.max_planes, vs.scene->dev.planes);
  }
  if (splats > kMaxSortItems)
    throw Error(Code::Unsupported, "splats over the views of one run exceed 2^30 - 1");
  if (tiles > (1u << 24) || bins > kMaxBins)
    throw Error(Code::Unsupported, "too many tiles in one run");
  l.total_splats = (uint32_t)splats;
  l.sets = (uint32_t)sets_host_.size();
  l.total_blocks = (uint32_t)blocks;
  l.key_blocks = (uint32_t)keys;
  l.total_tiles = (uint32_t)tiles;
  l.total_bins = (uint32_t)bins;
  l.bin_passes = bin_sort_passes(l.total_bins);
  return l;
}

void Pipeline::ensure_workspace(const Layout &l) {
  const uint32_t n = std::max<uint32_t>(l.total_splats, 1);
  if (l.views > view_cap_ || n > splat_cap_ || !view_ws_.get()) {
    const auto t_grow = std::chrono::steady_clock::now();
    GSR_CUDA(cudaStreamSynchronize(stream_));  // earlier runs may still use the old buffers
    drop_graph();
    // Growth is geometric: a reallocation synchronises the device (cudaFree),
    // so a stream of batches of varying size must not regrow every time.
    const uint32_t vcap = l.views > view_cap_
                              ? std::min<uint32_t>(std::max(l.views, view_cap_ + view_cap_ / 2),
                                                   kMaxViewsPerLaunch)
                              : view_cap_;
    const uint32_t ncap = n > splat_cap_
                              ? (uint32_t)std::min<uint64_t>(
                                    std::max<uint64_t>(n, splat_cap_ + (uint64_t)splat_cap_ / 2),
                                    kMaxSortItems)
                              : splat_cap_;
    // view workspace: [view counters | K1 status | emit status] zeroed, then the table.
    const uint64_t k1_words = key_blocks(ncap) + 1;  // + views: blocks round up per set
    const uint64_t k1_total = k1_words + vcap;
    const uint64_t emit_words = emit_status_words(ncap);
    uint64_t off = 0;
    const uint64_t o_vc = off; off += align256(sizeof(ViewCounters) * vcap);
    const uint64_t o_k1 = off; off += align256(8 * k1_total);
    const uint64_t o_em = off; off += align256(8 * emit_words);
    view_zero_bytes_ = off;
    // the table: view sets, then views (one host-to-device copy per run);
    // the sets region is sized for the largest launch, so the table's layout
    // (and the pinned staging slots that mirror it) never changes
    const uint64_t o_sets = off; off += align256(sizeof(ViewSetDev) * kMaxViewsPerLaunch);
    const uint64_t o_tab = off; off += align256(sizeof(ViewDev) * vcap);
    view_ws_.reset(off, stream_);
    sets_dev_ = view_ws_.as<ViewSetDev>(o_sets);
    view_counters_ = view_ws_.as<ViewCounters>(o_vc);
    k1_status_ = view_ws_.as<unsigned long long>(o_k1);
    emit_status_ = view_ws_.as<unsigned long long>(o_em);
    views_dev_ = view_ws_.as<ViewDev>(o_tab);
    view_cap_ = vcap;
    // A staging slot has the device table's layout (sets, then views at
    // o_tab). The pinned host arrays are pinned once, for the largest launch
    // (freeing pinned memory waits for the whole device, which would stall
    // a growing lane behind every other stream's work).
    if (!table_pinned_) {
      const uint64_t slot_bytes = (o_tab - o_sets) + align256(sizeof(ViewDev) * kMaxViewsPerLaunch);
      GSR_CUDA(cudaMallocHost(&view_counters_pinned_, sizeof(ViewCounters) * kMaxViewsPerLaunch));
      GSR_CUDA(cudaMallocHost((void **)&table_pinned_, slot_bytes * kViewSlots));
      view_counters_pinned_cap_ = kMaxViewsPerLaunch;
      table_slot_bytes_ = slot_bytes;
    }
    table_sets_bytes_ = o_tab - o_sets;
    if (n > splat_cap_) {
      const uint64_t words = sort_work_words(ncap, 4);
      off = 0;
      uint64_t o_k0 = off; off += align256(4ull * ncap);
      uint64_t o_v0 = off; off += align256(4ull * ncap);
      uint64_t o_k1b = off; off += align256(4ull * ncap);
      uint64_t o_v1 = off; off += align256(4ull * ncap);
      uint64_t o_rect = off; off += align256(8ull * ncap);
      uint64_t o_rec = off; off += align256(sizeof(Record) * (uint64_t)ncap);
      uint64_t o_work = off; off += align256(4 * words);
      splat_ws_.reset(off, stream_);
      sorted_valid_ = false;  // the sorted ids lived in the old buffers
      vis_keys0_ = splat_ws_.as<uint32_t>(o_k0);
      vis_vals0_ = splat_ws_.as<uint32_t>(o_v0);
      vis_keys1_ = splat_ws_.as<uint32_t>(o_k1b);
      vis_vals1_ = splat_ws_.as<uint32_t>(o_v1);
      rects_ = splat_ws_.as<uint2>(o_rect);
      records_ = splat_ws_.as<Record>(o_rec);
      depth_sort_work_ = splat_ws_.as<uint32_t>(o_work);
      splat_cap_ = ncap;
      projected_.reset(0, stream_);
      debug_cov_.reset(0, stream_);
    }
    note_regrowth(std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() -
                                                            t_grow).count());
  }
  if (l.total_bins > bin_cap_ || !bin_ws_.get()) {
    const auto t_grow = std::chrono::steady_clock::now();
    GSR_CUDA(cudaStreamSynchronize(stream_));
    drop_graph();
    bin_cap_ = std::max(l.total_bins, bin_cap_ + bin_cap_ / 2);
    bin_ws_.reset(align256(8ull * std::max<uint32_t>(bin_cap_, 1)), stream_);
    ranges_ = bin_ws_.as<uint2>();
    note_regrowth(std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() -
                                                            t_grow).count());
  }
  if (key_cap_ == 0)
    ensure_key_workspace(std::min<uint64_t>(std::max<uint64_t>(kInitialPairsPerSplat * n, 1u << 20),
                                            kMaxSortItems));
  if (debug_) {
    const uint64_t need = sizeof(ProjectedDev) * (uint64_t)splat_cap_;
    if (projected_.size() < need) {
      GSR_CUDA(cudaStreamSynchronize(stream_));
      drop_graph();
      projected_.reset(need, stream_);
    }
    if (debug_cov_.size() < 8ull * splat_cap_) {
      GSR_CUDA(cudaStreamSynchronize(stream_));
      drop_graph();
      debug_cov_.reset(8ull * splat_cap_, stream_);
    }
    if (debug_pairs_.size() < 8 * key_cap_) {
      GSR_CUDA(cudaStreamSynchronize(stream_));
      drop_graph();
      debug_pairs_.reset(8 * key_cap_, stream_);
    }
  }
}

void Pipeline::ensure_key_workspace(uint64_t capacity) {
  if (key_cap_ >= capacity && key_ws_.get()) return;
  if (capacity > kMaxSortItems)
    throw Error(Code::Unsupported, "tile pair count " + std::to_string(capacity) +
                                       " exceeds the renderer's limit of 2^30 - 1");
  const auto t_grow = std::chrono::steady_clock::now();
  GSR_CUDA(cudaStreamSynchronize(stream_));
  drop_graph();
  // geometric growth, as for the other workspaces
  const uint32_t cap = (uint32_t)std::min<uint64_t>(
      std::max<uint64_t>(capacity, key_cap_ + key_cap_ / 4), kMaxSortItems);
  const uint64_t words = sort_work_words(cap, kPairSortPasses);
  uint64_t off = 0;
  uint64_t o_k0 = off; off += align256(4ull * cap);
  uint64_t o_v0 = off; off += align256(4ull * cap);
  uint64_t o_k1 = off; off += align256(4ull * cap);
  uint64_t o_v1 = off; off += align256(4ull * cap);
  uint64_t o_work = off; off += align256(4 * words);
  key_ws_.reset(off, stream_);
  pair_keys0_ = key_ws_.as<uint32_t>(o_k0);
  pair_vals0_ = key_ws_.as<uint32_t>(o_v0);
  pair_keys1_ = key_ws_.as<uint32_t>(o_k1);
  pair_vals1_ = key_ws_.as<uint32_t>(o_v1);
  pair_sort_work_ = key_ws_.as<uint32_t>(o_work);
  key_cap_ = cap;
  debug_pairs_.reset(0, stream_);
  note_regrowth(std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() -
                                                          t_grow).count());
}

RunInit Pipeline::make_run_init(const Layout &l) const {
  RunInit init{};
  constexpr size_t kKept = offsetof(FrameCounters, k1_ticket);
  init.zero[0] = fixed_.as<uint32_t>(kKept);
  init.zero_words[0] = ((char *)depth_plan_ - (char *)fixed_.get() - kKept) / 4;
  init.phase_ns = counters_->phase_ns;
  init.zero[1] = view_ws_.as<uint32_t>();
  init.zero_words[1] = view_zero_bytes_ / 4;
  init.zero[2] = reinterpret_cast<uint32_t *>(ranges_);
  init.zero_words[2] = 2ull * l.total_bins;
  init.zero[3] = depth_sort_work_;
  init.zero_words[3] = kSortScratchHeadWords;
  init.zero[4] = pair_sort_work_;
  init.zero_words[4] = kSortScratchHeadWords;
  if (l.views <= kRunInlineViews && !batch_mode_) {
    init.inline_views = l.views;
    init.inline_sets = l.sets;
    init.sets_dst = sets_dev_;
    init.views_dst = views_dev_;
    std::memcpy(init.sets, sets_host_.data(), sizeof(ViewSetDev) * l.sets);
    std::memcpy(init.views, views_host_.data(), sizeof(ViewDev) * l.views);
  }
  return init;
}

void Pipeline::launch_all(const Layout &l, uint32_t *images, const HostSinks &sinks,
                          bool reuse, const ViewDev *views_dev, const ViewSetDev *sets_dev) {
  const uint32_t n = std::max<uint32_t>(l.total_splats, 1);
  launch_run_init(make_run_init(l), stream_);

  K1Buffers k1{vis_keys0_, vis_vals0_, rects_,         records_,
               k1_status_, counters_,  key_hist_,      view_counters_,
               debug_ ? projected_.as<ProjectedDev>() : nullptr, reuse};
  // The depth keys and their sort run on the side stream, beside the vertex
  // stage, and ahead of it where both want an SM (the sort's passes are few
  // blocks that wait for one another, the vertex stage many that do not). The
  // keys beside it too: 3M splats 1,495 -> 1,480 us, 64 thumbnails 457 -> 451.
  if (reuse) {  // a reused order keeps the last sort's ids and plan
    launch_keys(views_dev, sets_dev, l.sets, l.key_blocks, k1, std::nullopt, stream_);
  } else {
    GSR_CUDA(cudaEventRecord(fork_ev_, stream_));
    GSR_CUDA(cudaStreamWaitEvent(side_stream_, fork_ev_, 0));
    launch_keys(views_dev, sets_dev, l.sets, l.key_blocks, k1, side_priority_, side_stream_);
    SortBuffers ds{vis_keys0_, vis_vals0_, vis_keys1_, vis_vals1_, &counters_->visible, n, 0, 4,
                   depth_plan_, depth_sort_work_, &counters_->error, key_hist_, true};
    ds.priority = side_priority_;
    launch_sort(ds, side_stream_);
    GSR_CUDA(cudaEventRecord(join_ev_, side_stream_));
  }
  launch_preprocess(views_dev, sets_dev, l.sets, l.total_blocks, l.max_planes, k1, debug_,
                    stream_);
  if (!reuse) GSR_CUDA(cudaStreamWaitEvent(stream_, join_ev_, 0));

  EmitBuffers eb{depth_plan_, vis_vals0_,  vis_vals1_, rects_,        records_,
                 pair_keys0_, pair_vals0_, key_cap_,   emit_status_,  counters_,
                 view_counters_, bin_hist_, l.bin_passes, bin_wide_bits(l.total_bins),
                 l.total_splats, views_dev, l.views, tile_};
  launch_emit(eb, stream_);
  if (debug_) {
    GSR_CUDA(cudaMemcpyAsync(debug_pairs_.as<uint32_t>(), pair_keys0_, 4 * key_cap_,
                             cudaMemcpyDeviceToDevice, stream_));
    GSR_CUDA(cudaMemcpyAsync(debug_pairs_.as<uint32_t>(4 * key_cap_), pair_vals0_, 4 * key_cap_,
                             cudaMemcpyDeviceToDevice, stream_));
  }
  SortBuffers ts{pair_keys0_, pair_vals0_, pair_keys1_, pair_vals1_, &counters_->pairs,
                 (uint32_t)key_cap_, kBinCodeBits, l.bin_passes, bin_plan_, pair_sort_work_,
                 &counters_->error, bin_hist_, true};
  ts.expected = std::max<uint32_t>((uint32_t)(key_cap_ / kPairsPerBinPair), 1);
  ts.wide_bits = bin_wide_bits(l.total_bins);
  ts.start_ns = &counters_->phase_ns[kPhaseTileSort];
  launch_sort(ts, stream_);
  launch_ranges(bin_plan_, pair_keys0_, pair_keys1_, counters_, (uint32_t)key_cap_, ranges_,
                stream_);
  RasterArgs ra{views_dev,  l.views,  l.total_tiles, ranges_,   bin_plan_,
                pair_keys0_, pair_vals0_, pair_keys1_, pair_vals1_, records_, images, counters_,
                sticky_,     view_counters_, sinks.counters, sinks.views,
                batch_mode_ ? nullptr : &sinks.counters->phase_ns[kPhaseCount]};
  if (debug_) {
    GSR_CUDA(cudaMemsetAsync(debug_cov_.get(), 0xff, 8ull * std::max<uint32_t>(l.total_splats, 1),
                             stream_));
    ra.debug_cov = debug_cov_.as<float2>();
  }
  launch_raster(ra, tile_, blend_mode_, raster_cfg_, sm_count_, stream_);
}

void Pipeline::enqueue(const ViewSpec *views, uint32_t count, uint32_t *images,
                       const uint64_t *image_bases, HostSinks sinks) {
  GSR_CUDA(cudaSetDevice(device_));
  const Layout l = plan_views(views, count, image_bases);
  ensure_workspace(l);
  if (!sinks.counters) sinks = HostSinks{counters_host_, view_counters_pinned_};
  // The last sorted order can be reused only for the identical layout (same
  // scenes, sizes and tile grid) and while its buffers are intact.
  const bool reuse = reuse_request_ && sorted_valid_ && l == sorted_layout_ &&
                     std::equal(views, views + count, sorted_scenes_.begin(), sorted_scenes_.end(),
                                [](const ViewSpec &v, const DeviceScene *s) { return v.scene == s; });
  // A small view table rides in the zeroing kernel's parameters. A larger
  // one goes up from a pinned ring slot, ahead of the run on its stream
  // (outside the run's graph, so the graph serves every frame of the
  // layout); the slot's previous copy is long done in steady state.
  const bool inline_table = l.views <= kRunInlineViews;
  if (!inline_table) {
    const uint32_t slot = slot_;
    GSR_CUDA(cudaEventSynchronize(slot_ev_[slot]));
    unsigned char *staged = table_pinned_ + (uint64_t)slot * table_slot_bytes_;
    std::memcpy(staged, sets_host_.data(), sizeof(ViewSetDev) * l.sets);
    std::memcpy(staged + table_sets_bytes_, views_host_.data(), sizeof(ViewDev) * l.views);
    GSR_CUDA(cudaMemcpyAsync(sets_dev_, staged, table_sets_bytes_ + sizeof(ViewDev) * l.views,
                             cudaMemcpyHostToDevice, stream_));
    GSR_CUDA(cudaEventRecord(slot_ev_[slot], stream_));
    slot_ = (slot_ + 1) % kViewSlots;
  }
  ViewDev *run_views = views_dev_;
  ViewSetDev *run_sets = sets_dev_;

  if (!use_graph_) {
    launch_all(l, images, sinks, reuse, run_views, run_sets);
  } else {
    const GraphKey key{l,     images,      key_cap_,       tile_,       blend_mode_,
                       debug_, raster_cfg_, sinks.counters, sinks.views, reuse};
    GraphEntry *hit = nullptr;
    for (auto &g : graphs_)
      if (g.key == key) hit = &g;
    // A layout is captured the second time it is seen: one-off layouts (a
    // served batch of a new size) launch directly instead of paying for a
    // capture they would never replay.
    bool seen = false;
    if (!hit) {
      for (auto &k : seen_keys_)
        if (k == key) seen = true;
      if (!seen) {
        if (seen_keys_.size() >= kGraphCacheSize) seen_keys_.erase(seen_keys_.begin());
        seen_keys_.push_back(key);
      }
    }
    if (!hit && !seen) {
      launch_all(l, images, sinks, reuse, run_views, run_sets);
    } else if (!hit) {
      if (graphs_.size() >= kGraphCacheSize) {
        auto lru = std::min_element(graphs_.begin(), graphs_.end(),
                                    [](const GraphEntry &a, const GraphEntry &b) {
                                      return a.last_use < b.last_use;
                                    });
        cudaGraphExecDestroy(lru->exec);
        cudaGraphDestroy(lru->graph);
        graphs_.erase(lru);
      }
      cudaGraph_t g = nullptr;
      const auto t_capture = std::chrono::steady_clock::now();
      GSR_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
      try {
        launch_all(l, images, sinks, reuse, run_views, run_sets);
      } catch (...) {
        cudaStreamEndCapture(stream_, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        throw;
      }
      GSR_CUDA(cudaStreamEndCapture(stream_, &g));
      cudaGraphExec_t exec = nullptr;
      cudaError_t e = cudaGraphInstantiate(&exec, g, cudaGraphInstantiateFlagUseNodePriority);
      if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        throw Error(Code::Internal, std::string("CUDA graph instantiation failed: ") +
                                        cudaGetErrorString(e));
      }
      GraphEntry entry{key, exec, 0, g, nullptr, {}};
      size_t count = 0;
      GSR_CUDA(cudaGraphGetNodes(g, nullptr, &count));
      std::vector<cudaGraphNode_t> nodes(count);
      GSR_CUDA(cudaGraphGetNodes(g, nodes.data(), &count));
      for (cudaGraphNode_t node : nodes) {
        cudaGraphNodeType type;
        GSR_CUDA(cudaGraphNodeGetType(node, &type));
        if (type != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp{};
        GSR_CUDA(cudaGraphKernelNodeGetParams(node, &kp));
        if (kp.func == run_init_kernel_entry()) {
          entry.init_node = node;
          entry.init_params = kp;
          break;
        }
      }
      if (inline_table && !entry.init_node) {
        cudaGraphExecDestroy(exec);
        cudaGraphDestroy(g);
        throw Error(Code::Internal, "captured run has no zeroing kernel node");
      }
      graphs_.push_back(entry);
      hit = &graphs_.back();
      captures_.fetch_add(1, std::memory_order_relaxed);
      const double ms = std::chrono::duration<double, std::milli>(
                            std::chrono::steady_clock::now() - t_capture).count();
      capture_ms_.store(capture_ms_.load(std::memory_order_relaxed) + ms,
                        std::memory_order_relaxed);
    }
    if (hit) {
      hit->last_use = ++graph_clock_;
      if (inline_table) {
        // this run's view table, in the zeroing node's parameters
        RunInit init = make_run_init(l);
        void *args[] = {&init};
        cudaKernelNodeParams kp = hit->init_params;
        kp.kernelParams = args;
        kp.extra = nullptr;
        GSR_CUDA(cudaGraphExecKernelNodeSetParams(hit->exec, hit->init_node, &kp));
      }
      GSR_CUDA(cudaGraphLaunch(hit->exec, stream_));
    }
  }
  GSR_CUDA(cudaGetLastError());
  last_layout_ = l;
  last_sinks_ = sinks;
  has_run_ = true;
  last_reused_ = reuse;
  if (!reuse) {
    sorted_layout_ = l;
    sorted_valid_ = true;
    sorted_scenes_.clear();
    for (uint32_t v = 0; v < count; ++v) sorted_scenes_.push_back(views[v].scene);
  }
}

void Pipeline::enqueue_groups(const ViewSpec *views, uint32_t *images,
                              const uint64_t *image_bases, const std::vector<GroupRun> &groups) {
  GSR_CUDA(cudaSetDevice(device_));
  if (!use_graph_ || groups.empty()) {
    for (const GroupRun &g : groups)
      enqueue(views + g.first, g.count, images, image_bases + g.first, g.sinks);
    return;
  }
  // Size the workspace for every group first (growing it drops the graphs),
  // then stage every group's view table in the pinned area.
  std::vector<Layout> layouts;
  layouts.reserve(groups.size());
  for (const GroupRun &g : groups) {
    layouts.push_back(plan_views(views + g.first, g.count, image_bases + g.first));
    ensure_workspace(layouts.back());
  }
  std::vector<uint64_t> offs(groups.size());
  uint64_t total = 0;
  for (size_t k = 0; k < groups.size(); ++k) {
    offs[k] = total;
    total += (table_sets_bytes_ + sizeof(ViewDev) * layouts[k].views + 255) & ~uint64_t(255);
  }
  // the previous batch launch must have read the staging area
  if (batch_ev_) GSR_CUDA(cudaEventSynchronize(batch_ev_));
  else GSR_CUDA(cudaEventCreateWithFlags(&batch_ev_, cudaEventDisableTiming));
  if (total > batch_stage_bytes_) {
    drop_batch_graphs();  // the captured copies read the old area
    if (batch_stage_) cudaFreeHost(batch_stage_);
    batch_stage_ = nullptr;
    batch_stage_bytes_ = 0;
    GSR_CUDA(cudaMallocHost((void **)&batch_stage_, total + total / 4));
    batch_stage_bytes_ = total + total / 4;
  }
  for (size_t k = 0; k < groups.size(); ++k) {
    plan_views(views + groups[k].first, groups[k].count, image_bases + groups[k].first);
    std::memcpy(batch_stage_ + offs[k], sets_host_.data(), sizeof(ViewSetDev) * layouts[k].sets);
    std::memcpy(batch_stage_ + offs[k] + table_sets_bytes_, views_host_.data(),
                sizeof(ViewDev) * layouts[k].views);
  }
  BatchKey key{layouts, {}, {}, images, key_cap_, tile_, blend_mode_, debug_, raster_cfg_};
  for (const GroupRun &g : groups) {
    key.counters.push_back(g.sinks.counters);
    key.views.push_back(g.sinks.views);
  }
  // The groups in stream order: each copies its table into the device table
  // (no inline tables) and runs the frame pipeline over it.
  auto launch_groups = [&]() {
    for (size_t k = 0; k < groups.size(); ++k) {
      GSR_CUDA(cudaMemcpyAsync(sets_dev_, batch_stage_ + offs[k],
                               table_sets_bytes_ + sizeof(ViewDev) * layouts[k].views,
                               cudaMemcpyHostToDevice, stream_));
      launch_all(layouts[k], images, groups[k].sinks, false, views_dev_, sets_dev_);
    }
  };
  BatchGraph *hit = nullptr;
  for (auto &g : batch_graphs_)
    if (g.key == key) hit = &g;
  const bool seen = std::find(batch_seen_.begin(), batch_seen_.end(), key) != batch_seen_.end();
#ifdef GSR_BATCH_DEBUG
  fprintf(stderr, "batch: groups %zu hit %d seen %d graphs %zu seen_list %zu key_cap %llu images %p\n",
          groups.size(), hit != nullptr, (int)seen, batch_graphs_.size(), batch_seen_.size(),
          (unsigned long long)key_cap_, (void *)images);
  if (!batch_seen_.empty()) {
    const BatchKey &o = batch_seen_.back();
    fprintf(stderr, "  vs last seen: layouts %d counters %d views %d images %d cap %d tile %d blend %d dbg %d raster %d\n",
            o.layouts == key.layouts, o.counters == key.counters, o.views == key.views,
            o.images == key.images, o.key_cap == key.key_cap, o.tile == key.tile, o.blend == key.blend,
            o.debug == key.debug, o.raster == key.raster);
  }
#endif
  batch_mode_ = true;
  try {
    if (!hit && !seen) {
      // first sighting: direct launches (a one-off batch pays no capture)
      if (batch_seen_.size() >= kBatchGraphCacheSize) batch_seen_.erase(batch_seen_.begin());
      batch_seen_.push_back(key);
      launch_groups();
    } else {
      if (!hit) {
        if (batch_graphs_.size() >= kBatchGraphCacheSize) {
          auto lru = std::min_element(
              batch_graphs_.begin(), batch_graphs_.end(),
              [](const BatchGraph &a, const BatchGraph &b) { return a.last_use < b.last_use; });
          cudaGraphExecDestroy(lru->exec);
          cudaGraphDestroy(lru->graph);
          batch_graphs_.erase(lru);
        }
        const auto t_capture = std::chrono::steady_clock::now();
        cudaGraph_t g = nullptr;
        GSR_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
        try {
          launch_groups();
        } catch (...) {
          cudaStreamEndCapture(stream_, &g);
          if (g) cudaGraphDestroy(g);
          cudaGetLastError();
          throw;
        }
        GSR_CUDA(cudaStreamEndCapture(stream_, &g));
        cudaGraphExec_t exec = nullptr;
        const cudaError_t e = cudaGraphInstantiate(&exec, g, cudaGraphInstantiateFlagUseNodePriority);
        if (e != cudaSuccess) {
          cudaGraphDestroy(g);
          throw Error(Code::Internal, std::string("CUDA graph instantiation failed: ") +
                                          cudaGetErrorString(e));
        }
        batch_graphs_.push_back(BatchGraph{key, g, exec, 0});
        hit = &batch_graphs_.back();
        captures_.fetch_add(1, std::memory_order_relaxed);
        const double ms = std::chrono::duration<double, std::milli>(
                              std::chrono::steady_clock::now() - t_capture).count();
        capture_ms_.store(capture_ms_.load(std::memory_order_relaxed) + ms,
                          std::memory_order_relaxed);
      }
      hit->last_use = ++graph_clock_;
      GSR_CUDA(cudaGraphLaunch(hit->exec, stream_));
      ++batch_graph_launches_;
    }
  } catch (...) {
    batch_mode_ = false;
    throw;
  }
  batch_mode_ = false;
  GSR_CUDA(cudaEventRecord(batch_ev_, stream_));
  GSR_CUDA(cudaGetLastError());
  last_layout_ = layouts.back();
  last_sinks_ = groups.back().sinks;
  has_run_ = true;
  last_reused_ = false;
  sorted_valid_ = false;  // a batch never hands its order to a later frame
}

// By the kernels' own clock readings (the stream is synchronised).
void Pipeline::phase_times(float out[kPhaseCount]) const {
  unsigned long long at = last_sinks_.counters->phase_ns[0];
  for (int k = 0; k < kPhaseCount; ++k) {
    const unsigned long long next = std::max(at, last_sinks_.counters->phase_ns[k + 1]);
    out[k] = (float)((double)(next - at) * 1e-6);
    at = next;
  }
}

void Pipeline::collect(RunResult &r) {
  float t[kPhaseCount];
  phase_times(t);
  for (int k = 0; k < kPhaseCount; ++k) r.phase_ms[k] = t[k];
  r.preprocess_ms = t[kPhasePreprocess];
  r.sort_ms = t[kPhaseDepthSort] + t[kPhaseEmit] + t[kPhaseTileSort] + t[kPhaseRanges];
  r.raster_ms = t[kPhaseRaster];
  r.sorted = !last_reused_;
  r.visible = last_sinks_.counters->visible;
  r.drawn = last_sinks_.counters->drawn;
  r.keys = last_sinks_.counters->keys;
  view_counters_host_.assign(last_sinks_.views, last_sinks_.views + last_layout_.views);
}

// The error bits of the runs since the last call (the stream is synchronised),
// cleared on both sides.
uint32_t Pipeline::take_sticky() {
  const uint32_t sticky = last_sinks_.counters->sticky;
  if (sticky) {
    last_sinks_.counters->sticky = 0;
    GSR_CUDA(cudaMemsetAsync(sticky_, 0, 4, stream_));
  }
  return sticky;
}

RunResult Pipeline::run(const ViewSpec *views, uint32_t count, uint32_t *images,
                        const uint64_t *image_bases) {
  auto t0 = std::chrono::steady_clock::now();
  RunResult r;
  for (;;) {
    enqueue(views, count, images, image_bases);
    GSR_CUDA(cudaStreamSynchronize(stream_));
    if (counters_host_->error)
      throw Error(Code::Internal, "device wait limit reached in a look-back scan (error bits " +
                                      std::to_string(counters_host_->error) + ")");
    if (!counters_host_->overflow) break;
    // Grow the pair buffers to the exact need plus headroom and run again.
    const uint64_t need = counters_host_->keys;
    if (need > kMaxSortItems)
      throw Error(Code::Unsupported, "tile pair count " + std::to_string(need) +
                                         " exceeds the renderer's limit of 2^30 - 1");
    ensure_key_workspace(std::min<uint64_t>(need + need / 4 + 1024, kMaxSortItems));
    if (debug_) debug_pairs_.reset(8 * key_cap_, stream_);
    ++r.reruns;
  }
  take_sticky();
  collect(r);
  r.frame_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
  last_ = r;
  return r;
}

RunResult Pipeline::sync() {
  GSR_CUDA(cudaSetDevice(device_));
  GSR_CUDA(cudaStreamSynchronize(stream_));
  RunResult r;
  if (!has_run_) return r;
  const uint32_t sticky = take_sticky();
  collect(r);
  r.frame_ms = r.preprocess_ms + r.sort_ms + r.raster_ms;
  last_ = r;
  if (sticky & 0x7fffffffu)
    throw Error(Code::Internal, "device wait limit reached in a look-back scan");
  if (sticky & 0x80000000u)
    throw Error(Code::Internal,
                "an enqueued frame overflowed its tile-pair buffers; render it synchronously "
                "once to size them");
  return r;
}

uint32_t Pipeline::launches_per_run() const {
  // keys; preprocess; depth sort plan + 4 passes (histograms come from the
  // keys); emit; bin sort plan + passes (histograms from K2); ranges; raster.
  const uint32_t bin_passes = last_layout_.bin_passes;
  return 2 + (1 + 4) + 1 + (1 + bin_passes) + 1 + 1;
}

SortPlan Pipeline::read_plan(int which) {
  SortPlan plan;
  GSR_CUDA(cudaMemcpyAsync(&plan, which == 0 ? depth_plan_ : bin_plan_, sizeof(SortPlan),
                           cudaMemcpyDeviceToHost, stream_));
  GSR_CUDA(cudaStreamSynchronize(stream_));
  return plan;
}

std::vector<uint32_t> Pipeline::debug_order() {
  GSR_CUDA(cudaSetDevice(device_));
  SortPlan plan = read_plan(0);
  std::vector<uint32_t> out(plan.n);
  if (!out.empty())
    GSR_CUDA(cudaMemcpy(out.data(), plan.final_buffer == 0 ? vis_vals0_ : vis_vals1_,
                        4 * out.size(), cudaMemcpyDeviceToHost));
  return out;
}

std::vector<ProjectedDev> Pipeline::debug_projected(uint32_t count) {
  if (!debug_ || !projected_.get())
    throw Error(Code::InvalidArgument, "debug taps were not enabled for the last frame");
  GSR_CUDA(cudaSetDevice(device_));
  std::vector<ProjectedDev> out(count);
  if (count)
    GSR_CUDA(cudaMemcpy(out.data(), projected_.get(), sizeof(ProjectedDev) * count,
                        cudaMemcpyDeviceToHost));
  return out;
}

std::vector<float2> Pipeline::debug_coverage(uint32_t count) {
  if (!debug_ || !debug_cov_.get())
    throw Error(Code::InvalidArgument, "debug taps were not enabled for the last frame");
  GSR_CUDA(cudaSetDevice(device_));
  std::vector<float2> out(count);
  if (count)
    GSR_CUDA(cudaMemcpy(out.data(), debug_cov_.get(), sizeof(float2) * count,
                        cudaMemcpyDeviceToHost));
  return out;
}

// The (tile, splat) pairs of the frame in emission order (depth order, tile
// rows outer), from the (bin, splat) pairs: a splat's pairs lie together, bin
// rows outer, so its tile row r is row r % 4 of its bins of that bin row.
void Pipeline::debug_tile_pairs(std::vector<uint32_t> &tiles, std::vector<uint32_t> &ids) {
  if (!debug_ || !debug_pairs_.get())
    throw Error(Code::InvalidArgument, "debug taps were not enabled for the last frame");
  GSR_CUDA(cudaSetDevice(device_));
  const uint64_t n = std::min<uint64_t>(last_sinks_.counters->pairs, key_cap_);
  std::vector<uint32_t> keys(n), vals(n);
  if (n) {
    GSR_CUDA(cudaMemcpy(keys.data(), debug_pairs_.get(), 4 * n, cudaMemcpyDeviceToHost));
    GSR_CUDA(cudaMemcpy(vals.data(), debug_pairs_.as<uint32_t>(4 * key_cap_), 4 * n,
                        cudaMemcpyDeviceToHost));
  }
  tiles.clear();
  ids.clear();
  tiles.reserve(last_.keys);
  ids.reserve(last_.keys);
  const uint32_t tiles_x = views_host_[0].p.tiles_x, bins_x = bins_along(tiles_x);
  for (uint64_t i = 0; i < n;) {
    const uint32_t row = (keys[i] >> kBinCodeBits) / bins_x;
    uint64_t end = i;
    while (end < n && vals[end] == vals[i] && (keys[end] >> kBinCodeBits) / bins_x == row) ++end;
    for (uint32_t r = 0; r < kBinEdge; ++r)
      for (uint64_t k = i; k < end; ++k) {
        const uint32_t col = (keys[k] >> kBinCodeBits) % bins_x;
        for (uint32_t c = 0; c < kBinEdge; ++c)
          if (bin_code_tiles(keys[k]) >> (kBinEdge * r + c) & 1u) {
            tiles.push_back((row * kBinEdge + r) * tiles_x + col * kBinEdge + c);
            ids.push_back(vals[k]);
          }
      }
    i = end;
  }
}

// Every tile's list, from what the raster reads: the bins' ranges, the tiles'
// words (in the key buffer the sort has left free) and the sorted ids.
void Pipeline::debug_tile_ranges(uint32_t num_tiles, std::vector<uint32_t> &ranges,
                                 std::vector<uint32_t> &ids) {
  GSR_CUDA(cudaSetDevice(device_));
  SortPlan plan = read_plan(1);
  const bool first = plan.final_buffer == 0;
  const uint64_t n = std::min<uint64_t>(last_sinks_.counters->pairs, key_cap_);
  const FrameParams &p = views_host_[0].p;
  const uint32_t bins_x = bins_along(p.tiles_x);
  std::vector<uint32_t> words(tile_words(n)), sorted(n);
  std::vector<uint2> bin_ranges((size_t)bins_x * bins_along(p.tiles_y));
  auto fetch = [](auto &to, const void *from) {
    if (!to.empty())
      GSR_CUDA(cudaMemcpy(to.data(), from, sizeof(to[0]) * to.size(), cudaMemcpyDeviceToHost));
  };
  fetch(words, first ? pair_keys1_ : pair_keys0_);
  fetch(sorted, first ? pair_vals0_ : pair_vals1_);
  fetch(bin_ranges, ranges_);
  ranges.assign(2ull * num_tiles, 0);
  ids.clear();
  for (uint32_t t = 0; t < std::min(num_tiles, p.num_tiles); ++t) {
    const uint32_t tx = t % p.tiles_x, ty = t / p.tiles_x;
    const uint2 r = bin_ranges[ty / kBinEdge * bins_x + tx / kBinEdge];
    const uint32_t at = (uint32_t)ids.size();
    each_tile_position(words.data(), r.x, std::min<uint32_t>(r.y, (uint32_t)n),
                       ty % kBinEdge * kBinEdge + tx % kBinEdge,
                       [&](uint32_t i) { ids.push_back(sorted[i]); });
    if (ids.size() > at) {
      ranges[2ull * t] = at;
      ranges[2ull * t + 1] = (uint32_t)ids.size();
    }
  }
}

}  // namespace gsr
