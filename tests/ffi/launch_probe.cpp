// The kernels' launch code over a stand-in for the CUDA runtime with two
// devices: no GPU, no kernel runs. Prints one line per launch: the device, the
// dynamic shared memory it asks for, the limit raised for that kernel on that
// device (0: none), and the launch's priority attribute ("-": none).
//   launch_probe preprocess|emit|sort|sort-high
// "raster" prints the shape raster_shape names for every configuration and
// number of tiles, and the kernel (as a number) and grid launch_raster launches
// for it; "raster-tile" the chunk kept over changes of the tile size.
// "work" prints pair capacities, the words of their sort's scratch and the bytes
// a pair is counted with in place of launches.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <map>
#include <utility>

#include "device_types.h"
#include "kernels.h"

namespace {
int device = 0;
std::map<std::pair<int, const void *>, int> limits;

std::map<const void *, int> kernels;
int last_kernel = -1;
unsigned last_grid = 0;

void note(const void *func, size_t smem, const char *priority, dim3 grid) {
  last_kernel = kernels.emplace(func, (int)kernels.size()).first->second;
  last_grid = grid.x;
  auto it = limits.find({device, func});
  std::printf("launch %d %zu %d %s\n", device, smem, it == limits.end() ? 0 : it->second, priority);
}

struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} config;
}  // namespace

extern "C" {
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(cudaStream_t *)stream = config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *func, dim3 grid, dim3, void **, size_t smem, cudaStream_t) {
  note(func, smem, "-", grid);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *func, void **) {
  char priority[16] = "-";
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributePriority)
      std::snprintf(priority, sizeof priority, "%d", c->attrs[k].val.priority);
  note(func, c->dynamicSmemBytes, priority, c->gridDim);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *func, cudaFuncAttribute attr, int value) {
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) limits[{device, func}] = value;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *value, cudaDeviceAttr, int) {
  *value = 148;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                   unsigned) {
  *n = 3;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

using namespace gsr;

int main(int argc, char **argv) {
  const char *what = argc > 1 ? argv[1] : "";
  for (device = 0; device < 2; ++device) {
    if (!std::strcmp(what, "preprocess")) {
      // frames of every SH degree, with few blocks and with many
      K1Buffers b{};
      for (uint32_t planes : {1u, 3u, 7u, 12u, 19u})
        for (uint32_t blocks : {1u, 100000u})
          launch_preprocess(nullptr, nullptr, 1, blocks, planes, b, false, nullptr);
    } else if (!std::strcmp(what, "emit")) {
      // runs of the most views, with few ids and with many
      for (uint32_t n : {1000u, 10'000'000u}) {
        EmitBuffers b{};
        b.n = n;
        b.num_views = kMaxViewsPerLaunch;
        launch_emit(b, nullptr);
      }
    } else if (!std::strncmp(what, "sort", 4)) {
      const bool high = !std::strcmp(what, "sort-high");
      const uint32_t hist[1] = {};
      for (uint32_t bits : {0u, 9u, 10u})
        for (uint32_t capacity : {1000u, 1u << 22, 1u << 25}) {
          SortBuffers b{};
          b.capacity = capacity;
          if (high) {  // as a frame's depth sort: histograms given, a priority asked for
            b.hist = hist;
            b.priority = -5;
          }
          b.passes = bits ? 1 : 4;
          b.wide_bits = bits;
          launch_sort(b, nullptr);
        }
    } else if (!std::strcmp(what, "raster")) {
      for (uint32_t tiles : {1u, 592u, 593u, 1036u, 1037u, 2368u, 2369u, 8160u})
        for (uint32_t mode : {0u, 1u})
          for (uint32_t tile : {8u, 16u})
            for (uint32_t chunk : {32u, 64u, 128u, 256u})
              for (uint32_t bps : {0u, 2u}) {
                const RasterConfig cfg{chunk, bps, true};
                if (!raster_config_valid(tile, cfg)) continue;
                const RasterShape s = raster_shape(tiles, tile, mode, cfg, 148);
                RasterArgs a{};
                a.total_tiles = tiles;
                launch_raster(a, tile, mode, cfg, 148, nullptr);
                std::printf("raster %u %u %u %u %u %u %u %u %u %d %u\n", tiles, mode, tile, chunk,
                            bps, s.chunk, s.blocks, s.blocks_per_sm, s.tile + 100 * s.blend_mode,
                            last_kernel, last_grid);
              }
    } else if (!std::strcmp(what, "raster-tile")) {
      // chunk (0: never set) at a first tile size, then at the other, then back
      for (uint32_t tile : {16u, 8u})
        for (uint32_t chunk : {0u, 32u, 64u, 128u, 256u}) {
          RasterConfig c = raster_config_at(tile, RasterConfig{});
          if (chunk) c = {chunk, 3, true};
          if (!raster_config_valid(tile, c)) continue;
          const RasterConfig there = raster_config_at(24 - tile, c);
          const RasterConfig back = raster_config_at(tile, there);
          std::printf("raster-tile %u %u %u %u %u %u\n", tile, chunk, there.chunk, back.chunk,
                      there.blocks_per_sm, back.blocks_per_sm);
        }
    } else if (!std::strcmp(what, "work")) {
      for (uint32_t capacity : {1u << 20, 3'000'001u, 1u << 28})
        std::printf("work %u %llu %llu\n", capacity,
                    (unsigned long long)sort_work_words(capacity, kPairSortPasses),
                    (unsigned long long)kPairWorkspaceBytes);
    } else {
      return 2;
    }
  }
  return 0;
}
