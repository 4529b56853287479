// Layout of the tile passes' per-segment start tables and their level limits,
// shared by the kernels and the host planner (compiles with or without CUDA).
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define PWMGPU_HOST_DEVICE __host__ __device__
#else
#define PWMGPU_HOST_DEVICE
#endif

namespace pwmgpu {

constexpr int kTileMaxLevels = 4;
// A last pass whose finest-run prefixes are given (the histogram kernel's, for
// texts of at most 8 levels) neither counts nor looks back, and may split up
// to 7 times: all levels of such a text in one pass.
constexpr int kTileGivenMaxLevels = 8;

constexpr int kTileThreads = 256;
constexpr int kTileVectors = 4;  // 16-byte vectors per thread: 64 bytes of keys

// The histogram kernel reads a tile in equal units of at most kTileVectors
// vectors a thread, each loaded while the one before is counted: one for the
// usual tiles and smaller ones, 2 or 4 for those of 8 or 16 vectors.
PWMGPU_HOST_DEVICE constexpr uint32_t tile_hist_units(uint64_t tile_bytes) {
  return tile_bytes <= uint64_t(16 * kTileVectors) * kTileThreads
             ? 1u
             : uint32_t(tile_bytes / (uint64_t(16 * kTileVectors) * kTileThreads));
}

// Tiles of a histogram block: at most 16 (one-pass builds choose); else 16 of
// the usual size, and as many bytes of wider ones, so that a text keeps its
// number of blocks.
constexpr uint32_t kTileHistMaxTiles = 16;
PWMGPU_HOST_DEVICE constexpr uint32_t tile_hist_tiles_per_block(uint64_t tile_bytes) {
  return kTileHistMaxTiles / tile_hist_units(tile_bytes);
}

// Table entries of one segment: matrix starts (level j, run v) at
// (1 << j) - 1 + v, tree starts after them, then the S_out starts (2^K).
PWMGPU_HOST_DEVICE constexpr int tile_table_size(int K) { return 2 * ((1 << K) - 1) + (1 << K); }
PWMGPU_HOST_DEVICE constexpr int tile_wm_entry(int j, int v) { return (1 << j) - 1 + v; }
PWMGPU_HOST_DEVICE constexpr int tile_wt_entry(int K, int j, int v) { return (1 << K) - 1 + (1 << j) - 1 + v; }
PWMGPU_HOST_DEVICE constexpr int tile_out_entry(int K, int v) { return 2 * ((1 << K) - 1) + v; }

}  // namespace pwmgpu
