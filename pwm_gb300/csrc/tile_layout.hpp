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

// Keys of one tile for a key width and 16-byte vectors a thread (0: the usual).
PWMGPU_HOST_DEVICE constexpr uint32_t tile_pass_elems(uint32_t key_bytes, uint32_t vectors = 0) {
  return uint32_t(kTileThreads) * (vectors ? vectors : uint32_t(kTileVectors)) * (16 / key_bytes);
}

// The narrowest key width (1, 2 or 4 bytes) holding `bits` bits.
PWMGPU_HOST_DEVICE constexpr uint32_t tile_key_bytes(uint32_t bits) { return bits <= 8 ? 1u : (bits <= 16 ? 2u : 4u); }

// Whether launch_tile_pass has a kernel for a pass of K levels over keys of
// key_bytes in tiles of `vectors` a thread (0: the usual), with `out` writing
// S_{l+K} in keys of out_bytes; given: its prefixes come from the histogram
// kernel.
PWMGPU_HOST_DEVICE constexpr bool tile_pass_has_kernel(uint32_t key_bytes, uint32_t out_bytes, int K, bool out,
                                                       uint32_t vectors, bool given) {
  if ((key_bytes != 1 && key_bytes != 2 && key_bytes != 4) || K < 1) return false;
  const bool deep = K > kTileMaxLevels;
  if (out) {
    if (deep || (out_bytes != 1 && out_bytes != 2 && out_bytes != 4) || out_bytes > key_bytes) return false;
    // (4 levels over 4-byte keys only in the wider tiles: the usual ones are too small to sort by 4 bits at once)
    if (vectors == 0) return K < kTileMaxLevels || key_bytes < 4;
    return K == kTileMaxLevels && (vectors == 2 * kTileVectors || (key_bytes == 4 && vectors == 4 * kTileVectors));
  }
  // beyond 4 levels: only as the last pass of a text whose prefixes the histogram gives
  if (deep && (!given || K > kTileGivenMaxLevels)) return false;
  if (vectors == 0) return true;
  // half-size tiles: whole texts of 2 to 8 levels; double ones: those of up to 7, and last passes
  if (key_bytes != 1) return false;
  return vectors == kTileVectors / 2 ? K >= 2 : vectors == 2 * kTileVectors && K < kTileGivenMaxLevels;
}

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
