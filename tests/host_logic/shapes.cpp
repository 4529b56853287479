// The tiles' geometry (pwm_gb300/csrc/tile_layout.hpp): prints "ok", or what
// does not fit.
#include <cstdio>
#include <initializer_list>

#include "../../pwm_gb300/csrc/tile_layout.hpp"

using namespace pwmgpu;

// Every tile is whole units of whole vectors a thread, as many as the
// histogram kernel holds.
static int units() {
  for (int vectors : {1, 2, 4, 8, 16}) {
    const uint64_t bytes = uint64_t(vectors) * 16 * kTileThreads;
    const uint32_t u = tile_hist_units(bytes);
    if (u == 0 || bytes % u || bytes / u % (16 * kTileThreads) || bytes / u > uint64_t(16 * kTileVectors) * kTileThreads) {
      printf("tiles of %d vectors: %u units\n", vectors, u);
      return 1;
    }
  }
  return 0;
}

// A histogram block holds no more of a text in wide tiles than in the usual
// ones: the same number of blocks works on it.
static int blocks() {
  const uint64_t usual = uint64_t(kTileVectors) * 16 * kTileThreads;
  for (int vectors : {4, 8, 16}) {
    const uint64_t bytes = uint64_t(vectors) * 16 * kTileThreads;
    if (tile_hist_tiles_per_block(bytes) * bytes != tile_hist_tiles_per_block(usual) * usual) {
      printf("blocks of tiles of %d vectors: %u\n", vectors, tile_hist_tiles_per_block(bytes));
      return 1;
    }
  }
  return 0;
}

int main() {
  if (units() || blocks()) return 1;
  printf("ok\n");
  return 0;
}
