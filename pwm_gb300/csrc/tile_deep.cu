// Tile passes of 5..8 levels (a whole text of at most 8 levels in one pass,
// its finest-run prefixes given by the histogram kernel).
#include "kernels.cuh"
#include "tile_launch.cuh"

namespace pwmgpu {

namespace {

// 1-byte keys in the bit-plane form
template <typename KeyT>
void launch_deep_key(int K, const TileArgs& a, cudaStream_t s) {
  constexpr bool PL = sizeof(KeyT) == 1;
  switch (K) {
    case 5: launch_tile_one<KeyT, 5, false, KeyT, PL>(a, s); break;
    case 6: launch_tile_one<KeyT, 6, false, KeyT, PL>(a, s); break;
    case 7: launch_tile_one<KeyT, 7, false, KeyT, PL>(a, s); break;
    default: launch_tile_one<KeyT, 8, false, KeyT, PL>(a, s); break;
  }
}

// Tiles of V vectors a thread: half-size ones for short texts, which fill
// twice as many SMs (2 to 8 levels); double ones for long texts (1 to 7;
// tile_wide.cu says why, and 8 levels are no faster in them).
template <int V>
void launch_sized(int K, const TileArgs& a, cudaStream_t s) {
  switch (K) {
    case 2: launch_tile_one<uint8_t, 2, false, uint8_t, true, V>(a, s); break;
    case 3: launch_tile_one<uint8_t, 3, false, uint8_t, true, V>(a, s); break;
    case 4: launch_tile_one<uint8_t, 4, false, uint8_t, true, V>(a, s); break;
    case 5: launch_tile_one<uint8_t, 5, false, uint8_t, true, V>(a, s); break;
    case 6: launch_tile_one<uint8_t, 6, false, uint8_t, true, V>(a, s); break;
    case 7: launch_tile_one<uint8_t, 7, false, uint8_t, true, V>(a, s); break;
    default: launch_tile_one<uint8_t, V < kTileVectors ? 8 : 1, false, uint8_t, true, V>(a, s); break;
  }
}

}  // namespace

void launch_tile_pass_deep(uint32_t key_bytes, int K, const TileArgs& a, cudaStream_t s) {
  if (a.tile_vectors == kTileVectors / 2) launch_sized<kTileVectors / 2>(K, a, s);
  else if (a.tile_vectors) launch_sized<kTileVectors * 2>(K, a, s);
  else if (key_bytes == 1) launch_deep_key<uint8_t>(K, a, s);
  else if (key_bytes == 2) launch_deep_key<uint16_t>(K, a, s);
  else launch_deep_key<uint32_t>(K, a, s);
}

}  // namespace pwmgpu
