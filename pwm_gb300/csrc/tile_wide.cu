// Tile passes of 4 levels that write S_{l+K}, in tiles of twice the usual keys.
//
// Half of a tile's instructions do not grow with its keys: finding its
// segment, the barriers and scans of every split, the set-up of each of its 44
// runs.  With 8 vectors a thread (32768 keys of 8 bits, 16384 of 16, 8192 of
// 32; 80 registers, 3 CTAs an SM) they serve twice as many, and the runs are
// twice as long.  Measured (GB300), whole builds with keys split bit by bit:
// 2^30 bytes, both structures of 8 levels, 5.55 -> 5.00 ms; 2^28 16-bit
// symbols, 16 levels, 4.79 -> 4.40; 2^26 32-bit symbols, the matrix of 20
// levels, 1.87 -> 1.64 (with 4 CTAs an SM at 64 registers 16-bit 4.55, 32-bit
// 1.72).  Sorted by 4 bits at once (tile_rank_keys) passes in these tiles take
// 517 us for 2^28 8-bit keys and 211 for 2^26 16-bit ones, in the usual ones
// 563 and 270.  Texts too short to fill the SMs with such tiles keep those.
//
// 4-byte keys take tiles of 16 vectors (16384 keys, 128 registers, 2 CTAs an
// SM) in turn: with 32 keys a thread its scans and cursors weigh as much as its
// keys.  2^25 keys narrowed to 16 bits 169 -> 144 us, 2^26 symbols of 20 levels
// 1.25 -> 1.20 ms.  (2-byte keys in such tiles: 217 us against 211.)
#include "kernels.cuh"
#include "tile_launch.cuh"

namespace pwmgpu {

namespace {
template <typename KeyT, typename KeyO>
void launch(const TileArgs& a, cudaStream_t s) {
  if constexpr (sizeof(KeyT) == 4) {
    if (a.tile_vectors == 4 * uint32_t(kTileVectors)) {
      launch_tile_one<KeyT, kTileMaxLevels, true, KeyO, false, 4 * kTileVectors>(a, s);
      return;
    }
  }
  launch_tile_one<KeyT, kTileMaxLevels, true, KeyO, false, 2 * kTileVectors>(a, s);
}
}  // namespace

void launch_tile_pass_wide(uint32_t key_bytes, uint32_t out_bytes, const TileArgs& a, cudaStream_t s) {
  if (key_bytes == 1) launch<uint8_t, uint8_t>(a, s);
  else if (key_bytes == 2 && out_bytes == 1) launch<uint16_t, uint8_t>(a, s);
  else if (key_bytes == 2) launch<uint16_t, uint16_t>(a, s);
  else if (out_bytes == 1) launch<uint32_t, uint8_t>(a, s);
  else if (out_bytes == 2) launch<uint32_t, uint16_t>(a, s);
  else launch<uint32_t, uint32_t>(a, s);
}

}  // namespace pwmgpu
