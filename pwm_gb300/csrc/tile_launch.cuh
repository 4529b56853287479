// Launch of one tile-pass instantiation (shared by tile.cu and tile_deep.cu,
// which instantiate the pass widths in separate translation units so that
// they compile in parallel).
#pragma once
#include "tile.cuh"

namespace pwmgpu {

// PLANES: the bit-plane form of a pass without S_{l+K} over 1-byte keys.
template <typename KeyT, int K, bool OUT, typename KeyO = KeyT, bool PLANES = false, int V = kTileVectors>
void launch_tile_one(const TileArgs& a, cudaStream_t s) {
  using C = TileCfg<KeyT, K, OUT, kTileThreads, V>;
  auto kern = tile_pass_kernel<KeyT, K, OUT, kTileThreads, V, KeyO, PLANES>;
  constexpr size_t smem = PLANES ? C::plane_smem_bytes() : C::RANKABLE ? C::ranked_smem_bytes() : C::smem_bytes();
  static OncePerDevice allowed;
  if (allow_shared(allowed, reinterpret_cast<const void*>(kern), smem) != cudaSuccess) return;
  kern<<<a.launch_tiles, kTileThreads, smem, s>>>(a);
}

// Last passes of 5..8 levels with given prefixes (tile_deep.cu); with
// TileArgs::tile_vectors, last passes over 1-byte keys (half: 2..8 levels,
// double: 1..7).
void launch_tile_pass_deep(uint32_t key_bytes, int K, const TileArgs& a, cudaStream_t s);
// Passes of kTileMaxLevels levels that write S_{l+K}, double tiles
// (tile_wide.cu).
void launch_tile_pass_wide(uint32_t key_bytes, uint32_t out_bytes, const TileArgs& a, cudaStream_t s);

}  // namespace pwmgpu
