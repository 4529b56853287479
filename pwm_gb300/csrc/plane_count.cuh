// Symbol counts of 8-bit texts of 2 to 4 levels without an atomic a symbol:
// 32 symbols become one 32-bit plane a level (the order inside a plane is any,
// the same for all of them), and the count of every symbol value follows from
// popcounts of the planes' conjunctions, 2^L - 1 for 32 symbols.
#pragma once

#include "tile.cuh"

namespace pwmgpu {

// The first `valid` symbols of a 16-byte vector, the rest zero.
__device__ __forceinline__ uint4 keep_first(const uint4& v, int valid) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = valid - 4 * q;
    w[q] = k >= 4 ? w[q] : (k <= 0 ? 0u : w[q] & ((1u << (8 * k)) - 1u));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Adds the counts of the 32 symbols of two vectors (each below 2^L) to cnt.
template <int L>
__device__ __forceinline__ void count_planes(const uint4& a, const uint4& b, uint32_t (&cnt)[1 << L]) {
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  // symbols side by side in a byte: four bits each, and for two levels two
  uint32_t p[L];  // plane j: level j, the symbols' bit L - 1 - j
  if constexpr (L <= 2) {
    uint32_t x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) x[i] = w[4 * i] | (w[4 * i + 1] << 2) | (w[4 * i + 2] << 4) | (w[4 * i + 3] << 6);
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const int s = L - 1 - j;
      p[j] = ((x[0] >> s) & 0x55555555u) | (((x[1] >> s) & 0x55555555u) << 1);
    }
  } else {
    uint32_t x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = w[2 * i] | (w[2 * i + 1] << 4);
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const int s = L - 1 - j;
      p[j] = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) p[j] |= ((x[i] >> s) & 0x11111111u) << i;
    }
  }
  uint32_t m[1 << L], c[1 << L];
  m[0] = ~0u;
  c[0] = 32;
#pragma unroll
  for (int d = 0; d < L; ++d)
#pragma unroll
    for (int v = (1 << d) - 1; v >= 0; --v) {
      const uint32_t one = m[v] & p[d], n1 = __popc(one);
      m[2 * v + 1] = one;
      m[2 * v] = m[v] & ~p[d];
      c[2 * v + 1] = n1;
      c[2 * v] = c[v] - n1;
    }
#pragma unroll
  for (int v = 0; v < (1 << L); ++v) cnt[v] += c[v];
}

// The counts of one tile of n symbols at `p` (any alignment), by the CTA's
// THREADS threads of up to VMAX vectors each (nv of them): every warp's sums go
// to pairs[warp][i], value 2 i in the low half, 2 i + 1 in the high one.
// each(r, i, v): vector i (symbols 16 i.. of the tile; cut off at n, zero
// past it) is v, the thread's r-th; called by whole warps.  seen: OR of the
// symbols.  shift: the values counted are the symbols' bits shift .. shift +
// L - 1.
template <int L, int THREADS, int VMAX, typename F>
__device__ __forceinline__ void count_tile_planes(const unsigned char* p, uint32_t n, int nv, uint32_t& seen,
                                                  uint32_t (*pairs)[8], F&& each, uint32_t shift = 0) {
  const uint32_t tid = threadIdx.x, nvec = (n + 15) >> 4;
  const uint32_t off = uint32_t(reinterpret_cast<uintptr_t>(p) & 15);
  const uint4* av = reinterpret_cast<const uint4*>(p - off);
  const uint32_t last_block = uint32_t((uint64_t(off) + n + 15) >> 4) - 1;  // last aligned block holding tile symbols
  uint4 v[VMAX];
#pragma unroll
  for (int r = 0; r < VMAX; ++r) {
    const uint32_t i = tid + uint32_t(r) * THREADS;
    v[r] = make_uint4(0u, 0u, 0u, 0u);
    if (r < nv && i < nvec) {
      v[r] = __ldcs(av + i);
      if (off) v[r] = realign16(v[r], i + 1 <= last_block ? __ldcs(av + i + 1) : make_uint4(0u, 0u, 0u, 0u), off);
    }
  }
  // (a text may have more levels than 8: bits above a symbol's are 0)
  const uint32_t kBits = (shift + L <= 8 ? (1u << L) - 1u : (shift >= 8 ? 0u : (1u << (8 - shift)) - 1u)) * 0x01010101u;
  uint32_t cnt[1 << L], counted = 0, valid = 0;
#pragma unroll
  for (int k = 0; k < (1 << L); ++k) cnt[k] = 0;
#pragma unroll
  for (int r = 0; r < VMAX; ++r) {
    if (r >= nv) break;  // uniform
    const uint32_t i = tid + uint32_t(r) * THREADS;
    const int left = int(n) - int(16 * i), k = left >= 16 ? 16 : (left > 0 ? left : 0);
    if (k < 16) v[r] = keep_first(v[r], k);
    valid += uint32_t(k);
    each(r, i, v[r]);
    seen |= v[r].x | v[r].y | v[r].z | v[r].w;
    v[r] = make_uint4((v[r].x >> shift) & kBits, (v[r].y >> shift) & kBits, (v[r].z >> shift) & kBits,
                      (v[r].w >> shift) & kBits);
  }
#pragma unroll
  for (int r = 0; r < VMAX; r += 2) {
    if (r >= nv) break;
    count_planes<L>(v[r], r + 1 < VMAX && r + 1 < nv ? v[r + 1 < VMAX ? r + 1 : r] : make_uint4(0u, 0u, 0u, 0u), cnt);
    counted += 32;
  }
  cnt[0] -= counted - valid;  // the places that hold no symbol counted as 0
#pragma unroll
  for (int k = 0; k < (1 << L); k += 2) {
    const uint32_t x = __reduce_add_sync(0xFFFFFFFFu, cnt[k] | (cnt[k + 1] << 16));
    if ((tid & 31) == 0) pairs[tid >> 5][k / 2] = x;
  }
}

}  // namespace pwmgpu
