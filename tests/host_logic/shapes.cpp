// The tiles' geometry and the passes' shapes (pwm_gb300/csrc/tile_layout.hpp,
// host_tables.hpp): prints "ok", or what does not fit.
#include <cstdio>
#include <initializer_list>

#include "../../pwm_gb300/csrc/host_tables.hpp"

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

// Every pass of every plan has a kernel: each symbol width, 1 to 24 levels,
// every pass width, sizes on both sides of the ones where tiles change.
static int plans() {
  for (uint32_t width : {1u, 2u, 4u})
    for (uint32_t L = 1; L <= 24; ++L)
      for (int kmax = 1; kmax <= kTileGivenMaxLevels; ++kmax) {
        if (kmax > kTileMaxLevels && uint32_t(kmax) != L) continue;  // more than 4: a text in one pass
        for (int e = 0; e <= 34; ++e)
          for (int64_t d : {-1, 0, 1}) {
            const uint64_t n = (uint64_t(1) << e) + uint64_t(d);
            for (const PassPlan& p : plan_passes(L, kmax)) {
              const uint32_t l = p.level, kb = tile_pass_key_bytes(width, L, l);
              const uint32_t ob = tile_pass_key_bytes(width, L, l + uint32_t(p.K)), v = pass_vectors(width, L, kmax, l, n);
              const bool given = l == 0 && L >= 2 && L <= 8;
              if (!tile_pass_has_kernel(kb, ob, p.K, p.has_out, v, given)) {
                printf("no kernel: width %u, %u levels by %d, n %llu, level %u, %u vectors\n", width, L, kmax,
                       (unsigned long long)n, l, v);
                return 1;
              }
            }
          }
      }
  return 0;
}

// What has no kernel is refused: the launcher's switches would fall through.
static int refused() {
  struct Shape {
    uint32_t kb, ob;
    int K;
    bool out;
    uint32_t vectors;
    bool given;
  };
  const Shape none[] = {
      {4, 4, 4, true, 0, false},  // the usual tiles of 4-byte keys do not sort by 4 bits
      {4, 2, 4, true, 0, true},   {4, 4, 3, true, 8, false},  {2, 2, 4, true, 16, false}, {1, 1, 4, true, 2, false},
      {1, 2, 4, true, 0, false},  {2, 1, 4, false, 8, false}, {4, 1, 2, false, 2, false}, {1, 1, 4, false, 16, false},
      {1, 1, 5, false, 0, false},  // 5 levels and more with a look-back
      {1, 1, 5, true, 0, true},   {1, 1, 9, false, 0, true},  {1, 1, 0, false, 0, false}, {3, 1, 4, false, 0, false},
      {8, 1, 4, false, 0, false}, {4, 3, 4, true, 8, false},
      {1, 1, 1, false, 2, false}, {1, 1, 8, false, 8, true},
  };
  for (const Shape& s : none)
    if (tile_pass_has_kernel(s.kb, s.ob, s.K, s.out, s.vectors, s.given)) {
      printf("accepted: %u to %u bytes, %d levels, out %d, %u vectors, given %d\n", s.kb, s.ob, s.K, int(s.out), s.vectors,
             int(s.given));
      return 1;
    }
  return 0;
}

int main() {
  if (units() || blocks() || plans() || refused()) return 1;
  printf("ok\n");
  return 0;
}
