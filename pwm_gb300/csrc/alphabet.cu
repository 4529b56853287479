// Alphabet reduction of texts whose symbols index a table (8 and 16 bits,
// and 32-bit symbols below 2^24): first positions, their ranks and the
// renumbered text, all on the device.  (pwm's reduce_alphabet,
// include/util/alphabet_util.hpp:18-45.  Wider symbols go through the hash
// table in build_kernels.cu, whose slots are ranked here too.)
#include <algorithm>

#include "kernels.cuh"

namespace pwmgpu {

namespace {

// ---------------------------------------------------------------------------
// First positions.  first[c] holds ~(the first position of symbol c), 0 while
// c has not been seen, so that one zeroing prepares it and a larger value is
// an earlier position.
//
// Nearly every symbol occurs for the first time early, so the text's first
// kFirstPrefix symbols go first (every block still finds most symbols new),
// then the rest starts from the set seen there.  A block walks a contiguous
// chunk in tiles: positions ascend from tile to tile, so a symbol seen in an
// earlier tile cannot be new, and a tile is tested against the block's bitmap
// of those (shared memory: one load and a bit test a symbol instead of a
// 64-bit load of first[c], which at 65536 symbols lives in L2) before its own
// symbols join it.  Once all values have been seen nothing is left to find,
// and the rest of the text is not read.  Measured (GB300), 2^28 16-bit symbols
// (an 8-byte load of first[c] a symbol before): 710 -> 30 us where all 65536
// values occur early, -> 130 us with 1000 values (the whole text read, at 4
// TB/s); 2^29 bytes of 4 values 185 us.
// ---------------------------------------------------------------------------
constexpr int kFirstThreads = 512;
constexpr int kFirstUnroll = 4;                     // 16-byte vectors a thread and tile
constexpr uint64_t kFirstPrefix = uint64_t(1) << 21;  // symbols of the first sweep

// Vectors [v0, v1) of the text (16 bytes from the aligned block that holds its
// first symbol on; symbol i of the text is symbol i + lead of the vectors).
template <typename T>
__global__ void __launch_bounds__(kFirstThreads) first_positions_kernel(const T* text, const uint4* vecs, uint32_t lead,
                                                                        uint64_t n, uint64_t v0, uint64_t v1,
                                                                        unsigned long long* first,
                                                                        const uint32_t* seen, const uint32_t* seen_count) {
  constexpr uint32_t kSymbols = 1u << (8 * sizeof(T)), kWords = kSymbols / 32, kPer = 16 / sizeof(T);
  __shared__ uint32_t bits[kWords];
  if (seen) {
    if (*seen_count == kSymbols) return;
    for (uint32_t i = threadIdx.x; i < kWords; i += kFirstThreads) bits[i] = seen[i];
  } else {
    for (uint32_t i = threadIdx.x; i < kWords; i += kFirstThreads) bits[i] = 0;
  }
  __syncthreads();
  const uint64_t per = (v1 - v0 + gridDim.x - 1) / gridDim.x;
  const uint64_t b = v0 + per * blockIdx.x, e = b + per < v1 ? b + per : v1;
  for (uint64_t t = b; t < e; t += kFirstThreads * kFirstUnroll) {  // uniform over the block
    uint4 v[kFirstUnroll];
#pragma unroll
    for (int u = 0; u < kFirstUnroll; ++u) {
      const uint64_t i = t + uint64_t(u) * kFirstThreads + threadIdx.x;
      v[u] = i < e ? __ldg(vecs + i) : make_uint4(0u, 0u, 0u, 0u);
    }
    auto symbol = [&](int u, uint32_t k) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      return (w[k * sizeof(T) / 4] >> (8 * sizeof(T) * (k % (4 / sizeof(T))))) & (kSymbols - 1);
    };
    uint32_t known = 1u;  // bit 0: every symbol of the thread's vectors was seen before this tile
#pragma unroll
    for (int u = 0; u < kFirstUnroll; ++u)
#pragma unroll
      for (uint32_t k = 0; k < kPer; ++k) {
        const uint32_t c = symbol(u, k);
        known &= bits[c >> 5] >> (c & 31);
      }
    if (!__syncthreads_or(!(known & 1u))) continue;
    // (rare: symbol by symbol, read again)
    auto each_new = [&](auto f) {
      if (known & 1u) return;
#pragma unroll 1
      for (uint32_t x = 0; x < kFirstUnroll * kPer; ++x) {
        const uint64_t i = t + uint64_t(x / kPer) * kFirstThreads + threadIdx.x;
        const uint64_t at = i * kPer + x % kPer - lead;  // wraps below the text's first symbol
        if (i >= e || at >= n) continue;
        const uint32_t c = text[at];
        if (!((bits[c >> 5] >> (c & 31)) & 1u)) f(c, at);
      }
    };
    each_new([&](uint32_t c, uint64_t at) {
      if (~at > first[c]) atomicMax(first + c, ~(unsigned long long)at);
    });
    __syncthreads();  // the tile's tests are over
    each_new([&](uint32_t c, uint64_t) { atomicOr(bits + (c >> 5), 1u << (c & 31)); });
    __syncthreads();
  }
}

// The set of symbols seen so far, a bit each, and their number.
__global__ void seen_symbols_kernel(const unsigned long long* first, uint64_t nsym, uint32_t* seen, uint32_t* count) {
  const uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint32_t m = __ballot_sync(0xFFFFFFFFu, c < nsym && first[c] != 0);
  if ((threadIdx.x & 31) == 0) {
    seen[c >> 5] = m;
    if (m) atomicAdd(count, uint32_t(__popc(m)));
  }
}

// 32-bit symbols below nsym (up to 2^24), positions [from, to): those of the
// set `seen` (a bit each: 1/64 of the bytes of first[]) are not new; the
// others take an atomic where their position is earlier.
__global__ void first_positions_wide_kernel(const uint32_t* text, uint64_t from, uint64_t to, uint64_t nsym,
                                            unsigned long long* first, const uint32_t* seen) {
  for (uint64_t i = from + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < to;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t c = text[i];
    if (c >= nsym || (seen && ((__ldg(seen + (c >> 5)) >> (c & 31)) & 1u))) continue;
    if (~i > first[c]) atomicMax(first + c, ~(unsigned long long)i);
  }
}

// ---------------------------------------------------------------------------
// Ranks of the first positions: a bit a position, counted in groups of 1024
// (a thread) and chunks of 256 groups (a block); the last block to finish adds
// up the chunks, and a symbol's id is the bits before its own.  Chunks past
// the last first position are not read.
// ---------------------------------------------------------------------------
constexpr uint32_t kGroupLog = 10, kChunkLog = 18;
constexpr int kRankThreads = 1 << (kChunkLog - kGroupLog);

__global__ void mark_first_kernel(const unsigned long long* first, uint64_t nsym, uint32_t* marks,
                                  unsigned long long* last) {
  unsigned long long top = 0;
  for (uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < nsym; c += uint64_t(gridDim.x) * blockDim.x) {
    const unsigned long long f = first[c];
    if (!f) continue;
    const unsigned long long at = ~f;
    atomicOr(marks + (at >> 5), 0x80000000u >> (at & 31));
    top = max(top, at);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) top = max(top, (unsigned long long)__shfl_xor_sync(0xFFFFFFFFu, top, d));
  if ((threadIdx.x & 31) == 0 && top) atomicMax(last, top);
}

// Exclusive prefix over a block of kRankThreads threads, and the total.
__device__ __forceinline__ uint32_t block_prefix(uint32_t x, uint32_t* total) {
  __shared__ uint32_t ws[kRankThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t s = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, d);
    if (lane >= d) s += y;
  }
  __syncthreads();  // the words' last use is over
  if (lane == 31) ws[warp] = s;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kRankThreads / 32; ++w) {
    before += w < warp ? ws[w] : 0u;
    all += ws[w];
  }
  *total = all;
  return before + s - x;
}

// groups[g]: marks before group g inside its chunk; chunks[k]: marks before
// chunk k.  distinct (host-mapped): all of them.
__global__ void __launch_bounds__(kRankThreads) count_marks_kernel(const uint4* marks, const unsigned long long* last,
                                                                   uint32_t* groups, uint32_t* chunks, uint32_t* done, unsigned long long* distinct) {
  __shared__ bool is_last;
  const uint64_t used = (*last >> kChunkLog) + 1;  // chunks that hold marks
  for (uint64_t k = blockIdx.x; k < used; k += gridDim.x) {
    const uint4* m = marks + (k << (kChunkLog - 7)) + threadIdx.x * 8;
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 w = m[i];
      x += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
    }
    uint32_t total;
    groups[(k << (kChunkLog - kGroupLog)) + threadIdx.x] = block_prefix(x, &total);
    if (threadIdx.x == 0) chunks[k] = total;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  uint32_t run = 0;
  for (uint64_t k0 = 0; k0 < used; k0 += kRankThreads) {
    const uint64_t k = k0 + threadIdx.x;
    uint32_t total;
    const uint32_t p = block_prefix(k < used ? *static_cast<volatile uint32_t*>(chunks + k) : 0u, &total);
    if (k < used) chunks[k] = run + p;
    run += total;
  }
  if (threadIdx.x == 0) *distinct = run;
}

// map[c]: the id of symbol c, 0 where it does not occur.
__global__ void rank_symbols_kernel(const unsigned long long* first, uint64_t nsym, const uint32_t* marks,
                                    const uint32_t* groups, const uint32_t* chunks, uint32_t* map) {
  for (uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < nsym; c += uint64_t(gridDim.x) * blockDim.x) {
    const unsigned long long f = first[c];
    uint32_t id = 0;
    if (f) {
      const unsigned long long at = ~f;
      id = chunks[at >> kChunkLog] + groups[at >> kGroupLog];
      const uint64_t w1 = at >> 5;
      for (uint64_t w = (at >> kGroupLog) << (kGroupLog - 5); w < w1; ++w) id += __popc(marks[w]);
      const uint32_t r = uint32_t(at & 31);
      if (r) id += __popc(marks[w1] >> (32 - r));
    }
    map[c] = id;
  }
}

// ---------------------------------------------------------------------------
// The renumbered text of 8- and 16-bit symbols: a table of 65536 16-bit
// entries (for bytes, of every pair of them) in 128 KB of shared memory, so
// a 16-byte vector is 8 shared loads; the gather from L2 that 65536 entries
// otherwise are ran at 1.6 TB/s.  One block an SM; text and output read and
// written once.
// ---------------------------------------------------------------------------
constexpr int kRemapThreads = 1024;
constexpr int kRemapUnroll = 4;
constexpr uint32_t kRemapSmem = 65536 * 2;
// From here on the table pays for itself (a block fills its 128 KB in a few
// microseconds): whole calls on 4 / 8 / 32 MB of 16-bit text take 82 / 89 / 97
// us with it and 78 / 91 / 113 without, on 4 MB of bytes 83 and 85; 512 MB
// of 16-bit text is renumbered in 177 us (6.1 TB/s) against 676.
constexpr uint64_t kRemapTableMin = uint64_t(6) << 20;  // bytes of text

template <typename T>
__global__ void __launch_bounds__(kRemapThreads) remap_table_kernel(const T* text, uint64_t n, uint32_t head,
                                                                    const uint32_t* map, T* out) {
  extern __shared__ uint16_t table[];
  constexpr uint32_t kPer = 16 / sizeof(T);
  if constexpr (sizeof(T) == 2) {
    for (uint32_t c = threadIdx.x; c < 65536; c += kRemapThreads) table[c] = uint16_t(map[c]);
  } else {
    for (uint32_t c = threadIdx.x; c < 65536; c += kRemapThreads)
      table[c] = uint16_t((map[c & 255u] & 255u) | ((map[c >> 8] & 255u) << 8));
  }
  __syncthreads();
  auto two = [&](uint32_t w) { return uint32_t(table[w & 0xFFFFu]) | (uint32_t(table[w >> 16]) << 16); };
  auto one = [&](uint64_t i) { out[i] = T(table[text[i]]); };  // a byte's own entry is the low half of (byte, 0)
  const uint64_t nv = (n - head) / kPer;
  const uint4* in = reinterpret_cast<const uint4*>(text + head);
  uint4* to = reinterpret_cast<uint4*>(out + head);
  const uint64_t stride = uint64_t(gridDim.x) * kRemapThreads;
  uint64_t i = uint64_t(blockIdx.x) * kRemapThreads + threadIdx.x;
  for (; i + (kRemapUnroll - 1) * stride < nv; i += kRemapUnroll * stride) {
    uint4 v[kRemapUnroll];
#pragma unroll
    for (int u = 0; u < kRemapUnroll; ++u) v[u] = __ldcs(in + i + u * stride);
#pragma unroll
    for (int u = 0; u < kRemapUnroll; ++u)
      __stcs(to + i + u * stride, make_uint4(two(v[u].x), two(v[u].y), two(v[u].z), two(v[u].w)));
  }
  for (; i < nv; i += stride) {
    const uint4 v = __ldcs(in + i);
    __stcs(to + i, make_uint4(two(v.x), two(v.y), two(v.z), two(v.w)));
  }
  if (blockIdx.x == 0) {
    if (threadIdx.x < head) one(threadIdx.x);
    const uint64_t tail = head + nv * kPer;
    if (threadIdx.x < n - tail) one(tail + threadIdx.x);
  }
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 148;
}

template <typename T>
void first_positions(const void* text, uint64_t n, unsigned long long* first, uint32_t* seen, cudaStream_t s,
                     uint64_t* launches) {
  constexpr uint32_t kSymbols = 1u << (8 * sizeof(T));
  const uintptr_t at = reinterpret_cast<uintptr_t>(text);
  const uint32_t lead = uint32_t(at & 15) / sizeof(T);
  const auto* vecs = reinterpret_cast<const uint4*>(at & ~uintptr_t(15));
  constexpr uint32_t kPer = 16 / sizeof(T);
  const uint64_t nv = (lead + n + kPer - 1) / kPer, prefix = std::min<uint64_t>(nv, kFirstPrefix / kPer);
  // the first sweep a vector a thread (its atomics wait on one another), the rest in whole tiles
  constexpr uint64_t kTile = uint64_t(kFirstThreads) * kFirstUnroll;
  const uint64_t cap = uint64_t(sm_count()) * 4;
  auto blocks = [&](uint64_t v, uint64_t per) {
    return unsigned(std::max<uint64_t>(1, std::min((v + per - 1) / per, cap)));
  };
  first_positions_kernel<T><<<blocks(prefix, kFirstThreads), kFirstThreads, 0, s>>>(static_cast<const T*>(text), vecs,
                                                                                   lead, n, 0, prefix, first, nullptr,
                                                                                   nullptr);
  ++*launches;
  if (prefix == nv) return;
  seen_symbols_kernel<<<kSymbols / 256, 256, 0, s>>>(first, kSymbols, seen, seen + kSymbols / 32);
  first_positions_kernel<T><<<blocks(nv - prefix, kTile), kFirstThreads, 0, s>>>(static_cast<const T*>(text), vecs,
                                                                                lead, n, prefix, nv, first, seen,
                                                                                seen + kSymbols / 32);
  *launches += 2;
}

// Where each part of the scratch lies (bytes); all of it up to `zeroed` is
// zero before the first kernel.
struct RankScratch {
  uint64_t last, done, marks, zeroed, groups, chunks, end, nchunks;
  RankScratch(uint64_t n, uint64_t from) {
    auto align = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
    nchunks = (n + (uint64_t(1) << kChunkLog) - 1) >> kChunkLog;
    last = align(from);
    done = last + 8;
    marks = align(done + 4);
    zeroed = align(marks + (nchunks << (kChunkLog - 3)));
    groups = zeroed;
    chunks = align(groups + (nchunks << (kChunkLog - kGroupLog)) * 4);
    end = align(chunks + nchunks * 4);
  }
};
struct ScratchLayout {
  uint64_t seen, map, end;  // first positions lie at 0
  RankScratch rank;
  ScratchLayout(uint64_t n, uint64_t nsym)
      : seen((nsym * 8 + 255) & ~uint64_t(255)), map(0), end(0), rank(n, seen + (std::max<uint64_t>(nsym, 65536) + 255) / 8 + 8) {
    map = rank.end;
    end = map + nsym * 4;
  }
};

// ids[c] of the nsym symbols (or table slots) with first positions `first`;
// base: scratch of the layout, zeroed up to R.zeroed.
void rank_first_positions(const unsigned long long* first, uint64_t nsym, unsigned char* base, const RankScratch& R,
                          uint32_t* ids, unsigned long long* distinct, cudaStream_t s, uint64_t* launches) {
  auto* last = reinterpret_cast<unsigned long long*>(base + R.last);
  auto* marks = reinterpret_cast<uint32_t*>(base + R.marks);
  auto* groups = reinterpret_cast<uint32_t*>(base + R.groups);
  auto* chunks = reinterpret_cast<uint32_t*>(base + R.chunks);
  const unsigned gsym = unsigned(std::min<uint64_t>((nsym + 255) / 256, 2048));
  const unsigned gc = unsigned(std::min<uint64_t>(R.nchunks, uint64_t(sm_count()) * 4));
  mark_first_kernel<<<gsym, 256, 0, s>>>(first, nsym, marks, last);
  count_marks_kernel<<<gc, kRankThreads, 0, s>>>(reinterpret_cast<const uint4*>(marks), last, groups, chunks,
                                                 reinterpret_cast<uint32_t*>(base + R.done), distinct);
  rank_symbols_kernel<<<gsym, 256, 0, s>>>(first, nsym, marks, groups, chunks, ids);
  *launches += 3;
}

}  // namespace

uint64_t alphabet_rank_scratch_bytes(uint64_t n) { return RankScratch(n, 0).end; }

cudaError_t launch_rank_slots(const unsigned long long* first, uint64_t cap, uint64_t n, void* scratch, uint32_t* ids,
                              unsigned long long* distinct, cudaStream_t s, uint64_t* launches) {
  const RankScratch R(n, 0);
  const cudaError_t e = cudaMemsetAsync(scratch, 0, R.zeroed, s);
  if (e != cudaSuccess) return e;
  rank_first_positions(first, cap, static_cast<unsigned char*>(scratch), R, ids, distinct, s, launches);
  return cudaGetLastError();
}

uint64_t alphabet_scratch_bytes(uint64_t n, uint64_t nsym) { return ScratchLayout(n, nsym).end; }

void launch_first_positions(const void* text, uint64_t n, uint32_t width, uint64_t nsym, unsigned long long* first,
                            uint32_t* seen, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return;
  if (width == 1) {
    first_positions<uint8_t>(text, n, first, seen, s, launches);
  } else if (width == 2) {
    first_positions<uint16_t>(text, n, first, seen, s, launches);
  } else {
    auto blocks = [](uint64_t m) { return unsigned(std::min<uint64_t>((m + 255) / 256, 4096)); };
    const auto* t = static_cast<const uint32_t*>(text);
    const uint64_t prefix = std::min(n, std::max(kFirstPrefix, 8 * nsym));
    first_positions_wide_kernel<<<blocks(prefix), 256, 0, s>>>(t, 0, prefix, nsym, first, nullptr);
    ++*launches;
    if (prefix == n) return;
    const uint64_t words = (nsym + 255) / 256 * 8;  // whole blocks of 256 symbols
    seen_symbols_kernel<<<unsigned(words / 8), 256, 0, s>>>(first, nsym, seen, seen + words);
    first_positions_wide_kernel<<<blocks(n - prefix), 256, 0, s>>>(t, prefix, n, nsym, first, seen);
    *launches += 2;
  }
}

cudaError_t launch_reduce_alphabet(const void* text, uint64_t n, uint32_t width, uint64_t nsym, void* out,
                                   void* scratch, unsigned long long* distinct, uint32_t* status, cudaStream_t s,
                                   uint64_t* launches) {
  const ScratchLayout L(n, nsym);
  auto* base = static_cast<unsigned char*>(scratch);
  auto* first = reinterpret_cast<unsigned long long*>(base);
  auto* map = reinterpret_cast<uint32_t*>(base + L.map);
  cudaError_t e = cudaMemsetAsync(base, 0, L.rank.zeroed, s);
  if (e != cudaSuccess) return e;
  launch_first_positions(text, n, width, nsym, first, reinterpret_cast<uint32_t*>(base + L.seen), s, launches);
  rank_first_positions(first, nsym, base, L.rank, map, distinct, s, launches);
  const uintptr_t ti = reinterpret_cast<uintptr_t>(text), to = reinterpret_cast<uintptr_t>(out);
  const uint32_t head = uint32_t((16 - (ti & 15)) & 15) / width;
  if (width <= 2 && n * width >= kRemapTableMin && (ti & 15) == (to & 15) && ti % width == 0) {
    const unsigned g = unsigned(sm_count());
    if (width == 1) {
      e = cudaFuncSetAttribute(remap_table_kernel<uint8_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRemapSmem);
      if (e != cudaSuccess) return e;
      remap_table_kernel<uint8_t><<<g, kRemapThreads, kRemapSmem, s>>>(static_cast<const uint8_t*>(text), n, head,
                                                                       map, static_cast<uint8_t*>(out));
    } else {
      e = cudaFuncSetAttribute(remap_table_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRemapSmem);
      if (e != cudaSuccess) return e;
      remap_table_kernel<uint16_t><<<g, kRemapThreads, kRemapSmem, s>>>(static_cast<const uint16_t*>(text), n, head,
                                                                        map, static_cast<uint16_t*>(out));
    }
    ++*launches;
  } else {
    launch_remap(text, n, width, map, nsym, out, status, s, launches);
  }
  return cudaGetLastError();
}

}  // namespace pwmgpu
