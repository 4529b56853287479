// Device side of the Huffman-shaped builds: the text's code keys and the
// counts that the passes' start tables follow from.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"

namespace pwmgpu {

namespace {

// Key of symbol c with code (word, len), L the longest code: the code
// followed by a stop bit, ((word << 1) | 1) << (L - len), L + 1 bits (split.cuh
// HuffKeys); 0, which no code gives, where c has none.
__device__ __forceinline__ uint64_t code_key(const uint64_t* code_len, const uint64_t* code_word, uint64_t ncodes,
                                             uint64_t c, uint32_t L) {
  const uint64_t len = c < ncodes ? code_len[c] : 0;
  return len == 0 || len > L ? 0ull : ((code_word[c] << 1) | 1u) << (L - len);
}

// Any symbol width: two 8-byte gathers a symbol.
template <typename T, typename K>
__global__ void huffman_keys_kernel(const T* text, uint64_t n, const uint64_t* code_len, const uint64_t* code_word,
                                    uint64_t ncodes, uint32_t L, K* keys, uint32_t* status) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const uint64_t k = code_key(code_len, code_word, ncodes, uint64_t(text[i]), L);
    if (!k) atomicOr(status, kErrSymbol);
    keys[i] = K(k);
  }
}

// 8- and 16-bit symbols through a table in shared memory: for 16-bit ones the
// low 16 key bits of every symbol (128 KB) and, for keys of 17 to 24 bits, the
// next 8 (64 KB): one block an SM, two shared loads a symbol.  A thread takes
// the symbols of 16 bytes of keys, so that a warp reads and writes whole
// lines.  2^28 16-bit symbols of 18-bit keys (1.6 GB read and written): 1189
// us as gathers from L2 -> 272 us.
template <typename T, typename K, bool HI>
struct KeyTable {
  static constexpr uint32_t kSymbols = 1u << (8 * sizeof(T));
  using Low = typename std::conditional<sizeof(T) == 1, K, uint16_t>::type;
  static constexpr size_t bytes() { return kSymbols * (sizeof(Low) + (HI ? 1 : 0)); }
};
constexpr int kKeyUnroll = 4;

template <typename T, typename K, bool HI, int THREADS>
__global__ void __launch_bounds__(THREADS) huffman_keys_table_kernel(const T* text, uint64_t n, const uint64_t* code_len,
                                                                     const uint64_t* code_word, uint64_t ncodes,
                                                                     uint32_t L, K* keys, uint32_t* status) {
  using Tab = KeyTable<T, K, HI>;
  extern __shared__ __align__(16) unsigned char key_smem[];
  auto* low = reinterpret_cast<typename Tab::Low*>(key_smem);
  auto* high = reinterpret_cast<uint8_t*>(low + Tab::kSymbols);
  for (uint32_t c = threadIdx.x; c < Tab::kSymbols; c += THREADS) {
    const uint64_t k = code_key(code_len, code_word, ncodes, c, L);
    low[c] = typename Tab::Low(k);
    if constexpr (HI) high[c] = uint8_t(k >> 16);
  }
  __syncthreads();
  auto key = [&](uint32_t c) -> K {
    if constexpr (HI) return K(low[c]) | K(K(high[c]) << 16);
    else return K(low[c]);
  };
  constexpr uint32_t kPer = 16 / sizeof(K);  // symbols a thread and step
  struct alignas(kPer * sizeof(T)) Symbols {
    T s[kPer];
  };
  struct alignas(16) Keys {
    K k[kPer];
  };
  // (keys is aligned; a text off its vectors goes symbol by symbol)
  const uint64_t nv = reinterpret_cast<uintptr_t>(text) % sizeof(Symbols) == 0 ? n / kPer : 0;
  const auto* in = reinterpret_cast<const Symbols*>(text);
  auto* out = reinterpret_cast<Keys*>(keys);
  const uint64_t stride = uint64_t(gridDim.x) * THREADS;
  bool bad = false;
  auto put = [&](uint64_t i, const Symbols& v) {
    Keys o;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      o.k[k] = key(v.s[k]);
      bad |= o.k[k] == 0;
    }
    out[i] = o;
  };
  uint64_t i = uint64_t(blockIdx.x) * THREADS + threadIdx.x;
  for (; i + (kKeyUnroll - 1) * stride < nv; i += kKeyUnroll * stride) {
    Symbols v[kKeyUnroll];
#pragma unroll
    for (int u = 0; u < kKeyUnroll; ++u) v[u] = in[i + u * stride];
#pragma unroll
    for (int u = 0; u < kKeyUnroll; ++u) put(i + u * stride, v[u]);
  }
  for (; i < nv; i += stride) put(i, in[i]);
  for (uint64_t j = nv * kPer + uint64_t(blockIdx.x) * THREADS + threadIdx.x; j < n; j += stride) {
    const K k = key(text[j]);
    bad |= k == 0;
    keys[j] = k;
  }
  if (bad) atomicOr(status, kErrSymbol);
}

// Texts from here on fill the table (192 KB a block) for less than it saves.
constexpr uint64_t kKeyTableMin = uint64_t(1) << 20;

template <typename T, typename K, bool HI, int THREADS>
void launch_table(const void* text, uint64_t n, const uint64_t* code_len, const uint64_t* code_word, uint64_t ncodes,
                  uint32_t L, void* keys, uint32_t* status, int blocks, cudaStream_t s) {
  auto kern = huffman_keys_table_kernel<T, K, HI, THREADS>;
  constexpr size_t smem = KeyTable<T, K, HI>::bytes();
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  kern<<<blocks, THREADS, smem, s>>>(static_cast<const T*>(text), n, code_len, code_word, ncodes, L,
                                     static_cast<K*>(keys), status);
}

template <typename T>
void launch_gather(uint32_t key_bytes, const void* text, uint64_t n, const uint64_t* code_len,
                   const uint64_t* code_word, uint64_t ncodes, uint32_t L, void* keys, uint32_t* status,
                   cudaStream_t s) {
  const unsigned g = unsigned(std::min<uint64_t>((n + 255) / 256, 4096));
  const auto* t = static_cast<const T*>(text);
  switch (key_bytes) {
    case 1: huffman_keys_kernel<<<g, 256, 0, s>>>(t, n, code_len, code_word, ncodes, L, static_cast<uint8_t*>(keys), status); break;
    case 2: huffman_keys_kernel<<<g, 256, 0, s>>>(t, n, code_len, code_word, ncodes, L, static_cast<uint16_t*>(keys), status); break;
    case 4: huffman_keys_kernel<<<g, 256, 0, s>>>(t, n, code_len, code_word, ncodes, L, static_cast<uint32_t*>(keys), status); break;
    default: huffman_keys_kernel<<<g, 256, 0, s>>>(t, n, code_len, code_word, ncodes, L, static_cast<uint64_t*>(keys), status); break;
  }
}

// Counts of a weighted code table (kHuffCounts words of `out`, zeroed by the
// caller; symbol c occurs hist[c] times with code (word, len)): the symbols by
// code length, the zero bits of every level, and of every pass (l, K) the
// counts of its key_j values among the codes alive at l + j (key_j: code bits
// l..l+j-1, bit l least significant).  A warp takes 32 codes at a time, sums
// every counter over its lanes and keeps its totals in shared memory.
constexpr int kCountThreads = 256;

__global__ void __launch_bounds__(kCountThreads) huff_count_kernel(const unsigned long long* hist,
                                                                   const uint64_t* code_len, const uint64_t* code_word,
                                                                   uint64_t ncodes, uint32_t L, uint32_t K,
                                                                   unsigned long long* out) {
  extern __shared__ unsigned long long acc[];  // [warps][counters]
  const uint32_t C = (2u << K) - 2, counters = huff_count_words(L, K);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < counters * (kCountThreads / 32); i += kCountThreads) acc[i] = 0;
  __syncthreads();
  unsigned long long* mine = acc + warp * counters;
  auto add = [&](uint32_t id, unsigned long long x) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, d);
    if (lane == 0) mine[id] += x;
  };
  const uint64_t warps = uint64_t(gridDim.x) * (kCountThreads / 32);
  for (uint64_t c0 = (uint64_t(blockIdx.x) * (kCountThreads / 32) + warp) * 32; c0 < ncodes; c0 += warps * 32) {
    const uint64_t c = c0 + lane;
    const unsigned long long f = c < ncodes ? hist[c] : 0ull;
    const uint32_t len = f ? uint32_t(code_len[c]) : 0u;  // at most L
    const uint64_t rw = len ? __brevll(code_word[c]) >> (64 - len) : 0ull;  // code bit m at bit m
    for (uint32_t m = 0; m < L; ++m) {
      add(m, len == m + 1 ? f : 0ull);
      add(L + m, len > m && !((rw >> m) & 1u) ? f : 0ull);
    }
    uint32_t id = 2 * L;
    for (uint32_t l = 0; l < L; l += K, id += C)
      for (uint32_t j = 1; j <= K && l + j <= L; ++j) {
        const uint32_t v = uint32_t(rw >> l) & ((1u << j) - 1u);
        for (uint32_t x = 0; x < (1u << j); ++x) add(id + (1u << j) - 2 + x, len > l + j && v == x ? f : 0ull);
      }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < counters; i += kCountThreads) {
    unsigned long long t = 0;
    for (int w = 0; w < kCountThreads / 32; ++w) t += acc[w * counters + i];
    if (t) atomicAdd(out + i, t);
  }
}

}  // namespace

void launch_huffman_keys(const void* text, uint64_t n, uint32_t width, const uint64_t* code_len,
                         const uint64_t* code_word, uint64_t ncodes, uint32_t levels, uint32_t key_bytes, void* keys,
                         uint32_t* status, cudaStream_t s, uint64_t* launches) {
  if (n == 0) return;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  ++*launches;
  if (width == 1) {
    // (the grid covers short texts once)
    const int blocks = int(std::min<uint64_t>(uint64_t(sms) * 8, (n + 1023) / 1024));
    switch (key_bytes) {
      case 1: launch_table<uint8_t, uint8_t, false, 256>(text, n, code_len, code_word, ncodes, levels, keys, status, blocks, s); break;
      case 2: launch_table<uint8_t, uint16_t, false, 256>(text, n, code_len, code_word, ncodes, levels, keys, status, blocks, s); break;
      case 4: launch_table<uint8_t, uint32_t, false, 256>(text, n, code_len, code_word, ncodes, levels, keys, status, blocks, s); break;
      default: launch_table<uint8_t, uint64_t, false, 256>(text, n, code_len, code_word, ncodes, levels, keys, status, blocks, s); break;
    }
    return;
  }
  if (width == 2 && n >= kKeyTableMin && key_bytes == 2) {
    launch_table<uint16_t, uint16_t, false, 1024>(text, n, code_len, code_word, ncodes, levels, keys, status, sms, s);
    return;
  }
  if (width == 2 && n >= kKeyTableMin && key_bytes == 4 && levels + 1 <= 24) {
    launch_table<uint16_t, uint32_t, true, 1024>(text, n, code_len, code_word, ncodes, levels, keys, status, sms, s);
    return;
  }
  if (width == 2) launch_gather<uint16_t>(key_bytes, text, n, code_len, code_word, ncodes, levels, keys, status, s);
  else launch_gather<uint32_t>(key_bytes, text, n, code_len, code_word, ncodes, levels, keys, status, s);
}

void launch_huff_counts(const unsigned long long* hist, const uint64_t* code_len, const uint64_t* code_word,
                        uint64_t ncodes, uint32_t L, uint32_t K, unsigned long long* out, cudaStream_t s,
                        uint64_t* launches) {
  const unsigned blocks = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((ncodes + 255) / 256, 152)));
  const size_t smem = size_t(huff_count_words(L, K)) * (kCountThreads / 32) * 8;
  cudaFuncSetAttribute(huff_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  huff_count_kernel<<<blocks, kCountThreads, smem, s>>>(hist, code_len, code_word, ncodes, L, K, out);
  ++*launches;
}

}  // namespace pwmgpu
