// Popcount rank/select support in pwm's layout and batched queries.
//
// Layout (include/queries/bin_rank_popcnt.hpp:32-86, popcnt_traits.hpp:
// 12-21): per level, one l12 entry per L1 block of 32 words (2048 bits): the
// u32 count of ones before the block (wrapping like pwm's u32) and the ones
// of its first three 512-bit L2 blocks in 10-bit fields.  When the level has
// a multiple of 32 words pwm keeps one more, zeroed, entry; so does this
// layout.  l0 is all zero for levels below 2^32-1 bits (the only sizes
// accepted).  Select samples (bin_select_popcnt.hpp:38-107): the position of
// every 8192nd zero/one, taken in the L1 block where the running count first
// exceeds the next sample number.
#include <algorithm>
#include <mutex>

#include "kernels.cuh"

namespace pwmgpu {

namespace {

constexpr uint64_t kL1Bits = 2048, kL1Cover = 32, kL2Cover = 8, kSampleRate = 8192;
constexpr int kRsThreads = 512;

// Select-sample position inside L1 block b: the `rem`-th one (value 1) or
// zero (value 0) counted from the block's first word, found by one thread.
// pwm walks the L2 blocks and then the words of the block
// (bin_select_popcnt.hpp:55-99); skipping whole L2 blocks by their counts
// first does not change which word and rank it ends on, so this gives the
// same position.  Only words of the level count (the last block may be
// short).  rem == 0 is pwm's word_select1(first word, 0).  Returns false when
// the block ends before the rem-th bit (pwm then takes no sample).
__device__ __forceinline__ bool thread_block_select(const uint64_t* data, uint64_t nwords, uint32_t fields,
                                                    uint64_t b, int value, uint32_t rem, uint64_t* pos) {
  const uint64_t w0 = b * kL1Cover;
  if (rem == 0) {
    const uint64_t first = value ? data[w0] : ~data[w0];
    *pos = word_select1(first, 0) + 64 * w0;
    return true;
  }
  // skip whole L2 blocks (8 words) by their counts; the fourth has no field
  uint32_t sub = 0;
  for (; sub < 3; ++sub) {
    const uint64_t ws = w0 + kL2Cover * sub;
    const uint64_t left = ws >= nwords ? 0 : nwords - ws;
    const uint32_t words = uint32_t(left < kL2Cover ? left : kL2Cover);
    const uint32_t ones = (fields >> (10 * sub)) & 1023u;
    const uint32_t cnt = value ? ones : 64u * words - ones;
    if (rem <= cnt) break;
    rem -= cnt;
  }
  const uint64_t ws = w0 + kL2Cover * sub;
  if (ws + kL2Cover <= nwords && (reinterpret_cast<uintptr_t>(data) & 15) == 0) {
    // a whole L2 block: its words at once, the one that holds the bit by their counts
    const uint4* v = reinterpret_cast<const uint4*>(data + ws);
    uint64_t w[kL2Cover];
#pragma unroll
    for (uint32_t k = 0; k < kL2Cover / 2; ++k) {
      const uint4 x = v[k];
      w[2 * k] = uint64_t(x.y) << 32 | x.x;
      w[2 * k + 1] = uint64_t(x.w) << 32 | x.z;
    }
    uint32_t run = 0, at = kL2Cover, left = 0;
    uint64_t word = 0;
#pragma unroll
    for (uint32_t k = 0; k < kL2Cover; ++k) {
      const uint64_t y = value ? w[k] : ~w[k];
      const uint32_t pc = uint32_t(__popcll(y));
      if (rem > run && rem <= run + pc) {
        at = k;
        left = rem - run;
        word = y;
      }
      run += pc;
    }
    if (at < kL2Cover) {
      *pos = word_select1(word, left) + 64 * (ws + at);
      return true;
    }
    return false;
  }
  for (uint32_t k = 0; k < kL2Cover; ++k) {
    if (ws + k >= nwords) return false;
    const uint64_t w = value ? data[ws + k] : ~data[ws + k];
    const uint32_t pc = uint32_t(__popcll(w));
    if (pc >= rem) {
      *pos = word_select1(w, rem) + 64 * (ws + k);
      return true;
    }
    rem -= pc;
  }
  return false;
}

// One pass over the words: a CTA counts 512 L1 blocks (128 KB of a level),
// learns the ones before them by a decoupled look-back over the level's CTAs
// and writes the finished entries and the select samples that fall into its
// blocks, whose words are still in L2.  (Three kernels before: block counts
// into scratch, a scan of the CTA totals, and the entries and samples from
// the scratch and a second look at the words.  Both structures of 10^6 bytes,
// 8 levels: 12 us of kernels and two more launches -> 7 us; 8 levels of 2^30
// bits 261 -> 254 us, 171 of them the reading and counting, the rest waits on
// predecessors and samples.)  CTAs take their place in
// the level by ticket, so a CTA waits only for CTAs that already run; the wait
// is bounded: a CTA that gives up records kErrTimeout, goes on with a zero
// prefix and marks its own (kLost), as do all that build on it, and the last
// one writes all ones for the level's number of ones.  Consecutive CTAs belong to
// different levels: with the resident CTAs all in one level, prefixes reached
// them too slowly (8 levels of 2^30 bits 388 against 273 us, both with 256
// threads; 512 threads 254).  Looking back over 64 to 256 CTAs a step changed
// nothing: the wait is for the slowest loads.
//
// With few levels that wait has nothing to hide behind: all resident CTAs load,
// then all wait.  Up to 3 levels of 2^22 words and more therefore take two
// kernels: kRsCount leaves every block's ones before it in its CTA in its
// entry and the CTAs' totals in the state words; kRsFinish adds the totals up
// and finishes entries and samples from there.  One level alone, one kernel
// and two: 2^22 words 21.3 and 20.9 us, 2^23 29.9 and 24.2, 2^24 56.6 and
// 46.5, 33.4 million 98.7 and 80.9 (the three kernels 82.4).  Whole builds of
// 2^28 symbols: 2 levels of the matrix 200.1 and 197.1 us, 3 of both
// structures 219.5 and 215.9; 4 levels are even (2^30: 1487 and 1489), 7
// better in one (1681 and 1699).
//
// Counting: warp w reads its 32 blocks (8 KB) with coalesced 16-byte loads: in
// step i, lanes 0-15 read block 2i and lanes 16-31 block 2i+1, four lanes per
// 512-bit L2 block; the counts are then gathered so that lane b holds block
// b's.
constexpr uint64_t kLost = 1ull << 61;  // of a state word: the counts before it are incomplete
constexpr uint32_t kRsTwoKernelLevels = 3;                 // at most
constexpr uint64_t kRsTwoKernelWords = uint64_t(1) << 22;  // of the longest, at least
enum RsPart { kRsAll, kRsCount, kRsFinish };
template <RsPart PART>
__global__ void __launch_bounds__(kRsThreads, PART == kRsFinish ? 4 : 2) rank_select_kernel(const RankSelectArgs a) {
  chain_next();
  chain_wait();
  const uint32_t y = blockIdx.x;
  RankSelectLevel L, twin{};
  bool twinned = false;
  if (y < a.nfirst) {
    L = a.first ? a.first[a.first_lo + y] : a.one;
    twinned = a.twin && a.first_lo + y == 0;  // level 0 of a plain tree is the matrix's
    if (twinned) twin = a.second[0];
  } else {
    L = a.second[a.second_lo + y - a.nfirst];
  }
  const uint64_t nreal = (L.nwords + kL1Cover - 1) / kL1Cover, n12 = L.nwords / kL1Cover + 1;
  const uint64_t ctas = nreal ? (nreal + kRsThreads - 1) / kRsThreads : 1;
  const uint32_t withheld = a.withhold && ctas > 1 ? 1 : 0;  // the level's first CTA does not run
  if (blockIdx.y + withheld >= ctas) return;
  unsigned long long* state = a.state + uint64_t(y) * a.stride;  // a ticket, then a word a CTA
  uint32_t cta = blockIdx.y;
  if constexpr (PART == kRsAll) {
    __shared__ uint32_t s_cta;
    if (threadIdx.x == 0) s_cta = uint32_t(atomicAdd(state, 1ull)) + withheld;
    __syncthreads();
    cta = s_cta;
  }
  const uint64_t first = uint64_t(cta) * kRsThreads, b = first + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ uint32_t wsum[kRsThreads / 32];
  __shared__ unsigned long long s_before;
  __shared__ bool s_lost;
  uint32_t v, fields, total, before_block;  // the block's ones and L2 fields; the CTA's ones, and those before the block
  if constexpr (PART == kRsFinish) {
    // as kRsCount left them: the ones before the block in its CTA, and the CTAs' totals
    __shared__ uint32_t in_cta[kRsThreads + 1];
    __shared__ unsigned long long wbefore[kRsThreads / 32];
    total = uint32_t(state[1 + cta]);
    before_block = b < nreal ? L.l12[2 * b] : total;
    fields = b < nreal ? L.l12[2 * b + 1] : 0u;
    in_cta[threadIdx.x] = before_block;
    if (threadIdx.x == 0) in_cta[kRsThreads] = total;
    unsigned long long before = 0;
    for (uint32_t k = threadIdx.x; k < cta; k += kRsThreads) before += state[1 + k];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, d);
    if (lane == 0) wbefore[warp] = before;
    __syncthreads();
    v = in_cta[threadIdx.x + 1] - before_block;
    if (threadIdx.x == 0) {
      unsigned long long all = 0;
      for (int w = 0; w < kRsThreads / 32; ++w) all += wbefore[w];
      s_before = all;
      s_lost = false;
    }
  } else {
    uint32_t l2[4] = {0, 0, 0, 0};
    const uint64_t wb = first + 32 * uint64_t(warp);  // first block of this warp
    const uint64_t ww = wb * kL1Cover;                 // first word of this warp
    // 16-byte loads when the warp's words are all in the level and aligned
    const bool full = ww + 32 * kL1Cover <= L.nwords && (reinterpret_cast<uintptr_t>(L.data) & 15) == 0;
    auto gather = [&](int i, uint32_t c) {
      c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
      c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
      // lane 2i takes block 2i's four counts (lanes 0,4,8,12), lane 2i+1 block 2i+1's (16,20,24,28)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t x = __shfl_sync(0xFFFFFFFFu, c, (lane & 1) * 16 + 4 * k);
        if ((lane >> 1) == i) l2[k] = x;
      }
    };
    if (full) {
      // all 16 loads of the lane in flight before the first popcount
      uint32_t c[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint4 v = *reinterpret_cast<const uint4*>(L.data + ww + 2 * uint64_t(i * 32 + lane));
        c[i] = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) gather(i, c[i]);
    } else {
      for (int i = 0; i < 16; ++i) {
        const uint64_t w = ww + 2 * uint64_t(i * 32 + lane);  // first of this lane's two words
        gather(i, (w < L.nwords ? __popcll(L.data[w]) : 0) + (w + 1 < L.nwords ? __popcll(L.data[w + 1]) : 0));
      }
    }
    // exclusive scan of the block totals (past the level: 0)
    v = l2[0] + l2[1] + l2[2] + l2[3];
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t s = __shfl_up_sync(0xFFFFFFFFu, x, d);
      if (lane >= d) x += s;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t before_warp = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kRsThreads / 32; ++w) {
      before_warp += w < warp ? wsum[w] : 0u;
      total += wsum[w];
    }
    before_block = before_warp + x - v;
    fields = (l2[0] & 1023u) | ((l2[1] & 1023u) << 10) | ((l2[2] & 1023u) << 20);
    if constexpr (PART == kRsCount) {
      if (threadIdx.x == 0) state[1 + cta] = total;
      if (b < nreal) {
        L.l12[2 * b] = before_block;
        L.l12[2 * b + 1] = fields;
      }
      return;
    }
  }
  // publish, then look back 32 CTAs a step
  if (PART == kRsAll && warp == 0) {
    unsigned long long before = 0;
    bool lost = false;
    if (lane == 0) st_volatile(state + 1 + cta, (cta == 0 ? kFlagPrefix : kFlagAggregate) | total);
    for (int64_t at = int64_t(cta) - 1; at >= 0; at -= 32) {
      const int64_t k = at - lane;
      uint64_t w = kFlagPrefix;  // before the level: nothing
      if (k >= 0) {
        w = ld_volatile(state + 1 + k);
        for (uint32_t spins = 0; (w >> 62) == 0; ++spins) {
          if (spins >= a.spin_limit) {
            atomicOr(a.status, kErrTimeout);
            w = kFlagPrefix | kLost;
            break;
          }
          __nanosleep(32);
          w = ld_volatile(state + 1 + k);
        }
      }
      const uint32_t done = __ballot_sync(0xFFFFFFFFu, (w >> 62) == 2);
      const int stop = done ? __ffs(done) - 1 : 31;  // the nearest CTA with everything before it
      unsigned long long c = lane <= stop ? (w & (kLost - 1)) : 0ull;
      lost |= __any_sync(0xFFFFFFFFu, lane <= stop && (w & kLost));
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, d);
      before += c;
      if (done) break;
    }
    if (lane == 0) {
      if (cta) st_volatile(state + 1 + cta, kFlagPrefix | (lost ? kLost : 0) | (before + total));
      s_before = before;
      s_lost = lost;
    }
  }
  __syncthreads();
  const uint64_t level_before = s_before;
  auto finish = [&](const RankSelectLevel& R) {  // the outputs of one structure
    if (cta == 0) {
      // all zero below 2^32-1 bits per level (the only sizes built)
      for (uint64_t i = threadIdx.x; i < L.nwords / (4294967295ull / 64) + 1; i += kRsThreads) R.l0[i] = 0;
      if (threadIdx.x == 0) {
        if (n12 < 2) R.meta[0] = R.meta[1] = 0;  // too short for pwm to examine a block
        if (n12 > nreal) R.l12[2 * nreal] = R.l12[2 * nreal + 1] = 0;
      }
    }
    if (threadIdx.x == 0 && cta + 1 == ctas) R.meta[2] = s_lost ? ~0ull : level_before + total;  // ones of the level
  };
  finish(L);
  if (twinned) finish(twin);
  if (b >= nreal) return;
  const uint64_t ones_before = level_before + before_block, ones_through = ones_before + v;
  auto entry = [&](const RankSelectLevel& R) {
    R.l12[2 * b] = uint32_t(ones_before);
    R.l12[2 * b + 1] = fields;
  };
  entry(L);
  if (twinned) entry(twin);
  if (b + 1 >= n12) return;  // pwm examines blocks 0 .. n12-2
  // sample s is taken in the first block whose running count exceeds
  // 1 + 8192 s (bin_select_popcnt.hpp:55-99); pwm's count before the entry
  // that follows the last real block is 0
  const uint64_t through = b + 1 < nreal ? ones_through : 0;
  const uint64_t s1 = ones_before == 0 ? 0 : (ones_before - 1 + kSampleRate - 1) / kSampleRate;
  const uint64_t next1 = 1 + kSampleRate * s1;
  const uint64_t f_prev = b * kL1Bits - ones_before;
  const uint64_t f_here = (b + 1) * kL1Bits - through;
  const uint64_t s0 = f_prev == 0 ? 0 : (f_prev - 1 + kSampleRate - 1) / kSampleRate;
  const uint64_t next0 = 1 + kSampleRate * s0;
  uint64_t pos;
  auto sample = [&](int value, uint64_t s, uint64_t rem) -> uint32_t {
    if (!thread_block_select(L.data, L.nwords, fields, b, value, uint32_t(rem), &pos)) return 0;
    (value ? L.s1 : L.s0)[s] = uint32_t(pos);
    if (twinned) (value ? twin.s1 : twin.s0)[s] = uint32_t(pos);
    return 1;
  };
  const uint32_t got1 = through > next1 ? sample(1, s1, next1 - ones_before) : 0u;
  const uint32_t got0 = f_here > next0 ? sample(0, s0, next0 - f_prev) : 0u;
  // samples are taken in block order, so the count is fixed by the last
  // block pwm examines (n12 - 2): the samples before it plus its own
  if (b == n12 - 2) {
    L.meta[1] = s1 + got1;
    L.meta[0] = s0 + got0;
    if (twinned) {
      twin.meta[1] = s1 + got1;
      twin.meta[0] = s0 + got0;
    }
  }
}

// ---------------------------------------------------------------------------
// Queries (include/queries/query_support.hpp:39-178)
//
// A query walks one level after another, each step a few loads whose
// addresses come from the step before: latency bounds a small batch, scattered
// sectors a large one.  So a step asks for all it may need at once: a rank
// loads its block entry and the 512-bit L2 block (64 bytes, 64-byte aligned:
// levels start at multiples of 128) in one round trip, two 32-byte loads for
// the words, instead of walking up to 8 words one after the other; a select
// loads 8 block entries where the occurrence should lie and then one L2 block.
// A thread a query: pairs and quads of lanes sharing a query's words measured
// slower (5.0 and 7.2 against 4.2 ms for the large batch below), their
// exchanges costing more than the counting they save.  The level descriptors
// come from shared memory.  Measured (GB300): 3 x 10^4 queries on a tree of
// 10^6 bytes, 8 levels, 139 -> 52 us; 3 x 2^22 on the 2^28 16-bit matrix (16
// levels) 8.34 -> 4.22 ms (access 1.17, rank 1.32, select 1.72), bound by L1's
// scattered requests (80 % busy; DRAM 45 % of its peak).  128 threads a block
// spread a small batch over more SMs than 256 (50.7 against 54.5 us); 48
// registers a thread (10 blocks an SM) answered the large batch faster than 40
// (4.48 ms).
// ---------------------------------------------------------------------------
constexpr int kQueryThreads = 128;
constexpr uint32_t kQueryMaxLevels = 64;

// A level as the queries read it, in shared memory.
struct FastLevel {
  const uint64_t* data;
  const uint32_t* l12;
  const uint32_t* s0;
  const uint32_t* s1;
  uint32_t nwords;  // rank/select levels hold fewer than 2^32 - 64 bits
  uint32_t nreal;   // L1 blocks
  uint32_t total;   // ones
  uint32_t ns0, ns1;
  uint32_t zeros;   // matrix
  uint32_t bits;    // Huffman-shaped
};

// Four words, or four block entries (ones before the block in the low half,
// its L2 fields in the high one), by one 32-byte load.  The words go round L1
// and pull in no more than their 64 bytes of L2 (by default a miss fetched up
// to 128: 2^22 accesses took 13 % longer, ranks 68 %).
struct Four {
  uint64_t w[4];
};
__device__ __forceinline__ Four load_words(const uint64_t* p) {
  Four v;
  asm("ld.global.nc.L1::evict_first.L2::64B.v4.u64 {%0, %1, %2, %3}, [%4];"
      : "=l"(v.w[0]), "=l"(v.w[1]), "=l"(v.w[2]), "=l"(v.w[3])
      : "l"(p));
  return v;
}
__device__ __forceinline__ Four load_entries(const uint32_t* p) {
  Four v;
  asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(v.w[0]), "=l"(v.w[1]), "=l"(v.w[2]), "=l"(v.w[3]) : "l"(p));
  return v;
}

// ~0 << s with s >= 64 giving 0 (PTX clamps the shift amount).
__device__ __forceinline__ uint64_t high_mask(uint32_t s) {
  uint64_t r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(~0ull), "r"(s));
  return r;
}

// Ones of a level before `at` (bin_rank_popcnt::rank1, bin_rank_popcnt.hpp:
// 98-128).  The index of pwm's extra zeroed L1 entry answers with the level's
// total instead of 0, an index past the level with the whole level (the
// padding holds no ones), so that no index reads outside it.  BIT: also bit
// `at`.
struct Rank {
  uint32_t ones, bit;
};
template <bool BIT, typename I>
__device__ __forceinline__ Rank rank_at(const FastLevel& L, I at) {
  const uint32_t most = L.nwords * 64u - (BIT ? 1u : 0u);
  const uint32_t index = at > most ? most : uint32_t(at);
  const uint32_t l1 = index >> 11, l2 = (index >> 9) & 3u;
  if (l1 >= L.nreal) return Rank{L.total, 0u};
  const uint2 e = __ldg(reinterpret_cast<const uint2*>(L.l12) + l1);
  const int nb = int(index & 511u);
  const uint64_t* block = L.data + size_t(index >> 9) * 8;
  Rank r{0u, 0u};
  Four a = {}, b = {};
  if (BIT || nb > 0) a = load_words(block);
  if (BIT ? nb >= 256 : nb > 256) b = load_words(block + 4);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    r.ones += __popcll(a.w[k] & high_mask(uint32_t(max(64 * k + 64 - nb, 0))));
    r.ones += __popcll(b.w[k] & high_mask(uint32_t(max(64 * k + 320 - nb, 0))));
  }
  if (BIT) {
    const int k = nb & 255;
    const Four& h = nb < 256 ? a : b;
    const uint64_t w = k < 128 ? (k < 64 ? h.w[0] : h.w[1]) : (k < 192 ? h.w[2] : h.w[3]);
    r.bit = uint32_t(w >> (63 - (nb & 63))) & 1u;
  }
  // whole L2 blocks before it (at most 3)
  r.ones += e.x + (l2 > 0 ? e.y & 1023u : 0u) + (l2 > 1 ? (e.y >> 10) & 1023u : 0u) + (l2 > 2 ? (e.y >> 20) & 1023u : 0u);
  return r;
}
template <typename I>
__device__ __forceinline__ uint32_t ones_before(const FastLevel& L, I at) {
  return rank_at<false>(L, at).ones;
}

// bin_select_popcnt::select (bin_select_popcnt.hpp:112-117, 166-241), occ > 0:
// the sample of (occ - 1) / 8192 itself when occ is the one it was taken at,
// else the first L1 block from the sample's on whose successor's count
// reaches occ, then its L2 block and word.  The occ-th bit lies at or before
// the next sample; the block is looked for first where occ's share of the
// 8192 puts it (a window of 8 entries: found there for all but a few in a
// thousand selects of the 16-bit matrix, whose gaps between samples reach 300
// blocks), then between the bounds that leaves, four probes a step.  False
// past the count.  (pwm walks on past its arrays there.)
__device__ __forceinline__ bool select_bit(const FastLevel& L, bool value, uint32_t occ, uint32_t* pos) {
  if (L.nwords == 0) return false;
  const uint32_t ns = value ? L.ns1 : L.ns0;
  const uint32_t* samples = value ? L.s1 : L.s0;
  const uint32_t sidx = (occ - 1) / uint32_t(kSampleRate), share = (occ - 1) % uint32_t(kSampleRate);
  uint32_t lo = 0, hi = L.nreal - 1, guess = 0;
  if (ns) {
    const uint32_t s = __ldg(samples + min(sidx, ns - 1));
    uint32_t nx = 0;
    if (sidx + 1 < ns) nx = __ldg(samples + sidx + 1);
    if (sidx < ns && share == 0) {
      *pos = s;
      return true;
    }
    guess = lo = min(s >> 11, hi);
    if (sidx + 1 < ns) {
      hi = max(lo, min(hi, nx >> 11));
      guess = lo + uint32_t((uint64_t(hi - lo) * share) >> 13);
    }
  }
  // ones (or zeros) before block e, from its entry's ones
  auto before = [&](uint32_t e, uint32_t ones) { return value ? ones : e * uint32_t(kL1Bits) - ones; };
  // the last of blocks lo..hi with fewer than occ before it; lo is one
  uint32_t base = guess > lo + 2 ? (guess - 2) & ~3u : lo & ~3u;
  uint32_t l1;
  uint64_t entry = 0;
  for (;;) {
    const Four u = load_entries(L.l12 + 2 * size_t(base));
    Four v = {};
    if (base + 4 <= hi) v = load_entries(L.l12 + 2 * size_t(base + 4));
    // the entries ascend: the last one below occ is the answer, if the window holds it
    uint32_t n = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      const uint64_t e = k < 4 ? u.w[k & 3] : v.w[k & 3];
      if (base + k <= lo || (base + k <= hi && before(base + k, uint32_t(e)) < occ)) {
        n = k + 1;
        entry = e;
      }
    }
    if (n == 0) {
      hi = base - 1;
    } else if (n == 8 && base + 7 < hi) {
      lo = base + 7;
    } else {
      l1 = base + n - 1;
      break;
    }
    while (hi - lo > 4) {
      const uint64_t span = hi - lo;
      uint32_t e[4], x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) e[k] = lo + uint32_t(span * uint32_t(k + 1) / 5);
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = __ldg(L.l12 + 2 * size_t(e[k]));
#pragma unroll
      for (int k = 3; k >= 0; --k)
        if (before(e[k], x[k]) >= occ) hi = max(e[k] - 1, lo);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (e[k] <= hi) lo = e[k];
    }
    base = lo & ~3u;
  }
  occ -= before(l1, uint32_t(entry));
  // the L2 block: whole blocks skipped by their counts, the fourth has none
  uint32_t f = uint32_t(entry >> 32);
  f = value ? f : (512u | 512u << 10 | 512u << 20) - (f & 0x3FFFFFFFu);  // no borrows: a field is at most 512
  const uint32_t c0 = f & 1023u, c1 = c0 + ((f >> 10) & 1023u), c2 = c1 + ((f >> 20) & 1023u);
  const uint32_t l2 = (occ > c0 ? 1u : 0u) + (occ > c1 ? 1u : 0u) + (occ > c2 ? 1u : 0u);
  occ -= occ > c2 ? c2 : occ > c1 ? c1 : occ > c0 ? c0 : 0u;
  uint32_t word = l1 * 32 + l2 * 8;
  if (word >= L.nwords) return false;
  // the word (those past the level, inside its padding, hold no ones; a zero
  // found there lies past the count)
  const Four a = load_words(L.data + word), b = load_words(L.data + word + 4);
  const uint32_t pa0 = value ? __popcll(a.w[0]) : 64u - __popcll(a.w[0]);
  uint64_t x = a.w[0];
  uint32_t k = occ, run = pa0;
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    const uint64_t w = i < 4 ? a.w[i & 3] : b.w[i & 3];
    if (occ > run) {
      x = w;
      k = occ - run;
      word = l1 * 32 + l2 * 8 + i;
    }
    run += value ? __popcll(w) : 64u - __popcll(w);
  }
  if (occ > run || word >= L.nwords) return false;
  // the k-th bit of the word, halved from 32 down
  if (!value) x = ~x;
  uint32_t at = 64 * word;
  uint32_t c = uint32_t(x >> 32), n = __popc(c);
  if (k > n) {
    k -= n;
    at += 32;
    c = uint32_t(x);
  }
#pragma unroll
  for (int h = 16; h; h >>= 1) {
    n = __popc(c >> (32 - h));
    if (k > n) {
      k -= n;
      c <<= h;
      at += h;
    }
  }
  *pos = at;
  return true;
}

__device__ uint64_t huff_decode(const HuffQueryTables& h, uint32_t len, uint64_t word) {
  const uint64_t key = (uint64_t(len) << 56) | word;
  uint64_t lo = 0, hi = h.ndec;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (h.dec_key[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo < h.ndec && h.dec_key[lo] == key ? h.dec_sym[lo] : ~0ull;
}

// access(index): the symbol at a position below n.
template <bool TREE, bool HUFF>
__device__ __forceinline__ uint64_t query_access(const QueryStructure& S, const HuffQueryTables& h, const FastLevel* lv,
                                                 uint32_t index) {
  const uint32_t Lv = S.levels;
  uint64_t word = 0;
  uint32_t start = 0, end = uint32_t(S.n);
  for (uint32_t level = 0; level < Lv; ++level) {
    const FastLevel& L = lv[level];
    const Rank at = rank_at<true>(L, start + index);
    const bool one = at.bit != 0;
    word = (word << 1) | at.bit;
    if constexpr (TREE) {
      const uint32_t ra = ones_before(L, start), rb = ones_before(L, end);
      const uint32_t mid = end - rb + ra;  // where the node's zeros end: start + zeros inside it
      index = one ? at.ones - ra : start + index - at.ones - (start - ra);
      if (one) start = mid;
      else end = mid;
    } else {
      index = one ? L.zeros + at.ones : index - at.ones;
    }
    if (HUFF && (level + 1 == Lv || start + index >= lv[level + 1].bits)) return huff_decode(h, level + 1, word);
  }
  return word;
}

// rank(symbol, index): `len` bits of `code`, most significant first.  I =
// uint32_t: index at most n; uint64_t: any index.
template <bool TREE, bool HUFF, typename I>
__device__ __forceinline__ uint64_t query_rank(const QueryStructure& S, const FastLevel* lv, uint64_t code, uint32_t len,
                                               I index) {
  I start = 0, end = I(S.n);  // the symbol's node; a matrix uses start alone, its block's first position
  for (uint32_t level = 0; level < len; ++level) {
    const FastLevel& L = lv[level];
    const bool one = (code >> (len - 1 - level)) & 1;
    if constexpr (TREE) {
      if (HUFF && index == 0) break;
      const I at = ones_before(L, I(start + index)), ra = ones_before(L, start), rb = ones_before(L, end);
      const I mid = end - rb + ra;
      index = one ? at - ra : start + index - at - (start - ra);
      if (one) start = mid;
      else end = mid;
    } else {
      const I ra = ones_before(L, start), rb = ones_before(L, index);
      start = one ? L.zeros + ra : start - ra;
      index = one ? L.zeros + rb : index - rb;
    }
  }
  return TREE ? index : I(index - start);
}

// select(symbol, occ), occ > 0; node: words [2 * level] and [2 * level + 1] of
// this query in shared memory, blockDim.x apart (a tree's node starts and
// zero counts on the way down).  I = uint32_t: occ at most n; `bad` is set,
// with no answer, where a step leaves the level (an occurrence past the
// symbol's last).  uint64_t: any occ, such steps carried through as 64-bit
// numbers.
template <bool TREE, bool HUFF, typename I>
__device__ __forceinline__ uint64_t query_select(const QueryStructure& S, const FastLevel* lv, uint32_t* node,
                                                 uint64_t code, uint32_t len, I occ, bool* bad) {
  constexpr bool WIDE = sizeof(I) == 8;
  const uint32_t n = uint32_t(S.n);
  uint32_t start = 0, end = n;
  for (uint32_t level = 0; level < len; ++level) {
    const FastLevel& L = lv[level];
    const bool one = (code >> (len - 1 - level)) & 1;
    const uint32_t ra = ones_before(L, start);
    if constexpr (TREE) {
      const uint32_t rb = ones_before(L, end);
      node[(2 * level) * blockDim.x] = start;
      node[(2 * level + 1) * blockDim.x] = start - ra;
      const uint32_t mid = end - rb + ra;
      if (one) start = mid;
      else end = mid;
    } else {
      if constexpr (HUFF) {
        const uint32_t rb = ones_before(L, end);
        end = one ? L.zeros + rb : end - rb;
      }
      start = one ? L.zeros + ra : start - ra;
    }
  }
  if (HUFF && occ > I(end - start)) return ~0ull;  // the symbol's node holds its occurrences
  if constexpr (!TREE) {
    if (!WIDE && occ > n - start) {
      *bad = true;
      return 0;
    }
    occ += start;
  }
  for (int level = int(len) - 1; level >= 0; --level) {
    const FastLevel& L = lv[level];
    const uint32_t adj = level == 0 ? 0 : 1;
    const bool one = (code >> (len - 1 - uint32_t(level))) & 1;
    uint32_t off = one ? L.zeros : 0u, st = 0;  // the (occ - off)-th such bit of the level; its position less st
    if constexpr (TREE) {
      st = node[(2 * level) * blockDim.x];
      const uint32_t left = node[(2 * level + 1) * blockDim.x];
      off = 0u - (one ? st - left : left);
    }
    uint32_t pos = 0;
    if constexpr (WIDE) {
      const uint64_t o = TREE ? occ + uint32_t(0u - off) : occ - off;
      uint64_t at = 0;
      if (o != 0) at = (o >> 32) == 0 && select_bit(L, one, uint32_t(o), &pos) ? uint64_t(pos) : ~0ull;
      occ = at - st + adj;
    } else {
      // a matrix's one lies past the zeros, a tree's bit inside the level
      const uint32_t o = occ - off;
      if ((TREE ? (occ > n || o > n) : (one && occ <= off)) || !select_bit(L, one, o, &pos) || (TREE && pos < st)) {
        *bad = true;
        return 0;
      }
      occ = pos - st + adj;
    }
  }
  return occ;
}

// Operands past the text or the last occurrence: the 64-bit forms, out of the
// way of the ordinary ones.
template <bool TREE, bool HUFF>
__device__ __noinline__ uint64_t query_outside(const QueryStructure& S, const FastLevel* lv, uint32_t* node, int op,
                                               uint64_t code, uint32_t len, uint64_t arg) {
  bool bad = false;
  return op == 1 ? query_rank<TREE, HUFF, uint64_t>(S, lv, code, len, arg)
                 : query_select<TREE, HUFF, uint64_t>(S, lv, node, code, len, arg, &bad);
}

// A batch of queries, a thread each.  OP: 0 access, 1 rank, 2 select; -1: a
// mixed batch, ops[t] the kind of query t, and blockIdx.y the kind this block
// answers (a warp whose lanes hold different kinds runs them one after the
// other; a block a kind runs them side by side).
//
// Huffman-shaped structures (pwm's query_support has none: it prints "NOT YET
// IMPLEMENTED", include/queries/query_support.hpp:43,55,67): level l holds
// bit l of every code longer than l.  In both shapes the codes that end at a
// level sort behind all codes that go on: the matrix's codes (huff_codes.hpp:
// 204-245) take, length by length, the largest bit-reversed words, and the
// tree's are negated canonical codes (:246-283), the largest prefixes.  So
// level l + 1 is a prefix of level l's entries reordered as the plain
// structures reorder them (the matrix by its stable 0/1 partition, the tree
// within each node), and the plain position arithmetic holds; a code ends
// where its position falls past the next level's size.
template <int OP, bool TREE, bool HUFF>
__global__ void __launch_bounds__(kQueryThreads, 10) query_kernel(QueryStructure S, HuffQueryTables h,
                                                                 const uint8_t* __restrict__ ops,
                                                                 const uint64_t* __restrict__ a,
                                                                 const uint64_t* __restrict__ b, uint64_t count,
                                                                 uint64_t* __restrict__ out) {
  __shared__ FastLevel lv[kQueryMaxLevels];
  extern __shared__ uint32_t nodes[];  // a tree's selects: [2 * levels][threads]
  for (uint32_t l = threadIdx.x; l < S.levels; l += blockDim.x) {
    const QueryLevel L = S.lv[l];
    const uint64_t cap = L.nwords * 64 / kSampleRate + 2;  // entries of a sample array
    lv[l] = FastLevel{L.data, L.l12, L.s0, L.s1, uint32_t(L.nwords), uint32_t((L.nwords + kL1Cover - 1) / kL1Cover),
                      uint32_t(L.meta[2]), uint32_t(min(uint64_t(L.meta[0]), cap)),
                      uint32_t(min(uint64_t(L.meta[1]), cap)), TREE ? 0u : uint32_t(S.zeros[l]),
                      HUFF ? uint32_t(h.level_bits[l]) : 0u};
  }
  __syncthreads();
  const int op = OP >= 0 ? OP : int(blockIdx.y);
  uint32_t* node = nodes + threadIdx.x;
  for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < count; t += uint64_t(gridDim.x) * blockDim.x) {
    if (OP < 0 && int(ops[t]) != op) continue;
    uint64_t code = a[t], result = ~0ull;
    if (op == 0) {
      if (code < S.n) result = query_access<TREE, HUFF>(S, h, lv, uint32_t(code));
    } else {
      uint64_t arg = b[t];
      uint32_t len = S.levels;
      bool coded = true;
      if constexpr (HUFF) {
        len = code < h.nsym ? uint32_t(h.code_len[code]) : 0u;
        code = len ? h.code_word[code] : 0;
        coded = len != 0 && len <= S.levels;
        if (op == 1) arg = arg < S.n ? arg : S.n;
      }
      if (!coded) {
        result = (op == 1 || arg == 0) ? 0 : ~0ull;  // a symbol without a code does not occur
      } else if (arg == 0) {
        result = 0;
      } else {
        bool bad = arg > S.n;
        if (!bad && op == 1) result = query_rank<TREE, HUFF, uint32_t>(S, lv, code, len, uint32_t(arg));
        if (!bad && op == 2) result = query_select<TREE, HUFF, uint32_t>(S, lv, node, code, len, uint32_t(arg), &bad);
        if (bad) result = query_outside<TREE, HUFF>(S, lv, node, op, code, len, arg);
      }
    }
    out[t] = result;
  }
}

template <bool TREE, bool HUFF>
void start_queries(const QueryStructure& q, const HuffQueryTables& h, int op, const uint8_t* ops, const uint64_t* a,
                   const uint64_t* b, uint64_t count, uint64_t* out, cudaStream_t s) {
  // a tree's selects hold 2 words a level and thread in shared memory: fewer
  // threads a block for deep trees (at most 64 levels: 32 KB)
  const bool nodes_used = TREE && (ops || op == 2);
  unsigned threads = kQueryThreads;
  while (nodes_used && size_t(2) * q.levels * threads * 4 > 32768) threads /= 2;
  const size_t nodes = nodes_used ? size_t(2) * q.levels * threads * 4 : 0;
  const dim3 grid(unsigned(std::min<uint64_t>((count + threads - 1) / threads, 152 * 512)), ops ? 3 : 1);
  if constexpr (!HUFF) {  // mixed batches: plain structures
    if (ops) {
      query_kernel<-1, TREE, HUFF><<<grid, threads, nodes, s>>>(q, h, ops, a, b, count, out);
      return;
    }
  }
  if (op == 0) query_kernel<0, TREE, HUFF><<<grid, threads, 0, s>>>(q, h, nullptr, a, b, count, out);
  else if (op == 1) query_kernel<1, TREE, HUFF><<<grid, threads, 0, s>>>(q, h, nullptr, a, b, count, out);
  else query_kernel<2, TREE, HUFF><<<grid, threads, nodes, s>>>(q, h, nullptr, a, b, count, out);
}

}  // namespace

void launch_queries(const QueryStructure& q, int op, const uint64_t* a, const uint64_t* b, uint64_t count,
                    uint64_t* out, cudaStream_t s, uint64_t* launches, const uint8_t* ops) {
  if (count == 0) return;
  if (q.is_tree) start_queries<true, false>(q, HuffQueryTables{}, op, ops, a, b, count, out, s);
  else start_queries<false, false>(q, HuffQueryTables{}, op, ops, a, b, count, out, s);
  ++*launches;
}

void launch_huff_queries(const QueryStructure& q, const HuffQueryTables& h, int op, const uint64_t* a,
                         const uint64_t* b, uint64_t count, uint64_t* out, cudaStream_t s, uint64_t* launches) {
  if (count == 0) return;
  if (q.is_tree) start_queries<true, true>(q, h, op, nullptr, a, b, count, out, s);
  else start_queries<false, true>(q, h, op, nullptr, a, b, count, out, s);
  ++*launches;
}

uint64_t rank_select_state_words(uint64_t max_words) {
  const uint64_t nreal = (max_words + kL1Cover - 1) / kL1Cover;
  return 1 + std::max<uint64_t>(1, (nreal + kRsThreads - 1) / kRsThreads);
}

void launch_rank_select(const RankSelectArgs& a, uint64_t max_words, cudaStream_t s, uint64_t* launches) {
  const uint32_t levels = a.nfirst + a.nsecond;
  if (levels == 0) return;
  const dim3 grid(levels, unsigned(rank_select_state_words(max_words) - 1));  // at most 8192 CTAs a level (2^32 bits)
  if (levels <= kRsTwoKernelLevels && max_words >= kRsTwoKernelWords && !a.withhold) {
    launch_chained(rank_select_kernel<kRsCount>, grid, kRsThreads, 0, s, a);
    launch_chained(rank_select_kernel<kRsFinish>, grid, kRsThreads, 0, s, a);
    *launches += 2;
    return;
  }
  launch_chained(rank_select_kernel<kRsAll>, grid, kRsThreads, 0, s, a);
  ++*launches;
}

// ===========================================================================
// Allocation-free rank/select build (pwmgpu_rank_select_build_noalloc).
//
// For callers that must not allocate device memory while they run:
// allocator-less plugins that receive every buffer from their host framework,
// and latency-critical serving loops that cannot afford an allocator's
// implicit synchronisation.  The look-back state of the build lives in a
// fixed, file-scope device array instead of context scratch, resident on every
// GPU that loads this library until the process exits; the level descriptor
// travels as a kernel parameter.  Every call shares the array: calls that
// overlap on the GPU (different streams, or different host threads on one
// device) race and must be serialised by the caller.
// ===========================================================================
namespace {

// The level limit is the entry point's published one.  The array: a status
// word (and one to align), then the look-back state of the longest level, a
// ticket and a word a CTA: 16 KB.
constexpr uint64_t kNoAllocMaxL1Blocks = (uint64_t(1) << 20) - (uint64_t(1) << 12);
constexpr uint64_t kNoAllocStateWords = 1 + (kNoAllocMaxL1Blocks + kRsThreads - 1) / kRsThreads;

static __device__ __align__(256) uint32_t g_noalloc_rs_scratch[2 + 2 * kNoAllocStateWords];

struct NoAllocSymbols {
  bool ready = false;
  uint32_t* scratch = nullptr;
};

}  // namespace

// Device address of the file-scope array for the current device, looked
// up once per device (the first call on a device does it) and kept for the
// life of the process: after a cudaDeviceReset the module may load at other
// addresses, so the entry point must not be used across a device reset.
cudaError_t noalloc_rank_select_symbols(uint32_t** scratch) {
  static std::mutex mu;
  static NoAllocSymbols per_device[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  NoAllocSymbols& s = per_device[dev];
  if (!s.ready) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_rs_scratch);
    if (e != cudaSuccess) return e;
    s.scratch = static_cast<uint32_t*>(p);
    s.ready = true;
  }
  *scratch = s.scratch;
  return cudaSuccess;
}

uint64_t noalloc_rank_select_max_words() { return kNoAllocMaxL1Blocks * kL1Cover; }

// Enqueues the build of one level's blocks on `stream` using only the
// file-scope array; outputs that must start at zero (l0, counts) are cleared
// here.  Returns cudaErrorInvalidValue for levels above the limit.
cudaError_t noalloc_rank_select_build(const uint64_t* words, uint64_t nwords, uint64_t* l0, uint32_t* l12,
                                      uint32_t* s0, uint32_t* s1, unsigned long long* counts, cudaStream_t stream) {
  if (nwords > noalloc_rank_select_max_words()) return cudaErrorInvalidValue;
  uint32_t* scratch = nullptr;
  cudaError_t e = noalloc_rank_select_symbols(&scratch);
  if (e != cudaSuccess) return e;
  const uint64_t n0 = nwords / (4294967295ull / 64) + 1;
  e = cudaMemsetAsync(l0, 0, n0 * 8, stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(counts, 0, 3 * 8, stream);
  if (e != cudaSuccess) return e;
  if (nwords == 0) {
    // pwm keeps one zeroed l12 entry for an empty level; no kernel runs
    e = cudaMemsetAsync(l12, 0, 2 * sizeof(uint32_t), stream);
    return e;
  }
  RankSelectArgs a{};
  a.one = RankSelectLevel{words, nwords, l0, l12, s0, s1, counts};
  a.nfirst = 1;
  a.stride = rank_select_state_words(nwords);
  if (a.stride > kNoAllocStateWords) return cudaErrorInvalidValue;
  a.status = scratch;
  a.state = reinterpret_cast<unsigned long long*>(scratch + 2);
  a.spin_limit = kSpinLimit;
  e = cudaMemsetAsync(scratch, 0, 8 + a.stride * 8, stream);
  if (e != cudaSuccess) return e;
  uint64_t launches = 0;
  launch_rank_select(a, nwords, stream, &launches);
  return cudaGetLastError();
}

}  // namespace pwmgpu
