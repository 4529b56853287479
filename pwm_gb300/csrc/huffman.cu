// Huffman-shaped builds: the code table from the device's symbol histogram
// (pwm's builder restated on the host) and the warp-pass engine on packed
// code keys.
#include "engine.hpp"

using namespace pwmgpu;

namespace pwmgpu {


// Symbol histogram + first occurrences of a device text on the GPU, then the
// code builder on the host.  The counts stay in the context's scratch and in
// `counts`, for build_huffman.
HuffCodes huffman_codes_device(pwmgpu_ctx* ctx, const void* d_text, uint64_t n, uint32_t width, bool is_tree,
                               uint64_t* max_symbol_out, SymbolCounts* counts) {
  cudaStream_t s = ctx->stream;
  uint64_t nsym = width == 1 ? 256 : (width == 2 ? 65536 : 0);
  if (width == 4) {
    // bound the alphabet by the largest symbol (one histogram bin per value)
    throw Fail{PWMGPU_ERR_ARG, "Huffman codes for 32-bit texts: pass a code table"};
  }
  // counts, ~first positions and the scratch of the latter, zeroed together
  const uint64_t seen_bytes = 65536 / 8 + 8;
  auto* d_hist = static_cast<unsigned long long*>(ctx->grow("sym_first", nsym * 16 + seen_bytes));
  auto* d_first = d_hist + nsym;
  CUDA_TRY(cudaMemsetAsync(d_hist, 0, nsym * 16 + seen_bytes, s));
  CUDA_TRY(cudaMemsetAsync(ctx->d_status, 0, 4, s));
  {
    ProfScope ps(ctx, "symbol_histogram", n * width);
    launch_symbol_histogram(d_text, n, width, nsym, d_hist, ctx->d_status, s, &ctx->launches);
    if (width > 1)
      launch_first_positions(d_text, n, width, nsym, d_first, reinterpret_cast<uint32_t*>(d_first + nsym), s,
                             &ctx->launches);
  }
  std::vector<uint64_t> count(nsym), first(nsym);
  CUDA_TRY(cudaMemcpyAsync(count.data(), d_hist, nsym * 8, cudaMemcpyDeviceToHost, s));
  if (width > 1) CUDA_TRY(cudaMemcpyAsync(first.data(), d_first, nsym * 8, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  for (auto& f : first) f = ~f;
  uint64_t max_symbol = 0;
  for (uint64_t c = 0; c < nsym; ++c)
    if (count[c]) max_symbol = c;
  *max_symbol_out = max_symbol;
  auto entries = width == 1 ? histogram_order<uint8_t>(count, first, 1) : histogram_order<uint16_t>(count, first, 2);
  if (counts) {
    counts->host = std::move(count);
    counts->device = d_hist;
  }
  return build_huffman_codes(entries, max_symbol, is_tree);
}

// Huffman build of one structure (matrix, or tree through the matrix).
// known: the text's symbol counts where the codes were just built from them.
// while_running: host work that only needs the codes and the level sizes,
// done while the passes run.
void build_huffman(pwmgpu_ctx* ctx, const void* d_text, uint64_t n, uint32_t width, bool is_tree,
                   const std::vector<uint64_t>& code_len, const std::vector<uint64_t>& code_word, uint32_t levels,
                   Structure& wm, Structure* wt, bool rank_select, const SymbolCounts* known,
                   const std::function<void()>& while_running) {
  cudaStream_t s = ctx->stream;
  const uint64_t ncodes = code_len.size();
  CUDA_TRY(cudaMemsetAsync(ctx->d_status, 0, 4, s));
  // symbol counts for the weighted codes
  SymbolCounts own;
  if (!known) {
    // 8- and 16-bit texts count every value (symbols past the table fail below)
    const uint64_t bins =
        std::max<uint64_t>(width <= 2 ? uint64_t(1) << (8 * width) : ncodes, std::max<uint64_t>(ncodes, 1));
    own.device = static_cast<unsigned long long*>(ctx->grow("sym_hist", bins * 8));
    CUDA_TRY(cudaMemsetAsync(own.device, 0, bins * 8, s));
    {
      ProfScope ps(ctx, "symbol_histogram", n * width);
      launch_symbol_histogram(d_text, n, width, ncodes, own.device, ctx->d_status, s, &ctx->launches);
    }
    own.host.resize(ncodes);
    CUDA_TRY(cudaMemcpyAsync(own.host.data(), own.device, ncodes * 8, cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    known = &own;
  }
  const std::vector<uint64_t>& count = known->host;
  uint64_t counted = 0, maxlen = 0;
  for (uint64_t c = 0; c < ncodes; ++c) {
    counted += count[c];
    if (!count[c]) continue;
    if (code_len[c] == 0 || code_len[c] > 56) throw Fail{PWMGPU_ERR_ARG, "a text symbol has no usable code"};
    maxlen = std::max(maxlen, code_len[c]);
  }
  if (counted != n) throw Fail{PWMGPU_ERR_SYMBOL, "a text symbol is outside the code table"};
  if (levels == 0) levels = uint32_t(maxlen);  // the longest code of a symbol that occurs
  if (maxlen != levels) throw Fail{PWMGPU_ERR_ARG, "levels must equal the longest code length"};
  // keys: the code and a stop bit, levels + 1 bits (split.cuh HuffKeys)
  const uint32_t key_bytes = huff_key_bytes(levels + 1);
  const auto plan = plan_passes(levels, ctx->pass_levels);
  uint64_t* d_len = static_cast<uint64_t*>(ctx->grow("code_len", std::max<uint64_t>(ncodes, 1) * 8));
  uint64_t* d_word = static_cast<uint64_t*>(ctx->grow("code_word", std::max<uint64_t>(ncodes, 1) * 8));
  CUDA_TRY(cudaMemcpyAsync(d_len, code_len.data(), ncodes * 8, cudaMemcpyHostToDevice, s));
  CUDA_TRY(cudaMemcpyAsync(d_word, code_word.data(), ncodes * 8, cudaMemcpyHostToDevice, s));
  // a matrix's tables from counts the device sums; a tree's prefix groups on
  // the host, while the keys are made
  const uint32_t kmax = uint32_t(ctx->pass_levels), nc = huff_count_words(levels, kmax);
  std::vector<uint64_t> counts(nc);
  if (!wt) {
    auto* d_counts = static_cast<unsigned long long*>(ctx->grow("huff_counts", nc * 8));
    CUDA_TRY(cudaMemsetAsync(d_counts, 0, nc * 8, s));
    launch_huff_counts(known->device, d_len, d_word, ncodes, levels, kmax, d_counts, s, &ctx->launches);
    CUDA_TRY(cudaMemcpyAsync(counts.data(), d_counts, nc * 8, cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
  }
  void* keys = ctx->grow("huff_keys", std::max<uint64_t>(n, 1) * key_bytes);
  {
    ProfScope ps(ctx, "huffman_keys", n * (width + key_bytes));
    launch_huffman_keys(d_text, n, width, d_len, d_word, ncodes, levels, key_bytes, keys, ctx->d_status, s,
                        &ctx->launches);
  }
  LevelTables tabs;
  if (!wt) {
    tabs = build_tables_counts(counts.data(), levels, plan, int(kmax));
  } else {
    std::vector<WeightedCode> wc;
    wc.reserve(ncodes);
    for (uint64_t c = 0; c < ncodes; ++c)
      if (count[c]) wc.push_back({code_word[c], uint32_t(code_len[c]), count[c]});
    tabs = build_tables(wc, levels, plan, true);
  }
  // layouts
  alloc_structure(wm, tabs.level_bits, n, false, true, rank_select && !is_tree, s);
  wm.zeros = tabs.zeros;
  CUDA_TRY(cudaMemcpyAsync(wm.d_zeros, wm.zeros.data(), levels * 8, cudaMemcpyHostToDevice, s));
  if (wt) alloc_structure(*wt, tabs.level_bits, n, true, true, rank_select, s);
  run_passes(ctx, keys, key_bytes, width, true, levels, plan, tabs, wm, wt, true);
  build_rank_select(ctx, !is_tree ? &wm : nullptr, wt);
  if (while_running) while_running();
  check_device_status(ctx);
}

}  // namespace pwmgpu
