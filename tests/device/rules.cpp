// The rules of the dispatch on sizes that a test chooses, without CUDA.  Built by tests/device/__init__.py.
#include <algorithm>
#include <cstdint>

#include "cfm_b200.h"

namespace cfm {

// What the rules look at, under the names of cfm_reader.cu.
struct Layer {
  int H, I, E, K, F, N, B, R, global_experts, tensor_engine, row_engine;
  const int32_t* expert_map;
};
struct Bound {
  Layer L;
  int T;
};
constexpr int kScreenChannels = 128, kMixTokens = 16;
struct DownUnion {
  static constexpr int kColumns = 64;
};

#include "cfm_rules.cuh"

}  // namespace cfm

// out: tcgen05 screen, pairs per pass, gather by pairs, encoder rows shared, gather by unions.
extern "C" void dispatch(const cfm_layer* layer, int tokens, int32_t* out) {
  cfm::Bound b = {};
  b.L = {layer->hidden, layer->width, layer->experts, layer->top_k, layer->final_count, layer->top_k * layer->width,
         layer->hidden / 128, layer->rank, layer->global_experts, layer->tensor_engine, layer->row_engine,
         layer->global_experts ? out : nullptr};
  b.T = tokens;
  out[0] = cfm::screens_tc(b);
  out[1] = cfm::pass_pairs(b);
  out[2] = cfm::gathers_by_pair(b);
  out[3] = cfm::shares_encoder(b);
  out[4] = cfm::exact_by_union(b);
}
