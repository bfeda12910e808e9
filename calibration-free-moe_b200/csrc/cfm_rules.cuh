// Which kernels a call takes, by its sizes: the rules of the dispatch, host code only.
// `b` is a call: T tokens of a layer L.
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

// Experts that can have pairs.
static int busy_experts(const Bound& b) {
  return static_cast<int>(std::min<int64_t>(b.L.E, static_cast<int64_t>(b.T) * b.L.K));
}
// Pairs that this device's experts can expect of the call: all, or under expert parallelism their share.
static int64_t expected_pairs(const Bound& b) {
  const int64_t pairs = static_cast<int64_t>(b.T) * b.L.K;
  return b.L.expert_map && b.L.global_experts > 0 ? (pairs * b.L.E + b.L.global_experts - 1) / b.L.global_experts : pairs;
}
// More than 16/3 tokens per expert on average.
static bool shares_decode(const Bound& b) { return 3 * expected_pairs(b) > 16 * static_cast<int64_t>(b.L.E); }
// The tcgen05 screen on request, where several tokens share its decode, or where its CTAs of 128 channels
// give most SMs one or the rows are long.  Whole calls, us per layer, with it and with the warp-level kernel, which lets
// the selection be scheduled earlier: two tokens of the 128-expert layer (96 CTAs, 16 blocks) 36.7 and 34.8, of the
// 64-expert layer (128) 39.3 and 39.7; three and four of the 256-expert layer of width 512 (96, 128) 36.2 and 34.3, 37.3
// and 37.9, four with the recovery-aware score 41.0 and 45.4; three of the 128-expert layer (144) 38.9 and 40.0; four of a layer
// of 64 experts, hidden 1152 and width 704 (144, 9 blocks) 36.3 and 37.7; one token of hidden 4096 and width 1536 (96, 32 blocks) 54.9 and
// 54.8, three of hidden 4096, width 512 (96, 32) 46.1 and 50.1, two (64, 32) 43.6 and 39.0.  Its tables have to fit shared memory.
static bool screens_tc(const Bound& b) {
  const int64_t ctas = std::min<int64_t>(b.L.E, expected_pairs(b)) * ((b.L.I + kScreenChannels - 1) / kScreenChannels);
  if (b.L.tensor_engine == CFM_ENGINE_WARP) return false;
  return (b.L.tensor_engine == CFM_ENGINE_TCGEN05 || shares_decode(b) || ctas >= 128 || ctas * b.L.B >= 96 * 32) &&
         b.L.B <= 512;
}
// Its passes.  Of four tokens, five CTAs per SM and fewer instructions for empty places, up to four tokens per
// expert: 32 tokens of the 128-expert layer 24.5 us against 30.4 of passes of eight, 64 of them (4 per expert)
// 35.1 against 37.8, 50 of the 64-expert layer (6.3) 43 against 38.  Of sixteen from sixteen tokens per expert
// on: 256 tokens of hidden 4096 and width 1536 240 us against 269 of eight; 100 of the 64-expert layer (12.5)
// 50 against 47 (recovery-aware score 78 against 66), for fewer warps fit an SM and fewer passes are full.
// (One of eight ranks with 64 and 256 tokens of all of the 256-expert layer, two and eight per expert: passes of
// four 13.9 against 18.1 of sixteen, of eight 24.7 against 27.3.)
static int pass_pairs(const Bound& b) {
  if (!screens_tc(b)) return 8;
  const int64_t pairs = expected_pairs(b), experts = b.L.E;
  return pairs >= 16 * experts ? 16 : pairs <= 4 * experts ? 4 : 8;
}

// Batch size from which the down rows are read in expert order (the groups come from route and
// adopt); the gate and up rows see gathers_by_pair.
constexpr int kGroupedTokens = 8;
static bool pairs_grouped(const Bound& b) { return b.T >= kGroupedTokens; }

static bool encodes(const Bound& b) { return b.L.R > 0 && b.L.F < b.L.N; }

// The expert-major exact kernel, on request and from three tokens per expert and sixteen tokens on:
// below that the unions of an expert's kept channels are little smaller than their sum.  64 tokens of
// the 128-expert layer 67 us with the unions against 69 of the gathers, 100 of the 64-expert layer 100
// against 132, 256 of the 256-expert layer 96 against 155; at two tokens per expert 43 against 39 (32 of
// the 128-expert layer) and 141 against 120 (hidden 4096, width 1536).  Under expert parallelism the
// gathers per token stay, so that a token's bits do not depend on how the experts are spread.
static bool exact_by_union(const Bound& b) {
  if (!pairs_grouped(b) || b.L.expert_map || b.L.row_engine == CFM_ROWS_PER_TOKEN) return false;
  return b.L.row_engine == CFM_ROWS_EXPERT_MAJOR ||
         (b.T >= 16 && static_cast<int64_t>(b.T) * b.L.K >= 3 * static_cast<int64_t>(b.L.E));
}
// The expert-major down kernel, on request only: its sums depend in their last FP32 bits on what the
// other tokens of an expert kept, while the tiles give a token the same bits in every batch.  Where
// most experts have more than half a pass of sixteen tokens and there is a piece for every second
// warp: 64 tokens of the 128-expert layer 45 us with the output against 37 of the tiles, whole calls of
// 256 tokens 287 against 299 (256-expert layer) and 1535 against 1810 (hidden 4096, width 1536).
// (Repeating the sums that the distance could round otherwise, one in a hundred, costs more than the
// tiles: 3390 us there, most of it for single columns of rows that have left L2.)
static bool down_by_union(const Bound& b) {
  return exact_by_union(b) && b.L.row_engine == CFM_ROWS_EXPERT_MAJOR && shares_decode(b) &&
         static_cast<int64_t>(busy_experts(b)) * (b.L.H / DownUnion::kColumns) >= 148 * 8;
}
// Sixteen tokens per CTA of the output after it, and over the tiles of large batches while that gives
// every SM a CTA: 256 tokens of the 256-expert layer 15 us against 28, of hidden 4096 and width 1536 52
// against 127; 100 tokens of the 64-expert layer (112 CTAs) 21 against 15.
static bool mixes_tokens(const Bound& b) {
  return down_by_union(b) ||
         (exact_by_union(b) && (b.L.H / 128) * ((b.T + kMixTokens - 1) / kMixTokens) >= 148);
}
// The recovery encoder in the expert-major down launch.
static bool encodes_by_union(const Bound& b) { return down_by_union(b) && encodes(b); }
// Tokens per pass of the expert-major exact kernel, in eights: the next size up while the mean load
// is more than two thirds of the one before.  (The largest for all, leaving out tiles without tokens,
// spilled: 256 tokens of the 256-expert layer 97 us against 80, 64 of the 128-expert one 62 against 60.)
static int exact_union_tiles(const Bound& b) {
  int tiles = 1;
  while (tiles < 4 && 3 * static_cast<int64_t>(b.T) * b.L.K > 16 * tiles * static_cast<int64_t>(b.L.E)) tiles *= 2;
  return tiles;
}

// The gather that walks pairs in expert order, from twelve tokens and one token per expert on: below that the tokens
// share few rows, and every CTA's way to its rows is longer.  Whole calls, us per layer, this gather and the one that
// walks tokens: 9 tokens of the 128-expert layer (0.6 per expert) 58.3 and 56.2, of a layer of 32 experts (2.3) 52.7 and 51.1,
// of hidden 4096 and width 1536 132.3 and 129.8, of the 64-expert layer (1.1) 65.7 and 66.6; 12 of the 256-expert layer
// of width 512 (0.4) 53.5 and 52.4, 24 (0.8) 71.8 and 71.1, 40 (1.3) 94.0 and 94.4, 95 (3.0) 166.7 and 169.2; 16 of the
// 64-expert layer (2.0) 82.8 and 84.8; 12 of the 128-expert layer (0.8) 64.4 and 61.0, 24 (1.5) 87.9 and 86.9, 32 (2.0) 100.6 and 101.7,
// 47 (2.9) 126.0 and 129.2; 32 of hidden 4096 and width 1536 (2.0) 304.7 and 312.0.  Layers of few or short rows would
// rather walk tokens for longer: 12 tokens of 32 experts (3.0) 58.8 and 56.5, 28 of 100 experts of width 640 (1.7) 90.8 and 86.9.
static bool gathers_by_pair(const Bound& b) {
  return pairs_grouped(b) && (b.L.expert_map || (b.T >= 12 && static_cast<int64_t>(b.T) * b.L.K >= b.L.E));
}

// The encoder for four pairs of an expert at a time, from four tokens per expert on where the gathers beside
// it are long enough to cover its chain of loads, a quarter of a gigabyte: 96 tokens of the 128-expert layer
// (0.3 GB) 38 us against 45 of a pair at a time, 100 of the 64-expert layer 46 against 57, 243 of the 256-expert
// layer 52 against 70, hidden 4096 and width 1536 with 64 tokens 103 against 117 and with 256 522 against 597;
// 64 tokens of the 128-expert layer (0.2 GB) 34 against 33, 50 of the 64-expert layer 38 against 33.
static bool shares_encoder(const Bound& b) {
  const int64_t pairs = static_cast<int64_t>(b.T) * b.L.K;
  return pairs_grouped(b) && !b.L.expert_map && pairs >= 4 * static_cast<int64_t>(b.L.E) &&
         2 * static_cast<int64_t>(b.T) * b.L.F * b.L.H >= 240000000;
}
