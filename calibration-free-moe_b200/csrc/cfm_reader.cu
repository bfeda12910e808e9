// Sparse MoE decode reader for B200 (sm_100a): kernels and C ABI.
//
// One call processes T decode tokens of one MoE layer:
//   prepare  rotate the input (block Hadamard), keep the KEEP largest rotated
//            coordinates per 128-block, make a fixed-point copy of them
//   route    sort each token's K experts ascending, map to local ids
//   screen   exact integer dot products of the 2-bit ternary sketch with the
//            fixed-point rotated input -> projections -> selection scores
//   select   per token the F best scores, ties to the lower candidate index
//   exact    gathered BF16 gate/up rows of the kept channels, phi(g) * u
//   down     gathered channel-major down rows of the kept channels, and in the
//            same launch the low-rank recovery encoder over the skipped ones
//   output   router-weighted mix + decoder term, BF16 store, read-cost counters
//
// Selection depends only on integer dot products and pinned FP32 operations
// (see cfm_device.cuh), so it does not change with batch size, split count or
// launch shape.  No kernel waits on another: cross-CTA reductions use the
// "last CTA to arrive finishes" pattern with an atomic counter and no spin.
#include "cfm_device.cuh"

#include "cfm_b200.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <mutex>

namespace cfm {

// ---------------------------------------------------------------------------
// Workspace binding
// ---------------------------------------------------------------------------
struct Pass;
struct UnionWork;
struct Workspace {
  int32_t* ids;
  float* weights;
  float* norms;
  float* planes;
  int32_t* coordinates;
  int32_t* quantized;
  int32_t* exponents;
  float* parts;
  uint32_t* counters;
  float* partial;
  float* scores;
  uint8_t* selected;
  uint8_t* completed;
  int32_t* candidate_ids;
  int32_t* counts;
  int32_t* starts;
  int32_t* tile_starts;
  __nv_bfloat16* activations;
  __nv_bfloat16* features;
  float* exact;
  float* down_parts;
  float* encoder_parts;
  float* latent;
  int32_t* status;
  int8_t* limbs;
  int32_t* group_offsets;
  int32_t* group_pairs;
  int32_t* cuts;
  float* variances;
  Pass* pass_work;
  int32_t* busy_experts;
  int32_t* work_counts;
  int32_t* tile_list;
  int32_t* tile_count;
  uint32_t* kept_bits;
  uint16_t* kept_before;
  uint16_t* union_channels;
  __nv_bfloat16* union_activations;
  UnionWork* exact_work;
  UnionWork* down_work;
  int32_t parts_tokens;
  int32_t down_tiles;
  int32_t encoder_tiles;
  int32_t capacity;
};

struct Layer {  // device-visible copy of cfm_layer with typed pointers
  int H, I, E, K, F, KEEP, R, activation, score, global_experts, owner, tensor_engine, row_engine;
  int B, N, W;  // blocks, candidates, sketch words per coordinate
  uint32_t width_magic;  // floor(2^32 / I) + 1, or 0 where the multiplication is not exact
  const __nv_bfloat16* gate_up;
  const __nv_bfloat16* down;
  const uint32_t* sketch;
  const uint32_t* sketch_grouped;
  const __half* statistics;
  const float* norms;
  const float* geometry;
  const __nv_bfloat16* encoder;
  const __nv_bfloat16* decoder;
  const int8_t* signs;
  const int32_t* expert_map;
  double* read_work;
  const float* threshold;  // device scalar of the threshold mode, or nullptr
};

// Slot of candidate i, i / I, by multiplication where that is exact for the layer.
__device__ __forceinline__ int slot_of(const Layer& L, int i) {
  return L.width_magic ? static_cast<int>(__umulhi(static_cast<uint32_t>(i), L.width_magic))
                       : i / L.I;
}

static int64_t align256(int64_t v) { return (v + 255) / 256 * 256; }

// 32-bit words of a token's kept candidates as bits; one more, so that two in a row can be read.
__host__ __device__ inline int kept_words(int N) { return (N + 31) / 32 + 1; }

// Most candidates per token (N = K * I) the selection kernels take: their scans pack two
// counts of at most N into the halves of one 32-bit integer.
constexpr int64_t kMaxCandidates = 32767;

static int make_layout(const cfm_layer* l, int32_t capacity, cfm_workspace_layout* o) {
  if (!l || !o) return CFM_E_NULL;
  const int64_t H = l->hidden, I = l->width, K = l->top_k, F = l->final_count;
  const int64_t KEEP = l->keep, R = l->rank, C = capacity;
  if (H <= 0 || H % kBlock || I <= 0 || I % 16 || K <= 0 || K > 32 || KEEP < 1 ||
      KEEP > kBlock || R < 0 || R > 256 || (R % 8) || (R && (256 % R)) || F < 1 ||
      F > K * I || K * I > kMaxCandidates)
    return CFM_E_SHAPE;
  if (C < 1) return CFM_E_CAPACITY;
  const int64_t B = H / kBlock, N = K * I;
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    const int64_t here = at;
    at = align256(at + bytes);
    return here;
  };
  o->parts_tokens = static_cast<int32_t>(C < 16 ? C : 16);
  o->down_tiles = static_cast<int32_t>((F + kDownTileRows - 1) / kDownTileRows + K - 1);
  o->encoder_tiles = static_cast<int32_t>((I + kEncodeTileRows - 1) / kEncodeTileRows);
  o->reserved = 0;
  o->ids = take(4 * C * K);
  o->weights = take(4 * C * K);
  o->norms = take(4 * C * B);
  o->planes = take(4 * C * B * KEEP);
  o->coordinates = take(4 * C * B * KEEP);
  o->quantized = take(4 * C * B * KEEP);
  o->exponents = take(4 * C * B * 2);
  o->parts = take(4 * o->parts_tokens * K * B * 2 * I);
  o->counters = take(4 * (2 * C * K + 2 * C));
  o->partial = take(4 * C * 2 * N);
  o->scores = take(4 * C * N);
  o->selected = take(C * N);
  o->completed = take(C * N);
  o->candidate_ids = take(4 * C * F);
  o->counts = take(4 * C * K);
  o->starts = take(4 * C * K);
  o->tile_starts = take(4 * C * K);
  o->activations = take(2 * C * N);
  o->exact = take(4 * C * 2 * F);
  o->down_parts = take(4 * C * o->down_tiles * H);
  o->encoder_parts = take(4 * C * K * o->encoder_tiles * (R ? R : 1));
  o->latent = take(4 * C * (R ? R : 1));
  o->status = take(16);
  o->limbs = take(C * B * 3 * kBlock);
  o->group_offsets = take(4 * (static_cast<int64_t>(l->experts > 0 ? l->experts : 1) + 1));
  o->group_pairs = take(4 * C * K);
  o->cuts = take(4 * C * (K + 1));
  o->variances = take(4 * C * 2 * N);
  const int64_t E = std::max<int64_t>(l->experts, 1);
  o->features = take(2 * C * N);
  o->pass_work = take(16 * (C * K / 4 + std::min(E, C * K)));  // of at least four pairs
  o->busy_experts = take(4 * E);
  o->work_counts = take(32);
  o->tile_list = take(32 * C * ((F + kDownTileRows - 1) / kDownTileRows + K));
  o->tile_count = take(16);
  o->kept_bits = take(4 * C * kept_words(static_cast<int>(N)));
  o->kept_before = take(2 * C * kept_words(static_cast<int>(N)));
  o->union_channels = take(2 * E * I);
  o->union_activations = take(2 * C * N);
  const int64_t passes = C * K / 8 + std::min(E, C * K);  // of at least eight pairs
  o->exact_work = take(32 * passes * ((I + 31) / 32));  // tiles of 32 channels
  o->down_work = take(32 * passes);
  o->bytes = at;
  return 0;
}

static Workspace bind(const cfm_workspace_layout& o, void* base, int32_t capacity) {
  char* p = static_cast<char*>(base);
  Workspace w;
  w.ids = reinterpret_cast<int32_t*>(p + o.ids);
  w.weights = reinterpret_cast<float*>(p + o.weights);
  w.norms = reinterpret_cast<float*>(p + o.norms);
  w.planes = reinterpret_cast<float*>(p + o.planes);
  w.coordinates = reinterpret_cast<int32_t*>(p + o.coordinates);
  w.quantized = reinterpret_cast<int32_t*>(p + o.quantized);
  w.exponents = reinterpret_cast<int32_t*>(p + o.exponents);
  w.parts = reinterpret_cast<float*>(p + o.parts);
  w.counters = reinterpret_cast<uint32_t*>(p + o.counters);
  w.partial = reinterpret_cast<float*>(p + o.partial);
  w.scores = reinterpret_cast<float*>(p + o.scores);
  w.selected = reinterpret_cast<uint8_t*>(p + o.selected);
  w.completed = reinterpret_cast<uint8_t*>(p + o.completed);
  w.candidate_ids = reinterpret_cast<int32_t*>(p + o.candidate_ids);
  w.counts = reinterpret_cast<int32_t*>(p + o.counts);
  w.starts = reinterpret_cast<int32_t*>(p + o.starts);
  w.tile_starts = reinterpret_cast<int32_t*>(p + o.tile_starts);
  w.activations = reinterpret_cast<__nv_bfloat16*>(p + o.activations);
  w.exact = reinterpret_cast<float*>(p + o.exact);
  w.down_parts = reinterpret_cast<float*>(p + o.down_parts);
  w.encoder_parts = reinterpret_cast<float*>(p + o.encoder_parts);
  w.latent = reinterpret_cast<float*>(p + o.latent);
  w.status = reinterpret_cast<int32_t*>(p + o.status);
  w.limbs = reinterpret_cast<int8_t*>(p + o.limbs);
  w.group_offsets = reinterpret_cast<int32_t*>(p + o.group_offsets);
  w.group_pairs = reinterpret_cast<int32_t*>(p + o.group_pairs);
  w.cuts = reinterpret_cast<int32_t*>(p + o.cuts);
  w.variances = reinterpret_cast<float*>(p + o.variances);
  w.features = reinterpret_cast<__nv_bfloat16*>(p + o.features);
  w.pass_work = reinterpret_cast<Pass*>(p + o.pass_work);
  w.busy_experts = reinterpret_cast<int32_t*>(p + o.busy_experts);
  w.work_counts = reinterpret_cast<int32_t*>(p + o.work_counts);
  w.tile_list = reinterpret_cast<int32_t*>(p + o.tile_list);
  w.tile_count = reinterpret_cast<int32_t*>(p + o.tile_count);
  w.kept_bits = reinterpret_cast<uint32_t*>(p + o.kept_bits);
  w.kept_before = reinterpret_cast<uint16_t*>(p + o.kept_before);
  w.union_channels = reinterpret_cast<uint16_t*>(p + o.union_channels);
  w.union_activations = reinterpret_cast<__nv_bfloat16*>(p + o.union_activations);
  w.exact_work = reinterpret_cast<UnionWork*>(p + o.exact_work);
  w.down_work = reinterpret_cast<UnionWork*>(p + o.down_work);
  w.parts_tokens = o.parts_tokens;
  w.down_tiles = o.down_tiles;
  w.encoder_tiles = o.encoder_tiles;
  w.capacity = capacity;
  return w;
}

static Layer device_layer(const cfm_layer* l) {
  Layer d;
  d.H = l->hidden;
  d.I = l->width;
  d.E = l->experts;
  d.K = l->top_k;
  d.F = l->final_count;
  d.KEEP = l->keep;
  d.R = l->rank;
  d.activation = l->activation;
  d.score = l->score;
  d.global_experts = l->global_experts;
  d.owner = l->recovery_owner;
  d.tensor_engine = l->tensor_engine;
  d.row_engine = l->row_engine;
  d.B = d.H / kBlock;
  d.N = d.K * d.I;
  d.W = 2 * d.I / kWordRows;
  // i / I == umulhi(i, magic) for every candidate i < N as long as N * I <= 2^32.
  const uint64_t width = static_cast<uint64_t>(d.I);
  d.width_magic = static_cast<uint64_t>(d.N) * width <= (1ull << 32)
                      ? static_cast<uint32_t>((1ull << 32) / width + 1) : 0u;
  d.gate_up = static_cast<const __nv_bfloat16*>(l->gate_up);
  d.down = static_cast<const __nv_bfloat16*>(l->down);
  d.sketch = l->sketch;
  d.sketch_grouped = l->sketch_grouped;
  d.statistics = static_cast<const __half*>(l->statistics);
  d.norms = l->norms;
  d.geometry = l->geometry;
  d.encoder = static_cast<const __nv_bfloat16*>(l->encoder);
  d.decoder = static_cast<const __nv_bfloat16*>(l->decoder);
  d.signs = l->signs;
  d.expert_map = l->expert_map;
  d.read_work = l->read_work;
  d.threshold = l->selection_threshold;
  return d;
}

#include "cfm_exchange.cuh"
#include "cfm_prepare.cuh"
#include "cfm_screen.cuh"
#include "cfm_screen_tc.cuh"

// ---------------------------------------------------------------------------
// adopt: a selection made on the token's home rank, cut down to this rank's experts
// ---------------------------------------------------------------------------
// grid (T), 256 threads.  Expert parallelism with a replicated sketch: the home
// rank of a token has chosen its kept channels and sent them as a list of
// candidate ids (slot * I + channel, slots in ascending expert order; ascending,
// -1 after the last).  This rank orders and maps the router's experts exactly as
// k_route does, keeps the entries of the slots it owns in their order, and
// derives the per-slot counts, list starts and down-tile starts for them.
// With `peers` the lists are those the home ranks stored into this rank's exchange
// block; the CTA first waits (bounded) until the lists of its row's home rank have
// landed for the current epoch.
__global__ void __launch_bounds__(256) k_adopt(Layer L, Workspace ws, const void* ids, int ids64,
                                               const void* weights, int wbf16,
                                               const uint8_t* padding, const int32_t* lists,
                                               Exchange x, int peers) {
  __shared__ int route[32];
  __shared__ int count[32];
  __shared__ int warp_total[8];
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool padded = padding && padding[t];
  if (peers) {
    uint32_t* header = exchange_header(x, x.rank);
    if (tid == 0)
      exchange_wait(header + kExchangeListsFlag + t / x.tokens, header[kExchangeEpoch] + 1u,
                    header + kExchangeStatus, 1u);
    lists = reinterpret_cast<const int32_t*>(x.block[x.rank] + exchange_lists_offset());
    __syncthreads();
  }
  if (warp == 0) {
    long long id = 0x7fffffffffffffffLL;
    float w = 0.0f;
    if (lane < L.K) {
      const size_t at = static_cast<size_t>(t) * L.K + lane;
      id = ids64 ? static_cast<const long long*>(ids)[at]
                 : static_cast<long long>(static_cast<const int32_t*>(ids)[at]);
      w = wbf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(weights)[at])
                : static_cast<const float*>(weights)[at];
    }
    int rank = 0;
    for (int j = 0; j < L.K; ++j) {
      const long long o = __shfl_sync(kFull, id, j);
      rank += (o < id) || (o == id && j < lane);
    }
    count[lane] = 0;
    if (lane < L.K) {
      int local = -1;
      if (L.expert_map) {
        if (id >= 0 && id < L.global_experts) local = L.expert_map[id];
      } else if (id >= 0 && id < L.E) {
        local = static_cast<int>(id);
      }
      if (local >= L.E) local = -1;
      const size_t out = static_cast<size_t>(t) * L.K + rank;
      ws.ids[out] = local;
      ws.weights[out] = w;
      route[rank] = padded ? -1 : local;
    }
  }
  __syncthreads();
  const int32_t* in = lists + static_cast<size_t>(t) * L.F;
  int32_t* out = ws.candidate_ids + static_cast<size_t>(t) * L.F;
  int kept = 0;
  for (int base = 0; base < L.F; base += 256) {
    const int i = base + tid;
    const int cid = i < L.F ? __ldcg(in + i) : -1;  // past L1: a peer may have written it
    const int slot = cid >= 0 ? min(cid / L.I, L.K - 1) : 0;
    const bool keep = cid >= 0 && route[slot] >= 0;
    const unsigned ballot = __ballot_sync(kFull, keep);
    if (lane == 0) warp_total[warp] = __popc(ballot);
    __syncthreads();
    int before = kept, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      before += w < warp ? warp_total[w] : 0;
      all += warp_total[w];
    }
    if (keep) {
      out[before + __popc(ballot & ((1u << lane) - 1))] = cid;
      atomicAdd(&count[slot], 1);
    }
    kept += all;
    __syncthreads();
  }
  for (int i = kept + tid; i < L.F; i += 256) out[i] = -1;
  {  // the same channels as bits, with the number of them before every word
    const int words = kept_words(L.N);
    uint32_t* bits = ws.kept_bits + static_cast<size_t>(t) * words;
    for (int w = tid; w < words; w += 256) bits[w] = 0;
    __syncthreads();
    for (int i = tid; i < kept; i += 256) {
      const int w = out[i] >> 5;
      if (i > 0 && out[i - 1] >> 5 == w) continue;  // the word's first entry writes it
      uint32_t word = 0;
      for (int j = i; j < kept && out[j] >> 5 == w; ++j) word |= 1u << (out[j] & 31);
      bits[w] = word;
      ws.kept_before[static_cast<size_t>(t) * words + w] = static_cast<uint16_t>(i);
    }
  }
  if (warp == 0) {
    const bool live = lane < L.K;
    const int mine = live ? count[lane] : 0;
    const int tiles = (mine + kDownTileRows - 1) / kDownTileRows;
    int rows = mine, scan = tiles;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const int r = __shfl_up_sync(kFull, rows, w), o = __shfl_up_sync(kFull, scan, w);
      if (lane >= w) {
        rows += r;
        scan += o;
      }
    }
    if (live) {
      const size_t pair = static_cast<size_t>(t) * L.K + lane;
      ws.counts[pair] = mine;
      ws.starts[pair] = rows - mine;
      ws.tile_starts[pair] = scan - tiles;
    }
  }
}

// ---------------------------------------------------------------------------
// screen of layers without a row-major sketch: sketch GEMV + score
// ---------------------------------------------------------------------------
// grid (T*K pairs, S splits of the rotation blocks), W*CG threads.  Thread
// (cg, wi) owns sketch word wi (16 rows) and the kept coordinates j = cg mod CG
// of each block.  Integer partial dots are summed across coordinate groups in
// shared memory; each thread then finishes 16/CG rows.
template <int CG>
__global__ void __launch_bounds__(512) k_screen(Layer L, Workspace ws, const uint8_t* padding, int S) {
  grid_dependency_wait();     // the kept values and the routes are complete
  grid_dependency_release();  // the selection may be scheduled; it waits for this grid
  constexpr int RPT = kWordRows / CG;  // rows a thread finishes per block
  constexpr int U = 8;                 // words in flight per thread
  extern __shared__ int smem[];
  const int rows = 2 * L.I, W = L.W, threads = W * CG;
  int* sq = smem;              // [128] fixed-point values of the block
  int* sc = sq + kBlock;       // [128] their coordinates
  int* red = sc + kBlock;      // [CG * 16 * W] partial dots (CG > 1)
  __shared__ int s_last;

  const int pair = blockIdx.x, split = blockIdx.y;
  const int t = pair / L.K, slot = pair - t * L.K;
  const int tid = threadIdx.x, wi = tid % W, cg = tid / W;
  const int e = ws.ids[pair];
  if ((padding && padding[t]) || e < 0) {
    if (split == 0) {
      for (int c = tid; c < L.I; c += threads) {
        ws.partial[static_cast<size_t>(t) * 2 * L.N + slot * L.I + c] = 0.0f;
        ws.partial[static_cast<size_t>(t) * 2 * L.N + L.N + slot * L.I + c] = 0.0f;
      }
    }
    return;
  }
  const int per = (L.B + S - 1) / S;
  const int b0 = split * per, b1 = min(L.B, b0 + per);
  float run[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) run[r] = 0.0f;
  const int row0 = wi * kWordRows + cg * RPT;  // first row this thread finishes

  for (int b = b0; b < b1; ++b) {
    const size_t tb = static_cast<size_t>(t) * L.B + b;
    __syncthreads();
    for (int j = tid; j < L.KEEP; j += threads) {
      sq[j] = ws.quantized[tb * L.KEEP + j];
      sc[j] = ws.coordinates[tb * L.KEEP + j];
    }
    // Scales of the rows this thread finishes, fetched ahead of the dots.
    float scale[RPT];
    {
      const __half* st = L.statistics +
                         (static_cast<size_t>(e) * L.B + b) * 2 * rows + row0;
#pragma unroll
      for (int r = 0; r < RPT; ++r) scale[r] = __half2float(st[r]);
    }
    const int be = ws.exponents[2 * tb], qsum = ws.exponents[2 * tb + 1];
    __syncthreads();

    int acc[kWordRows];
#pragma unroll
    for (int j = 0; j < kWordRows; ++j) acc[j] = 0;
    const uint32_t* base =
        L.sketch + (static_cast<size_t>(e) * L.H + static_cast<size_t>(b) * kBlock) * W + wi;
    for (int j0 = cg; j0 < L.KEEP; j0 += CG * U) {
      uint32_t word[U];
      int q[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + u * CG;
        if (j < L.KEEP) {
          word[u] = load_stream4(base + static_cast<size_t>(sc[j]) * W);
          q[u] = sq[j];
        } else {
          word[u] = 0;
          q[u] = 0;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int j = 0; j < kWordRows; ++j)
          acc[j] += static_cast<int>((word[u] >> (2 * j)) & 3u) * q[u];
      }
    }
    int dot[RPT];
    if (CG > 1) {
#pragma unroll
      for (int j = 0; j < kWordRows; ++j) red[(cg * kWordRows + j) * W + wi] = acc[j];
      __syncthreads();
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        int s = 0;
#pragma unroll
        for (int g = 0; g < CG; ++g) s += red[(g * kWordRows + cg * RPT + r) * W + wi];
        dot[r] = s;
      }
    } else {
#pragma unroll
      for (int r = 0; r < RPT; ++r) dot[r] = acc[r];
    }
    // code = trit + 1, so sum(trit * q) = sum(code * q) - sum(q).
    const float unscale = __uint_as_float(static_cast<uint32_t>(127 + be - kQuantBits) << 23);
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const float d = __fmul_rn(__int2float_rn(dot[r] - qsum), unscale);
      const float prod = __fmul_rn(scale[r], d);
      if (S == 1) {
        run[r] = __fadd_rn(run[r], prod);
      } else {
        ws.parts[(static_cast<size_t>(pair) * L.B + b) * rows + row0 + r] = prod;
      }
    }
  }

  float* gate_out = ws.partial + static_cast<size_t>(t) * 2 * L.N + static_cast<size_t>(slot) * L.I;
  float* up_out = gate_out + L.N;
  // Scores and features of the pair, once the CTA's threads have written its projections (the
  // library-scratch screen has no place for them).
  auto finish = [&]() {
    if (!ws.scores) return;
    __syncthreads();
    const float* variance = ws.variances + static_cast<size_t>(t) * 2 * L.N +
                            static_cast<size_t>(slot) * L.I;
    const bool risk = L.score != CFM_SCORE_POINT;
    for (int c = tid; c < L.I; c += threads)
      finish_candidate(L, ws, pair, c, candidate_factors(L, e, c), gate_out[c], up_out[c],
                       risk ? variance[c] : 0.0f, risk ? variance[L.N + c] : 0.0f);
  };
  if (S == 1) {
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int row = row0 + r;
      (row < L.I ? gate_out[row] : up_out[row - L.I]) = run[r];
    }
    finish();
    return;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned old = atomicAdd(&ws.counters[pair], 1u);
    s_last = (old == static_cast<unsigned>(S - 1));
    if (s_last) ws.counters[pair] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // The last split to arrive sums the per-block products in block order.
  for (int row = tid; row < rows; row += threads) {
    float s = 0.0f;
    const float* p = ws.parts + static_cast<size_t>(pair) * L.B * rows + row;
    for (int b = 0; b < L.B; ++b) s = __fadd_rn(s, __ldcg(p + static_cast<size_t>(b) * rows));
    (row < L.I ? gate_out[row] : up_out[row - L.I]) = s;
  }
  finish();
}

#include "cfm_build.cuh"

// grid (T, ceil(N / 256)), 256 threads: zero the scores of remote or padded slots (used when the
// scores are exchanged between ranks before selection; the screen has written the others).
__global__ void k_score(Layer L, Workspace ws, const uint8_t* padding) {
  const int t = blockIdx.x, i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= L.N) return;
  const int slot = i / L.I;
  if ((padding && padding[t]) || ws.ids[static_cast<size_t>(t) * L.K + slot] < 0)
    ws.scores[static_cast<size_t>(t) * L.N + i] = 0.0f;
}

// Residual variance of every candidate's sketch projections (recovery-aware
// score): sum over blocks, in block order, of the row's FP16 residual variance
// times the energy of the token's kept coordinates in that block.
// grid (T*K pairs, ceil(2I / 256)), 256 threads, one sketch row per thread.
__global__ void __launch_bounds__(256) k_variance(Layer L, Workspace ws, const uint8_t* padding) {
  const int pair = blockIdx.x, row = blockIdx.y * 256 + threadIdx.x;
  const int rows = 2 * L.I;
  if (row >= rows) return;
  const int t = pair / L.K, slot = pair - t * L.K;
  const int e = ws.ids[pair];
  float sum = 0.0f;
  if (e >= 0 && !(padding && padding[t])) {
    const __half* variance = L.statistics + (static_cast<size_t>(e) * L.B * 2 + 1) * rows + row;
    const float* energy = ws.norms + static_cast<size_t>(t) * L.B;
    for (int b = 0; b < L.B; ++b)
      sum = __fadd_rn(sum, __fmul_rn(__half2float(variance[static_cast<size_t>(b) * 2 * rows]),
                                     energy[b]));
  }
  float* out = ws.variances + static_cast<size_t>(t) * 2 * L.N + static_cast<size_t>(slot) * L.I;
  (row < L.I ? out[row] : out[L.N + row - L.I]) = sum;
}

// ---------------------------------------------------------------------------
// select: top-F per token, read-cost counters
// ---------------------------------------------------------------------------
constexpr int kSelectThreads = 1024;

#include "cfm_select.cuh"

__device__ __forceinline__ int64_t sector_run(int64_t bytes) { return (bytes + 31) / 32 * 32; }

// Read-cost counters of one token (integers, so FP64 atomics are exact): lane
// `lane` of one warp adds slot `lane` of `read_work`.  `local_slots` of the
// token's experts are held here and `kept_local` of its kept channels are theirs.
__device__ __forceinline__ void account_reads(const Layer& L, int lane, int local_slots,
                                              int kept_local, bool screened) {
  const int I = L.I, K = L.K;
  if (L.read_work && lane < CFM_READ_WORK_SLOTS) {
    const bool ep = L.expert_map != nullptr;
    const int64_t H = L.H, R = L.R;
    const int64_t candidates = static_cast<int64_t>(local_slots) * I;
    const int64_t native = 2 * (2 * kept_local * H + kept_local * H);
    const int64_t dense_slot = 6 * static_cast<int64_t>(I) * H;
    const int64_t reference = ep ? local_slots * dense_slot : K * dense_slot;
    const int64_t recovery = 2 * R * (candidates - kept_local + (L.owner ? H : 0));
    const bool residual = L.score != CFM_SCORE_POINT;
    const int64_t code = 2 * ((I + 4) / 5), plane = 4 * I;
    const int64_t sketch_exact =
        screened ? local_slots * L.B * (L.KEEP * code + plane * (1 + residual)) : 0;
    const int64_t sketch_sector =
        screened ? local_slots * L.B *
                       (L.KEEP * sector_run(code) + sector_run(plane) * (1 + residual))
                 : 0;
    // Bytes the screen kernel itself requests: 2-bit codes (I / 2 bytes per
    // kept coordinate) and the FP16 scale plane.
    const int64_t sketch_issued =
        screened ? local_slots * L.B * (static_cast<int64_t>(L.KEEP) * (I / 2) + plane) : 0;
    const int64_t selection =
        screened ? ((L.geometry ? 12 : 4) * candidates) : 0;
    // Threshold mode: every token also reads the FP32 layer threshold (one sector).
    const int64_t threshold_exact = L.threshold ? 4 : 0, threshold_sector = L.threshold ? 32 : 0;
    int64_t value = 0;
    switch (lane) {
      case 0: case 6: value = native; break;
      case 1: value = reference; break;
      case 3: case 7: value = recovery; break;
      case 4: value = selection + threshold_exact; break;
      case 9: value = selection + threshold_sector; break;
      case 19: value = L.threshold ? 1 : 0; break;
      case 5: value = sketch_exact; break;
      case 10: value = screened ? H : 0; break;
      case 11: value = sketch_issued; break;
      case 17: value = sketch_sector; break;
      case 12: value = 4 * H * kept_local; break;
      case 13: value = 2 * H * kept_local; break;
      case 14: value = 2 * R * (candidates - kept_local); break;
      default: value = 0;
  }
    if (value) atomicAdd(L.read_work + lane, static_cast<double>(value));
  }
}

// The same from one slot per lane: whether it is held here and how many channels it kept.
__device__ __forceinline__ void account_token(const Layer& L, int lane, bool local, int count,
                                              bool screened) {
  const int local_slots = __popc(__ballot_sync(kFull, local));
  const int kept_local = __reduce_add_sync(kFull, local ? count : 0);
  account_reads(L, lane, local_slots, kept_local, screened);
}

// Sums over the warps before this one and over all of them of a warp-uniform value; `slots` holds
// 32 values; one barrier.
__device__ __forceinline__ uint2 warp_prefix(uint32_t mine, uint32_t* slots) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) slots[warp] = mine;
  __syncthreads();
  const uint32_t v = slots[lane];
  return make_uint2(__reduce_add_sync(kFull, lane < warp ? v : 0u), __reduce_add_sync(kFull, v));
}

constexpr int kSelectListed = 256;  // keys that one warp finishes the search among
// Bins of keys by their upper thirteen bits but the sign, which scores do not have (keys with it share
// the last bin).
constexpr int kSelectBins = 8192, kSelectShift = 18;
__device__ __forceinline__ uint32_t select_bin(uint32_t key) {
  return min(key >> kSelectShift, static_cast<uint32_t>(kSelectBins - 1));
}

// grid (T), 1024 threads, up to PER keys each in registers: candidate 32 (PER warp + j) + lane.
// The F-th largest key is found by its bin first: 8192 counters in shared memory, one addition per key
// (equal addresses of a warp are added by the hardware), and a sum over them from the top.  The few
// keys of its bin (some ten of 6144) are listed and one warp compares each with each; bins with more go
// on two bits or one bit at a time.  Then ballots give every warp its keys' places in candidate order.
// Bound by the latency of one CTA per token, most of it code and data that are met for the first time:
// what only ties, remote slots or budgets need is branched around, and the read-cost counters are left
// to the output kernel where one follows (`account`).  One token of 6144 candidates 5.2 us with its
// launch, of 8192 5.6, 32 tokens of 12288 7.2, 256 of them 16.4; by bits from the top, three counts of
// the whole CTA per two bits, with stores of single bytes and entries, 8.8, 11.3, 17.3 and 31.8.
// With `peers` (expert parallelism over peer memory; row_offset 0, T = x.tokens) a
// CTA ends by storing its token's kept list into slot [rank] of every rank's exchange
// block; the last CTA to arrive releases each destination's flag with the call's epoch.
// Without PEERS the exchange argument is a dummy, so that the single-GPU kernel carries
// neither the parameter block nor the code of the hand-over.
struct NoExchange {
  int world, rank, tokens;
  char* block[1];
};
template <bool PEERS, int PER>
__global__ void __launch_bounds__(kSelectThreads, PER <= 4 ? 2 : 1)
    k_select(Layer L, Workspace ws, const uint8_t* padding, int scores_ready, int row_offset, int account,
             int clear, typename std::conditional<PEERS, Exchange, NoExchange>::type x) {
  constexpr bool peers = PEERS;
  grid_dependency_release();  // the exact gather may be scheduled; it waits for this grid
  __shared__ __align__(16) uint32_t s_bins[kSelectBins];
  __shared__ uint2 s_counts[2][32];
  __shared__ uint32_t s_slots[3][32], s_listed[kSelectListed];
  __shared__ uint32_t s_cut;
  __shared__ int s_take, s_count, s_bin, s_above, s_inside;
  __shared__ int s_route[32], s_tie_start[33], s_budget[32];
  __shared__ uint32_t s_chunk[32 * PER];   // kept candidates of every 32, as bits
  __shared__ uint16_t s_before[32 * PER];  // kept candidates before them
  const int t = blockIdx.x + row_offset, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = L.N, F = L.F, K = L.K, I = L.I;
  constexpr int kOwnBins = kSelectBins / kSelectThreads;
#pragma unroll
  for (int j = 0; j < kOwnBins; j += 4)
    *reinterpret_cast<uint4*>(s_bins + 4 * tid + 4 * kSelectThreads * (j / 4)) = make_uint4(0, 0, 0, 0);
  if (tid == 0) s_count = s_inside = 0;
  grid_dependency_wait();  // the screen's projections are complete
  const bool cut_given = scores_ready == 2, cut_only = scores_ready == 3;
  int32_t* counts = ws.counts + static_cast<size_t>(t) * K;
  int32_t* starts = ws.starts + static_cast<size_t>(t) * K;
  int32_t* tile_starts = ws.tile_starts + static_cast<size_t>(t) * K;
  // All threads of the CTA call this once the token's list is complete (or has
  // nothing to say: a padding row, whose list the owners ignore).
  auto publish = [&](bool send) {
    if constexpr (PEERS) {
    __syncthreads();  // the list is complete in global memory for this CTA's threads
    uint32_t* header = exchange_header(x, x.rank);
    const uint32_t epoch = header[kExchangeEpoch] + 1u;
    if (send) {
      const int32_t* mine = ws.candidate_ids + static_cast<size_t>(t) * F;
      const size_t at = (static_cast<size_t>(x.rank) * x.tokens + t) * F;
      if (F % 4 == 0) {
        const int quads = F / 4;
        for (int j = tid; j < x.world * quads; j += kSelectThreads) {
          const int d = j / quads, i = j - d * quads;
          int4* out = reinterpret_cast<int4*>(
              reinterpret_cast<int32_t*>(x.block[d] + exchange_lists_offset()) + at);
          out[i] = reinterpret_cast<const int4*>(mine)[i];
        }
      } else {
        for (int j = tid; j < x.world * F; j += kSelectThreads) {
          const int d = j / F, i = j - d * F;
          (reinterpret_cast<int32_t*>(x.block[d] + exchange_lists_offset()) + at)[i] = mine[i];
        }
      }
    }
    // The CTA barrier orders every thread's stores before the fences of the few threads
    // that announce; a system-scope fence is cumulative.
    __syncthreads();
    if (tid < x.world) {
      __threadfence_system();
      uint32_t* counter = header + kExchangeListsArrive + tid;
      if (atomicAdd(counter, 1u) == gridDim.x - 1) {
        *counter = 0;
        __threadfence_system();
        store_release_system(exchange_header(x, tid) + kExchangeListsFlag + x.rank, epoch);
      }
    }
    }
  };
  if (padding && padding[t]) {
    if (tid < K) counts[tid] = starts[tid] = tile_starts[tid] = 0;
    if (tid <= K) ws.cuts[static_cast<size_t>(t) * (K + 1) + tid] = 0;
    if (peers) publish(false);
    return;
  }
  const bool screened = F < N;
  if (tid < 32) {
    s_route[tid] = tid < K ? ws.ids[static_cast<size_t>(t) * K + tid] : -1;
  }
  const int first = 32 * PER * warp + lane;  // this thread's candidates: first, first + 32, ...
  float* score = ws.scores + static_cast<size_t>(t) * N;
  uint32_t key[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int i = first + 32 * j;
    key[j] = screened && i < N ? __float_as_uint(score[i]) : 0u;
  }
  __syncthreads();
  const bool remote = __any_sync(kFull, lane < K && s_route[lane] < 0);
  if (screened && !scores_ready && remote) {
#pragma unroll
    for (int j = 0; j < PER; ++j) {  // the screen's scores; zero for remote slots
      const int i = first + 32 * j;
      if (i < N && s_route[slot_of(L, i)] < 0) {
        key[j] = 0u;
        score[i] = 0.0f;
      }
    }
  }
  uint32_t cut = 0;
  int take_ties = 0;
  if (screened && !cut_given) {
    // The bin of the F-th largest key: the thread whose bins, from the top, take the count past F.
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (first + 32 * j < N && key[j]) atomicAdd(&s_bins[select_bin(key[j])], 1u);
    __syncthreads();
    uint32_t own[kOwnBins], sum = 0;  // counts, from the top
#pragma unroll
    for (int j = 0; j < kOwnBins; j += 4) {
      const uint4 four = *reinterpret_cast<const uint4*>(s_bins + kSelectBins - kOwnBins * (tid + 1) + kOwnBins - 4 - j);
      own[j] = four.w;
      own[j + 1] = four.z;
      own[j + 2] = four.y;
      own[j + 3] = four.x;
      sum += (four.x + four.y) + (four.z + four.w);
    }
    uint32_t scan = sum;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const uint32_t o = __shfl_up_sync(kFull, scan, w);
      if (lane >= w) scan += o;
    }
    const uint2 totals = warp_prefix(__shfl_sync(kFull, scan, 31), s_slots[2]);
    uint32_t upto = totals.x + scan - sum;  // keys in higher bins
    if (upto < static_cast<uint32_t>(F) && upto + sum >= static_cast<uint32_t>(F)) {
#pragma unroll
      for (int j = 0; j < kOwnBins; ++j) {
        if (upto < static_cast<uint32_t>(F) && upto + own[j] >= static_cast<uint32_t>(F)) {
          s_bin = kSelectBins - 1 - kOwnBins * tid - j;
          s_above = upto;
          s_inside = own[j];
        }
        upto += own[j];
      }
    }
    __syncthreads();
    int above = s_above, reached = above + s_inside;  // keys beyond the bounds, keys from `cut` up
    int shift = kSelectShift;
    bool found = false;
    if (s_inside == 0) {  // fewer than F keys differ from zero: zeros tie for the rest
      above = totals.y;
      shift = 0;
    } else {
      cut = static_cast<uint32_t>(s_bin) << kSelectShift;
      if (reached == F) {  // exactly the keys from the cut up, none of them zero
        cut = max(cut, 1u) - 1u;
        found = true;
      } else if (s_bin == kSelectBins - 1 || s_inside > kSelectListed) {
        if (s_bin == kSelectBins - 1) {  // whatever has its sign
          cut = 0;
          above = 0;
          reached = N;
          shift = 32;
        }
        // Two bits per step: three counts of the whole CTA, one barrier.
        for (int step = 0; shift > 0; ++step) {
          shift -= 2;
          uint32_t low = 0, high = 0;  // counts from one and two steps up, from three steps up
#pragma unroll
          for (int j = 0; j < PER; ++j) {
            low += (key[j] >= (cut | (1u << shift)) ? 1u : 0u) + (key[j] >= (cut | (2u << shift)) ? 0x10000u : 0u);
            high += key[j] >= (cut | (3u << shift)) ? 1u : 0u;
          }
          low = __reduce_add_sync(kFull, low);
          high = __reduce_add_sync(kFull, high);
          if (lane == 0) s_counts[step & 1][warp] = make_uint2(low, high);
          __syncthreads();
          const uint2 c = s_counts[step & 1][lane];
          low = __reduce_add_sync(kFull, c.x);
          const int c3 = __reduce_add_sync(kFull, c.y), c2 = low >> 16, c1 = low & 0xffff;
          if (c3 >= F) {
            cut |= 3u << shift;
            reached = c3;
          } else if (c2 >= F) {
            cut |= 2u << shift;
            reached = c2;
            above = c3;
          } else if (c1 >= F) {
            cut |= 1u << shift;
            reached = c1;
            above = c2;
          } else {
            above = c1;
          }
          if (reached == F) {  // exactly the keys from the cut up
            cut -= 1;
            found = true;
            break;
          }
          if (shift > 0 && reached - above <= kSelectListed) break;
        }
      }
    }
    if (!found && shift <= 0) {
      take_ties = F - above;  // the cut is the F-th largest key
    } else if (!found) {
      const uint32_t low = max(cut, 1u), top = cut + ((1u << shift) - 1);  // bounds; the cut is no zero
      int inside = 0;
#pragma unroll
      for (int j = 0; j < PER; ++j)
        inside += key[j] >= low && key[j] <= top;
      if (inside) {  // any order will do
        int at = atomicAdd(&s_count, inside);
#pragma unroll
        for (int j = 0; j < PER; ++j)
          if (key[j] >= low && key[j] <= top) s_listed[at++] = key[j];
      }
      __syncthreads();
      if (warp == 0) {
        const int listed = s_count, wanted = F - above;
        if (listed <= 32) {
          // Every key against every other: the one that `wanted` keys reach is the cut.
          const uint32_t own_key = lane < listed ? s_listed[lane] : 0u;
          int more = 0, same = 0;
          for (int i = 0; i < listed; ++i) {
            const uint32_t other = s_listed[i];
            more += other > own_key;
            same += other == own_key;
          }
          if (more < wanted && more + same >= wanted) {  // one lane, or several with the same key
            const bool all = more + same == wanted;
            s_cut = all ? own_key - 1 : own_key;
            s_take = all ? 0 : wanted - more;
          }
        } else {
          uint32_t k[kSelectListed / 32];
#pragma unroll
          for (int j = 0; j < kSelectListed / 32; ++j) k[j] = 32 * j + lane < listed ? s_listed[32 * j + lane] : 0u;
          auto count_from = [&](uint32_t bound) {
            int n = 0;
#pragma unroll
            for (int j = 0; j < kSelectListed / 32; ++j) n += k[j] >= bound;
            return __reduce_add_sync(kFull, n);
          };
          for (int bit = shift - 1; bit >= 0 && !found; --bit) {
            const uint32_t trial = cut | (1u << bit);
            const int n = count_from(trial);
            if (n >= wanted) cut = trial;
            found = n == wanted;
          }
          const int ties = found ? 0 : wanted - count_from(cut + 1);
          if (lane == 0) {
            s_cut = found ? cut - 1 : cut;
            s_take = ties;
          }
        }
      }
      __syncthreads();
      cut = s_cut;
      take_ties = s_take;
    }
    if (L.threshold) {
      // Threshold mode: every score at or above the layer threshold, at most F (best first).
      // When fewer than F reach it, the cut moves up to just below the threshold's key and no
      // tie budget is needed.
      const uint32_t floor_key = __float_as_uint(__fadd_rn(*L.threshold, 0.0f));
      if (cut < floor_key) {
        cut = floor_key - 1u;
        take_ties = 0;
      }
    }
  }

  // Ties at the cut are kept in candidate order; that rule is applied slot by slot with a
  // per-slot tie budget, so that a rank holding only some of a token's slots can
  // repeat the selection from the cut and the budgets alone.
  int32_t* cuts = ws.cuts + static_cast<size_t>(t) * (K + 1);
  if (cut_given) cut = static_cast<uint32_t>(cuts[0]);
  const bool budgets = cut_given || cut_only;
  const unsigned before = (1u << lane) - 1;
  const bool tied_keys = screened && (budgets || take_ties > 0);
  uint32_t mine = 0;
  uint2 ties = make_uint2(0, 0);  // before this warp, in all
  if (tied_keys) {
#pragma unroll
    for (int j = 0; j < PER; ++j)
      mine += __popc(__ballot_sync(kFull, first + 32 * j < N && key[j] == cut));
    ties = warp_prefix(mine, s_slots[0]);
  }
  if (budgets) {
    uint32_t running = ties.x;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = first + 32 * j, slot = slot_of(L, min(i, N - 1));
      const unsigned tied = __ballot_sync(kFull, screened && i < N && key[j] == cut);
      if (i < N && i == slot * I) s_tie_start[slot] = running + __popc(tied & before);
      running += __popc(tied);
    }
    if (tid == 0) s_tie_start[K] = ties.y;
    __syncthreads();
    if (tid < K) {
      int budget;
      if (cut_given) {
        budget = cuts[1 + tid];
      } else {
        const int in_slot = s_tie_start[tid + 1] - s_tie_start[tid];
        budget = max(0, min(in_slot, take_ties - s_tie_start[tid]));
        cuts[1 + tid] = budget;
        if (tid == 0) cuts[0] = static_cast<int32_t>(cut);
      }
      s_budget[tid] = budget;
    }
    if (cut_only) return;  // the token's home rank only publishes the cut and the budgets
    __syncthreads();
  }
  uint32_t kept = 0;  // bit j: this thread keeps its candidate j
#pragma unroll
  for (int j = 0; j < PER; ++j)
    kept |= static_cast<uint32_t>(screened ? key[j] > cut : first + 32 * j < N) << j;
  if (tied_keys) {
    uint32_t running = ties.x;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int i = first + 32 * j;
      const bool tie = i < N && key[j] == cut;
      const unsigned tied = __ballot_sync(kFull, tie);
      const int tie_index = running + __popc(tied & before);
      running += __popc(tied);
      if (tie) {
        const int slot = slot_of(L, i);
        const bool keep = budgets ? tie_index - s_tie_start[slot] < s_budget[slot] : tie_index < take_ties;
        kept |= static_cast<uint32_t>(keep) << j;
      }
    }
  }
  if (cut_given && remote) {  // other ranks' slots
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (first + 32 * j < N && s_route[slot_of(L, first + 32 * j)] < 0) kept &= ~(1u << j);
  }
  // Lane j of a warp goes on with the mask of its candidates 32 j ..: the masks' places, then masks,
  // lists and bytes by as many threads as there are words of each.  (Byte and entry at a time from the
  // candidates' threads, stores took half of the kernel's time.)
  uint32_t word = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const uint32_t ballot = __ballot_sync(kFull, (kept >> j) & 1u);
    if (lane == j) word = ballot;
  }
  uint32_t scan = __popc(word);
#pragma unroll
  for (int w = 1; w < PER; w <<= 1) {
    const uint32_t o = __shfl_up_sync(kFull, scan, w);
    if (lane >= w) scan += o;
  }
  const uint2 kept_counts = warp_prefix(__shfl_sync(kFull, scan, PER - 1), s_slots[1]);
  const int total_kept = kept_counts.y;
  if (lane < PER) {
    s_chunk[warp * PER + lane] = word;
    s_before[warp * PER + lane] = static_cast<uint16_t>(kept_counts.x + scan - __popc(word));
  }
  __syncthreads();
  int32_t* list = ws.candidate_ids + static_cast<size_t>(t) * F;
  if (32 * tid < N) {
    uint32_t bits = s_chunk[tid];
    int at = s_before[tid];
    ws.kept_bits[static_cast<size_t>(t) * kept_words(N) + tid] = bits;
    ws.kept_before[static_cast<size_t>(t) * kept_words(N) + tid] = static_cast<uint16_t>(at);
    for (; bits; bits &= bits - 1, ++at) {
      const int i = 32 * tid + __ffs(bits) - 1;
      list[at] = i;
      if (clear) ws.features[static_cast<size_t>(t) * N + i] = __float2bfloat16_rn(0.0f);
    }
  }
  for (int i = total_kept + tid; i < F; i += kSelectThreads) list[i] = -1;
  // Sixteen candidates' bytes at a time, from the last thread on: N = K I is a multiple of sixteen, and
  // a slot's first candidate too.
  for (int i = 16 * (kSelectThreads - 1 - tid); i < N; i += 16 * kSelectThreads) {
    const uint32_t bits = s_chunk[i >> 5] >> (i & 16);
    auto bytes = [&](int from) {  // four bits to four bytes
      return (((bits >> from) & 15u) * 0x00204081u) & 0x01010101u;
    };
    const uint4 four = make_uint4(bytes(0), bytes(4), bytes(8), bytes(12));
    *reinterpret_cast<uint4*>(ws.selected + static_cast<size_t>(t) * N + i) = four;
    *reinterpret_cast<uint4*>(ws.completed + static_cast<size_t>(t) * N + i) =
        !remote || s_route[slot_of(L, i)] >= 0 ? four : make_uint4(0, 0, 0, 0);
  }
  if (warp == 0) {
    const bool live = lane < K;
    const int from = min(lane, K) * I, chunk = from / 32;  // the slot's first candidate
    int start = total_kept;
    if (lane < K) start = s_before[chunk] + __popc(s_chunk[chunk] & ((1u << (from & 31)) - 1));
    const int next = __shfl_down_sync(kFull, start, 1);
    const int count = live ? (lane == 31 || lane + 1 >= K ? total_kept : next) - start : 0;
    const bool local = live && s_route[lane] >= 0;
    const int tiles = local ? (count + kDownTileRows - 1) / kDownTileRows : 0;
    int scan = tiles;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const int o = __shfl_up_sync(kFull, scan, w);
      if (lane >= w) scan += o;
    }
    if (live) {
      counts[lane] = count;
      starts[lane] = start;
      tile_starts[lane] = scan - tiles;
    }
    if (account) account_token(L, lane, local, count, screened);
  }
  if (peers) publish(true);
}

// ---------------------------------------------------------------------------
// exact: gathered gate/up rows
// ---------------------------------------------------------------------------
constexpr int kExactWarps = 4;

// One warp's dot products of a gate row and an up row with the input staged in
// shared memory (`xs`, `chunks` 16-byte pieces): eight pieces of each row in
// flight per lane (2048 columns per sweep), FP32 FMAs in a fixed order, then a
// butterfly over the lanes.  Every lane returns the sums.  The loads of a sweep and
// the arithmetic on them are separate steps, so that a kernel can issue a row's
// first sweep before the barrier that publishes `xs`.
constexpr int kExactSweep = 8;  // 16-byte pieces of each row per lane and sweep

__device__ __forceinline__ void exact_load(const uint4* gate, const uint4* up, int base, int chunks,
                                           uint4 (&gw)[kExactSweep], uint4 (&uw)[kExactSweep]) {
  if (base + 32 * (kExactSweep - 1) < chunks) {
#pragma unroll
    for (int k = 0; k < kExactSweep; ++k) {
      gw[k] = load_stream16(gate + base + 32 * k);
      uw[k] = load_stream16(up + base + 32 * k);
    }
  } else {
#pragma unroll
    for (int k = 0; k < kExactSweep; ++k) {
      const int i = base + 32 * k;
      gw[k] = uw[k] = make_uint4(0, 0, 0, 0);
      if (i < chunks) {
        gw[k] = load_stream16(gate + i);
        uw[k] = load_stream16(up + i);
      }
    }
  }
}

__device__ __forceinline__ void exact_consume(const uint4 (&gw)[kExactSweep],
                                              const uint4 (&uw)[kExactSweep], const uint4* xs,
                                              int base, int chunks, float& g, float& u) {
#pragma unroll
  for (int k = 0; k < kExactSweep; ++k) {
    const int i = min(base + 32 * k, chunks - 1);
    const uint4 xw = xs[i];
    g = fmaf(bf16_lo(gw[k].x), bf16_lo(xw.x), g);
    g = fmaf(bf16_hi(gw[k].x), bf16_hi(xw.x), g);
    g = fmaf(bf16_lo(gw[k].y), bf16_lo(xw.y), g);
    g = fmaf(bf16_hi(gw[k].y), bf16_hi(xw.y), g);
    g = fmaf(bf16_lo(gw[k].z), bf16_lo(xw.z), g);
    g = fmaf(bf16_hi(gw[k].z), bf16_hi(xw.z), g);
    g = fmaf(bf16_lo(gw[k].w), bf16_lo(xw.w), g);
    g = fmaf(bf16_hi(gw[k].w), bf16_hi(xw.w), g);
    u = fmaf(bf16_lo(uw[k].x), bf16_lo(xw.x), u);
    u = fmaf(bf16_hi(uw[k].x), bf16_hi(xw.x), u);
    u = fmaf(bf16_lo(uw[k].y), bf16_lo(xw.y), u);
    u = fmaf(bf16_hi(uw[k].y), bf16_hi(xw.y), u);
    u = fmaf(bf16_lo(uw[k].z), bf16_lo(xw.z), u);
    u = fmaf(bf16_hi(uw[k].z), bf16_hi(xw.z), u);
    u = fmaf(bf16_lo(uw[k].w), bf16_lo(xw.w), u);
    u = fmaf(bf16_hi(uw[k].w), bf16_hi(xw.w), u);
  }
}

// The rest of a row pair whose first sweep (`gw`, `uw`) is loaded already when
// `loaded`, else the whole pair; same order of operations either way.
__device__ __forceinline__ void exact_dot(const uint4* gate, const uint4* up, const uint4* xs,
                                          int chunks, int lane, bool loaded,
                                          uint4 (&gw)[kExactSweep], uint4 (&uw)[kExactSweep],
                                          float& g_out, float& u_out) {
  float g = 0.0f, u = 0.0f;
  for (int base = lane; base < chunks; base += 32 * kExactSweep) {
    if (!(loaded && base == lane)) exact_load(gate, up, base, chunks, gw, uw);
    exact_consume(gw, uw, xs, base, chunks, g, u);
  }
#pragma unroll
  for (int w = 16; w; w >>= 1) {
    g += __shfl_xor_sync(kFull, g, w);
    u += __shfl_xor_sync(kFull, u, w);
  }
  g_out = g;
  u_out = u;
}

// grid (ceil(F / 4), T), 128 threads; one warp per kept candidate.  With `list` one more CTA row, the
// first, lists the down tiles meanwhile.  Five CTAs per SM, at the price of two registers spilled: whole calls of
// 10 tokens of the 128-expert layer 59.7 us against 60.6 with four, of the 64-expert layer 69.3 against 69.4, of 100 experts of
// hidden 2816 53.8 against 55.4; up to 7 tokens the same within 0.5 us, four or five.
__global__ void __launch_bounds__(kExactWarps * 32, 5) k_exact(Layer L, Workspace ws,
                                                            const __nv_bfloat16* hidden,
                                                            const uint8_t* padding, int list_tiles) {
  grid_dependency_wait();     // the selection is complete
  grid_dependency_release();  // the down kernel may be scheduled: its encoder needs no more than that
  extern __shared__ uint4 xs[];  // H bf16 values of the token
  if (list_tiles && blockIdx.y == 0) {
    if (blockIdx.x == 0) list_down_tiles(L, ws, reinterpret_cast<int*>(xs));
    return;
  }
  const int t = blockIdx.y - list_tiles, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (padding && padding[t]) return;
  const int32_t* list = ws.candidate_ids + static_cast<size_t>(t) * L.F;
  const bool strided = gridDim.x * kExactWarps < L.F;  // CTAs walk the list in strides
  if (L.expert_map) {
    // Expert parallel: leave before staging the input when this CTA has nothing
    // to do.  A list cut down to the local slots ends with -1 entries; a full list
    // is probed for candidates of local experts.
    if (list[blockIdx.x * kExactWarps] < 0) return;
    if (!strided) {
      const int probe = blockIdx.x * kExactWarps + warp;
      bool mine = false;
      if (probe < L.F) {
        const int cid = list[probe];
        mine = cid >= 0 && ws.ids[static_cast<size_t>(t) * L.K + cid / L.I] >= 0;
      }
      if (!__syncthreads_or(mine)) return;
    }
  }
  const int chunks = L.H / 8;
  const size_t up_offset = static_cast<size_t>(L.I) * L.H / 8;
  // The rows of a candidate of a local expert, or null.
  auto rows_of = [&](int index) -> const uint4* {
    if (index >= L.F) return nullptr;
    const int cid = list[index];
    if (cid < 0) return nullptr;
    const int slot = cid / L.I, c = cid - slot * L.I;
    const int e = ws.ids[static_cast<size_t>(t) * L.K + slot];
    if (e < 0) return nullptr;
    return reinterpret_cast<const uint4*>(L.gate_up + (static_cast<size_t>(e) * 2 * L.I + c) * L.H);
  };
  // The first row pair's first sweep is on its way while the input row is staged.
  const int first = blockIdx.x * kExactWarps + warp;
  uint4 gw[kExactSweep], uw[kExactSweep];
  const uint4* first_rows = rows_of(first);
  if (first_rows) exact_load(first_rows, first_rows + up_offset, lane, chunks, gw, uw);
  const uint4* x = reinterpret_cast<const uint4*>(hidden + static_cast<size_t>(t) * L.H);
  for (int i = tid; i < chunks; i += kExactWarps * 32) xs[i] = x[i];
  __syncthreads();
  for (int index = first; index < L.F; index += gridDim.x * kExactWarps) {
  const int cid = list[index];
  if (cid < 0) break;  // lists end with -1 entries
  const uint4* gate = index == first ? first_rows : rows_of(index);
  if (!gate) continue;
  float g, u;
  exact_dot(gate, gate + up_offset, xs, chunks, lane, index == first, gw, uw, g, u);
  if (lane == 0) {
    ws.activations[static_cast<size_t>(t) * L.N + cid] =
        __float2bfloat16_rn(exact_feature(g, u, L.activation));
    ws.exact[static_cast<size_t>(t) * 2 * L.F + index] = g;
    ws.exact[static_cast<size_t>(t) * 2 * L.F + L.F + index] = u;
  }
  }
}

// The same gather with the (token, expert) pairs walked in expert order:
// grid (X, T * K), 128 threads.  CTA row y takes the y-th pair of the list
// grouped by expert (k_group), so the tokens of one expert run next to each
// other in time and a row several of them kept comes from HBM once and from L2
// after that.  The X CTAs of a pair share its kept rows, one warp per row.  Same
// arithmetic, same order, same bits as k_exact.
// The kept rows of the y-th pair of the list grouped by expert, for the CTA column
// blockIdx.x; all threads of the CTA call it with the staged row `xs` free.
__device__ __forceinline__ void exact_pair(const Layer& L, const Workspace& ws,
                                           const __nv_bfloat16* hidden, uint4* xs, int y) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pair = ws.group_pairs[y];
  const int count = ws.counts[pair];
  if (static_cast<int>(blockIdx.x) * kExactWarps >= count) return;  // the whole CTA
  const int t = pair / L.K, slot = pair - t * L.K, e = ws.ids[pair];
  const int start = ws.starts[pair];
  const int32_t* list = ws.candidate_ids + static_cast<size_t>(t) * L.F + start;
  const int chunks = L.H / 8;
  const size_t up_offset = static_cast<size_t>(L.I) * L.H / 8;
  const uint4* expert_rows =
      reinterpret_cast<const uint4*>(L.gate_up + static_cast<size_t>(e) * 2 * L.I * L.H);
  // The first row pair's first sweep is on its way while the input row is staged.
  const int first = blockIdx.x * kExactWarps + warp;
  uint4 gw[kExactSweep], uw[kExactSweep];
  if (first < count) {
    const uint4* gate = expert_rows + static_cast<size_t>(list[first] - slot * L.I) * chunks;
    exact_load(gate, gate + up_offset, lane, chunks, gw, uw);
  }
  const uint4* x = reinterpret_cast<const uint4*>(hidden + static_cast<size_t>(t) * L.H);
  for (int i = tid; i < chunks; i += kExactWarps * 32) xs[i] = x[i];
  __syncthreads();
  for (int index = first; index < count; index += gridDim.x * kExactWarps) {
    const int cid = list[index];
    const uint4* gate = expert_rows + static_cast<size_t>(cid - slot * L.I) * chunks;
    float g, u;
    exact_dot(gate, gate + up_offset, xs, chunks, lane, index == first, gw, uw, g, u);
    if (lane == 0) {
      ws.activations[static_cast<size_t>(t) * L.N + cid] =
          __float2bfloat16_rn(exact_feature(g, u, L.activation));
      ws.exact[static_cast<size_t>(t) * 2 * L.F + start + index] = g;
      ws.exact[static_cast<size_t>(t) * 2 * L.F + L.F + start + index] = u;
    }
  }
}

// With `list` one more CTA row, the first, lists the down tiles meanwhile.  Five CTAs per SM, at the price of
// six registers spilled: 32 tokens of the 128-expert layer 40.0 us against 41.7 with four, 19 tokens of a layer
// of hidden 1152 26.8 against 29.1, 8 of the former 14.9 against 15.1.
// STRIDED: under expert parallelism fewer CTA rows than (token, slot) pairs are launched,
// since a rank owns few of them; row y then takes pairs y, y + gridDim.y, ...
template <bool STRIDED>
__global__ void __launch_bounds__(kExactWarps * 32, STRIDED ? 4 : 5) k_exact_pairs(Layer L, Workspace ws,
                                                                  const __nv_bfloat16* hidden,
                                                                  int list) {
  grid_dependency_wait();     // the selection is complete
  grid_dependency_release();  // the down kernel may be scheduled: its encoder needs no more than that
  extern __shared__ uint4 xs[];  // H bf16 values of the token
  __shared__ int scratch[33];
  if (list && blockIdx.y == 0) {
    if (blockIdx.x == 0) list_down_tiles(L, ws, scratch);
    return;
  }
  const int pairs = ws.group_offsets[L.E], first = blockIdx.y - list;
  if (!STRIDED) {
    if (first < pairs) exact_pair(L, ws, hidden, xs, first);
    return;
  }
  for (int y = first; y < pairs; y += gridDim.y - list) {
    exact_pair(L, ws, hidden, xs, y);
    __syncthreads();  // the staged row may be overwritten by the next pair
  }
}

// ---------------------------------------------------------------------------
// encode: recovery encoder over skipped channels, then the latent
// ---------------------------------------------------------------------------
// 128 threads.  A CTA owns 256 channels of one (token, expert) pair: index = pair * tiles + tile.
// The sketch features of the skipped channels (0 for kept ones) go to shared memory; then the
// encoder rows stream: LPR = R / 8 lanes cover one row (16 bytes each), 128 / LPR row groups walk
// the channels with eight rows in flight per thread; last, the row groups fold (shuffles inside a
// warp, shared memory across warps).  L2 and latency bound, and needed by nothing before the output
// mix, so its CTAs ride at the head of the down kernel's launch, beside the gathers (a stream of
// its own cost two events and, for one token, 7 us at its end).  The last CTA of a token to arrive
// mixes the latent, hidden there as well (in every CTA of the output it took 4 us for one token and
// 13 us for 64).  `shared`: 256 + 4 * 256 floats.
constexpr int kEncodeThreads = 128;

// The latent of a token whose encoder sums are all there, by 128 threads.
__device__ __forceinline__ void mix_latent(const Layer& L, const Workspace& ws, int t) {
  const int tid = threadIdx.x, R = L.R;
  // Per slot the sums in tile order, rounded to BF16, times the router weight, in slot order.
  const int parts_of_slot = ws.encoder_tiles, all_parts = L.K * parts_of_slot;
  const size_t pair0 = static_cast<size_t>(t) * L.K;
  for (int r = tid; r < R; r += kEncodeThreads) {
    const float* p = ws.encoder_parts + pair0 * parts_of_slot * R + r;
    float latent = 0.0f, sum = 0.0f;
    int slot2 = 0, left = parts_of_slot;
    for (int n0 = 0; n0 < all_parts; n0 += 8) {
      float v[8];  // on their way together
#pragma unroll
      for (int n = 0; n < 8; ++n)
        v[n] = n0 + n < all_parts ? __ldcg(p + static_cast<size_t>(n0 + n) * R) : 0.0f;
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        if (n0 + n >= all_parts) break;
        sum += v[n];
        if (--left == 0) {
          if (ws.ids[pair0 + slot2] >= 0)
            latent = fmaf(bf16_round(sum), ws.weights[pair0 + slot2], latent);
          sum = 0.0f;
          left = parts_of_slot;
          ++slot2;
        }
      }
    }
    ws.latent[static_cast<size_t>(t) * R + r] = latent;
  }
}

__device__ __forceinline__ void encode_tile(const Layer& L, const Workspace& ws,
                                            const uint8_t* padding, int index, float* shared) {
  float* feature = shared;
  float(*red)[256] = reinterpret_cast<float(*)[256]>(shared + kEncodeTileRows);
  const int pair = index / ws.encoder_tiles, tile = index - pair * ws.encoder_tiles;
  const int tid = threadIdx.x, t = pair / L.K, slot = pair - t * L.K;
  const int R = L.R, lpr = R / 8, groups = kEncodeThreads / lpr;
  const int e = ws.ids[pair];
  if (padding && padding[t]) {
    if (slot == 0 && tile == 0)
      for (int r = tid; r < R; r += kEncodeThreads) ws.latent[static_cast<size_t>(t) * R + r] = 0.0f;
    return;
  }
  const int c0 = tile * kEncodeTileRows, c1 = e < 0 ? c0 : min(L.I, c0 + kEncodeTileRows);
  const int group = tid / lpr, col = (tid - group * lpr) * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
  {
    const size_t first = static_cast<size_t>(t) * L.N + slot * L.I;
    for (int c = c0 + tid; c < c1; c += kEncodeThreads)
      feature[c - c0] = ws.selected[first + c] ? 0.0f : __bfloat162float(ws.features[first + c]);
    __syncthreads();
    const __nv_bfloat16* enc = L.encoder + static_cast<size_t>(e) * L.I * R + col;
    constexpr int U = 8;
    for (int base = c0 + group; base < c1; base += groups * U) {
      uint4 w[U];
      float p[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = base + u * groups;
        p[u] = 0.0f;
        w[u] = make_uint4(0, 0, 0, 0);
        if (c < c1) {
          p[u] = feature[c - c0];
          w[u] = *reinterpret_cast<const uint4*>(enc + static_cast<size_t>(c) * R);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        acc[0] = fmaf(bf16_lo(w[u].x), p[u], acc[0]);
        acc[1] = fmaf(bf16_hi(w[u].x), p[u], acc[1]);
        acc[2] = fmaf(bf16_lo(w[u].y), p[u], acc[2]);
        acc[3] = fmaf(bf16_hi(w[u].y), p[u], acc[3]);
        acc[4] = fmaf(bf16_lo(w[u].z), p[u], acc[4]);
        acc[5] = fmaf(bf16_hi(w[u].z), p[u], acc[5]);
        acc[6] = fmaf(bf16_lo(w[u].w), p[u], acc[6]);
        acc[7] = fmaf(bf16_hi(w[u].w), p[u], acc[7]);
      }
    }
  }
  // Fold the row groups that share a warp (lanes lpr apart hold the same columns).
  for (int w = lpr; w < 32; w <<= 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(kFull, acc[j], w);
  }
  const int lane = tid & 31, warp = tid >> 5;
  if (lane < lpr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) red[warp][col + j] = acc[j];
  }
  __syncthreads();
  float* parts = ws.encoder_parts + static_cast<size_t>(index) * R;
  for (int r = tid; r < R; r += kEncodeThreads)
    parts[r] = ((red[0][r] + red[1][r]) + red[2][r]) + red[3][r];
  __threadfence();
  __syncthreads();
  uint32_t* counter = ws.counters + 2 * static_cast<size_t>(ws.capacity) * L.K + t;
  if (tid == 0) {
    const bool last = atomicAdd(counter, 1u) == static_cast<unsigned>(L.K * ws.encoder_tiles - 1);
    if (last) *counter = 0;
    shared[0] = last ? 1.0f : 0.0f;
  }
  __syncthreads();
  if (shared[0] == 0.0f) return;
  __threadfence();
  mix_latent(L, ws, t);
}

// The same sums for up to four pairs of an expert at a time: its rows are read and widened once for all
// of them (a pair at a time they came from L2 once per pair, 0.8 GB for 256 tokens of hidden 4096 and width
// 1536), and a pair's product is one packed instruction per two columns.  Rows, their order and every
// rounding are encode_tile's.  `index` = (pass * subs + part of the pass) * tiles + tile; after those, CTAs
// whose threads zero the latents of tokens without a live pair.  `shared`: 4 x 256 pairs of floats, 4 x 4 x
// 256 floats, 4 words.
constexpr int kEncodePairs = 4;
constexpr int kEncodeGroupBytes = kEncodePairs * (kEncodeTileRows * 8 + 4 * 256 * 4) + 16;

template <int N>
__device__ __forceinline__ void encode_rows(const __nv_bfloat16* rows, const Pair* feature, int c0, int c1, int R,
                                            int group, int groups, float (*red)[4][256], int col, int lpr) {
  constexpr int U = 8;
  Pair acc[N][4];
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[n][j] = 0;
  for (int base = c0 + group; base < c1; base += groups * U) {
    uint4 w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = base + u * groups;
      w[u] = c < c1 ? *reinterpret_cast<const uint4*>(rows + static_cast<size_t>(c) * R) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = min(base + u * groups, c1 - 1) - c0;
      const bool there = base + u * groups < c1;
      const Pair v[4] = {pair_of(bf16_lo(w[u].x), bf16_hi(w[u].x)), pair_of(bf16_lo(w[u].y), bf16_hi(w[u].y)),
                         pair_of(bf16_lo(w[u].z), bf16_hi(w[u].z)), pair_of(bf16_lo(w[u].w), bf16_hi(w[u].w))};
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const Pair a = there ? feature[n * kEncodeTileRows + c] : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = pair_fma(v[j], a, acc[n][j]);
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    float sum[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) pair_split(acc[n][j], sum[2 * j], sum[2 * j + 1]);
    for (int w = lpr; w < 32; w <<= 1) {  // the row groups that share a warp
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[j] += __shfl_xor_sync(kFull, sum[j], w);
    }
    if (lane < lpr) {
#pragma unroll
      for (int j = 0; j < 8; ++j) red[n][warp][col + j] = sum[j];
    }
  }
}

__device__ __forceinline__ void encode_group(const Layer& L, const Workspace& ws, const uint8_t* padding, int index,
                                             int subs, int group_ctas, int tokens, uint8_t* shared) {
  const int tid = threadIdx.x, R = L.R, I = L.I, tiles = ws.encoder_tiles;
  if (index >= group_ctas) {
    const int t = (index - group_ctas) * kEncodeThreads + tid;
    bool live = t >= tokens;
    for (int k = 0; k < L.K && !live; ++k)
      live = !(padding && padding[t]) && ws.ids[static_cast<size_t>(t) * L.K + k] >= 0;
    if (!live)
      for (int r = 0; r < R; ++r) ws.latent[static_cast<size_t>(t) * R + r] = 0.0f;
    return;
  }
  const int tile = index % tiles, part = index / tiles % subs, number = index / tiles / subs;
  if (number >= ws.work_counts[kPassCount]) return;
  const int4 pass = *reinterpret_cast<const int4*>(ws.pass_work + number);
  const int e = pass.x, first = pass.y + kEncodePairs * part, count = min(kEncodePairs, pass.z - kEncodePairs * part);
  if (count <= 0) return;
  Pair* feature = reinterpret_cast<Pair*>(shared);
  float(*red)[4][256] = reinterpret_cast<float(*)[4][256]>(shared + kEncodePairs * kEncodeTileRows * 8);
  int* last = reinterpret_cast<int*>(shared + kEncodePairs * (kEncodeTileRows * 8 + 4 * 256 * 4));
  const int c0 = tile * kEncodeTileRows, c1 = min(I, c0 + kEncodeTileRows);
  int pairs[kEncodePairs];
#pragma unroll
  for (int n = 0; n < kEncodePairs; ++n) pairs[n] = ws.group_pairs[first + min(n, count - 1)];
#pragma unroll
  for (int i = 0; i < kEncodeTileRows / kEncodeThreads; ++i) {
    const int c = min(c0 + tid + i * kEncodeThreads, c1 - 1);
    uint8_t kept[kEncodePairs];
    __nv_bfloat16 f[kEncodePairs];
#pragma unroll
    for (int n = 0; n < kEncodePairs; ++n) {
      const size_t at = static_cast<size_t>(pairs[n]) * I + c;  // (t K + slot) I = t N + slot I
      kept[n] = ws.selected[at];
      f[n] = ws.features[at];
    }
#pragma unroll
    for (int n = 0; n < kEncodePairs; ++n) {
      const float v = kept[n] ? 0.0f : __bfloat162float(f[n]);
      feature[n * kEncodeTileRows + c - c0] = pair_of(v, v);
    }
  }
  __syncthreads();
  const int lpr = R / 8, groups = kEncodeThreads / lpr, group = tid / lpr, col = (tid - group * lpr) * 8;
  const __nv_bfloat16* rows = L.encoder + static_cast<size_t>(e) * I * R + col;
  switch (count) {
    case 1: encode_rows<1>(rows, feature, c0, c1, R, group, groups, red, col, lpr); break;
    case 2: encode_rows<2>(rows, feature, c0, c1, R, group, groups, red, col, lpr); break;
    default: encode_rows<4>(rows, feature, c0, c1, R, group, groups, red, col, lpr); break;
  }
  __syncthreads();
  for (int i = tid; i < count * R; i += kEncodeThreads) {
    const int n = i / R, r = i - n * R;
    const float(*own)[256] = red[n];
    const int pair = n == 0 ? pairs[0] : n == 1 ? pairs[1] : n == 2 ? pairs[2] : pairs[3];
    ws.encoder_parts[(static_cast<size_t>(pair) * tiles + tile) * R + r] =
        ((own[0][r] + own[1][r]) + own[2][r]) + own[3][r];
  }
  __threadfence();
  __syncthreads();
  // The last to arrive of a token's live pairs and their tiles mixes its latent.
  if (tid < count) {
    const int t = (tid == 0 ? pairs[0] : tid == 1 ? pairs[1] : tid == 2 ? pairs[2] : pairs[3]) / L.K;
    int live = 0;
    for (int k = 0; k < L.K; ++k) live += ws.ids[static_cast<size_t>(t) * L.K + k] >= 0;
    uint32_t* counter = ws.counters + 2 * static_cast<size_t>(ws.capacity) * L.K + t;
    const bool done = atomicAdd(counter, 1u) == static_cast<unsigned>(live * tiles - 1);
    if (done) *counter = 0;
    last[tid] = done ? t : -1;
  }
  __syncthreads();
  for (int n = 0; n < count; ++n) {
    if (last[n] < 0) continue;
    __threadfence();
    mix_latent(L, ws, last[n]);
  }
}

// The encoder on its own: grid (pairs * tiles), 128 threads.
__global__ void __launch_bounds__(kEncodeThreads) k_encode(Layer L, Workspace ws,
                                                           const uint8_t* padding) {
  __shared__ float shared[kEncodeTileRows + 4 * 256];
  encode_tile(L, ws, padding, blockIdx.x, shared);
}

// ---------------------------------------------------------------------------
// down: gathered channel-major down rows
// ---------------------------------------------------------------------------
constexpr int kDownRingBytes = 32 * 1024;  // per CTA
static_assert(kEncodeGroupBytes <= kDownRingBytes, "the encoder's arrays lie in the ring");

// 128 threads, kDownRingBytes of dynamic shared memory.  A CTA sums up to 64 kept rows of one
// expert, each scaled by its activation, over 256 CHUNKS output columns.  A warp takes every fourth
// row of the tile.  Rows travel through a ring in shared memory, 16 / CHUNKS per warp in flight:
// per row a lane copies CHUNKS 16-byte pieces 512 bytes apart with cp.async and later reads back
// exactly the pieces it copied, so a lane only ever waits for its own copy groups and the ring
// needs no barrier.  The row is accumulated into 8 CHUNKS FP32 registers per lane in row order;
// the four warps' sums are added in warp order through shared memory (the ring's, once
// all copies have landed): same bits for every CHUNKS.  Calls with few tiles split the columns
// finer, so that their rows come in over more SMs.
// One tile: `rows` (at most 64) kept rows of slot `slot` of token t, an expert-e
// slot, whose candidate ids start at `list`, summed into down tile `tile`, columns from `column`.
// Called by all 128 threads of a CTA; begins and ends with the shared arrays free.
template <int CHUNKS>
__device__ __forceinline__ void down_tile(const Layer& L, const Workspace& ws, int t, int slot,
                                          int e, int rows, const int32_t* list, int tile,
                                          int column, int* tile_channel, float* tile_activation,
                                          uint8_t* ring) {
  constexpr int STAGES = 16 / CHUNKS, kColumns = 256 * CHUNKS, kRowBytes = 2 * kColumns;
  static_assert(4 * STAGES * kRowBytes == kDownRingBytes, "ring");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int column0 = column + lane * 8;  // this lane's first column
  const __nv_bfloat16* act = ws.activations + static_cast<size_t>(t) * L.N;
  if (tid < rows) {
    const int cid = list[tid];
    tile_channel[tid] = cid - slot * L.I;
    tile_activation[tid] = __bfloat162float(act[cid]);
  }
  __syncthreads();
  const __nv_bfloat16* base = L.down + static_cast<size_t>(e) * L.I * L.H + column0;
  bool live[CHUNKS];
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j) live[j] = column0 + 256 * j < L.H;
  float acc[CHUNKS][8];
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[j][i] = 0.0f;
  // This lane's pieces of ring slot s of its warp.
  uint8_t* mine = ring + warp * (STAGES * kRowBytes) + lane * 16;
  auto fetch = [&](int r, int s) {  // row r of the tile into slot s; one copy group
    if (r < rows) {
      const __nv_bfloat16* row = base + static_cast<size_t>(tile_channel[r]) * L.H;
#pragma unroll
      for (int j = 0; j < CHUNKS; ++j)
        if (live[j]) copy_async16(shared_u32(mine + s * kRowBytes + 512 * j), row + 256 * j);
    }
    copy_async_commit();  // also when empty: the group count per iteration stays fixed
  };
  auto add = [&](int r, int s) {
    const float a = tile_activation[r];
#pragma unroll
    for (int j = 0; j < CHUNKS; ++j) {
      const uint4 w = live[j] ? *reinterpret_cast<const uint4*>(mine + s * kRowBytes + 512 * j)
                              : make_uint4(0, 0, 0, 0);
      acc[j][0] = fmaf(bf16_lo(w.x), a, acc[j][0]);
      acc[j][1] = fmaf(bf16_hi(w.x), a, acc[j][1]);
      acc[j][2] = fmaf(bf16_lo(w.y), a, acc[j][2]);
      acc[j][3] = fmaf(bf16_hi(w.y), a, acc[j][3]);
      acc[j][4] = fmaf(bf16_lo(w.z), a, acc[j][4]);
      acc[j][5] = fmaf(bf16_hi(w.z), a, acc[j][5]);
      acc[j][6] = fmaf(bf16_lo(w.w), a, acc[j][6]);
      acc[j][7] = fmaf(bf16_hi(w.w), a, acc[j][7]);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES; ++s) fetch(warp + 4 * s, s);
  int s = 0;
  for (int r = warp; r < rows; r += 4) {
    copy_async_wait<STAGES - 1>();  // the oldest group, row r, has landed
    add(r, s);
    fetch(r + 4 * STAGES, s);  // the slot is free again: its pieces are in registers
    s = s + 1 == STAGES ? 0 : s + 1;
  }
  copy_async_wait<0>();
  __syncthreads();  // every warp is done with the ring: it now holds the warps' sums
  float(*red)[kColumns] = reinterpret_cast<float(*)[kColumns]>(ring);
#pragma unroll
  for (int j = 0; j < CHUNKS; ++j) {
    float4* out = reinterpret_cast<float4*>(&red[warp][256 * j + lane * 8]);
    out[0] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
    out[1] = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
  }
  __syncthreads();
  float* parts = ws.down_parts + (static_cast<size_t>(t) * ws.down_tiles + tile) * L.H + column;
  for (int c = tid * 4; c < kColumns; c += 128 * 4) {
    if (column + c < L.H) {
      const float4 a = *reinterpret_cast<const float4*>(&red[0][c]);
      const float4 b = *reinterpret_cast<const float4*>(&red[1][c]);
      const float4 d = *reinterpret_cast<const float4*>(&red[2][c]);
      const float4 g = *reinterpret_cast<const float4*>(&red[3][c]);
      *reinterpret_cast<float4*>(parts + c) =
          make_float4(((a.x + b.x) + d.x) + g.x, ((a.y + b.y) + d.y) + g.y,
                      ((a.z + b.z) + d.z) + g.z, ((a.w + b.w) + d.w) + g.w);
    }
  }
  __syncthreads();  // the shared arrays may be reused
}

// What a launch of a down kernel does: `encode_ctas` CTAs of the recovery encoder first, then
// `columns` CTAs per tile.
struct DownGrid {
  int encode_ctas, columns, tiles;
  int encode_subs, group_ctas, tokens;  // parts of a screen pass that share encoder rows (0: none do)
};

// The tiles of every token in turn: 1D grid of encode_ctas + T * tiles * columns CTAs.  Under expert
// parallelism (STRIDED) fewer CTAs than tiles are launched per token, since a rank owns few of a
// token's slots; they walk the tiles in strides.
template <bool STRIDED, int CHUNKS>
__global__ void __launch_bounds__(128, 4) k_down(Layer L, Workspace ws, const uint8_t* padding,
                                                 DownGrid d) {
  extern __shared__ __align__(128) uint8_t down_ring[];
  __shared__ int tile_channel[kDownTileRows];
  __shared__ float tile_activation[kDownTileRows];
  __shared__ int s_slot, s_first;
  if (static_cast<int>(blockIdx.x) < d.encode_ctas) {
    grid_dependency_release();
    encode_tile(L, ws, padding, blockIdx.x, reinterpret_cast<float*>(down_ring));
    return;
  }
  grid_dependency_wait();     // the activations are complete
  grid_dependency_release();  // the output may be scheduled; it waits for this grid
  int at = blockIdx.x - d.encode_ctas;
  const int column = at % d.columns * (256 * CHUNKS);
  at /= d.columns;
  const int t = at / d.tiles, tid = threadIdx.x;
  int tile = at - t * d.tiles;
  if (padding && padding[t]) return;
  const size_t token_pairs = static_cast<size_t>(t) * L.K;
  int used;
  {
    // Tiles are laid out slot after slot; leave at once beyond the last one.
    const size_t last = token_pairs + L.K - 1;
    const int tail =
        ws.ids[last] >= 0 ? (ws.counts[last] + kDownTileRows - 1) / kDownTileRows : 0;
    used = ws.tile_starts[last] + tail;
  }
  if (tile >= used) return;
  do {
    if (tid == 0) s_slot = -1;
    __syncthreads();
    if (tid < L.K) {  // the slot whose tile range holds this tile, if any
      const int e = ws.ids[token_pairs + tid];
      const int tiles =
          e >= 0 ? (ws.counts[token_pairs + tid] + kDownTileRows - 1) / kDownTileRows : 0;
      const int begin = ws.tile_starts[token_pairs + tid];
      if (tile >= begin && tile < begin + tiles) {
        s_slot = tid;
        s_first = (tile - begin) * kDownTileRows;
      }
    }
    __syncthreads();
    const int slot = s_slot, first = s_first;
    if (slot < 0) continue;  // uniform: every thread read the same slot
    down_tile<CHUNKS>(L, ws, t, slot, ws.ids[token_pairs + slot],
              min(kDownTileRows, ws.counts[token_pairs + slot] - first),
              ws.candidate_ids + static_cast<size_t>(t) * L.F + ws.starts[token_pairs + slot] + first,
              tile, column, tile_channel, tile_activation, down_ring);
  } while (STRIDED && (tile += d.tiles) < used);
}

// The same tiles from the list of the call's tiles in expert order
// (cfm_select.cuh): 1D grid of encode_ctas + tiles * columns CTAs.  A CTA reads its 32-byte record
// and goes straight to the tile's rows.  Same tiles, same sums, same bits as k_down.  Five CTAs per SM: whole
// calls of 64 tokens of the 128-expert layer 155.9 us against 158.1 with four, 32 tokens 101.0 and 101.3, 8 tokens 53.1 and
// 52.1; of the 256-expert layer 64 tokens 122.6 and 124.0, 8 tokens 43.2 and 43.9.
template <int CHUNKS>
__global__ void __launch_bounds__(128, 5) k_down_tiles(Layer L, Workspace ws, const uint8_t* padding,
                                                       DownGrid d) {
  extern __shared__ __align__(128) uint8_t down_ring[];
  __shared__ int tile_channel[kDownTileRows];
  __shared__ float tile_activation[kDownTileRows];
  if (static_cast<int>(blockIdx.x) < d.encode_ctas) {
    grid_dependency_release();
    if (d.encode_subs)
      encode_group(L, ws, padding, blockIdx.x, d.encode_subs, d.group_ctas, d.tokens, down_ring);
    else
      encode_tile(L, ws, padding, blockIdx.x, reinterpret_cast<float*>(down_ring));
    return;
  }
  grid_dependency_wait();     // the activations and the list are complete
  grid_dependency_release();  // the output may be scheduled; it waits for this grid
  const int at = blockIdx.x - d.encode_ctas, tiles = ws.tile_count[0];
  const int column = at % d.columns * (256 * CHUNKS);
  for (int y = at / d.columns; y < tiles; y += d.tiles) {  // strides under expert parallelism
    const int4* record = reinterpret_cast<const int4*>(ws.tile_list) + 2 * y;
    const int4 a = record[0], b = record[1];  // t, slot, expert, rows | list, tile
    down_tile<CHUNKS>(L, ws, a.x, a.y, a.z, a.w, ws.candidate_ids + b.x, b.y, column, tile_channel,
                      tile_activation, down_ring);
  }
}

// grid (T), 128 threads: latent = 0 (no skipped channels, or no map).
__global__ void k_zero_latent(Layer L, Workspace ws) {
  for (int r = threadIdx.x; r < L.R; r += blockDim.x)
    ws.latent[static_cast<size_t>(blockIdx.x) * L.R + r] = 0.0f;
}

#include "cfm_union.cuh"

// ---------------------------------------------------------------------------
// output: router mix + decoder term
// ---------------------------------------------------------------------------
// One output column of one token: the per-slot sums of its down-tile partials in
// tile order, each rounded to BF16 and mixed with the slot's router weight in slot
// order.  `parts` points at the column in the token's first tile; `slot_end` and
// `slot_weight` are the token's slot table in shared memory.  Sixteen tile loads are
// in flight at a time; the additions keep their order.
__device__ __forceinline__ float mix_down_tiles(const float* parts, int used, size_t stride,
                                                const int* slot_end, const float* slot_weight) {
  constexpr int kInFlight = 16;
  float routed = 0.0f, sum = 0.0f;
  int slot = 0;
  for (int base = 0; base < used; base += kInFlight) {
    float v[kInFlight];
#pragma unroll
    for (int j = 0; j < kInFlight; ++j)
      v[j] = base + j < used ? __ldcg(parts + static_cast<size_t>(base + j) * stride) : 0.0f;
#pragma unroll
    for (int j = 0; j < kInFlight; ++j) {
      const int tile = base + j;
      if (tile < used) {
        while (tile >= slot_end[slot]) {  // close the finished slots
          routed = fmaf(bf16_round(sum), slot_weight[slot], routed);
          sum = 0.0f;
          ++slot;
        }
        sum += v[j];
      }
    }
  }
  if (used > 0) routed = fmaf(bf16_round(sum), slot_weight[slot], routed);
  return routed;
}

// The same for four adjacent columns (16-byte loads); each column's additions keep
// the order of the one-column version.
__device__ __forceinline__ float4 mix_down_tiles4(const float* parts, int used, size_t stride,
                                                  const int* slot_end, const float* slot_weight) {
  constexpr int kInFlight = 8;
  float4 routed = make_float4(0.0f, 0.0f, 0.0f, 0.0f), sum = routed;
  int slot = 0;
  auto close = [&]() {
    const float w = slot_weight[slot];
    routed.x = fmaf(bf16_round(sum.x), w, routed.x);
    routed.y = fmaf(bf16_round(sum.y), w, routed.y);
    routed.z = fmaf(bf16_round(sum.z), w, routed.z);
    routed.w = fmaf(bf16_round(sum.w), w, routed.w);
    sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    ++slot;
  };
  for (int base = 0; base < used; base += kInFlight) {
    float4 v[kInFlight];
#pragma unroll
    for (int j = 0; j < kInFlight; ++j)
      v[j] = base + j < used
                 ? __ldcg(reinterpret_cast<const float4*>(parts + static_cast<size_t>(base + j) * stride))
                 : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < kInFlight; ++j) {
      const int tile = base + j;
      if (tile < used) {
        while (tile >= slot_end[slot]) close();  // close the finished slots
        sum.x += v[j].x;
        sum.y += v[j].y;
        sum.z += v[j].z;
        sum.w += v[j].w;
      }
    }
  }
  if (used > 0) close();
  return routed;
}

// grid (H / 128, T), 128 threads, one output column per thread; with one more column of CTAs that
// add the tokens' read-cost counters.
// `latents` false: there are none (the workspace's are set to zero).
__global__ void __launch_bounds__(128) k_output(Layer L, Workspace ws, const uint8_t* padding,
                                                __nv_bfloat16* out, int latents, int early) {
  __shared__ float latent[256];
  __shared__ int slot_end[32];       // one past the last down tile of every slot
  __shared__ float slot_weight[32];
  const int t = blockIdx.y, tid = threadIdx.x, h = blockIdx.x * 128 + tid;
  if (!early) grid_dependency_wait();
  if (h >= L.H) {  // the token's read-cost counters
    if (tid < 32 && !(padding && padding[t])) {
      const size_t pair = static_cast<size_t>(t) * L.K + tid;
      const bool local = tid < L.K && ws.ids[pair] >= 0;
      account_token(L, tid, local, local ? ws.counts[pair] : 0, L.F < L.N);
    }
    return;
  }
  if (padding && padding[t]) {
    if (early) grid_dependency_wait();
    out[static_cast<size_t>(t) * L.H + h] = __float2bfloat16_rn(0.0f);
    return;
  }
  const bool recover = L.R > 0 && L.owner && L.decoder;
  // With `early` the down kernel is the launch before this one, so the selection is complete when
  // this grid starts; the decoder row and the slot table are read while the last tiles are summed.
  constexpr int kAhead = 8;  // 16-byte chunks of the decoder row fetched ahead (R <= 64: all)
  float correction = 0.0f;
  const uint4* decoder_row = reinterpret_cast<const uint4*>(L.decoder + static_cast<size_t>(h) * L.R);
  uint4 ahead[kAhead];
  if (recover) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      ahead[i] = i < L.R / 8 ? decoder_row[i] : make_uint4(0, 0, 0, 0);
  }
  if (tid < L.K) {
    const size_t pair = static_cast<size_t>(t) * L.K + tid;
    slot_end[tid] = down_slot_end(L, ws, t, tid);
    slot_weight[tid] = ws.weights[pair];
  }
  if (early) grid_dependency_wait();  // the sums are complete
  for (int r = tid; r < L.R; r += 128) {
    float* kept = ws.latent + static_cast<size_t>(t) * L.R + r;
    if (!latents && blockIdx.x == 0) *kept = 0.0f;
    latent[r] = latents ? bf16_round(*kept) : 0.0f;
  }
  __syncthreads();
  const int used = slot_end[L.K - 1];  // tiles are laid out slot after slot
  const float routed = mix_down_tiles(
      ws.down_parts + static_cast<size_t>(t) * ws.down_tiles * L.H + h, used, L.H, slot_end,
      slot_weight);
  if (recover) {
    float dot = 0.0f;
    auto fold = [&](const uint4 w, int i) {
      const float* z = latent + i * 8;
      dot = fmaf(bf16_lo(w.x), z[0], dot);
      dot = fmaf(bf16_hi(w.x), z[1], dot);
      dot = fmaf(bf16_lo(w.y), z[2], dot);
      dot = fmaf(bf16_hi(w.y), z[3], dot);
      dot = fmaf(bf16_lo(w.z), z[4], dot);
      dot = fmaf(bf16_hi(w.z), z[5], dot);
      dot = fmaf(bf16_lo(w.w), z[6], dot);
      dot = fmaf(bf16_hi(w.w), z[7], dot);
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (i < L.R / 8) fold(ahead[i], i);
    for (int i0 = kAhead; i0 < L.R / 8; i0 += 4) {
      uint4 row[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        row[i] = i0 + i < L.R / 8 ? decoder_row[i0 + i] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i0 + i < L.R / 8) fold(row[i], i0 + i);
    }
    correction = bf16_round(dot);
  }
  out[static_cast<size_t>(t) * L.H + h] = __float2bfloat16_rn(routed + correction);
}

// Expert parallelism splits the output stage in two.  k_partial_output runs on
// the rank that owns experts: the router-weighted FP32 sum of its local slots'
// BF16-rounded expert sums, no decoder term.  k_finish runs on the token's home
// rank after the partial sums and latents of all ranks have been added: decoder
// term and BF16 store.  grid (H / 128, T), 128 threads each.
// With `peers` row t goes straight into slot [this rank] of the `rows` of its home
// rank's exchange block (no latent: the home rank computes its own), and the last
// CTA of a home rank's rows announces the epoch there.
__global__ void __launch_bounds__(128) k_partial_output(Layer L, Workspace ws,
                                                        const uint8_t* padding, float* combined,
                                                        int by_union, Exchange x, int peers) {
  __shared__ int slot_end[32];
  __shared__ float slot_weight[32];
  const int t = blockIdx.y, tid = threadIdx.x, h = blockIdx.x * 128 + tid;
  float* routed_out = combined + static_cast<size_t>(t) * (L.H + L.R);
  const bool padded = padding && padding[t];
  if (peers) {
    // grid (ceil(H / 512), T): four adjacent columns per thread, so that a row crosses
    // NVLink in 16-byte stores and a quarter of the CTAs fence and arrive.
    const int h4 = (blockIdx.x * 128 + tid) * 4;
    const int home = t / x.tokens, row = t - home * x.tokens;
    routed_out = reinterpret_cast<float*>(x.block[home] +
                                          exchange_rows_offset(x.world, x.tokens, L.F)) +
                 (static_cast<size_t>(x.rank) * x.tokens + row) * L.H;
    float4 routed = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!padded && by_union) {
      if (h4 < L.H)
        routed = make_float4(mix_sums(L, ws, t, h4), mix_sums(L, ws, t, h4 + 1),
                             mix_sums(L, ws, t, h4 + 2), mix_sums(L, ws, t, h4 + 3));
    } else if (!padded) {
      if (tid < L.K) {
        slot_end[tid] = down_slot_end(L, ws, t, tid);
        slot_weight[tid] = ws.weights[static_cast<size_t>(t) * L.K + tid];
      }
      __syncthreads();
      if (h4 < L.H)
        routed = mix_down_tiles4(
            ws.down_parts + static_cast<size_t>(t) * ws.down_tiles * L.H + h4, slot_end[L.K - 1],
            L.H, slot_end, slot_weight);
    }
    if (h4 < L.H) *reinterpret_cast<float4*>(routed_out + h4) = routed;
    uint32_t* header = exchange_header(x, x.rank);
    exchange_announce(header + kExchangeRowsArrive + home, gridDim.x * x.tokens,
                      exchange_header(x, home) + kExchangeRowsFlag + x.rank,
                      header[kExchangeEpoch] + 1u);
    return;
  }
  if (blockIdx.x == 0)  // this rank's share of the latent rides behind the H outputs
    for (int r = tid; r < L.R; r += 128)
      routed_out[L.H + r] = padded ? 0.0f : ws.latent[static_cast<size_t>(t) * L.R + r];
  if (padded) {
    routed_out[h] = 0.0f;
    return;
  }
  if (by_union) {
    routed_out[h] = mix_sums(L, ws, t, h);
    return;
  }
  if (tid < L.K) {
    const size_t pair = static_cast<size_t>(t) * L.K + tid;
    slot_end[tid] = down_slot_end(L, ws, t, tid);
    slot_weight[tid] = ws.weights[pair];
  }
  __syncthreads();
  routed_out[h] = mix_down_tiles(
      ws.down_parts + static_cast<size_t>(t) * ws.down_tiles * L.H + h, slot_end[L.K - 1], L.H,
      slot_end, slot_weight);
}

__global__ void __launch_bounds__(128) k_finish(Layer L, const float* combined,
                                                const float* latent_rows, __nv_bfloat16* out) {
  __shared__ float latent[256];
  const int t = blockIdx.y, tid = threadIdx.x, h = blockIdx.x * 128 + tid;
  // The latent rides behind the H sums of a row unless it is given on its own.
  const float* row_in = combined + static_cast<size_t>(t) * (latent_rows ? L.H : L.H + L.R);
  const float* latent_in = latent_rows ? latent_rows + static_cast<size_t>(t) * L.R : row_in + L.H;
  const bool recover = L.R > 0 && L.decoder;
  float correction = 0.0f;
  if (recover) {
    for (int r = tid; r < L.R; r += 128)
      latent[r] = bf16_round(latent_in[r]);
    __syncthreads();
    const uint4* row = reinterpret_cast<const uint4*>(L.decoder + static_cast<size_t>(h) * L.R);
    float dot = 0.0f;
    for (int i = 0; i < L.R / 8; ++i) {
      const uint4 w = row[i];
      const float* z = latent + i * 8;
      dot = fmaf(bf16_lo(w.x), z[0], dot);
      dot = fmaf(bf16_hi(w.x), z[1], dot);
      dot = fmaf(bf16_lo(w.y), z[2], dot);
      dot = fmaf(bf16_hi(w.y), z[3], dot);
      dot = fmaf(bf16_lo(w.z), z[4], dot);
      dot = fmaf(bf16_hi(w.z), z[5], dot);
      dot = fmaf(bf16_lo(w.w), z[6], dot);
      dot = fmaf(bf16_hi(w.w), z[7], dot);
    }
    correction = bf16_round(dot);
  }
  out[static_cast<size_t>(t) * L.H + h] =
      __float2bfloat16_rn(row_in[h] + correction);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct Bound {
  Layer L;
  Workspace ws;
  cudaStream_t stream;
  int T;
  int row_offset;  // first workspace row of the call (cfm_select only)
  const uint8_t* padding;
};

static bool screens_grouped(const Bound& b);

static int bind_call(const cfm_layer* layer, void* workspace, int32_t capacity,
                     const cfm_call* call, void* stream, Bound* b) {
  if (!layer || !workspace || !call) return CFM_E_NULL;
  cfm_workspace_layout layout;
  const int rc = make_layout(layer, capacity, &layout);
  if (rc) return rc;
  if (call->tokens < 1 || call->row_offset < 0 || call->tokens + call->row_offset > capacity)
    return CFM_E_CAPACITY;
  if (layer->experts < 1) return CFM_E_SHAPE;
  if (layer->activation != CFM_ACT_SILU && layer->activation != CFM_ACT_GELU_TANH)
    return CFM_E_UNSUPPORTED;
  if (layer->score != CFM_SCORE_POINT && layer->score != CFM_SCORE_RECOVERY_AWARE)
    return CFM_E_UNSUPPORTED;
  if (layer->row_engine < CFM_ROWS_AUTO || layer->row_engine > CFM_ROWS_EXPERT_MAJOR)
    return CFM_E_UNSUPPORTED;
  const bool screened = layer->final_count < layer->top_k * layer->width;
  if (screened && (!layer->statistics || !layer->norms || !layer->signs)) return CFM_E_NULL;
  if (layer->rank && (!layer->encoder || !layer->decoder)) return CFM_E_NULL;
  b->L = device_layer(layer);
  b->ws = bind(layout, workspace, capacity);
  b->stream = static_cast<cudaStream_t>(stream);
  b->T = call->tokens;
  b->row_offset = call->row_offset;
  b->padding = call->padding;
  // Without a row-major sketch that the expert-major screen can read, the coordinate-major one is.
  if (screened && !layer->sketch && !screens_grouped(*b)) return CFM_E_NULL;
  return 0;
}

// Launch with programmatic stream serialisation: the kernel may be scheduled while its
// predecessor in the stream is finishing and waits for it at grid_dependency_wait().
// Used for every launch of a whole call (measured for two of them: 0.6 to 1.3 us per call).  CFM_PDL=0 in the environment makes these ordinary
// launches.
template <typename... Params, typename... Args>
static void launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, Args... args) {
  static const bool on = [] {
    const char* v = std::getenv("CFM_PDL");
    return !v || std::atoi(v) != 0;
  }();
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = on ? 1 : 0;
  (void)cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

static int launched() {
  const cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? 0 : static_cast<int>(err);
}

// Layers that have a row-major sketch screen expert-major (the kernels read it 16 bytes at a time).
static bool screens_grouped(const Bound& b) {
  return b.L.F < b.L.N && b.L.sketch_grouped &&
         ((reinterpret_cast<uintptr_t>(b.L.sketch_grouped) | reinterpret_cast<uintptr_t>(b.L.statistics)) & 15) == 0;
}
#include "cfm_rules.cuh"

static int group_smem(const Bound& b, size_t* smem) {
  *smem = std::max<size_t>(sizeof(int) * b.L.E, sizeof(float) * kPrepareThreads * 4);
  return *smem > 200 * 1024 ? CFM_E_SHAPE : 0;
}
static Routes routes_of(const Bound& b, const cfm_call* call) {
  Routes r = {};
  if (call) r = Routes{call->ids, call->weights, call->ids_are_int64, call->weights_are_bf16, 1, 0};
  r.lanes = 1;
  while (r.lanes < b.L.K) r.lanes *= 2;
  r.pass = pass_pairs(b);
  return r;
}

// Rotation of the input, or routing and grouping, or both in one launch.
static int run_prepare(const Bound& b, const cfm_call* call, bool rotate, bool group) {
  rotate = rotate && b.L.F < b.L.N;
  if (!rotate && !group) return 0;
  if (rotate && !call->hidden) return CFM_E_NULL;
  if (group && (!call->ids || !call->weights)) return CFM_E_NULL;
  size_t smem;
  const int rc = group_smem(b, &smem);
  if (rc) return rc;
  if (smem > 40 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(
        k_prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  constexpr int kPerCta = kPrepareThreads / 32;
  const int64_t ctas = rotate ? (static_cast<int64_t>(b.T) * b.L.B + kPerCta - 1) / kPerCta : 0;
  launch_dependent(k_prepare, dim3(static_cast<unsigned>(ctas + group)), dim3(kPrepareThreads), smem,
                   b.stream, b.L, b.ws, static_cast<const __nv_bfloat16*>(call->hidden), b.padding, b.T,
                   static_cast<int>(group), routes_of(b, call));
  return launched();
}

// Grouping after routes that another kernel wrote.
static int run_group(const Bound& b) {
  size_t smem;
  const int rc = group_smem(b, &smem);
  if (rc) return rc;
  if (smem > 40 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(
        k_group, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  k_group<<<1, kPrepareThreads, smem, b.stream>>>(b.L, b.ws, b.padding, b.T, routes_of(b, nullptr));
  return launched();
}

template <int CG>
static int launch_screen(const Bound& b, int S) {
  const int threads = b.L.W * CG;
  const size_t smem = sizeof(int) * (2 * kBlock + (CG > 1 ? CG * kWordRows * b.L.W : 0));
  if (smem > 48 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(
        k_screen<CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  k_screen<CG><<<dim3(b.T * b.L.K, S), threads, smem, b.stream>>>(b.L, b.ws, b.padding, S);
  return launched();
}

// As many CTAs as run at a time, at most `work` of them.
template <typename... Params, typename... Args>
static int launch_persistent(void (*kernel)(Params...), int64_t work, int per_sm, int threads, size_t smem,
                             cudaStream_t stream, Args... args) {
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
  if (err != cudaSuccess) return static_cast<int>(err);
  const unsigned ctas = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(work, 148 * per_sm)));
  launch_dependent(kernel, dim3(ctas), dim3(threads), smem, stream, args...);
  return launched();
}

// Rows of CTAs that clear dead pairs, eight pairs per CTA: with one row, six CTAs of the 128-expert layer walked
// all pairs of the call, and that was most of the screen on a rank of eight (256 tokens: 409 us, 28 now; 32 tokens 54 and 17).
static int dead_rows(int pairs, int columns) {
  return pairs ? std::min(std::max((pairs + 8 * columns - 1) / (8 * columns), 1), 64) : 0;
}

// `rows`: most passes of the call; `dead`: its pairs, where some may be dead.
template <int TOKENS, bool RISK>
static int launch_screen_tc(const Bound& b, int rows, int dead) {
  const size_t smem = Screen<TOKENS, RISK>::shared_bytes(b.L.B);
  const cudaError_t err = cudaFuncSetAttribute(
      k_screen_tc<TOKENS, RISK>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (err != cudaSuccess) return static_cast<int>(err);
  const int columns = (b.L.I + kScreenChannels - 1) / kScreenChannels, clearing = dead_rows(dead, columns);
  launch_dependent(k_screen_tc<TOKENS, RISK>, dim3(columns, rows + clearing), dim3(kScreenThreads), smem, b.stream,
                   b.L, b.ws, b.padding, dead, clearing);
  return launched();
}

template <int W>
static int launch_screen_tiles(const Bound& b, int rows, int dead) {
  using S = ScreenTiles<W>;
  const size_t smem = S::shared_bytes(b.L.B);
  if (smem > 40 * 1024) {
    const cudaError_t err = cudaFuncSetAttribute(
        k_screen_tiles<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  const int channels = 16 * S::kTiles, columns = (b.L.I + channels - 1) / channels, clearing = dead_rows(dead, columns);
  launch_dependent(k_screen_tiles<W>, dim3(columns, rows + clearing), dim3(S::kThreads), smem, b.stream, b.L, b.ws,
                   b.padding, dead, clearing);
  return launched();
}

static int run_screen_grouped(const Bound& b) {
  const int64_t pairs = static_cast<int64_t>(b.T) * b.L.K;
  const int dead = b.padding || b.L.expert_map ? static_cast<int>(pairs) : 0;
  const int pass = pass_pairs(b);
  const int rows = static_cast<int>(pairs / pass) + busy_experts(b);  // passes, at most
  if (screens_tc(b)) {
    const bool risk = b.L.score == CFM_SCORE_RECOVERY_AWARE;
    switch (pass) {
      case 4: return risk ? launch_screen_tc<4, true>(b, rows, dead) : launch_screen_tc<4, false>(b, rows, dead);
      case 8: return risk ? launch_screen_tc<8, true>(b, rows, dead) : launch_screen_tc<8, false>(b, rows, dead);
      default: return risk ? launch_screen_tc<16, true>(b, rows, dead) : launch_screen_tc<16, false>(b, rows, dead);
    }
  }
  // Four warps per tile: the calls that come here would not give every SM its sixteen with one each (one token
  // of the 128-expert layer 6.9 us against 12.3).  The products of a tile have to fit shared memory.
  if (b.L.B <= 128) return launch_screen_tiles<4>(b, rows, dead);
  return launch_screen_tiles<1>(b, rows, dead);
}

static int run_screen_projections(const Bound& b);

static int run_screen(const Bound& b) {
  if (b.L.F >= b.L.N) return 0;
  if (b.L.score == CFM_SCORE_RECOVERY_AWARE && !screens_grouped(b)) {
    k_variance<<<dim3(b.T * b.L.K, (2 * b.L.I + 255) / 256), 256, 0, b.stream>>>(b.L, b.ws,
                                                                                 b.padding);
    const int rc = launched();
    if (rc) return rc;
  }
  return run_screen_projections(b);
}

static int run_screen_projections(const Bound& b) {
  if (screens_grouped(b)) return run_screen_grouped(b);
  // Split the rotation blocks across CTAs while the batch is too small to fill
  // the 148 SMs; large batches keep each pair's blocks in one CTA.
  const int pairs = b.T * b.L.K;
  int S = 1;
  if (b.T <= b.ws.parts_tokens) {
    while (S < b.L.B && pairs * S < 2 * 148) S *= 2;
    if (S > b.L.B) S = b.L.B;
  }
  // Coordinate groups: as many as keep the CTA within 512 threads, at most 4.
  int cg = 4;
  while (cg > 1 && b.L.W * cg > 512) cg >>= 1;
  if (b.L.W > 512) return CFM_E_SHAPE;  // I > 4096
  switch (cg) {
    case 4: return launch_screen<4>(b, S);
    case 2: return launch_screen<2>(b, S);
    default: return launch_screen<1>(b, S);
  }
}

template <int PER>
static int launch_select(const Bound& b, int scores_ready, const Exchange* exchange, int account) {
  if (exchange)
    launch_dependent(k_select<true, PER>, dim3(b.T), dim3(kSelectThreads), 0, b.stream, b.L, b.ws,
                     b.padding, scores_ready, b.row_offset, account, static_cast<int>(encodes_by_union(b)), *exchange);
  else
    launch_dependent(k_select<false, PER>, dim3(b.T), dim3(kSelectThreads), 0, b.stream, b.L, b.ws,
                     b.padding, scores_ready, b.row_offset, account, static_cast<int>(encodes_by_union(b)), NoExchange{});
  return launched();
}

static int run_select(const Bound& b, int scores_ready, const Exchange* exchange, bool account) {
  const int per = (b.L.N + kSelectThreads - 1) / kSelectThreads;  // keys per thread
  if (per <= 2) return launch_select<2>(b, scores_ready, exchange, account);
  if (per <= 4) return launch_select<4>(b, scores_ready, exchange, account);
  if (per <= 6) return launch_select<6>(b, scores_ready, exchange, account);
  if (per <= 8) return launch_select<8>(b, scores_ready, exchange, account);
  if (per <= 12) return launch_select<12>(b, scores_ready, exchange, account);
  return launch_select<32>(b, scores_ready, exchange, account);
}

// The down tiles of the call in expert order, once the selection is done.
static int run_list_tiles(const Bound& b) {
  if (!pairs_grouped(b) || !b.L.down) return 0;  // a layer without native rows has no down stage
  k_list_tiles<<<1, 1024, 0, b.stream>>>(b.L, b.ws);
  return launched();
}

static int run_score(const Bound& b) {
  if (b.L.F >= b.L.N) return 0;
  k_score<<<dim3(b.T, (b.L.N + 255) / 256), 256, 0, b.stream>>>(b.L, b.ws, b.padding);
  return launched();
}

// `whole`: part of a whole call, which grouped the pairs and cleared the lists' lengths.
static int run_exact_union(const Bound& b, const cfm_call* call, bool whole) {
  if (!whole) {
    const cudaError_t err = cudaMemsetAsync(b.ws.work_counts + kExactCount, 0, 2 * sizeof(int32_t), b.stream);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  const int tiles = exact_union_tiles(b);
  const bool early = whole && b.L.F < b.L.N;  // a screen stands between the grouping and the selection
  launch_dependent(k_union, dim3(busy_experts(b)), dim3(kUnionThreads), 0, b.stream, b.L, b.ws, 8 * tiles,
                   DownUnion::kPass, static_cast<int>(early));
  const int rc = launched();
  if (rc) return rc;
  const int64_t pairs = static_cast<int64_t>(b.T) * b.L.K;
  const int64_t work = (pairs / (8 * tiles) + busy_experts(b)) * ((b.L.I + kUnionTile - 1) / kUnionTile);
  const int by_union = down_by_union(b), list = whole && !by_union;
  const auto* hidden = static_cast<const __nv_bfloat16*>(call->hidden);
  auto launch = [&](auto tile) {
    constexpr int NT = decltype(tile)::value;
    using X = ExactUnion<NT>;
    return launch_persistent(k_exact_union<NT>, work + list, X::kPerSm, X::kThreads, X::kSharedBytes, b.stream,
                             b.L, b.ws, hidden, by_union, list);
  };
  switch (tiles) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    default: return launch(std::integral_constant<int, 4>{});
  }
}

static int run_down_union(const Bound& b, bool encode, bool whole) {
  using X = DownUnion;
  if (!whole) {
    const cudaError_t err = cudaMemsetAsync(b.ws.work_counts + kDownNext, 0, sizeof(int32_t), b.stream);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  const int encoder_blocks = encode && encodes_by_union(b) ? (b.L.R + X::kColumns - 1) / X::kColumns : 0;
  const int64_t passes = static_cast<int64_t>(b.T) * b.L.K / X::kPass + busy_experts(b);
  return launch_persistent(k_down_union, (passes * (b.L.H / X::kColumns + encoder_blocks) + 3) / 4, X::kPerSm,
                           X::kThreads, X::kSharedBytes, b.stream, b.L, b.ws, encoder_blocks,
                           static_cast<uint32_t>((1ull << 32) / (b.L.H / X::kColumns) + 1));
}

// `whole`: part of a whole call; the down tiles are listed too where the down kernel needs them.
static int run_exact(const Bound& b, const cfm_call* call, bool whole) {
  if (!call->hidden || !b.L.gate_up) return CFM_E_NULL;
  if (exact_by_union(b)) return run_exact_union(b, call, whole);
  const size_t smem = static_cast<size_t>(b.L.H) * 2;
  if (smem > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(
        k_exact, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(k_exact_pairs<false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem));
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(k_exact_pairs<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem));
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  if (gathers_by_pair(b)) {
    const bool list = whole;
    // One warp per kept row of a pair when the pair keeps the mean number of rows.
    const int per_pair = (b.L.F + b.L.K - 1) / b.L.K;
    const int ctas = std::max(1, (per_pair + kExactWarps - 1) / kExactWarps);
    int64_t rows = static_cast<int64_t>(b.T) * b.L.K;
    if (b.L.expert_map && b.L.global_experts > 0)  // twice the expected share of the pairs
      rows = std::max<int64_t>(8, std::min<int64_t>(
                                      rows, (2 * rows * b.L.E + b.L.global_experts - 1) /
                                                b.L.global_experts));
    if (rows < static_cast<int64_t>(b.T) * b.L.K)
      launch_dependent(k_exact_pairs<true>, dim3(ctas, static_cast<unsigned>(rows + list)),
                       dim3(kExactWarps * 32), smem, b.stream, b.L, b.ws,
                       static_cast<const __nv_bfloat16*>(call->hidden),
                       static_cast<int>(list));
    else
      launch_dependent(k_exact_pairs<false>, dim3(ctas, static_cast<unsigned>(rows + list)),
                       dim3(kExactWarps * 32), smem, b.stream, b.L, b.ws,
                       static_cast<const __nv_bfloat16*>(call->hidden),
                       static_cast<int>(list));
    return launched();
  }
  int ctas = (b.L.F + kExactWarps - 1) / kExactWarps;
  if (b.L.expert_map && b.L.global_experts > 0) {
    // Expert parallel: a rank holds E of the global experts, so about that share
    // of a token's kept channels; CTAs stride through the list, twice the
    // expected share of them are launched.
    const int64_t share = (2LL * ctas * b.L.E + b.L.global_experts - 1) / b.L.global_experts;
    ctas = static_cast<int>(std::max<int64_t>(8, std::min<int64_t>(ctas, share)));
  }
  const int list = whole && pairs_grouped(b);
  launch_dependent(k_exact, dim3(ctas, b.T + list), dim3(kExactWarps * 32), smem, b.stream, b.L, b.ws,
                   static_cast<const __nv_bfloat16*>(call->hidden), b.padding, list);
  return launched();
}

// `encode`: run the recovery encoder too.  `whole`: part of a whole call.
static int run_down(const Bound& b, bool encode, bool whole) {
  if (!b.L.down) return CFM_E_NULL;
  if (down_by_union(b)) return run_down_union(b, encode, whole);
  // Tiles per token (T < 8) or of the call, at most; twice the expected share under expert
  // parallelism, walked in strides.
  const bool listed = pairs_grouped(b);
  int64_t tiles = listed ? static_cast<int64_t>(b.T) * ((b.L.F + kDownTileRows - 1) / kDownTileRows + b.L.K)
                         : (b.L.F + kDownTileRows - 1) / kDownTileRows + b.L.K - 1;
  const int64_t all = tiles;
  if (b.L.expert_map && b.L.global_experts > 0)
    tiles = std::max<int64_t>(listed ? 8 : 2, std::min<int64_t>(
        tiles, (2 * tiles * b.L.E + b.L.global_experts - 1) / b.L.global_experts));
  // Columns per CTA: finer until every SM has two CTAs of the tiles there will be about.
  const int64_t expected = static_cast<int64_t>(b.T) * (b.L.F / kDownTileRows + b.L.K / 2 + 1);
  int chunks = 4;
  while (chunks > 1 && expected * ((b.L.H + 256 * chunks - 1) / (256 * chunks)) < 2 * 148) chunks /= 2;
  DownGrid d = {};
  d.encode_ctas = encode ? b.T * b.L.K * b.ws.encoder_tiles : 0;
  if (encode && whole && shares_encoder(b)) {
    const int pass = pass_pairs(b);
    const int64_t passes = static_cast<int64_t>(b.T) * b.L.K / pass + busy_experts(b);
    d.encode_subs = pass / kEncodePairs;
    d.group_ctas = static_cast<int>(passes * d.encode_subs * b.ws.encoder_tiles);
    d.tokens = b.T;
    d.encode_ctas = d.group_ctas + (b.T + kEncodeThreads - 1) / kEncodeThreads;
  }
  d.columns = (b.L.H + 256 * chunks - 1) / (256 * chunks);
  d.tiles = static_cast<int>(tiles);
  const unsigned ctas = static_cast<unsigned>(d.encode_ctas + tiles * d.columns * (listed ? 1 : b.T));
  auto launch = [&](auto chunk) {
    constexpr int C = decltype(chunk)::value;
    if (listed)
      launch_dependent(k_down_tiles<C>, dim3(ctas), dim3(128), kDownRingBytes, b.stream, b.L, b.ws,
                       b.padding, d);
    else if (tiles < all)
      launch_dependent(k_down<true, C>, dim3(ctas), dim3(128), kDownRingBytes, b.stream, b.L, b.ws,
                       b.padding, d);
    else
      launch_dependent(k_down<false, C>, dim3(ctas), dim3(128), kDownRingBytes, b.stream, b.L, b.ws,
                       b.padding, d);
    return launched();
  };
  switch (chunks) {
    case 1: return launch(std::integral_constant<int, 1>{});
    case 2: return launch(std::integral_constant<int, 2>{});
    default: return launch(std::integral_constant<int, 4>{});
  }
}

static int run_encode(const Bound& b) {
  if (b.L.R == 0) return 0;
  if (b.L.F >= b.L.N) {
    k_zero_latent<<<b.T, 128, 0, b.stream>>>(b.L, b.ws);
    return launched();
  }
  k_encode<<<b.T * b.L.K * b.ws.encoder_tiles, kEncodeThreads, 0, b.stream>>>(b.L, b.ws, b.padding);
  return launched();
}

// `whole`: the last launch of a whole call.
static int run_output(const Bound& b, const cfm_call* call, bool whole) {
  if (!call->out) return CFM_E_NULL;
  const int latents = !whole || encodes(b);
  auto* out = static_cast<__nv_bfloat16*>(call->out);
  if (!mixes_tokens(b)) {
    launch_dependent(k_output, dim3(b.L.H / 128 + whole, b.T), dim3(128), 0, b.stream, b.L, b.ws, b.padding,
                     out, latents, static_cast<int>(whole));
    return launched();
  }
  const int mixed = whole && encodes_by_union(b) ? kLatentsFromSums : latents ? kLatentsGiven : kLatentsNone;
  const dim3 grid(b.L.H / 128 + whole, (b.T + kMixTokens - 1) / kMixTokens);
  if (down_by_union(b))
    launch_dependent(k_mix<false>, grid, dim3(128), 0, b.stream, b.L, b.ws, b.padding, b.T, out, mixed,
                     static_cast<int>(whole));
  else
    launch_dependent(k_mix<true>, grid, dim3(128), 0, b.stream, b.L, b.ws, b.padding, b.T, out, mixed,
                     static_cast<int>(whole));
  return launched();
}

// Checks an exchange description against the layer and the call (`rows` = tokens
// of all ranks) and makes the device-visible copy.
static int bind_exchange(const cfm_exchange* e, const cfm_layer* layer, int rows, Exchange* out) {
  if (!e || !layer) return CFM_E_NULL;
  if (e->world < 1 || e->world > CFM_MAX_RANKS || e->rank < 0 || e->rank >= e->world ||
      e->tokens < 1)
    return CFM_E_SHAPE;
  if (rows != e->world * e->tokens) return CFM_E_CAPACITY;
  out->world = e->world;
  out->rank = e->rank;
  out->tokens = e->tokens;
  for (int p = 0; p < CFM_MAX_RANKS; ++p) {
    out->block[p] = p < e->world ? static_cast<char*>(e->blocks[p]) : nullptr;
    if (p < e->world && !e->blocks[p]) return CFM_E_NULL;
  }
  return 0;
}

}  // namespace cfm

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace cfm;

extern "C" {

int cfm_abi_version(void) { return CFM_ABI_VERSION; }

const char* cfm_error_string(int code) {
  switch (code) {
    case 0: return "success";
    case CFM_E_NULL: return "a required pointer is NULL";
    case CFM_E_SHAPE: return "a dimension violates the layer contract";
    case CFM_E_CAPACITY: return "token count outside the workspace capacity";
    case CFM_E_UNSUPPORTED: return "option not supported by this build";
    case CFM_E_STATIC_CAPACITY: return "batch exceeds the library-owned scratch of cfm_screen_static";
    default: return code > 0 ? cudaGetErrorString(static_cast<cudaError_t>(code)) : "unknown error";
  }
}

int cfm_workspace_layout_for(const cfm_layer* layer, int32_t capacity,
                             cfm_workspace_layout* layout) {
  return make_layout(layer, capacity, layout);
}

#define CFM_STAGE(name, body)                                                      \
  int name(const cfm_layer* layer, void* workspace, int32_t capacity,             \
           const cfm_call* call, void* stream) {                                   \
    Bound b;                                                                       \
    const int rc = bind_call(layer, workspace, capacity, call, stream, &b);        \
    if (rc) return rc;                                                             \
    body                                                                           \
  }

CFM_STAGE(cfm_prepare_input, return run_prepare(b, call, true, false);)
CFM_STAGE(cfm_route, return run_prepare(b, call, false, true);)
CFM_STAGE(cfm_screen, return run_screen(b);)
CFM_STAGE(cfm_select, {
  // With an exchange in the call (home rank of an expert-parallel layer, plain
  // selection of its own rows) the kernel also sends the kept lists to all ranks.
  Exchange x = {};
  const bool send = call->exchange != nullptr && call->scores_ready == 0;
  if (send) {
    const int bound = bind_exchange(call->exchange, layer, call->exchange->world * b.T, &x);
    if (bound) return bound;
    if (b.row_offset != 0) return CFM_E_CAPACITY;
  }
  const int code = run_select(b, call->scores_ready, send ? &x : nullptr, true);
  // Mode 3 only publishes the cut; every other mode leaves final counts behind.
  return code || call->scores_ready == 3 ? code : run_list_tiles(b);
})
CFM_STAGE(cfm_score, return run_score(b);)
CFM_STAGE(cfm_list_tiles, return run_list_tiles(b);)
CFM_STAGE(cfm_exact, return run_exact(b, call, false);)
CFM_STAGE(cfm_down, return run_down(b, false, false);)
CFM_STAGE(cfm_encode, return run_encode(b);)
CFM_STAGE(cfm_output, return run_output(b, call, false);)

int cfm_partial_output(const cfm_layer* layer, void* workspace, int32_t capacity,
                       const cfm_call* call, void* stream) {
  Bound b;
  const int rc = bind_call(layer, workspace, capacity, call, stream, &b);
  if (rc) return rc;
  Exchange x = {};
  const int peers = call->exchange != nullptr;
  if (peers) {
    const int code = bind_exchange(call->exchange, layer, b.T, &x);
    if (code) return code;
  } else if (!call->out) {
    return CFM_E_NULL;
  }
  k_partial_output<<<dim3(peers ? (b.L.H + 511) / 512 : b.L.H / 128, b.T), 128, 0, b.stream>>>(
      b.L, b.ws, b.padding, static_cast<float*>(call->out),
      static_cast<int>(down_by_union(b)), x, peers);
  return launched();
}

int cfm_finish(const cfm_layer* layer, int32_t tokens, const float* combined,
               const float* latent, void* out, void* stream) {
  if (!layer || !combined || !out) return CFM_E_NULL;
  cfm_workspace_layout layout;
  const int rc = make_layout(layer, 1, &layout);  // validates the dimensions
  if (rc) return rc;
  if (tokens < 1) return CFM_E_CAPACITY;
  const Layer L = device_layer(layer);
  k_finish<<<dim3(L.H / 128, tokens), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      L, combined, latent, static_cast<__nv_bfloat16*>(out));
  return launched();
}

int cfm_adopt(const cfm_layer* layer, void* workspace, int32_t capacity, const cfm_call* call,
              void* stream) {
  Bound b;
  const int rc = bind_call(layer, workspace, capacity, call, stream, &b);
  if (rc) return rc;
  if (!call->ids || !call->weights || (!call->lists && !call->exchange)) return CFM_E_NULL;
  Exchange x = {};
  const int peers = call->exchange != nullptr;
  if (peers) {
    const int bound = bind_exchange(call->exchange, layer, b.T, &x);
    if (bound) return bound;
  }
  k_adopt<<<b.T, 256, 0, b.stream>>>(b.L, b.ws, call->ids, call->ids_are_int64, call->weights,
                                     call->weights_are_bf16, b.padding, call->lists, x, peers);
  const int code = launched();
  // The exact and down kernels read the pairs grouped by expert; the down tiles are
  // listed by cfm_list_tiles, which may run beside cfm_exact.
  return code || !pairs_grouped(b) ? code : run_group(b);
}

int cfm_build_sketch(const cfm_layer* layer, const void* gate_up, const int8_t* signs,
                     uint32_t* sketch, uint32_t* sketch_grouped, void* statistics, void* stream) {
  if (!layer || !gate_up || !signs || !sketch || !sketch_grouped || !statistics) return CFM_E_NULL;
  const int64_t H = layer->hidden, I = layer->width, E = layer->experts;
  if (H <= 0 || H % kBlock || I <= 0 || I % 16 || E < 1 || E > 65535 || 2 * I / kBuildRows > 65535)
    return CFM_E_SHAPE;
  const int64_t row_tiles = (2 * I / kBuildRows + kBuildWarps - 1) / kBuildWarps;
  const dim3 grid(static_cast<unsigned>(H / kBlock), static_cast<unsigned>(row_tiles),
                  static_cast<unsigned>(E));
  k_build_sketch<<<grid, kBuildWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<int>(H), static_cast<int>(I), static_cast<const __nv_bfloat16*>(gate_up), signs,
      sketch, sketch_grouped, static_cast<__half*>(statistics));
  return launched();
}

int64_t cfm_exchange_bytes(const cfm_layer* layer, int32_t world, int32_t tokens) {
  if (!layer || world < 1 || world > CFM_MAX_RANKS || tokens < 1) return 0;
  return static_cast<int64_t>(
      exchange_bytes(world, tokens, layer->final_count, layer->hidden));
}

int cfm_peer_alloc(int64_t bytes, void** block) {
  if (!block || bytes < 1) return CFM_E_NULL;
  cudaError_t err = cudaMalloc(block, static_cast<size_t>(bytes));
  if (err == cudaSuccess) err = cudaMemset(*block, 0, static_cast<size_t>(bytes));
  if (err == cudaSuccess) err = cudaDeviceSynchronize();
  return static_cast<int>(err);
}

int cfm_peer_export(void* block, void* handle) {
  if (!block || !handle) return CFM_E_NULL;
  static_assert(sizeof(cudaIpcMemHandle_t) == CFM_PEER_HANDLE_BYTES, "handle size");
  return static_cast<int>(
      cudaIpcGetMemHandle(static_cast<cudaIpcMemHandle_t*>(handle), block));
}

int cfm_peer_import(const void* handle, void** block) {
  if (!block || !handle) return CFM_E_NULL;
  cudaIpcMemHandle_t copy;
  memcpy(&copy, handle, sizeof(copy));
  return static_cast<int>(cudaIpcOpenMemHandle(block, copy, cudaIpcMemLazyEnablePeerAccess));
}

int cfm_peer_release(void* block, int32_t imported) {
  if (!block) return 0;
  return static_cast<int>(imported ? cudaIpcCloseMemHandle(block) : cudaFree(block));
}

int cfm_exchange_status(const cfm_exchange* exchange, int32_t* status) {
  if (!exchange || !status || exchange->rank < 0 || exchange->rank >= CFM_MAX_RANKS ||
      !exchange->blocks[exchange->rank])
    return CFM_E_NULL;
  uint32_t word = 0;
  const cudaError_t err = cudaMemcpy(
      &word, static_cast<const uint32_t*>(exchange->blocks[exchange->rank]) + kExchangeStatus,
      sizeof(word), cudaMemcpyDeviceToHost);
  *status = static_cast<int32_t>(word);
  return static_cast<int>(err);
}

int cfm_finish_rows(const cfm_layer* layer, const cfm_exchange* exchange, const float* latent,
                    void* out, void* stream) {
  if (!layer || !exchange || !out) return CFM_E_NULL;
  cfm_workspace_layout layout;
  const int rc = make_layout(layer, 1, &layout);  // validates the dimensions
  if (rc) return rc;
  Exchange x = {};
  const int bound = bind_exchange(exchange, layer, exchange->world * exchange->tokens, &x);
  if (bound) return bound;
  const Layer L = device_layer(layer);
  k_finish_rows<<<dim3(L.H / 128, x.tokens), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      L, x, latent, static_cast<__nv_bfloat16*>(out));
  return launched();
}

int cfm_reader_forward(const cfm_layer* layer, void* workspace, int32_t capacity,
                       const cfm_call* call, void* stream) {
  Bound b;
  int rc = bind_call(layer, workspace, capacity, call, stream, &b);
  if (rc) return rc;
  if (!layer->gate_up || !layer->down) return CFM_E_NULL;
  if ((rc = run_prepare(b, call, !call->input_prepared, true))) return rc;
  if ((rc = run_screen(b))) return rc;
  if ((rc = run_select(b, 0, nullptr, false))) return rc;
  if ((rc = run_exact(b, call, true))) return rc;
  if ((rc = run_down(b, encodes(b), true))) return rc;
  return run_output(b, call, true);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Screen with library-owned scratch (no allocation by anyone at call time)
// ---------------------------------------------------------------------------
// Scratch of cfm_screen_static: the per-block products of the split screen and
// its arrival counters.  The arrays live in the library image, so every GPU
// that loads the library holds them (4 MiB + 4 KiB) until the process exits.
// All calls on a device share them.
static __device__ __align__(256) float g_static_parts[CFM_STATIC_PARTS_FLOATS];
static __device__ __align__(256) unsigned int g_static_counters[CFM_STATIC_MAX_PAIRS];

namespace {
constexpr int kMaxDevices = 64;
struct StaticScratch {
  float* parts;
  unsigned int* counters;
  bool ready;
};
StaticScratch g_scratch[kMaxDevices];
std::mutex g_scratch_lock;

// Resolves the device addresses of the two arrays for the current device.  In
// host code the array names are only handles; kernels need the addresses
// cudaGetSymbolAddress returns for the device that is current.
int static_scratch(StaticScratch* out) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return static_cast<int>(err);
  if (device < 0 || device >= kMaxDevices) return CFM_E_UNSUPPORTED;
  std::lock_guard<std::mutex> guard(g_scratch_lock);
  StaticScratch& slot = g_scratch[device];
  if (!slot.ready) {
    void* parts = nullptr;
    void* counters = nullptr;
    err = cudaGetSymbolAddress(&parts, g_static_parts);
    if (err != cudaSuccess) return static_cast<int>(err);
    err = cudaGetSymbolAddress(&counters, g_static_counters);
    if (err != cudaSuccess) return static_cast<int>(err);
    slot.parts = static_cast<float*>(parts);
    slot.counters = static_cast<unsigned int*>(counters);
    slot.ready = true;
  }
  *out = slot;
  return 0;
}
}  // namespace

extern "C" int cfm_screen_static(const cfm_layer* layer, const cfm_static_screen* io,
                                 void* stream) {
  if (!layer || !io) return CFM_E_NULL;
  if (!io->ids || !io->quantized || !io->coordinates || !io->exponents || !io->partial ||
      !layer->sketch || !layer->statistics)
    return CFM_E_NULL;
  cfm_workspace_layout layout;
  int rc = make_layout(layer, 1, &layout);  // validates the dimensions
  if (rc) return rc;
  const Layer L = device_layer(layer);
  if (L.F >= L.N) return CFM_E_SHAPE;  // unscreened plans have no screen
  if (L.W > 512) return CFM_E_SHAPE;
  if (io->tokens < 1) return CFM_E_CAPACITY;
  const int64_t pairs = static_cast<int64_t>(io->tokens) * L.K;
  if (pairs > CFM_STATIC_MAX_PAIRS ||
      pairs * L.B * 2 * L.I > static_cast<int64_t>(CFM_STATIC_PARTS_FLOATS))
    return CFM_E_STATIC_CAPACITY;
  StaticScratch scratch;
  if ((rc = static_scratch(&scratch))) return rc;

  Workspace ws = {};
  ws.ids = const_cast<int32_t*>(io->ids);
  ws.quantized = const_cast<int32_t*>(io->quantized);
  ws.coordinates = const_cast<int32_t*>(io->coordinates);
  ws.exponents = const_cast<int32_t*>(io->exponents);
  ws.parts = scratch.parts;
  ws.counters = scratch.counters;
  ws.partial = io->partial;
  ws.parts_tokens = io->tokens;
  ws.capacity = io->tokens;
  Bound b;
  b.L = L;
  b.ws = ws;
  b.stream = static_cast<cudaStream_t>(stream);
  b.T = io->tokens;
  b.row_offset = 0;
  b.padding = io->padding;
  // The arrival counters must start at zero; the products need no clearing
  // (every entry that is read has been written by this call).
  const cudaError_t err = cudaMemsetAsync(scratch.counters, 0, sizeof(unsigned int) * pairs,
                                          b.stream);
  if (err != cudaSuccess) return static_cast<int>(err);
  // The recovery-aware score also reads the residual variances of the projections;
  // that kernel needs no scratch and runs when the caller asks for them.
  if (io->variances) {
    if (!io->energies) return CFM_E_NULL;
    b.ws.norms = const_cast<float*>(io->energies);
    b.ws.variances = io->variances;
    k_variance<<<dim3(b.T * L.K, (2 * L.I + 255) / 256), 256, 0, b.stream>>>(b.L, b.ws, b.padding);
    if ((rc = launched())) return rc;
  }
  // Always split the rotation blocks across CTAs, so the scratch is what joins them.
  int S = 2;
  while (S < L.B && pairs * S < 2 * 148) S *= 2;
  if (S > L.B) S = L.B;
  if (L.B == 1) S = 1;
  int cg = 4;
  while (cg > 1 && L.W * cg > 512) cg >>= 1;
  switch (cg) {
    case 4: return launch_screen<4>(b, S);
    case 2: return launch_screen<2>(b, S);
    default: return launch_screen<1>(b, S);
  }
}
