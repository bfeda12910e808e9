// Expert-major screen: int8 tensor-core dots of sketch rows with fixed-point tokens (sm_100a).
//
// The (token, expert) pairs are grouped by expert into passes (k_prepare).  A pass's tokens are
// the columns of the product, three base-256 digits each; the sketch rows' 2-bit codes are its
// rows, as unsigned bytes 0, 1, 2 (trit + 1), so decoding is a mask and a shift per four codes,
// and the product is corrected by the sum of the token's values.  Products are exact int32 sums;
// each rotation block's is rescaled in FP32 and added in block order, as the reference does, so
// results do not depend on which kernel or split computed them.  A kernel here has both
// projections of its channels in hand at the end, so it also computes what follows from them
// alone: the selection score and the feature the recovery encoder takes for a skipped channel
// (one CTA per token did that in the selection: 10 us of its 25 for one token).
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

// Codes of four coordinates as bytes; m = 0 .. 3 gives coordinates {0, 2, 8, 10}, {4, 6, 12, 14},
// {1, 3, 9, 11}, {5, 7, 13, 15} of a word of the row-major layout.  The digits of a token are
// stored in the same order (digit_byte).
__device__ __forceinline__ uint32_t codes_of(uint32_t word, int m) {
  return (word >> (2 * m)) & 0x03030303u;
}

// d += (A: unsigned codes) x (B: signed digits), m16n8k32.
__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 2^(e - 21): undoes the fixed point of a block.
__device__ __forceinline__ float unscale_of(int e) {
  return __uint_as_float(static_cast<uint32_t>(127 + e - kQuantBits) << 23);
}

// What a channel brings to its candidates' scores.
struct CandidateFactors {
  float norm;
  float2 geometry;
};
__device__ __forceinline__ CandidateFactors candidate_factors(const Layer& L, int e, int c) {
  const size_t channel = static_cast<size_t>(e) * L.I + c;
  return CandidateFactors{L.norms[channel],
                          L.score != CFM_SCORE_POINT && L.geometry
                              ? reinterpret_cast<const float2*>(L.geometry)[channel]
                              : make_float2(0.0f, 0.0f)};
}

// What the selection and the recovery encoder take from a live candidate's projections (and
// their residual variances): channel c, slot `pair` = (token, slot).
__device__ __forceinline__ void finish_candidate(const Layer& L, const Workspace& ws, int pair, int c,
                                                 const CandidateFactors& f, float gate, float up,
                                                 float gate_variance, float up_variance) {
  const size_t at = static_cast<size_t>(pair) * L.I + c;  // N = K I: candidate slot * I + c of the token
  const float weight = ws.weights[pair];
  const float active = pinned_activate(bf16_round(gate), L.activation);
  ws.features[at] = __float2bfloat16_rn(sketch_feature(active, up));
  ws.scores[at] = L.score == CFM_SCORE_POINT
                      ? point_score(active, up, f.norm, weight)
                      : risk_score(gate, active, up, gate_variance, up_variance, f.norm, f.geometry.x, f.geometry.y,
                                   weight, L.activation);
}

// Residual variances of a channel's projections: per block, in block order, the row's FP16
// residual variance times the energy of the token's kept coordinates.
__device__ __forceinline__ float2 channel_variance(const Layer& L, const Workspace& ws, int t, int e,
                                                   int c) {
  const size_t rows = 2 * static_cast<size_t>(L.I);
  const __half* gate = L.statistics + (static_cast<size_t>(e) * L.B * 2 + 1) * rows + c;
  const float* energy = ws.norms + static_cast<size_t>(t) * L.B;
  float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll 4
  for (int b = 0; b < L.B; ++b, gate += 2 * rows) {
    sum.x = __fadd_rn(sum.x, __fmul_rn(__half2float(gate[0]), energy[b]));
    sum.y = __fadd_rn(sum.y, __fmul_rn(__half2float(gate[L.I]), energy[b]));
  }
  return sum;
}

// Stores the projections of channel c for a pair and finishes the candidate.
__device__ __forceinline__ void store_candidate(const Layer& L, const Workspace& ws, int pair, int t,
                                                int e, int c, float gate, float up) {
  // Projections of a token: gate plane, up plane, N = K I each; (t K + slot) I = pair I.
  const size_t at = static_cast<size_t>(t) * L.N + static_cast<size_t>(pair) * L.I + c;
  ws.partial[at] = gate;
  ws.partial[at + L.N] = up;
  float2 variance = make_float2(0.0f, 0.0f);
  if (L.score != CFM_SCORE_POINT) {
    variance = channel_variance(L, ws, t, e, c);
    ws.variances[at] = variance.x;
    ws.variances[at + L.N] = variance.y;
  }
  finish_candidate(L, ws, pair, c, candidate_factors(L, e, c), gate, up, variance.x, variance.y);
}

// The last rows of CTAs of a screen, `rows` of them: zero the projections of every remote or padded pair
// of the call, a pair at a time by all threads of a CTA.
__device__ __forceinline__ void clear_dead(const Layer& L, const Workspace& ws, const uint8_t* padding, int pairs,
                                           int rows) {
  const int row = blockIdx.y - (gridDim.y - rows);
  for (int p = row * gridDim.x + blockIdx.x; p < pairs; p += rows * gridDim.x) {
    const int t = p / L.K;
    if (ws.ids[p] >= 0 && !(padding && padding[t])) continue;
    // I is a multiple of 16, and so is the offset of a pair.
    float4* gate = reinterpret_cast<float4*>(ws.partial + static_cast<size_t>(t) * L.N + static_cast<size_t>(p) * L.I);
    for (int i = threadIdx.x; i < L.I / 4; i += blockDim.x)
      gate[i] = gate[L.N / 4 + i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// ---------------------------------------------------------------------------
// warp-level products (mma.sync)
// ---------------------------------------------------------------------------
// A tile is sixteen channels of an expert, their gate and up rows, against up to eight tokens.
// W warps share it, warp w taking rotation blocks w, w + W, ...; lane (g, tq) holds coordinates
// 32 tq .. + 31 of rows g and g + 8 of both and of token g's digits.  Digits come straight from
// global memory (L1 resident, 32 contiguous bytes each), codes and scales through a ring of the
// warp's own in shared memory, four blocks deep, filled with cp.async.  (Requested from L2 with
// bulk prefetches they cost some 25 cycles of the SM's copy engine per 512 bytes: 25 us at 8
// tokens of the 128-expert layer.)  With W = 1 the projections stay in registers; otherwise the
// blocks' products meet in shared memory and are added there in block order.
// Bound by the integer ALU (58 % busy), the L1 reads of the digits and the latency between them:
// some 160 cycles of an SM per 32 rows x 128 coordinates x 8 tokens, whatever the split.
template <int W>
struct ScreenTiles {
  static constexpr int kWarps = 4;
  static constexpr int kTiles = kWarps / W;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kStages = 4;
  static constexpr int kStageBytes = 1024 + 64;  // codes of 32 rows, their scales
  static constexpr int kRingBytes = kWarps * kStages * kStageBytes;
  static size_t shared_bytes(int B) {
    return kRingBytes + (W > 1 ? static_cast<size_t>(kTiles) * B * 256 * sizeof(float) : 0);
  }
};

// grid (ceil(I / (16 tiles)), most passes of eight tokens); `dead_rows` more rows of CTAs clear the
// projections of the dead ones of the call's `pairs`.
template <int W>
__global__ void __launch_bounds__(ScreenTiles<W>::kThreads, 16 / ScreenTiles<W>::kWarps)
    k_screen_tiles(Layer L, Workspace ws, const uint8_t* padding, int pairs, int dead_rows) {
  using S = ScreenTiles<W>;
  extern __shared__ __align__(128) uint8_t tiles_shared[];
  float* products = reinterpret_cast<float*>(tiles_shared + S::kRingBytes);  // [tile][block][8][lane]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  grid_dependency_wait();     // the digits and the passes are complete
  grid_dependency_release();  // the selection may be scheduled; it waits for this grid
  const int I = L.I, B = L.B, rows = 2 * I;
  if (blockIdx.y + dead_rows >= gridDim.y) {
    clear_dead(L, ws, padding, pairs, dead_rows);
    return;
  }
  if (static_cast<int>(blockIdx.y) >= ws.work_counts[kPassCount]) return;
  const int4 pass = *reinterpret_cast<const int4*>(ws.pass_work + blockIdx.y);
  const int e = pass.x, first = pass.y, count = pass.z;
  const int part = warp % W, c0 = (blockIdx.x * S::kTiles + warp / W) * 16;
  const bool inside = c0 < I;
  if (W == 1 && !inside) return;

  // This lane's 16-byte pieces of a block: of the gate and the up codes (512 contiguous bytes
  // each), and, in four lanes, of the scales.
  const size_t code_step = static_cast<size_t>(rows) * 32, scale_step = static_cast<size_t>(rows) * 4;
  const uint8_t* codes = reinterpret_cast<const uint8_t*>(L.sketch_grouped) +
                         (static_cast<size_t>(e) * B + part) * code_step + c0 * 32 + lane * 16;
  const uint8_t* scales = reinterpret_cast<const uint8_t*>(L.statistics) +
                          (static_cast<size_t>(e) * B + part) * scale_step +
                          ((lane & 2 ? I : 0) + c0 + 8 * (lane & 1)) * 2;
  uint8_t* ring = tiles_shared + warp * (S::kStages * S::kStageBytes);
  const uint32_t ring_address = shared_u32(ring) + lane * 16;
  int fetched = part, fetch_stage = 0;
  auto fetch = [&]() {  // the next block of this warp
    if (inside && fetched < B) {
      const uint32_t to = ring_address + fetch_stage * S::kStageBytes;
      copy_async16(to, codes);
      copy_async16(to + 512, codes + static_cast<size_t>(I) * 32);
      if (lane < 4) copy_async16(to + 1024, scales);
      codes += W * code_step;
      scales += W * scale_step;
      fetched += W;
    }
    fetch_stage = (fetch_stage + 1) % S::kStages;
    copy_async_commit();  // also when empty: one group per block
  };
#pragma unroll
  for (int i = 0; i < S::kStages - 1; ++i) fetch();
  // Columns beyond the pass repeat its first token.
  const int pair_g = ws.group_pairs[first + (g < count ? g : 0)];
  const int token_g = pair_g / L.K;
  const int pair_0 = __shfl_sync(kFull, pair_g, 8 * tq), pair_1 = __shfl_sync(kFull, pair_g, 8 * tq + 4);
  const int token_0 = __shfl_sync(kFull, token_g, 8 * tq), token_1 = __shfl_sync(kFull, token_g, 8 * tq + 4);

  const uint4* digits = reinterpret_cast<const uint4*>(
      ws.limbs + (static_cast<size_t>(token_g) * B + part) * 3 * kBlock + 32 * tq);
  const int2* factors_0 = reinterpret_cast<const int2*>(ws.exponents) + static_cast<size_t>(token_0) * B + part;
  const int2* factors_1 = reinterpret_cast<const int2*>(ws.exponents) + static_cast<size_t>(token_1) * B + part;
  float run[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  float* mine = products + (static_cast<size_t>(warp / W) * B + part) * 256 + lane;
  auto compute = [&](const uint8_t* stage) {
    uint4 digit[3][2];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      digit[j][0] = digits[j * (kBlock / 16)];
      digit[j][1] = digits[j * (kBlock / 16) + 1];
    }
    const int2 f0 = *factors_0, f1 = *factors_1;  // exponent, sum of the values
    digits += W * 3 * kBlock / 16;
    factors_0 += W;
    factors_1 += W;
    const float unscale[2] = {unscale_of(f0.x), unscale_of(f1.x)};
#pragma unroll
    for (int tile = 0; tile < 2; ++tile) {
      const uint8_t* from = stage + 512 * tile + g * 32 + tq * 8;
      const uint2 a = *reinterpret_cast<const uint2*>(from);
      const uint2 b = *reinterpret_cast<const uint2*>(from + 256);
      const __half* scale = reinterpret_cast<const __half*>(stage + 1024) + 16 * tile + g;
      const float scales[2] = {__half2float(scale[0]), __half2float(scale[8])};
      // code = trit + 1: the sum of the values is taken off where the first sum starts.
      int acc[3][4] = {{-f0.y, -f1.y, -f0.y, -f1.y}, {0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t a0 = codes_of(a.x, m), a1 = codes_of(b.x, m);
        const uint32_t a2 = codes_of(a.y, m), a3 = codes_of(b.y, m);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const uint4 lo = digit[j][0], hi = digit[j][1];
          mma_u8s8(acc[j], a0, a1, a2, a3, m == 0 ? lo.x : m == 1 ? lo.y : m == 2 ? lo.z : lo.w,
                   m == 0 ? hi.x : m == 1 ? hi.y : m == 2 ? hi.z : hi.w);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int dot = acc[0][i] + acc[1][i] * 256 + acc[2][i] * 65536;
        const float d = __fmul_rn(__int2float_rn(dot), unscale[i & 1]);
        const float product = __fmul_rn(scales[i >> 1], d);
        if (W == 1) run[4 * tile + i] = __fadd_rn(run[4 * tile + i], product);
        else mine[(4 * tile + i) * 32] = product;
      }
    }
    if (W > 1) mine += W * 256;
  };
  if (inside) {
    int stage = 0;
    for (int b = part; b < B; b += W) {
      copy_async_wait<S::kStages - 2>();
      __syncwarp();  // the block has landed, for all lanes; all have read the one before it
      fetch();       // into that one's place
      compute(ring + stage * S::kStageBytes);
      stage = (stage + 1) % S::kStages;
    }
  }
  if (W == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (2 * tq + (i & 1) < count)
        store_candidate(L, ws, (i & 1) ? pair_1 : pair_0, (i & 1) ? token_1 : token_0, e,
                        c0 + g + 8 * (i >> 1), run[i], run[4 + i]);
    return;
  }
  __syncthreads();
  // Warp `part` of a tile finishes registers part, part + W of the tile's lanes.
  if (!inside) return;
  for (int i = part; i < 4; i += W) {
    if (2 * tq + (i & 1) >= count) continue;
    const float* from = products + static_cast<size_t>(warp / W) * B * 256 + i * 32 + lane;
    float gate = 0.0f, up = 0.0f;
#pragma unroll 8
    for (int b = 0; b < B; ++b, from += 256) {
      gate = __fadd_rn(gate, from[0]);
      up = __fadd_rn(up, from[128]);
    }
    store_candidate(L, ws, (i & 1) ? pair_1 : pair_0, (i & 1) ? token_1 : token_0, e,
                    c0 + g + 8 * (i >> 1), gate, up);
  }
}
