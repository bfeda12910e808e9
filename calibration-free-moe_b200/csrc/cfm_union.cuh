// Expert-major exact gate/up, down and recovery-encoder products on the tensor cores (sm_100a).
//
// The (token, expert) pairs of a call are grouped by expert.  The kernels here walk one expert at
// a time: a row of its weights that several of its tokens kept is read once, as one operand of
// m16n8k16 BF16 matrix instructions whose other operand holds the tokens, eight to a tile.
// Products for tokens that did not keep the row come out of the same instruction and are dropped.
//
//   k_union         per expert the union of its tokens' kept channels; work lists
//   k_exact_union   gate and up rows of the unions
//   k_down_union    channel-major down rows of the unions; recovery-encoder rows
//   k_mix           router mix of the expert sums, latent, decoder term, BF16 store
//
// The tensor cores are not there for their rate (they idle nine tenths of the time) but for their
// instruction count: per row and eight tokens a matrix instruction replaces some fifty loads,
// conversions and FMAs, which is what gathers per token are bound by once tokens share experts.
// A token's gate and up sums depend on its own row and the weights only, in an order fixed by H
// (quarters of H, columns ascending inside a quarter); its down sums go sixteen union rows at a
// time and depend in their last FP32 bits on the channels the other tokens of an expert kept.
// The exact and down kernels are persistent and take their work from flat lists, so experts of
// very different load keep all SMs busy, and their copies run ahead from one piece of work into
// the next.  Included by cfm_reader.cu inside namespace cfm.
#pragma once

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 8 bytes global -> shared memory in the thread's current cp.async group.
__device__ __forceinline__ void copy_async8(uint32_t shared, const void* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(shared), "l"(global) : "memory");
}
__device__ __forceinline__ uint2 load_shared8(uint32_t address) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(address) : "memory");
  return v;
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t (&a)[4], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(address)
               : "memory");
}

// ---------------------------------------------------------------------------
// unions and work lists
// ---------------------------------------------------------------------------
constexpr int kUnionThreads = 128;
constexpr int kUnionStagedPairs = 128;  // pairs of an expert whose numbers a CTA stages

// One piece of work of the exact kernel (tile `tile` of expert e's union for `count` pairs from
// `first` of the grouped list) or of the down kernel (`tile` unused).  The union has `rows`
// channels.
struct __align__(32) UnionWork {
  int e, first, count, tile, rows;
};

__device__ __forceinline__ UnionWork load_work(const UnionWork* p) {
  const int4 a = *reinterpret_cast<const int4*>(p);
  return UnionWork{a.x, a.y, a.z, a.w, reinterpret_cast<const int*>(p)[4]};
}

// Word w (channels 32 w ..) of the kept channels of slot `slot` of a token whose kept candidates
// are `bits`; the slot's candidates begin at a multiple of sixteen.
__device__ __forceinline__ uint32_t slot_word(const uint32_t* bits, int I, int slot, int w) {
  const int at = slot * I + 32 * w;
  uint32_t word = bits[at >> 5];
  if (at & 31) word = __funnelshift_r(word, bits[(at >> 5) + 1], 16);
  return 32 * w + 32 > I ? word & 0xffffu : word;
}

// grid (busy experts), 128 threads.  A CTA makes the union of its expert's kept channels from the
// tokens' masks (one OR and one scan over I / 32 words), leaves the channels behind and appends the
// expert's tiles of sixteen channels x passes of `exact_pass` tokens and its passes of `down_pass`
// tokens to the work lists.  With `early` the grouping is known to be complete when this grid can
// start at all, and is read while the selection still runs.  (When every exact CTA made its
// expert's union itself, the dependent loads and the scan cost each of them some 5 us, a third of
// its life at 64 tokens of the 128-expert layer.)
__global__ void __launch_bounds__(kUnionThreads)
    k_union(Layer L, Workspace ws, int exact_pass, int down_pass, int early) {
  __shared__ int scratch[33];
  __shared__ int staged[kUnionStagedPairs];
  __shared__ int s_base[2];
  const int tid = threadIdx.x, words = (L.I + 31) / 32, token_words = kept_words(L.N);
  if (!early) grid_dependency_wait();
  const bool live = static_cast<int>(blockIdx.x) < ws.work_counts[kBusyCount];
  int e = 0, first = 0, total = 0;
  if (live) {
    e = ws.busy_experts[blockIdx.x];
    first = ws.group_offsets[e];
    total = ws.group_offsets[e + 1] - first;
  }
  for (int j = tid; j < min(total, kUnionStagedPairs); j += kUnionThreads)
    staged[j] = ws.group_pairs[first + j];
  if (early) grid_dependency_wait();  // the selection is complete
  grid_dependency_release();
  if (!live) return;
  __syncthreads();
  auto word_of = [&](int pair, int w) {
    const int t = pair / L.K;
    return slot_word(ws.kept_bits + static_cast<size_t>(t) * token_words, L.I, pair - t * L.K, w);
  };
  uint16_t* channels = ws.union_channels + static_cast<size_t>(e) * L.I;
  int rows = 0;
  for (int w0 = 0; w0 < words; w0 += kUnionThreads) {
    const int w = w0 + tid;
    uint32_t mask = 0;
    if (w < words) {
      const int quick = min(total, kUnionStagedPairs);
#pragma unroll 8
      for (int j = 0; j < quick; ++j) mask |= word_of(staged[j], w);
      for (int j = quick; j < total; ++j) mask |= word_of(ws.group_pairs[first + j], w);
    }
    int all = 0;
    int at = rows + block_exclusive_scan(__popc(mask), scratch, &all);
    for (; mask; mask &= mask - 1, ++at)
      channels[at] = static_cast<uint16_t>(32 * w + __ffs(mask) - 1);
    rows += all;
  }
  const int tiles = (rows + 15) / 16;
  const int exact_passes = (total + exact_pass - 1) / exact_pass;
  const int down_passes = (total + down_pass - 1) / down_pass;
  if (tid == 0) {
    s_base[0] = atomicAdd(ws.work_counts + kExactCount, tiles * exact_passes);
    s_base[1] = atomicAdd(ws.work_counts + kDownCount, down_passes);
  }
  __syncthreads();
  for (int i = tid; i < tiles * exact_passes; i += kUnionThreads) {
    const int pass = i % exact_passes;  // the passes of a tile run next to each other
    ws.exact_work[s_base[0] + i] =
        UnionWork{e, first + pass * exact_pass, min(exact_pass, total - pass * exact_pass),
                  i / exact_passes, rows};
  }
  for (int i = tid; i < down_passes; i += kUnionThreads)
    ws.down_work[s_base[1] + i] =
        UnionWork{e, first + i * down_pass, min(down_pass, total - i * down_pass), 0, rows};
}

// ---------------------------------------------------------------------------
// exact
// ---------------------------------------------------------------------------
// A tile is sixteen union rows of gate and up against NT x 8 tokens; its columns are cut into
// quarters of H, one per warp.  Per step of 32 columns lane (g, tq) takes 16 bytes (eight columns)
// of rows g and g + 8, gate and up, and of its tokens' rows, copies them into a ring in shared
// memory with cp.async and reads them back itself: it waits for its own copies only, and the ring
// needs no barrier.  The instruction's column order is free as long as both operands agree, so the
// eight columns serve as columns 2 tq, 2 tq + 1, 2 tq + 8, 2 tq + 9 of two instructions.  The
// tokens' rows travel with the weights because the ring leaves L1 too small to hold them.  (Loads
// straight into registers were issued one by one: 76 us at 64 tokens of the 128-expert layer, 54
// with the ring; the gathers per token take 69.)
template <int NT>
struct ExactUnion {
  static constexpr int kThreads = 128;
  static constexpr int kPass = 8 * NT;
  static constexpr int kSlots = 4;    // steps in the ring
  static constexpr int kStepBytes = (4 + NT) * 512;
  static constexpr int kRingBytes = 4 * kSlots * kStepBytes;
  static constexpr int kSumFloats = NT * 2 * 4 * 32;  // of a quarter
  static constexpr int kSharedBytes = kRingBytes + 4 * kSumFloats * 4;
  // CTAs per SM: bound by shared memory (227 KB, 1 KB of it per CTA) and registers.
  static constexpr int kPerSm = NT == 1 ? 5 : NT == 2 ? 3 : 2;
};

// Where a lane's pieces of a tile come from.
template <int NT>
struct ExactSource {
  const char *a, *b, *x[NT];
};

// `by_candidate`: activations go to their candidates' places, for the tile-wise down kernel.
template <int NT>
__global__ void __launch_bounds__(ExactUnion<NT>::kThreads, ExactUnion<NT>::kPerSm)
    k_exact_union(Layer L, Workspace ws, const __nv_bfloat16* hidden, int by_candidate) {
  using X = ExactUnion<NT>;
  constexpr int kSlots = X::kSlots;
  extern __shared__ __align__(1024) uint8_t union_shared[];
  grid_dependency_wait();     // the work list is complete
  grid_dependency_release();  // the down kernel may be scheduled: it reads the lists at once
  const int work_count = ws.work_counts[kExactCount];
  int index = blockIdx.x;
  if (index >= work_count) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  const int column = warp * (L.H / 4) + 8 * tq;
  const int steps = L.H / 128;  // of a quarter
  const int padded = (steps + kSlots - 1) / kSlots * kSlots;
  const size_t up_bytes = static_cast<size_t>(L.I) * L.H * 2;
  const int token_words = kept_words(L.N);
  const uint32_t mine = shared_u32(union_shared) + warp * (kSlots * X::kStepBytes) + lane * 16;
  float* red = reinterpret_cast<float*>(union_shared + X::kRingBytes);

  auto read_work = [&](int i) {
    return i < work_count ? load_work(ws.exact_work + i) : UnionWork{0, 0, 0, 0, 0};
  };
  auto locate = [&](const UnionWork& w) {  // rows beyond the union repeat its last one
    ExactSource<NT> s;
    const uint16_t* channels = ws.union_channels + static_cast<size_t>(w.e) * L.I;
    const int last = w.rows - 1, row = w.tile * 16 + g;
    const char* weights = reinterpret_cast<const char*>(
        L.gate_up + static_cast<size_t>(w.e) * 2 * L.I * L.H + column);
    s.a = weights + static_cast<size_t>(channels[min(row, last)]) * L.H * 2;
    s.b = weights + static_cast<size_t>(channels[min(row + 8, last)]) * L.H * 2;
#pragma unroll
    for (int n = 0; n < NT; ++n) {  // columns beyond the pass repeat its last token
      const int pair = ws.group_pairs[w.first + min(8 * n + g, w.count - 1)];
      s.x[n] = reinterpret_cast<const char*>(hidden + static_cast<size_t>(pair / L.K) * L.H + column);
    }
    return s;
  };
  auto copy = [&](int slot, const ExactSource<NT>& s, int offset) {
    const uint32_t to = mine + slot * X::kStepBytes;
    copy_async16(to, s.a + offset);
    copy_async16(to + 512, s.b + offset);
    copy_async16(to + 1024, s.a + up_bytes + offset);
    copy_async16(to + 1536, s.b + up_bytes + offset);
#pragma unroll
    for (int n = 0; n < NT; ++n) copy_async16(to + 512 * (4 + n), s.x[n] + offset);
  };

  UnionWork work = read_work(index), next = read_work(index + gridDim.x);
  ExactSource<NT> source = locate(work);
#pragma unroll
  for (int j = 0; j < kSlots - 1; ++j) {
    if (j < steps) copy(j, source, 64 * j);
    copy_async_commit();  // also when empty: the group count per step stays fixed
  }
  for (;;) {
    const bool more = index + static_cast<int>(gridDim.x) < work_count;
    // What the end of the tile needs, and where the next one's rows are, on their way early.
    const int at = work.tile * 16 + g + 8 * (warp >> 1);
    const bool finishes = at < work.rows;
    const int channel =
        finishes ? ws.union_channels[static_cast<size_t>(work.e) * L.I + at] : 0;
    uint32_t bits[NT];
    int pairs[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int token = 8 * n + 2 * tq + (warp & 1);
      bits[n] = 0;
      pairs[n] = 0;
      if (finishes && token < work.count) {
        pairs[n] = ws.group_pairs[work.first + token];
        const int t = pairs[n] / L.K, candidate = (pairs[n] - t * L.K) * L.I + channel;
        bits[n] = ws.kept_bits[static_cast<size_t>(t) * token_words + (candidate >> 5)] >> (candidate & 31);
      }
    }
    ExactSource<NT> next_source = source;
    if (more) next_source = locate(next);
    const UnionWork after = read_work(index + 2 * gridDim.x);

    float acc[NT][2][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][0][i] = acc[n][1][i] = 0.0f;
#pragma unroll 1
    for (int s = 0; s < padded; s += kSlots) {
      const bool last = s + kSlots >= padded;
#pragma unroll
      for (int j = 0; j < kSlots; ++j) {
        copy_async_wait<kSlots - 2>();  // this lane's copies of step s + j have landed
        const bool live = s + j < steps;
        uint4 w[4], t[NT];
        if (live) {
          const uint32_t from = mine + j * X::kStepBytes;
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] = load_shared16(from + 512 * i);
#pragma unroll
          for (int n = 0; n < NT; ++n) t[n] = load_shared16(from + 512 * (4 + n));
        }
        // Refill the place read one step ago.
        if (j == 0) {
          if (s + kSlots - 1 < steps) copy(kSlots - 1, source, 64 * (s + kSlots - 1));
        } else if (!last) {
          if (s + kSlots + j - 1 < steps) copy(j - 1, source, 64 * (s + kSlots + j - 1));
        } else if (more && j - 1 < steps) {
          copy(j - 1, next_source, 64 * (j - 1));
        }
        copy_async_commit();
        if (live) {
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            mma_bf16(acc[n][0], w[0].x, w[1].x, w[0].y, w[1].y, t[n].x, t[n].y);
            mma_bf16(acc[n][1], w[2].x, w[3].x, w[2].y, w[3].y, t[n].x, t[n].y);
            mma_bf16(acc[n][0], w[0].z, w[1].z, w[0].w, w[1].w, t[n].z, t[n].w);
            mma_bf16(acc[n][1], w[2].z, w[3].z, w[2].w, w[3].w, t[n].z, t[n].w);
          }
        }
      }
    }
    // Sums of the quarters: [quarter][tile of tokens][gate, up][accumulator register][lane].
    float* own = red + warp * X::kSumFloats + lane;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        own[(n * 8 + i) * 32] = acc[n][0][i];
        own[(n * 8 + 4 + i) * 32] = acc[n][1][i];
      }
    __syncthreads();
    // Thread (register, lane): the quarters in order, then the feature, or zero for a channel the
    // token did not keep.
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int token = 8 * n + 2 * tq + (warp & 1);
      if (!finishes || token >= work.count) continue;
      const bool kept = bits[n] & 1u;
      float feature = 0.0f;
      if (kept) {
        float gate = 0.0f, up = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* sums = red + q * X::kSumFloats + lane;
          gate += sums[(n * 8 + warp) * 32];
          up += sums[(n * 8 + 4 + warp) * 32];
        }
        feature = exact_feature(gate, up, L.activation);
      }
      if (!by_candidate)
        ws.activations[static_cast<size_t>(work.first + token) * L.I + at] = __float2bfloat16_rn(feature);
      else if (kept)
        ws.activations[static_cast<size_t>(pairs[n]) * L.I + channel] = __float2bfloat16_rn(feature);
    }
    if (!more) break;
    __syncthreads();  // the sums may be overwritten
    index += gridDim.x;
    work = next;
    next = after;
    source = next_source;
  }
}
