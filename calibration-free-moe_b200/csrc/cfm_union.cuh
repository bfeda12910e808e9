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
//   k_mix           output of large batches: router mix, latent, decoder term, BF16 store, counters
//
// The tensor cores are not there for their rate (they idle nine tenths of the time) but for their
// instruction count: per row and eight tokens a matrix instruction replaces some fifty loads,
// conversions and FMAs, which is what gathers per token are bound by once tokens share experts.
// A token's gate and up sums depend on its own row and the weights only, in an order fixed by H
// (quarters of H, columns ascending inside a quarter), and round as the gathers' do; its down and
// encoder sums go sixteen union rows at a time and depend in their last FP32 bits on the channels
// the other tokens of an expert kept, which is why k_down_union runs on request only.
// The exact and down kernels are persistent and take their work from flat lists, so experts of
// very different load keep all SMs busy, and their copies run ahead from one piece of work into
// the next.  Included by cfm_reader.cu inside namespace cfm.
#pragma once

// d = a b, and d += a b.
__device__ __forceinline__ void mma_bf16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
               "{%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
               "{%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Copies and loads at a fixed distance from a shared-memory address, which the instruction adds.
// (With `bytes` 0 instead of 16 nothing is read and zeros are written.)
template <int AT, int FROM>
__device__ __forceinline__ void copy_async16_at(uint32_t shared, const void* global, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0+%2], [%1+%3], 16, %4;" ::"r"(shared), "l"(global), "n"(AT), "n"(FROM),
               "r"(bytes)
               : "memory");
}
template <int AT>
__device__ __forceinline__ void copy_async16_at(uint32_t shared, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0+%2], [%1], 16;" ::"r"(shared), "l"(global), "n"(AT) : "memory");
}
template <int AT>
__device__ __forceinline__ void copy_async8_at(uint32_t shared, const void* global) {
  asm volatile("cp.async.ca.shared.global [%0+%2], [%1], 8;" ::"r"(shared), "l"(global), "n"(AT) : "memory");
}
template <int AT>
__device__ __forceinline__ uint2 load_shared8_at(uint32_t address) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(address), "n"(AT) : "memory");
  return v;
}
template <int AT>
__device__ __forceinline__ void load_matrices_at(uint32_t (&a)[4], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4+%5];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(address), "n"(AT)
               : "memory");
}
template <int AT>
__device__ __forceinline__ void load_matrices_transposed_at(uint32_t (&a)[4], uint32_t address) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4+%5];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(address), "n"(AT)
               : "memory");
}
template <int I>
struct Index {
  static constexpr int value = I;
  __host__ __device__ constexpr operator int() const { return I; }
};
// f(0), f(1), ... f(N - 1) with the index as a constant.
template <int N, int I = 0, typename F>
__device__ __forceinline__ void repeat(F&& f) {
  if constexpr (I < N) {
    f(Index<I>{});
    repeat<N, I + 1>(f);
  }
}

// ---------------------------------------------------------------------------
// unions and work lists
// ---------------------------------------------------------------------------
constexpr int kUnionTile = 32;  // rows of a tile of the exact kernel
constexpr int kUnionThreads = 512;
constexpr int kUnionStagedPairs = 512;  // pairs of an expert whose numbers a CTA stages

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

// grid (busy experts), 512 threads.  A CTA makes the union of its expert's kept channels from the
// tokens' masks (one OR and one scan over I / 32 words), leaves the channels behind and appends the
// expert's tiles of 32 channels x passes of `exact_pass` tokens and its passes of `down_pass`
// tokens to the work lists.  With `early`, in whole calls with a screen, the grouping is read while
// the selection still runs: this grid cannot start before every CTA of the selection has, those not
// before every CTA of the screen has released them, and the screen's CTAs release after their wait
// for k_prepare.  The selection itself releases before it waits, so without a screen nothing orders
// this grid's start behind the grouping, and the wait comes first.  (When every exact CTA made its
// expert's union itself, the dependent loads and the scan cost each of them some 5 us, a third of
// its life at 64 tokens of the 128-expert layer.)
__global__ void __launch_bounds__(kUnionThreads)
    k_union(Layer L, Workspace ws, int exact_pass, int down_pass, int early) {
  __shared__ int scratch[33];
  __shared__ int staged[kUnionStagedPairs];
  __shared__ uint32_t masks[kUnionThreads];
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
  // Few words leave threads over: groups of them share the pairs.
  int lanes = 32;
  while (lanes < words && lanes < kUnionThreads) lanes *= 2;
  const int groups = kUnionThreads / lanes, group = tid / lanes;
  int rows = 0;
  for (int w0 = 0; w0 < words; w0 += kUnionThreads) {
    const int w = w0 + tid - group * lanes;
    uint32_t mask = 0;
    if (w < words) {
      const int quick = min(total, kUnionStagedPairs);
      int j = group;
#pragma unroll 8
      for (; j < quick; j += groups) mask |= word_of(staged[j], w);
      for (; j < total; j += groups) mask |= word_of(ws.group_pairs[first + j], w);
    }
    if (groups > 1) {
      masks[tid] = mask;
      __syncthreads();
      mask = 0;
      if (group == 0)
        for (int i = 0; i < groups; ++i) mask |= masks[i * lanes + tid];
    }
    int all = 0;
    int at = rows + block_exclusive_scan(__popc(mask), scratch, &all);
    for (; mask; mask &= mask - 1, ++at)
      channels[at] = static_cast<uint16_t>(32 * w + __ffs(mask) - 1);
    rows += all;
  }
  const int tiles = (rows + kUnionTile - 1) / kUnionTile;
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
// A tile is 32 union rows of gate and up against NT x 8 tokens; its columns are cut into
// quarters of H, one per warp.  Per step of 32 columns lane (g, tq) copies 16 bytes (eight columns)
// of rows g, g + 8, g + 16 and g + 24, gate and up, and of its tokens' rows into a ring of the warp's own with
// cp.async; the matrix loads read them from there as the instruction wants them.  A row's four
// pieces are permuted by the row, so that the eight rows of a matrix lie in different banks.  The
// tokens' rows travel with the weights because the ring leaves L1 too small to hold them.  The
// instruction truncates where an FMA rounds, so a sum leaves it after 128 columns and goes on by
// ordinary additions (RMS error of a gate sum of 2048 columns against FP64: 8.0e-7 without, 4.1e-7
// with, 2.1e-7 the gathers').  The sums are rounded to BF16 next; where the distance between the two
// ways of summing could change a rounding (kExactMargin), the CTA lists the row and repeats the
// product as the gathers do it when the list is full and at its end, so that the activations are
// those of the gathers.
// Bound by the latency of its copies: two warps per scheduler, of 13 cycles per issued instruction four
// waiting for copies, three for the queue of memory instructions, half a one at barriers; 15 % of the
// way from L2 to the SMs, DRAM 57 % at 64 tokens of the 128-expert layer (63 us; 69 the gathers per
// token).  100 tokens of the 64-expert layer 95 us (132), 256 of the 256-expert layer 90 (155), 256 of
// hidden 4096 and width 1536 616 at 5 TB/s of HBM (1431); without the repeats 61, 89, 80 and 580.
template <int NT>
struct ExactUnion {
  static constexpr int kThreads = 128;
  static constexpr int kPass = 8 * NT;
  static constexpr int kSlots = 4;    // steps in the ring
  static constexpr int kStepBytes = (8 + NT) * 512;
  static constexpr int kRingBytes = 4 * kSlots * kStepBytes;
  static constexpr int kSumFloats = NT * 2 * 4 * 32;  // of a quarter, for half of the rows
  static constexpr int kSharedBytes = kRingBytes + 4 * kSumFloats * 4;
  static constexpr int kPerSm = 2;  // CTAs per SM: bound by shared memory (227 KB, 1 KB of it per CTA)
};

// Where a lane's pieces of a tile come from: rows g, g + 8, g + 16, g + 24 and the tokens, as
// numbers and as pointers.
template <int NT>
struct ExactRows {
  int e, channel[4], token[NT];
};
template <int NT>
struct ExactSource {
  const char *gate[4], *x[NT];
};

// Rows to be repeated that a CTA lists before it repeats them.
constexpr int kRepeats = 64;

// Largest distance of the two ways of summing a gate or up row that is provided for, in units of the
// row sums' size: per token the largest sum, over eight rows and both matrices, of the quarters'
// magnitudes.  Other rows than the sum's own count because a quarter whose large terms cancel would
// say nothing about the roundings inside it.  A measured margin, not a bound: over hidden sizes of
// 1024 to 4096 the distance was 0.04 of it RMS and 0.37 at most in seven million sums of normal, outlier
// and Student-t inputs, 0.94 where 98 % of every two adjacent terms of all rows cancel.  One row in a
// hundred is repeated for it.
constexpr float kExactMargin = 1.0f / (1 << 19);

// Whether an error of `margin` could round v to another BF16 value.
__device__ __forceinline__ bool rounds_either_way(float v, float margin) {
  return bf16_round(v - margin) != bf16_round(v + margin);
}

// `by_union`: activations also go to their union rows, for k_down_union.  With `list` one more CTA,
// the first, lists the down tiles for the tile-wise down kernel.
template <int NT>
__global__ void __launch_bounds__(ExactUnion<NT>::kThreads, ExactUnion<NT>::kPerSm)
    k_exact_union(Layer L, Workspace ws, const __nv_bfloat16* hidden, int by_union, int list) {
  using X = ExactUnion<NT>;
  constexpr int kSlots = X::kSlots;
  extern __shared__ __align__(128) uint8_t union_shared[];
  __shared__ int2 repeats[kRepeats];  // place in the grouped list; channel, and row of the union above it
  __shared__ int repeat_count;
  static_assert(sizeof(repeats) >= 33 * sizeof(int), "scratch of the listing");
  grid_dependency_wait();     // the work list is complete
  grid_dependency_release();  // the down kernel may be scheduled: its encoder needs no more than that
  if (list && blockIdx.x == 0) {
    list_down_tiles(L, ws, reinterpret_cast<int*>(repeats));
    return;
  }
  const int work_count = ws.work_counts[kExactCount], stride = gridDim.x - list;
  int index = blockIdx.x - list;
  if (index >= work_count) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  const int column = warp * (L.H / 4) + 8 * tq;
  const int steps = L.H / 128;  // of a quarter
  const int padded = (steps + kSlots - 1) / kSlots * kSlots;
  const size_t up_bytes = static_cast<size_t>(L.I) * L.H * 2;
  const int token_words = kept_words(L.N);
  const uint32_t ring = shared_u32(union_shared) + warp * (kSlots * X::kStepBytes);
  const uint32_t mine = ring + 64 * g + 16 * (tq ^ ((g >> 1) & 3));
  // Where this lane's row of a matrix lies: of the first operand (rows 0 to 7 and 8 to 15 of the
  // first eight columns, then of the next; the other sixteen columns 32 bytes away by xor), and of
  // the second (a token's four pieces).
  const int r = lane & 7, matrix = lane >> 3;
  const uint32_t weights_at = ring + (matrix & 1) * 512 + 64 * r + 16 * ((matrix >> 1) ^ ((r >> 1) & 3));
  const uint32_t weights_at2 = weights_at ^ 32;
  const uint32_t tokens_at = ring + 64 * r + 16 * (matrix ^ ((r >> 1) & 3));
  float* red = reinterpret_cast<float*>(union_shared + X::kRingBytes);

  auto read_work = [&](int i) {
    return i < work_count ? load_work(ws.exact_work + i) : UnionWork{0, 0, 0, 0, 0};
  };
  auto locate = [&](const UnionWork& w) {  // rows beyond the union repeat its last one
    ExactRows<NT> at;
    const uint16_t* channels = ws.union_channels + static_cast<size_t>(w.e) * L.I;
    at.e = w.e;
#pragma unroll
    for (int i = 0; i < 4; ++i) at.channel[i] = channels[min(w.tile * kUnionTile + 8 * i + g, w.rows - 1)];
#pragma unroll
    for (int n = 0; n < NT; ++n)  // columns beyond the pass repeat its last token
      at.token[n] = ws.group_pairs[w.first + min(8 * n + g, w.count - 1)];
    return at;
  };
  auto point = [&](const ExactRows<NT>& at) {
    ExactSource<NT> s;
    const char* weights = reinterpret_cast<const char*>(
        L.gate_up + static_cast<size_t>(at.e) * 2 * L.I * L.H + column);
    const uint32_t row_bytes = 2 * L.H;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      s.gate[i] = weights + static_cast<uint64_t>(static_cast<uint32_t>(at.channel[i])) * row_bytes;
#pragma unroll
    for (int n = 0; n < NT; ++n)
      s.x[n] = reinterpret_cast<const char*>(hidden + column) +
               static_cast<uint64_t>(static_cast<uint32_t>(at.token[n]) / static_cast<uint32_t>(L.K)) * row_bytes;
    return s;
  };
  // Step `step` from where the source's pointers stand, into place `slot` of the ring
  // (zeros where the quarter has no such step).
  auto copy = [&](auto slot, const ExactSource<NT>& s, auto step, bool there) {
    const int bytes = there ? 16 : 0;
    constexpr int kTo = decltype(slot)::value * X::kStepBytes, kFrom = 64 * decltype(step)::value;
    repeat<4>([&](auto i) {
      constexpr int kPlace = kTo + 512 * ((decltype(i)::value >> 1) * 4 + (decltype(i)::value & 1));
      copy_async16_at<kPlace, kFrom>(mine, s.gate[i], bytes);
      copy_async16_at<kPlace + 1024, kFrom>(mine, s.gate[i] + up_bytes, bytes);
    });
    repeat<NT>([&](auto n) { copy_async16_at<kTo + 512 * (8 + decltype(n)::value), kFrom>(mine, s.x[n], bytes); });
  };

  // The first `count` rows on the list, one per warp at a time, as the gathers do them.
  auto repeat_listed = [&](int count) {
    for (int i = warp; i < count; i += 4) {
      const int position = repeats[i].x, channel = repeats[i].y & 0xffff, at = repeats[i].y >> 16;
      const int pair = ws.group_pairs[position], t = pair / L.K;
      const int candidate = (pair - t * L.K) * L.I + channel;
      const size_t word = static_cast<size_t>(t) * token_words + (candidate >> 5);
      const int place = ws.kept_before[word] + __popc(ws.kept_bits[word] & ((1u << (candidate & 31)) - 1));
      const int chunks = L.H / 8;
      const uint4* gate = reinterpret_cast<const uint4*>(L.gate_up) +
                          (static_cast<size_t>(ws.ids[pair]) * 2 * L.I + channel) * chunks;
      uint4 gw[kExactSweep], uw[kExactSweep];
      float g_sum, u_sum;
      exact_dot(gate, gate + static_cast<size_t>(L.I) * chunks,
                reinterpret_cast<const uint4*>(hidden) + static_cast<size_t>(t) * chunks, chunks, lane, false, gw,
                uw, g_sum, u_sum);
      if (lane == 0) {
        const __nv_bfloat16 feature = __float2bfloat16_rn(exact_feature(g_sum, u_sum, L.activation));
        ws.activations[static_cast<size_t>(pair) * L.I + channel] = feature;
        if (by_union) ws.union_activations[static_cast<size_t>(position) * L.I + at] = feature;
        float* exact = ws.exact + static_cast<size_t>(t) * 2 * L.F + place;
        exact[0] = g_sum;
        exact[L.F] = u_sum;
      }
    }
  };
  if (tid == 0) repeat_count = 0;  // ordered by the barriers of the first tile
  UnionWork work = read_work(index), next = read_work(index + stride);
  ExactRows<NT> rows = locate(work);
  ExactSource<NT> source = point(rows);
  repeat<kSlots - 1>([&](auto j) {
    copy(j, source, j, j < steps);
    copy_async_commit();
  });
  for (;;) {
    const bool more = index + stride < work_count;
    // What the end of the tile needs, and where the next one's rows are, on their way early.  There
    // this thread has row g or g + 8 and a token that another lane has located.
    int pairs[NT];
    uint32_t bits[2][NT];    // the kept bits of the candidate's word
    uint16_t before[2][NT];  // kept channels of the token before the word
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      pairs[n] = __shfl_sync(kFull, rows.token[n], 4 * (2 * tq + (warp & 1)));
      const int t = pairs[n] / L.K;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int channel = warp < 2 ? rows.channel[2 * half] : rows.channel[2 * half + 1];
        const int candidate = (pairs[n] - t * L.K) * L.I + channel;
        const size_t word = static_cast<size_t>(t) * token_words + (candidate >> 5);
        bits[half][n] = ws.kept_bits[word];
        before[half][n] = ws.kept_before[word];
      }
    }
    ExactRows<NT> next_rows = {};
    if (more) next_rows = locate(next);
    const UnionWork after = read_work(index + 2 * stride);

    uint32_t doubt = 0;  // of this thread's sums: bit half * NT + n
    float acc[2][NT][2][4];  // [rows][tokens][gate, up]
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[half][n][0][i] = acc[half][n][1][i] = 0.0f;
#pragma unroll 1
    for (int s = 0; s < padded; s += kSlots) {
      const bool last = s + kSlots >= padded;
      float part[2][NT][2][4];  // of this turn of the ring
      // The last turn's copies, but for its first, are the next tile's: the pointers go on there.
      repeat<kSlots>([&](auto turn) {
        constexpr int j = decltype(turn)::value;
        constexpr Index<(j + kSlots - 1) % kSlots> free{};
        copy_async_wait<kSlots - 2>();
        __syncwarp();  // every lane's copies of step s + j have landed; the step before has been read
        // Refill the place read one step ago.
        if (j == 1 && last && more) source = point(next_rows);
        if (j == 0 || !last) {
          copy(free, source, Index<kSlots + j - 1>{}, s + kSlots + j - 1 < steps);
        } else if (more) {
          copy(free, source, Index<(j > 0 ? j - 1 : 0)>{}, j - 1 < steps);
        }
        copy_async_commit();
        constexpr int kFrom = j * X::kStepBytes;
        uint32_t t[NT][4];
        repeat<NT>([&](auto n) { load_matrices_at<kFrom + 512 * (8 + decltype(n)::value)>(t[n], tokens_at); });
        repeat<2>([&](auto h) {
          constexpr int half = decltype(h)::value, kRows = kFrom + 2048 * half;
          uint32_t w[4][4];
          load_matrices_at<kRows>(w[0], weights_at);
          load_matrices_at<kRows + 1024>(w[1], weights_at);
          load_matrices_at<kRows>(w[2], weights_at2);
          load_matrices_at<kRows + 1024>(w[3], weights_at2);
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            if (j == 0) {
              mma_bf16_first(part[half][n][0], w[0], t[n][0], t[n][1]);
              mma_bf16_first(part[half][n][1], w[1], t[n][0], t[n][1]);
            } else {
              mma_bf16(part[half][n][0], w[0], t[n][0], t[n][1]);
              mma_bf16(part[half][n][1], w[1], t[n][0], t[n][1]);
            }
            mma_bf16(part[half][n][0], w[2], t[n][2], t[n][3]);
            mma_bf16(part[half][n][1], w[3], t[n][2], t[n][3]);
          }
        });
      });
      if (!last) {
#pragma unroll
        for (int i = 0; i < 4; ++i) source.gate[i] += 64 * kSlots;
#pragma unroll
        for (int n = 0; n < NT; ++n) source.x[n] += 64 * kSlots;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            acc[half][n][0][i] += part[half][n][0][i];
            acc[half][n][1][i] += part[half][n][1][i];
          }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      // Sums of the quarters: [quarter][tile of tokens][gate, up][accumulator register][lane].
      float* own = red + warp * X::kSumFloats + lane;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          own[(n * 8 + i) * 32] = acc[half][n][0][i];
          own[(n * 8 + 4 + i) * 32] = acc[half][n][1][i];
        }
      __syncthreads();
      // Thread (register, lane): the quarters in order, then the feature, or zero for a channel the
      // token did not keep.
      const int at = work.tile * kUnionTile + 16 * half + g + 8 * (warp >> 1);
      const int channel = warp < 2 ? rows.channel[2 * half] : rows.channel[2 * half + 1];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int token = 8 * n + 2 * tq + (warp & 1);
        float gate[4], up[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float* sums = red + q * X::kSumFloats + lane;
          gate[q] = sums[(n * 8 + warp) * 32];
          up[q] = sums[(n * 8 + 4 + warp) * 32];
        }
        float size = fmaxf((fabsf(gate[0]) + fabsf(gate[1])) + (fabsf(gate[2]) + fabsf(gate[3])),
                           (fabsf(up[0]) + fabsf(up[1])) + (fabsf(up[2]) + fabsf(up[3])));
#pragma unroll
        for (int w = 4; w < 32; w <<= 1) size = fmaxf(size, __shfl_xor_sync(kFull, size, w));
        if (at >= work.rows || token >= work.count) continue;
        __nv_bfloat16 feature = __float2bfloat16_rn(0.0f);
        const int t = pairs[n] / L.K, bit = ((pairs[n] - t * L.K) * L.I + channel) & 31;
        if ((bits[half][n] >> bit) & 1u) {
          const float g_sum = (gate[0] + gate[1]) + (gate[2] + gate[3]);
          const float u_sum = (up[0] + up[1]) + (up[2] + up[3]);
          feature = __float2bfloat16_rn(exact_feature(g_sum, u_sum, L.activation));
          ws.activations[static_cast<size_t>(pairs[n]) * L.I + channel] = feature;
          float* exact = ws.exact + static_cast<size_t>(t) * 2 * L.F + before[half][n] +
                         __popc(bits[half][n] & ((1u << bit) - 1));
          exact[0] = g_sum;
          exact[L.F] = u_sum;
          const float margin = kExactMargin * size;
          if (rounds_either_way(g_sum, margin) || rounds_either_way(u_sum, margin))
            doubt |= 1u << (half * NT + n);
        }
        if (by_union) ws.union_activations[static_cast<size_t>(work.first + token) * L.I + at] = feature;
      }
      if (half == 0) __syncthreads();  // the sums may be overwritten
    }
    for (;;) {
      for (; doubt; doubt &= doubt - 1) {
        const int place = atomicAdd(&repeat_count, 1);
        if (place >= kRepeats) break;
        const int bit = __ffs(doubt) - 1, half = bit / NT, n = bit - half * NT;
        const int channel = warp < 2 ? (half ? rows.channel[2] : rows.channel[0])
                                     : (half ? rows.channel[3] : rows.channel[1]);
        repeats[place] = make_int2(work.first + 8 * n + 2 * tq + (warp & 1),
                                   channel | (work.tile * kUnionTile + 16 * half + g + 8 * (warp >> 1)) << 16);
      }
      // The sums may be overwritten, the list is complete, what the tile left for its rows is written.
      __syncthreads();
      const int listed = repeat_count;
      if (more && listed <= kRepeats) break;
      repeat_listed(min(listed, kRepeats));
      if (listed <= kRepeats) return;
      __syncthreads();
      if (tid == 0) repeat_count = 0;
      __syncthreads();
    }
    index += stride;
    work = next;
    next = after;
    rows = next_rows;
  }
}

// ---------------------------------------------------------------------------
// down, and the recovery encoder
// ---------------------------------------------------------------------------
// D[token][column] = sum over union rows: sixteen tokens' activations (zero where a token did not
// keep the row) of sixteen rows are the instruction's first operand, the rows' weights of eight
// columns the second.  A warp takes one piece of work on its own: 64 columns of one pass over one
// expert, all the union's rows, sixteen (a unit) at a time through a ring of cp.async copies that
// runs on into its next piece.  The matrix loads transpose the weights on their way to registers;
// rows lie 144 bytes apart, which keeps the eight of a matrix in different banks.  Union row
// 4 a + 2 b + i of a unit is the instruction's row 8 b + 2 a + i, so that a lane's four activations
// are adjacent in memory.  Rows beyond the union are another row's weights and meet zeros.
// The instruction truncates, so a sum leaves it after four units and goes on by ordinary additions
// (of 786,432 sums over 1536 rows 92 round to another BF16 value than the sum in 64 bits does, 90 of
// the gathers' and 819 of one chain).
// The recovery encoder is the same product with an expert's whole width as its rows and the sketch
// features (zero for kept channels, k_select) as activations; its pieces, the longest, come first.
// Pieces differ in length with the unions and the number of passes, so warps claim them one at a
// time (the next one while the current one's copies run): with fixed strides half of the SMs were
// idle while the longest pieces ended (85 us at 256 tokens of the 256-expert layer, 55 with claims;
// the tiles per token take 79).  Bound by latency and instruction issue: 126 instructions per unit of
// 2 KB.  256 tokens of hidden 4096 and width 1536 373 us at 4.7 TB/s of HBM (651 the tiles per token).
// A row with a weight that is not finite would meet the zeros of tokens that did not keep it and leave
// them NaN: sums that are NaN are repeated over the token's own rows, as the tiles add them.
struct DownUnion {
  static constexpr int kThreads = 128;
  static constexpr int kPass = 16;
  static constexpr int kColumns = 64;
  static constexpr int kPerSm = 3;  // four would spill in the loop: 1577 us for 1525 at the widest, 297 for 285
  static constexpr int kSlots = 5;
  static constexpr int kRowBytes = 144;
  static constexpr int kUnitBytes = 16 * kRowBytes;
  static constexpr int kFold = 4;  // units after which a sum leaves the tensor cores
  static constexpr int kSlotBytes = kUnitBytes + 512;
  static constexpr int kSharedBytes = 4 * kSlots * kSlotBytes;
};

// The lane with the `index`-th of the bits, or -1.
__device__ __forceinline__ int lane_of_bit(unsigned bits, int index) {
  for (; index > 0; --index) bits &= bits - 1;
  return __ffs(bits) - 1;
}

// One column of a pair's down sum as down_tile and the output add it: tiles of 64 of the `rows` kept
// candidates of `list`, four chains of every fourth row in a tile.  Four adjacent lanes per sum, one
// chain each; all lanes of the warp call it (with no rows: for nothing).  `weights`: the column in the
// row of candidate 0.
__device__ __forceinline__ float repeat_down_sum(const int32_t* list, const __nv_bfloat16* values,
                                              const __nv_bfloat16* weights, int H, int rows) {
  const int lane = threadIdx.x & 31, base = lane & ~3;
  const int most = __reduce_max_sync(kFull, rows);
  float sum = 0.0f;
  for (int r0 = 0; r0 < most; r0 += kDownTileRows) {
    float chain = 0.0f;
    for (int r = r0 + (lane & 3); r < min(rows, r0 + kDownTileRows); r += 4) {
      const int candidate = list[r];
      chain = fmaf(__bfloat162float(weights[static_cast<int64_t>(candidate) * H]), __bfloat162float(values[candidate]),
                   chain);
    }
    __syncwarp();
    const float c0 = __shfl_sync(kFull, chain, base), c1 = __shfl_sync(kFull, chain, base + 1);
    const float c2 = __shfl_sync(kFull, chain, base + 2), c3 = __shfl_sync(kFull, chain, base + 3);
    if (r0 < rows) sum += ((c0 + c1) + c2) + c3;
  }
  return sum;
}

// `encoder_blocks`: column blocks of the recovery encoder, or 0 without it; `blocks_magic`:
// floor(2^32 / (H / 64)) + 1, which divides piece numbers exactly.
__global__ void __launch_bounds__(DownUnion::kThreads, DownUnion::kPerSm)
    k_down_union(Layer L, Workspace ws, int encoder_blocks, uint32_t blocks_magic) {
  using X = DownUnion;
  constexpr int kSlots = X::kSlots;
  extern __shared__ __align__(128) uint8_t union_shared[];
  grid_dependency_wait();     // the activations are complete
  grid_dependency_release();  // the output may be scheduled; it waits for this grid
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  const int blocks = L.H / X::kColumns, passes = ws.work_counts[kDownCount];
  const int encoder_pieces = passes * encoder_blocks, pieces = encoder_pieces + passes * blocks;
  const uint32_t ring = shared_u32(union_shared) + warp * (kSlots * X::kSlotBytes);
  const int copy_row = lane >> 3, copy_column = (lane & 7) * 8;
  const uint32_t copy_to = ring + ((copy_row >> 1) * 8 + (copy_row & 1)) * X::kRowBytes + (lane & 7) * 16;
  const uint32_t values_at = ring + X::kUnitBytes + 8 * lane;
  int ahead = blockIdx.x * 4 + warp;
  if (ahead >= pieces) return;

  // ---- the copies, some units ahead of the sums ----
  // Piece `ahead` is block `block` of `source`; the piece after it is claimed when this one's copies
  // begin, its record read after two units and its first channels after four.
  int claimed = 0, block = 0, next_block = 0, next_piece = 0, stage = 0, unit = 0, units = 0;
  uint32_t channels = 0, more_channels = 0, first_channels = 0, row_bytes = 0;
  bool live = false;
  const char* rows = nullptr;
  const __nv_bfloat16* values[2];
  UnionWork source = {}, next = {};
  // Lane i has what the sums need to know of pieces i, 32 + i, ... of this warp.
  int piece_of = 0, first_of = 0, count_of = 0, rows_of = 0, started = 0;

  auto read_piece = [&](int piece) {
    int pass = piece;
    next_piece = piece;
    next_block = 0;  // blocks of the encoder come before those of the down rows
    if (piece < encoder_pieces) {
      for (; pass >= passes; pass -= passes) ++next_block;
    } else {
      const int at = piece - encoder_pieces;
      pass = __umulhi(static_cast<uint32_t>(at), blocks_magic);
      next_block = encoder_blocks + at - pass * blocks;
    }
    if (piece < pieces) next = load_work(ws.down_work + pass);
  };
  // Channels of union rows 32 `window` .. of a piece, one per lane; any for rows beyond the last.
  auto channel_window = [&](const UnionWork& w, bool encoder, int window) -> uint32_t {
    const int row = 32 * window + lane;
    if (encoder) return row;
    return row < w.rows ? ws.union_channels[static_cast<size_t>(w.e) * L.I + row] : 0;
  };
  auto start_piece = [&]() {
    ahead = next_piece;
    block = next_block;
    source = next;
    const bool encoder = block < encoder_blocks;
    if (encoder) source.rows = L.I;
    if (lane == (started & 31)) {
      piece_of = ahead < pieces ? block : -1;
      first_of = source.first;
      count_of = source.count;
      rows_of = source.rows;
    }
    ++started;
    unit = units = 0;
    if (ahead >= pieces) return;
    if (lane == 0) claimed = atomicAdd(ws.work_counts + kDownNext, 1) + gridDim.x * 4;
    stage = 0;
    const int width = encoder ? L.R : L.H;
    const int column = (encoder ? block : block - encoder_blocks) * X::kColumns + copy_column;
    live = column < width;
    row_bytes = 2 * width;
    rows = reinterpret_cast<const char*>((encoder ? L.encoder : L.down) +
                                         static_cast<size_t>(source.e) * L.I * width + column);
#pragma unroll
    for (int n = 0; n < 2; ++n) {  // tokens beyond the pass repeat its last one
      const int at = source.first + min(8 * n + g, source.count - 1);
      values[n] = (encoder ? ws.features + static_cast<size_t>(ws.group_pairs[at]) * L.I
                           : ws.union_activations + static_cast<size_t>(at) * L.I) + 4 * tq;
    }
    units = max(1, (source.rows + 15) / 16);
    channels = first_channels;
    more_channels = units > 2 ? channel_window(source, encoder, 1) : 0;
  };
  uint32_t put = 0;  // where the next unit goes in the ring
  auto fetch = [&]() {
    if (unit < units) {
      const uint32_t to = copy_to + put;
      const int from = 16 * (unit & 1) + copy_row;
      repeat<4>([&](auto i) {
        constexpr int kRow = decltype(i)::value;
        const uint32_t channel = __shfl_sync(kFull, channels, from + 4 * kRow);
        if (live)
          copy_async16_at<2 * kRow * X::kRowBytes>(to, rows + static_cast<uint64_t>(channel) * row_bytes);
      });
      copy_async8_at<0>(values_at + put, values[0]);
      copy_async8_at<256>(values_at + put, values[1]);
      values[0] += 16;
      values[1] += 16;
      ++unit;
      const bool done = unit == units;
      if (stage == 0 && (done || unit == 2)) {
        read_piece(__shfl_sync(kFull, claimed, 0));
        stage = 1;
      }
      if (stage == 1 && (done || unit == 4)) {
        if (next_piece < pieces) first_channels = channel_window(next, next_block < encoder_blocks, 0);
        stage = 2;
      }
      if (done) {
        start_piece();
      } else if ((unit & 1) == 0) {
        channels = more_channels;
        if (unit + 2 < units) more_channels = channel_window(source, block < encoder_blocks, unit / 2 + 1);
      }
    }
    copy_async_commit();  // also when empty: the group count per step stays fixed
    put = put == (kSlots - 1) * X::kSlotBytes ? 0 : put + X::kSlotBytes;
  };
  read_piece(ahead);
  first_channels = channel_window(next, next_block < encoder_blocks, 0);
  start_piece();
#pragma unroll 1
  for (int s = 0; s < kSlots - 1; ++s) fetch();

  // ---- the sums ----
  // The row whose address this lane gives to the matrix loads: rows 0 to 7 and 8 to 15 of eight
  // columns, then of the next eight.
  const uint32_t load_from = ring + (((lane >> 3) & 1) * 8 + (lane & 7)) * X::kRowBytes + (lane >> 4) * 16;
  uint32_t get = 0;  // where the next unit lies in the ring
  for (int done = 0;; ++done) {
    const int piece = __shfl_sync(kFull, piece_of, done & 31);
    if (piece < 0) break;
    const int first = __shfl_sync(kFull, first_of, done & 31), count = __shfl_sync(kFull, count_of, done & 31);
    int left = __shfl_sync(kFull, rows_of, done & 31);
    int pairs[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) pairs[n] = 8 * n + g < count ? ws.group_pairs[first + 8 * n + g] : -1;
    float acc[8][4], part[8][4];  // of all the rows, of the last few units
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][i] = part[n][i] = 0.0f;
    int turn = 0;
    do {
      copy_async_wait<kSlots - 2>();
      __syncwarp();  // every lane's copies of the unit have landed; the unit before has been read
      fetch();
      uint2 v[2];
      v[0] = load_shared8_at<0>(values_at + get);
      v[1] = load_shared8_at<256>(values_at + get);
      if (left < 16) {  // rows beyond the union weigh nothing
        const int mine = left - 4 * tq;
        const uint32_t x = mine > 1 ? ~0u : mine > 0 ? 0xffffu : 0u;
        const uint32_t y = mine > 3 ? ~0u : mine > 2 ? 0xffffu : 0u;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          v[n].x &= x;
          v[n].y &= y;
        }
      }
      const uint32_t a[4] = {v[0].x, v[1].x, v[0].y, v[1].y};
      repeat<4>([&](auto m) {
        constexpr int kPart = decltype(m)::value;
        uint32_t w[4];
        load_matrices_transposed_at<32 * kPart>(w, load_from + get);
        mma_bf16(part[2 * kPart], a, w[0], w[1]);
        mma_bf16(part[2 * kPart + 1], a, w[2], w[3]);
      });
      get = get == (kSlots - 1) * X::kSlotBytes ? 0 : get + X::kSlotBytes;
      left -= 16;
      if (++turn == X::kFold || left <= 0) {
        turn = 0;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            acc[n][i] += part[n][i];
            part[n][i] = 0.0f;
          }
      }
    } while (left > 0);
    // A token's sum over the expert, rounded to BF16 as the mix takes it.
    const bool encoder = piece < encoder_blocks;
    const int width = encoder ? L.R : L.H;
    const int column = (encoder ? piece : piece - encoder_blocks) * X::kColumns;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(encoder ? ws.encoder_parts : ws.down_parts) + column;
    uint32_t repeat = 0;  // bit 16 n + 2 c + b: column 8 c + 2 tq + b of token 8 n + g
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      if (pairs[n] < 0) continue;
      __nv_bfloat16* row = out + static_cast<size_t>(pairs[n]) * width + 2 * tq;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (column + 8 * c < width) {
          *reinterpret_cast<__nv_bfloat162*>(row + 8 * c) = __floats2bfloat162_rn(acc[c][2 * n], acc[c][2 * n + 1]);
          repeat |= static_cast<uint32_t>(isnan(acc[c][2 * n])) << (16 * n + 2 * c);
          repeat |= static_cast<uint32_t>(isnan(acc[c][2 * n + 1])) << (16 * n + 2 * c + 1);
        }
    }
    if (encoder) continue;  // the encoder rows meet every token's zeros in encode_tile too
    __syncwarp();           // the sums stored above may be replaced
    for (;;) {
      const unsigned any = __ballot_sync(kFull, repeat != 0);
      if (!any) break;
      // The first of the sums of up to eight lanes, each for four lanes.
      const int source = lane_of_bit(any, lane >> 2), from = max(source, 0);
      const uint32_t bits = __shfl_sync(kFull, repeat, from);
      const int low = __shfl_sync(kFull, pairs[0], from), high = __shfl_sync(kFull, pairs[1], from);
      const int bit = __ffs(bits) - 1, pair = source < 0 ? -1 : bit & 16 ? high : low;
      const int of = column + 8 * ((bit >> 1) & 7) + 2 * (from & 3) + (bit & 1);
      const int p = max(pair, 0), t = p / L.K;
      const float sum = repeat_down_sum(
          ws.candidate_ids + static_cast<size_t>(t) * L.F + ws.starts[p], ws.activations + static_cast<size_t>(t) * L.N,
          L.down + (static_cast<int64_t>(ws.ids[p]) - (p - t * L.K)) * L.I * L.H + of, L.H, pair < 0 ? 0 : ws.counts[p]);
      if (pair >= 0 && (lane & 3) == 0)
        out[static_cast<size_t>(pair) * width + of - column] = __float2bfloat16_rn(sum);
      if (__popc(any & ((1u << lane) - 1)) < 8) repeat &= repeat - 1;
    }
  }
}

// ---------------------------------------------------------------------------
// output of large batches
// ---------------------------------------------------------------------------
// Router mix of the BF16 expert sums of token t at column h, in slot order.
__device__ __forceinline__ float mix_sums(const Layer& L, const Workspace& ws, int t, int h) {
  const unsigned short* sums = reinterpret_cast<const unsigned short*>(ws.down_parts) +
                               static_cast<size_t>(t) * L.K * L.H + h;
  float routed = 0.0f;
#pragma unroll 8
  for (int s = 0; s < L.K; ++s) {
    const size_t pair = static_cast<size_t>(t) * L.K + s;
    if (ws.ids[pair] >= 0)
      routed = fmaf(__bfloat162float(__ushort_as_bfloat16(__ldcg(sums + static_cast<size_t>(s) * L.H))),
                    ws.weights[pair], routed);
  }
  return routed;
}

// grid (H / 128, or one more for the tokens' read-cost counters; ceil(T / 16)), 128 threads: sixteen
// tokens, 32 output columns per warp.  The decoder term is a product of the tokens' latents (BF16)
// with decoder rows, done by the tensor cores; a sum leaves them after 32 columns of the latent and
// goes on by ordinary additions, and one whose rounding to BF16 the distance to k_output's chain of
// FMAs could change is repeated as that chain: the bits are those of k_output.  Columns are dealt to
// the instruction so that a thread ends up with eight adjacent ones of two tokens, and the order
// inside sixteen latent columns so that it loads eight adjacent ones of a decoder row.  The expert
// sums are BF16, one per slot (of the expert-major down kernel; the first slots' are on their way
// meanwhile), or with TILES the FP32 sums of the down tiles.  Bound by latency, over tiles by their
// traffic: 256 tokens of the 256-expert layer 9.2 us (tiles 15.4, one token per CTA 27.8), of hidden
// 4096 and rank 128 13.8 (52, 4.2 TB/s; 127).
// `latents`: none, the workspace's, or to be mixed here from the encoder's sums.
constexpr int kLatentsNone = 0, kLatentsGiven = 1, kLatentsFromSums = 2;
constexpr int kMixTokens = 16;

// z += w * (the eight BF16 values of v).
__device__ __forceinline__ void add_scaled8(float (&z)[8], const uint4& v, float w) {
  z[0] = fmaf(bf16_lo(v.x), w, z[0]);
  z[1] = fmaf(bf16_hi(v.x), w, z[1]);
  z[2] = fmaf(bf16_lo(v.y), w, z[2]);
  z[3] = fmaf(bf16_hi(v.y), w, z[3]);
  z[4] = fmaf(bf16_lo(v.z), w, z[4]);
  z[5] = fmaf(bf16_hi(v.z), w, z[5]);
  z[6] = fmaf(bf16_lo(v.w), w, z[6]);
  z[7] = fmaf(bf16_hi(v.w), w, z[7]);
}
// Eight adjacent columns of a token from its down tiles: per slot the tiles in order, their sum rounded
// to BF16 times the router weight, slots in order (mix_down_tiles).
__device__ __forceinline__ void mix_tiles(float (&routed)[8], const float* parts, int H, int used,
                                          const int* slot_end, const float* slot_weight) {
  float sum[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  int slot = 0;
  auto close = [&]() {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      routed[c] = fmaf(bf16_round(sum[c]), slot_weight[slot], routed[c]);
      sum[c] = 0.0f;
    }
    ++slot;
  };
  constexpr int kTiles = 4;  // on their way at a time
  for (int base = 0; base < used; base += kTiles) {
    float4 v[kTiles][2];
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      const float4* from = reinterpret_cast<const float4*>(parts + static_cast<size_t>(base + i) * H);
#pragma unroll
      for (int c = 0; c < 2; ++c) v[i][c] = base + i < used ? __ldcg(from + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      if (base + i >= used) break;
      while (base + i >= slot_end[slot]) close();
      sum[0] += v[i][0].x;
      sum[1] += v[i][0].y;
      sum[2] += v[i][0].z;
      sum[3] += v[i][0].w;
      sum[4] += v[i][1].x;
      sum[5] += v[i][1].y;
      sum[6] += v[i][1].z;
      sum[7] += v[i][1].w;
    }
  }
  if (used > 0) close();
}
__device__ __forceinline__ uint4 pack_bf16x8(const float (&z)[8]) {
  uint4 v;
  uint32_t* out = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 two = __floats2bfloat162_rn(z[2 * i], z[2 * i + 1]);
    out[i] = *reinterpret_cast<const uint32_t*>(&two);
  }
  return v;
}

// Largest distance to a chain of FMAs that is provided for, in units of the token's largest running sum
// over the columns of a warp: 0.27 of it at most and 0.02 RMS in seventeen million sums of latents as
// the encoder leaves them for normal, outlier and Student-t inputs.
constexpr float kMixMargin = 1.0f / (1 << 19);

// One past the last down tile of slot `slot` of token t: a token's tiles lie slot after slot,
// ceil(count / 64) per local slot, from `tile_starts`.
__device__ __forceinline__ int down_slot_end(const Layer& L, const Workspace& ws, int t, int slot) {
  const size_t pair = static_cast<size_t>(t) * L.K + slot;
  const int tiles = ws.ids[pair] >= 0 ? (ws.counts[pair] + kDownTileRows - 1) / kDownTileRows : 0;
  return ws.tile_starts[pair] + tiles;
}

// Without tiles (after the union down kernel) seven registers are spilled for the four CTAs per SM.
template <bool TILES>
__global__ void __launch_bounds__(128, 4) k_mix(Layer L, Workspace ws, const uint8_t* padding, int tokens,
                                                __nv_bfloat16* out, int latents, int early) {
  __shared__ __align__(16) __nv_bfloat16 latent[kMixTokens][256 + 32];
  __shared__ float weight[kMixTokens][32];
  __shared__ uint32_t valid[kMixTokens];  // the slots that have sums
  __shared__ int slot_end[TILES ? kMixTokens : 1][32];  // one past a slot's last down tile
  const int t0 = blockIdx.y * kMixTokens, count = min(kMixTokens, tokens - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
  if (!early) grid_dependency_wait();
  if (static_cast<int>(blockIdx.x) * 128 >= L.H) {  // the read-cost counters
    for (int j = warp; j < count; j += 4) {
      const int t = t0 + j;
      if (padding && padding[t]) continue;
      const size_t pair = static_cast<size_t>(t) * L.K + lane;
      const bool local = lane < L.K && ws.ids[pair] >= 0;
      account_token(L, lane, local, local ? ws.counts[pair] : 0, L.F < L.N);
    }
    return;
  }
  const int pieces = L.R / 8;  // of a latent
  const bool recover = L.R > 0 && L.owner && L.decoder;
  // The instruction's column g of tile n is this warp's column 8 (g / 2) + 2 n + g % 2; a decoder
  // row is loaded 64 columns ahead.
  const uint4* rows = reinterpret_cast<const uint4*>(
      L.decoder + static_cast<size_t>(blockIdx.x * 128 + 32 * warp + 8 * (g >> 1) + (g & 1)) * L.R);
  uint4 decoder[2][4];
  auto load_decoder = [&](uint4 (&d)[4], int k) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
      d[n] = recover && k + tq < pieces ? rows[2 * n * pieces + k + tq] : make_uint4(0, 0, 0, 0);
  };
  load_decoder(decoder[0], 0);
  load_decoder(decoder[1], 4);
  for (int j = warp; j < kMixTokens; j += 4) {
    bool here = false;
    if (j < count && lane < L.K) {
      const size_t pair = static_cast<size_t>(t0 + j) * L.K + lane;
      here = ws.ids[pair] >= 0 && !(padding && padding[t0 + j]);
      weight[j][lane] = ws.weights[pair];
      if (TILES) slot_end[j][lane] = down_slot_end(L, ws, t0 + j, lane);
    }
    const unsigned slots = __ballot_sync(kFull, here);
    if (lane == 0) valid[j] = slots;
  }
  if (early) grid_dependency_wait();
  __syncthreads();
  // This thread's columns h .. h + 7 of tokens g and g + 8.
  const int h = blockIdx.x * 128 + 32 * warp + 8 * tq;
  constexpr int kSums = 4;  // slots on their way at a time
  uint4 sums[2][kSums];
  const uint4* from[2];
#pragma unroll
  for (int i = 0; i < 2 && !TILES; ++i) {
    from[i] = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(ws.down_parts) +
                                             static_cast<size_t>(t0 + min(8 * i + g, count - 1)) * L.K * L.H + h);
#pragma unroll
    for (int s = 0; s < kSums; ++s)
      sums[i][s] = s < L.K ? __ldcg(from[i] + static_cast<size_t>(s) * (L.H / 8)) : make_uint4(0, 0, 0, 0);
  }
  if (L.R > 0) {
    const int padded = (pieces + 3) & ~3;
    for (int i = tid; i < kMixTokens * padded; i += 128) {
      const int j = i / padded, piece = i - j * padded;
      const bool live = j < count && piece < pieces;
      float z[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      const size_t at = static_cast<size_t>(t0 + j) * L.R + 8 * piece;
      if (live && valid[j] && latents == kLatentsFromSums) {
        const uint4* parts = reinterpret_cast<const uint4*>(ws.encoder_parts) +
                             static_cast<size_t>(t0 + j) * L.K * pieces + piece;
        for (int s0 = 0; s0 < L.K; s0 += 8) {
          uint4 part[8];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            part[s] = s0 + s < L.K ? __ldcg(parts + (s0 + s) * pieces) : make_uint4(0, 0, 0, 0);
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if ((valid[j] >> (s0 + s)) & 1u) add_scaled8(z, part[s], weight[j][s0 + s]);
        }
      } else if (live && valid[j] && latents == kLatentsGiven) {
#pragma unroll
        for (int k = 0; k < 8; ++k) z[k] = ws.latent[at + k];
      }
      *reinterpret_cast<uint4*>(&latent[j][8 * piece]) = pack_bf16x8(z);
      if (live && blockIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) ws.latent[at + k] = z[k];
      }
    }
    __syncthreads();
  }
  float size[2] = {0.0f, 0.0f};  // largest running sums of tokens g and g + 8
  float dot[4][4];  // [n][token g, g + 8][columns 2 n, 2 n + 1 of this thread's eight]
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) dot[n][i] = 0.0f;
  if (recover) {
    auto fold = [&](const uint4 (&d)[4], int k) {
      const uint4 lo = *reinterpret_cast<const uint4*>(&latent[g][8 * (k + tq)]);
      const uint4 hi = *reinterpret_cast<const uint4*>(&latent[g + 8][8 * (k + tq)]);
      const uint32_t a[2][4] = {{lo.x, hi.x, lo.y, hi.y}, {lo.z, hi.z, lo.w, hi.w}};
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        float part[4];
        mma_bf16_first(part, a[0], d[n].x, d[n].y);
        mma_bf16(part, a[1], d[n].z, d[n].w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dot[n][i] += part[i];
          size[i >> 1] = fmaxf(size[i >> 1], fabsf(dot[n][i]));
        }
      }
    };
    for (int k = 0; k < pieces; k += 8) {
      fold(decoder[0], k);
      load_decoder(decoder[0], k + 8);
      if (k + 4 < pieces) fold(decoder[1], k + 4);
      load_decoder(decoder[1], k + 12);
    }
    // Sums in doubt again, a column after the other as the output of the tiles adds them.
    uint32_t doubt = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float margin = size[i];
      margin = fmaxf(margin, __shfl_xor_sync(kFull, margin, 1));
      margin = kMixMargin * fmaxf(margin, __shfl_xor_sync(kFull, margin, 2));
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int b = 0; b < 2; ++b)
          doubt |= static_cast<uint32_t>(rounds_either_way(dot[n][2 * i + b], margin)) << (4 * n + 2 * i + b);
    }
    for (; doubt; doubt &= doubt - 1) {
      const int bit = __ffs(doubt) - 1, j = g + 4 * (bit & 2);
      const uint4* row = reinterpret_cast<const uint4*>(
          L.decoder + static_cast<size_t>(h + 2 * (bit >> 2) + (bit & 1)) * L.R);
      const uint4* z = reinterpret_cast<const uint4*>(latent[j]);
      float sum = 0.0f;
#pragma unroll 4
      for (int k = 0; k < pieces; ++k) {
        const uint4 d = row[k], v = z[k];
        sum = fmaf(bf16_lo(d.x), bf16_lo(v.x), sum);
        sum = fmaf(bf16_hi(d.x), bf16_hi(v.x), sum);
        sum = fmaf(bf16_lo(d.y), bf16_lo(v.y), sum);
        sum = fmaf(bf16_hi(d.y), bf16_hi(v.y), sum);
        sum = fmaf(bf16_lo(d.z), bf16_lo(v.z), sum);
        sum = fmaf(bf16_hi(d.z), bf16_hi(v.z), sum);
        sum = fmaf(bf16_lo(d.w), bf16_lo(v.w), sum);
        sum = fmaf(bf16_hi(d.w), bf16_hi(v.w), sum);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i == bit) dot[i >> 2][i & 3] = sum;
    }
  }
  const bool aligned = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int j = 8 * i + g;
    if (j >= count) continue;
    float routed[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (TILES) mix_tiles(routed, ws.down_parts + static_cast<size_t>(t0 + j) * ws.down_tiles * L.H + h, L.H,
                         slot_end[j][L.K - 1], slot_end[j], weight[j]);
#pragma unroll
    for (int s = 0; s < kSums && !TILES; ++s)
      if ((valid[j] >> s) & 1u) add_scaled8(routed, sums[i][s], weight[j][s]);
    for (int s0 = kSums; s0 < L.K && !TILES; s0 += kSums) {
#pragma unroll
      for (int s = 0; s < kSums; ++s)
        if (s0 + s < L.K) sums[i][s] = __ldcg(from[i] + static_cast<size_t>(s0 + s) * (L.H / 8));
#pragma unroll
      for (int s = 0; s < kSums; ++s)
        if (s0 + s < L.K && ((valid[j] >> (s0 + s)) & 1u)) add_scaled8(routed, sums[i][s], weight[j][s0 + s]);
    }
    if (!(padding && padding[t0 + j])) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        routed[2 * n] += bf16_round(dot[n][2 * i]);
        routed[2 * n + 1] += bf16_round(dot[n][2 * i + 1]);
      }
    }
    __nv_bfloat16* to = out + static_cast<size_t>(t0 + j) * L.H + h;
    if (aligned) {
      *reinterpret_cast<uint4*>(to) = pack_bf16x8(routed);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) to[c] = __float2bfloat16_rn(routed[c]);
    }
  }
}
