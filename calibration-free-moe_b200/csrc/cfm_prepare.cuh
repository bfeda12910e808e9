// The start of a call (sm_100a): input rotation, routing, the pairs grouped by expert.
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

constexpr int kPrepareThreads = 512;

// Lengths of the work lists.
constexpr int kPassCount = 0, kBusyCount = 1, kExactCount = 2, kDownCount = 3;
// Pieces of the expert-major down kernel claimed so far.
constexpr int kDownNext = 4;

// Up to `pass` pairs of one expert, `first .. first + count - 1` of the grouped list.
struct __align__(16) Pass {
  int e, first, count, reserved;
};

// Coordinate c of sixteen goes to this byte of its digits: the order in which the masked shifts
// of a code word (cfm_screen.cuh) give its codes.  Lane j of four holds coordinates 4 j .. 4 j + 3;
// its even ones are the bytes `digit_byte(j)` and the next, its odd ones those eight further on.
__device__ __forceinline__ int digit_byte(int j) { return 4 * (j & 1) + 2 * (j >> 1); }

// One rotation block of one token by one warp, lane l holding coordinates 4 l .. 4 l + 3: signs,
// 128-point butterfly, the KEEP largest magnitudes (ties to the lower coordinate), the fixed-point
// copy of what is kept and its base-256 digits.  Latency bound (a thread per coordinate ranked
// itself against all 128 before, and one of them added the energies: 3.5 us for one token, 24.6 us
// for 256 of hidden size 2048); here the cut is searched two bits at a time from the top, three
// counts in one warp reduction, until it separates exactly KEEP values.
__device__ __forceinline__ void rotate_block(const Layer& L, const Workspace& ws,
                                             const __nv_bfloat16* hidden, int t, int b,
                                             float* squares) {
  const int lane = threadIdx.x & 31;
  const size_t row = static_cast<size_t>(t) * L.B + b;
  const uint2 raw = *reinterpret_cast<const uint2*>(hidden + static_cast<size_t>(t) * L.H +
                                                    b * kBlock + 4 * lane);
  const char4 sign = *reinterpret_cast<const char4*>(L.signs + b * kBlock + 4 * lane);
  float v[4] = {__fmul_rn(bf16_lo(raw.x), static_cast<float>(sign.x)),
                __fmul_rn(bf16_hi(raw.x), static_cast<float>(sign.y)),
                __fmul_rn(bf16_lo(raw.y), static_cast<float>(sign.z)),
                __fmul_rn(bf16_hi(raw.y), static_cast<float>(sign.w))};
  {  // half-widths 1 and 2: the lower member takes the sum, the upper one the difference
    const float a = __fadd_rn(v[0], v[1]), d = __fsub_rn(v[0], v[1]);
    const float c = __fadd_rn(v[2], v[3]), f = __fsub_rn(v[2], v[3]);
    v[0] = __fadd_rn(a, c);
    v[2] = __fsub_rn(a, c);
    v[1] = __fadd_rn(d, f);
    v[3] = __fsub_rn(d, f);
  }
#pragma unroll
  for (int w = 1; w < 32; w <<= 1)  // half-widths 4 .. 64
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float o = __shfl_xor_sync(kFull, v[i], w);
      v[i] = (lane & w) ? __fsub_rn(o, v[i]) : __fadd_rn(v[i], o);
    }
  uint32_t key[4], most = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = __fmul_rn(v[i], 0.0883883461f);  // float(1 / sqrt(128))
    key[i] = __float_as_uint(v[i]) & 0x7fffffffu;
    most = max(most, key[i]);
  }
  most = __reduce_max_sync(kFull, most);

  unsigned kept[4] = {kFull, kFull, kFull, kFull};  // ballots
  if (L.KEEP < kBlock) {
    uint32_t cut = 0;  // at least KEEP keys reach it
    bool exact = false;
    for (int s = 30; s >= 0 && !exact; s -= 2) {
      // Counts at or above cut + 1, 2, 3 steps, ten bits each.
      uint32_t counts = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        counts += (key[i] >= (cut | (1u << s)) ? 1u : 0u) + (key[i] >= (cut | (2u << s)) ? 1u << 10 : 0u) +
                  (key[i] >= (cut | (3u << s)) ? 1u << 20 : 0u);
      counts = __reduce_add_sync(kFull, counts);
      const int c1 = counts & 1023, c2 = (counts >> 10) & 1023, c3 = counts >> 20;
      const int digit = c3 >= L.KEEP ? 3 : c2 >= L.KEEP ? 2 : c1 >= L.KEEP ? 1 : 0;
      const int reached = digit == 3 ? c3 : digit == 2 ? c2 : digit == 1 ? c1 : 0;
      cut |= static_cast<uint32_t>(digit) << s;
      exact = reached == L.KEEP;  // everything from the cut up, no ties left over
    }
    unsigned above[4], tied[4];
    int taken = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      above[i] = __ballot_sync(kFull, exact ? key[i] >= cut : key[i] > cut);
      tied[i] = __ballot_sync(kFull, !exact && key[i] == cut);
      taken += __popc(above[i]);
    }
    const unsigned before = (1u << lane) - 1;
    int ties = 0;  // at lower coordinates
#pragma unroll
    for (int i = 0; i < 4; ++i) ties += __popc(tied[i] & before);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool tie = (tied[i] >> lane) & 1u;
      kept[i] = __ballot_sync(kFull, ((above[i] >> lane) & 1u) || (tie && taken + ties < L.KEEP));
      ties += tie;
    }
  }
  int position = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) position += __popc(kept[i] & ((1u << lane) - 1));

  // Fixed point: q = rint(v * 2^(21 - e)), e = floor(log2 max|v|) clamped to +-100.
  int e = static_cast<int>(most >> 23) - 127;
  e = max(-100, min(100, e));
  const float scale = __uint_as_float(static_cast<uint32_t>(127 + kQuantBits - e) << 23);
  int qsum = 0;
  uint32_t digits[3][2] = {{0, 0}, {0, 0}, {0, 0}};  // [digit][even, odd coordinates], two bytes each
  float square[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool keep = (kept[i] >> lane) & 1u;
    int q = 0;
    square[i] = 0.0f;
    if (keep) {
      q = most ? __float2int_rn(__fmul_rn(v[i], scale)) : 0;
      q = max(-(1 << 22), min(1 << 22, q));
      square[i] = __fmul_rn(v[i], v[i]);
      const size_t out = row * L.KEEP + position++;
      ws.planes[out] = v[i];
      ws.coordinates[out] = 4 * lane + i;
      ws.quantized[out] = q;
    }
    qsum += q;
    // Balanced base-256 digits (zero for dropped coordinates): q = l0 + 256 l1 + 65536 l2.
    const int l0 = static_cast<int8_t>(q & 0xff), q1 = (q - l0) >> 8;
    const int l1 = static_cast<int8_t>(q1 & 0xff), l2 = (q1 - l1) >> 8;
    digits[0][i & 1] |= (static_cast<uint32_t>(l0) & 0xffu) << (8 * (i >> 1));
    digits[1][i & 1] |= (static_cast<uint32_t>(l1) & 0xffu) << (8 * (i >> 1));
    digits[2][i & 1] |= (static_cast<uint32_t>(l2) & 0xffu) << (8 * (i >> 1));
  }
  int8_t* limb = ws.limbs + row * 3 * kBlock + 16 * (lane >> 2) + digit_byte(lane & 3);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    *reinterpret_cast<uint16_t*>(limb + j * kBlock) = static_cast<uint16_t>(digits[j][0]);
    *reinterpret_cast<uint16_t*>(limb + j * kBlock + 8) = static_cast<uint16_t>(digits[j][1]);
  }
  qsum = __reduce_add_sync(kFull, qsum);
  if (lane == 0) reinterpret_cast<int2*>(ws.exponents)[row] = make_int2(e, qsum);
  // Energy of the kept coordinates, summed in coordinate order (pinned); only the
  // recovery-aware score reads it.
  if (L.score != CFM_SCORE_POINT) {
    *reinterpret_cast<float4*>(squares + 4 * lane) =
        make_float4(square[0], square[1], square[2], square[3]);
    __syncwarp();
    if (lane == 0) {
      float total = 0.0f;
#pragma unroll 8
      for (int j = 0; j < kBlock / 4; ++j) {
        const float4 s = reinterpret_cast<const float4*>(squares)[j];
        total = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(total, s.x), s.y), s.z), s.w);
      }
      ws.norms[row] = total;
    }
  }
}

// Exclusive scan over the CTA of three counts packed in 64 bits (pairs: 24 bits, experts that have
// any: 20, passes: 20); `scratch` holds 33 of them.
__device__ __forceinline__ unsigned long long block_scan_packed(unsigned long long value,
                                                                unsigned long long* scratch,
                                                                unsigned long long* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  unsigned long long scan = value;
#pragma unroll
  for (int w = 1; w < 32; w <<= 1) {
    const unsigned long long o = __shfl_up_sync(kFull, scan, w);
    if (lane >= w) scan += o;
  }
  __syncthreads();  // earlier users of the scratch are done
  if (lane == 31) scratch[warp] = scan;
  __syncthreads();
  unsigned long long before = 0, all = 0;
  for (int w = 0; w < warps; ++w) {
    const unsigned long long s = scratch[w];
    before += w < warp ? s : 0;
    all += s;
  }
  *total = all;
  return before + scan - value;
}

// What the router gave.
struct Routes {
  const void* ids;
  const void* weights;
  int ids64, weights16;
  int lanes;  // power of two that holds K: lanes per token
  int pass;   // pairs per pass of the screen
};

// One CTA: with `route` every token's K experts are sorted ascending (stable) and mapped to local
// ids; then the active (token, slot) pairs are listed by expert, and the experts' passes of
// `pass` pairs.  The order of an expert's pairs is whatever the atomics produce; every pair's
// result is independent of it.  `count` holds E ints.
__device__ __forceinline__ void group_pairs(const Layer& L, const Workspace& ws, const Routes& r,
                                            bool route, const uint8_t* padding, int T, int* count) {
  __shared__ unsigned long long scratch[33];
  const int tid = threadIdx.x, threads = blockDim.x, lane = tid & 31, pairs = T * L.K;
  for (int e = tid; e < L.E; e += threads) count[e] = 0;
  __syncthreads();
  if (route) {
    const int j = lane & (r.lanes - 1), per_cta = threads / r.lanes, base = lane - j;
    for (int t0 = 0; t0 < T; t0 += per_cta) {  // every lane takes part in the shuffles
      const int t = t0 + tid / r.lanes;
      const bool live = t < T && j < L.K;
      long long id = 0x7fffffffffffffffLL;
      float w = 0.0f;
      if (live) {
        const size_t at = static_cast<size_t>(t) * L.K + j;
        id = r.ids64 ? static_cast<const long long*>(r.ids)[at]
                     : static_cast<long long>(static_cast<const int32_t*>(r.ids)[at]);
        w = r.weights16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(r.weights)[at])
                        : static_cast<const float*>(r.weights)[at];
      }
      int rank = 0;
      for (int i = 0; i < L.K; ++i) {
        const long long o = __shfl_sync(kFull, id, base + i);
        rank += (o < id) || (o == id && i < j);
      }
      if (live) {
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
        if (local >= 0 && !(padding && padding[t])) atomicAdd(&count[local], 1);
      }
    }
  } else {
    for (int p = tid; p < pairs; p += threads) {
      const int e = ws.ids[p];
      if (e >= 0 && !(padding && padding[p / L.K])) atomicAdd(&count[e], 1);
    }
  }
  __syncthreads();
  unsigned long long base = 0;
  for (int e0 = 0; e0 < L.E; e0 += threads) {
    const int e = e0 + tid, mine = e < L.E ? count[e] : 0, passes = (mine + r.pass - 1) / r.pass;
    unsigned long long all;
    const unsigned long long at =
        base + block_scan_packed(static_cast<unsigned long long>(mine) |
                                     static_cast<unsigned long long>(mine > 0) << 24 |
                                     static_cast<unsigned long long>(passes) << 44,
                                 scratch, &all);
    base += all;
    if (e < L.E) {
      const int first = static_cast<int>(at & 0xffffff), place = static_cast<int>(at >> 44);
      ws.group_offsets[e] = count[e] = first;
      for (int j = 0; j < passes; ++j)
        ws.pass_work[place + j] = Pass{e, first + j * r.pass, min(r.pass, mine - j * r.pass), 0};
      if (mine) ws.busy_experts[(at >> 24) & 0xfffff] = e;
    }
  }
  if (tid == 0) {
    ws.group_offsets[L.E] = static_cast<int>(base & 0xffffff);
    ws.work_counts[kPassCount] = static_cast<int>(base >> 44);
    ws.work_counts[kBusyCount] = static_cast<int>((base >> 24) & 0xfffff);
    ws.work_counts[kExactCount] = ws.work_counts[kDownCount] = ws.work_counts[kDownNext] = 0;
  }
  __syncthreads();
  for (int p = tid; p < pairs; p += threads) {
    const int e = ws.ids[p];
    if (e >= 0 && !(padding && padding[p / L.K])) ws.group_pairs[atomicAdd(&count[e], 1)] = p;
  }
}

// 512 threads.  With `group` CTA 0 routes and groups; the other CTAs rotate sixteen blocks each.
// One launch for what were three on two streams: they do not depend on one another.
__global__ void __launch_bounds__(kPrepareThreads)
    k_prepare(Layer L, Workspace ws, const __nv_bfloat16* hidden, const uint8_t* padding, int T,
              int group, Routes r) {
  extern __shared__ __align__(16) uint8_t prepare_shared[];  // E counters | 16 x 128 squares
  grid_dependency_wait();     // the workspace and the inputs may still be in use, or in the making
  grid_dependency_release();  // the screen may be scheduled; it waits for this grid
  if (group && blockIdx.x == 0) {
    group_pairs(L, ws, r, true, padding, T, reinterpret_cast<int*>(prepare_shared));
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int block = (blockIdx.x - group) * (kPrepareThreads / 32) + warp;
  const int t = block / L.B;
  if (t >= T || (padding && padding[t])) return;
  rotate_block(L, ws, hidden, t, block - t * L.B,
               reinterpret_cast<float*>(prepare_shared) + warp * kBlock);
}

// One CTA of 512 threads: the grouping alone, after routes that another kernel wrote.
__global__ void __launch_bounds__(kPrepareThreads)
    k_group(Layer L, Workspace ws, const uint8_t* padding, int T, Routes r) {
  extern __shared__ __align__(16) uint8_t prepare_shared[];
  group_pairs(L, ws, r, false, padding, T, reinterpret_cast<int*>(prepare_shared));
}
