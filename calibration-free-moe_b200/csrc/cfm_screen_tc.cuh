// Expert-major screen on the 5th-generation tensor cores (sm_100a), for passes of many tokens.
//
// A CTA takes 64 channels of one expert, their gate and up rows (128 sketch rows, one per
// thread, the M of the instruction), and a pass of up to TOKENS tokens.  Per rotation block the
// exact integer dots are one M128 x N x K128 product of bytes (cfm_screen.cuh):
//
//   * a thread decodes its row's 128 codes from 32 bytes into 32 registers and stores them
//     straight into tensor memory, where the instruction takes its first operand;
//   * the digits go to shared memory as they lie in the workspace, 16 bytes at a time, in the
//     canonical K-major layout of the second operand;
//   * one thread issues the product of a block, whose int32 accumulators in tensor memory every
//     thread reads back for its row, combines the digits, rescales, and adds to the FP32
//     projections in block order.
//
// Codes, digits and scales travel through a ring of three blocks in shared memory with cp.async.
// A block is a chain of waits (copies, product, barrier); six CTAs per SM (four with sixteen
// tokens, by their tensor memory) cover each other's.  Bound by instruction issue: some 60
// instructions decode a row's block, 7 per token rescale it.
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

constexpr int kScreenThreads = 128;
constexpr int kScreenChannels = 64;
constexpr int kScreenRing = 3;  // blocks

template <int TOKENS>
struct Screen {
  static constexpr int kColumns = TOKENS == 8 ? 32 : 3 * TOKENS;  // N: three digits per token
  static constexpr int kDigitStep = kColumns * 32;             // bytes of one K = 32 step
  static constexpr int kCodeBytes = kScreenThreads * 32;       // two planes of 16 bytes per row
  static constexpr int kScaleBytes = kScreenThreads * 2;
  static constexpr int kStageBytes = kCodeBytes + 4 * kDigitStep + 2 * kScaleBytes;
  static constexpr int kAhead = kScreenRing - 1;               // blocks whose copies are under way
  static constexpr int kTmemColumns = TOKENS == 8 ? 64 : 128;
  static constexpr int kSumsColumn = 32;                       // accumulators; before them the rows
  static constexpr int kPerSm = TOKENS == 8 ? 6 : 4;
  static constexpr int kStride = kScreenThreads + 4;           // floats per token of the exchange
  static constexpr size_t kRing = static_cast<size_t>(kScreenRing) * kStageBytes;
  static constexpr size_t kExchange = static_cast<size_t>(2) * TOKENS * kStride * sizeof(float);
  static constexpr size_t kFirst = kRing > kExchange ? kRing : kExchange;
  static size_t shared_bytes(int B) {
    return kFirst + static_cast<size_t>(3) * TOKENS * B * sizeof(float);
  }
};

namespace tc {

__device__ __forceinline__ void barrier_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Waits for the phase with the given parity; false when the wait ran out (about a second) or
// another thread already gave up.
__device__ __forceinline__ bool barrier_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
  long long start = 0;
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (!start) start = clock64();
    if (*abort || clock64() - start > 2000000000LL) {
      *abort = 1;
      return false;
    }
  }
}

// Shared-memory matrix descriptor: K-major, no swizzle, 128 bytes between the two 16-byte K
// chunks of a core-matrix row group, 256 bytes between row groups.
__device__ __forceinline__ uint64_t matrix_descriptor(uint32_t address) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((address & 0x3ffffu) >> 4);  // start address
  d |= static_cast<uint64_t>(128 >> 4) << 16;             // leading (K) byte offset
  d |= static_cast<uint64_t>(256 >> 4) << 32;             // stride (N) byte offset
  d |= static_cast<uint64_t>(1) << 46;                    // descriptor version of sm_100
  return d;
}

// Instruction descriptor: int32 accumulate, A unsigned and B signed int8, both K-major, M = 128.
__host__ __device__ constexpr uint32_t instruction_descriptor(int columns) {
  return (2u << 4) | (0u << 7) | (1u << 10) | (static_cast<uint32_t>(columns >> 3) << 17) |
         (static_cast<uint32_t>(128 >> 4) << 24);
}

// First operand in tensor memory.
__device__ __forceinline__ void mma_i8(uint32_t d, uint32_t a, uint64_t b, uint32_t descriptor,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(d), "r"(a), "l"(b), "r"(descriptor), "r"(accumulate), "r"(0)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void store_row(uint32_t address, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          address),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
      "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
      "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
      "r"(v[30]), "r"(v[31])
      : "memory");
}

// 24 columns of this thread's row: eight tokens' digits.
__device__ __forceinline__ void load_accumulators(uint32_t address, int (&c)[24]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]),
        "=r"(c[7]), "=r"(c[8]), "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]),
        "=r"(c[14]), "=r"(c[15])
      : "r"(address)
      : "memory");
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(c[16]), "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]), "=r"(c[21]), "=r"(c[22]),
        "=r"(c[23])
      : "r"(address + 16)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace tc

// grid (ceil(I / 64), most passes of TOKENS tokens), 128 threads; with `pairs` one more row of CTAs
// that clears the projections of the call's dead pairs.
template <int TOKENS, bool RISK>
__global__ void __launch_bounds__(kScreenThreads, Screen<TOKENS>::kPerSm)
    k_screen_tc(Layer L, Workspace ws, const uint8_t* padding, int pairs) {
  using S = Screen<TOKENS>;
  using namespace tc;
  extern __shared__ __align__(1024) uint8_t screen_shared[];
  __shared__ uint64_t barrier;
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag, s_pair[TOKENS], s_token[TOKENS];
  volatile int* abort = &abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5;
  grid_dependency_wait();  // the digits and the passes are complete
  if (pairs && blockIdx.y == gridDim.y - 1) {
    const int c = blockIdx.x * kScreenChannels;
    clear_dead(L, ws, padding, pairs, c, min(L.I, c + kScreenChannels));
    return;
  }
  if (static_cast<int>(blockIdx.y) >= ws.work_counts[kPassCount]) return;
  const int4 pass = *reinterpret_cast<const int4*>(ws.pass_work + blockIdx.y);
  const int e = pass.x, first = pass.y, count = pass.z;
  const int I = L.I, B = L.B, rows = 2 * I, c0 = blockIdx.x * kScreenChannels;
  const int channel = c0 + (tid & 63), row = tid < 64 ? channel : I + channel;
  const bool inside = channel < I;

  const uint32_t bar = shared_u32(&barrier);
  if (tid < TOKENS) {
    const int pair = ws.group_pairs[first + min(tid, count - 1)];
    s_pair[tid] = pair;
    s_token[tid] = pair / L.K;
  }
  if (tid == 0) {
    abort_flag = 0;
    barrier_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     shared_u32(&tmem_holder)),
                 "r"(S::kTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;
  const uint32_t tmem_lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);

  const uint32_t ring = shared_u32(screen_shared);
  float* exchange = reinterpret_cast<float*>(screen_shared);
  // Per block the tokens' scales of the fixed point and sums of their values, and energies.
  int2* factor = reinterpret_cast<int2*>(screen_shared + S::kFirst);
  float* energy = reinterpret_cast<float*>(factor + TOKENS * B);
  for (int i = tid; i < TOKENS * B; i += kScreenThreads) {
    const int b = i / TOKENS, t = i % TOKENS;
    const size_t at = static_cast<size_t>(s_token[t]) * B + b;
    const int2 f = reinterpret_cast<const int2*>(ws.exponents)[at];
    factor[i] = make_int2(__float_as_int(unscale_of(f.x)), f.y);
    if (RISK) energy[i] = ws.norms[at];
  }
  // Codes and scales of block b: this thread's 32 bytes, and 16-byte pieces of the planes.
  const uint8_t* next_codes = reinterpret_cast<const uint8_t*>(L.sketch_grouped) +
                              (static_cast<size_t>(e) * B * rows + row) * 32;
  const int plane = tid >> 4, plane_row = (tid & 8 ? I : 0) + c0 + 8 * (tid & 7);
  const bool copies_plane = tid < (RISK ? 32 : 16) && c0 + 8 * (tid & 7) < I;
  const uint8_t* next_planes = reinterpret_cast<const uint8_t*>(
      L.statistics + (static_cast<size_t>(e) * B * 2 + (plane & 1)) * rows + plane_row);
  const uint32_t code_step = rows * 32, plane_step = 4 * rows;  // bytes per block
  constexpr int kPieces = (3 * TOKENS * 8 + kScreenThreads - 1) / kScreenThreads;  // of digits
  const int8_t* digits[kPieces];
  uint32_t digit_place[kPieces];
#pragma unroll
  for (int i = 0; i < kPieces; ++i) {
    const int piece = tid + i * kScreenThreads, column = piece >> 3, chunk = piece & 7;
    const int t = column / 3;
    digits[i] = t < count ? ws.limbs + (static_cast<size_t>(s_token[t]) * B * 3 + (column - 3 * t)) * kBlock +
                                16 * chunk
                          : nullptr;
    digit_place[i] = S::kCodeBytes + (chunk >> 1) * S::kDigitStep + (column >> 3) * 256 +
                     (chunk & 1) * 128 + (column & 7) * 16;
  }
  int fetched = 0;
  uint32_t fetch_stage = ring;
  auto fetch = [&]() {  // the next block
    if (fetched < B) {
      if (inside) {
        copy_async16(fetch_stage + 16 * tid, next_codes);
        copy_async16(fetch_stage + 2048 + 16 * tid, next_codes + 16);
      }
#pragma unroll
      for (int i = 0; i < kPieces; ++i)
        if (digits[i]) {
          copy_async16(fetch_stage + digit_place[i], digits[i]);
          digits[i] += 3 * kBlock;
        }
      if (copies_plane)
        copy_async16(fetch_stage + S::kCodeBytes + 4 * S::kDigitStep + plane * S::kScaleBytes +
                         16 * (tid & 15),
                     next_planes);
      next_codes += code_step;
      next_planes += plane_step;
      fetch_stage = fetch_stage + S::kStageBytes == ring + S::kRing ? ring : fetch_stage + S::kStageBytes;
      ++fetched;
    }
    copy_async_commit();  // also when empty: one group per block
  };
  float run[TOKENS], spread[RISK ? TOKENS : 1], scale = 0.0f, variance = 0.0f;
#pragma unroll
  for (int t = 0; t < TOKENS; ++t) {
    run[t] = 0.0f;
    if (RISK) spread[t] = 0.0f;
  }
  // Adds block b, whose product is under way, to the projections, two tokens at a time.
  auto rescale = [&](int b) {
    barrier_wait(bar, b & 1, abort);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int half = 0; half < TOKENS / 8; ++half) {
      if (8 * half >= count) break;
      int c[24];
      load_accumulators(tmem_lane + S::kSumsColumn + 24 * half, c);
      const int4* factors = reinterpret_cast<const int4*>(factor + b * TOKENS + 8 * half);
      const float2* energies = reinterpret_cast<const float2*>(energy + b * TOKENS + 8 * half);
#pragma unroll
      for (int two = 0; two < 4; ++two) {
        if (8 * half + 2 * two >= count) break;
        const int4 f = factors[two];
        const float2 en = RISK ? energies[two] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = 8 * half + 2 * two + i, j = 3 * (2 * two + i);
          // code = trit + 1: the sum of the values comes off.
          const int dot = (c[j] - (i ? f.w : f.y)) + c[j + 1] * 256 + c[j + 2] * 65536;
          const float d = __fmul_rn(__int2float_rn(dot), __int_as_float(i ? f.z : f.x));
          run[t] = __fadd_rn(run[t], __fmul_rn(scale, d));
          if (RISK) spread[t] = __fadd_rn(spread[t], __fmul_rn(variance, i ? en.y : en.x));
        }
      }
    }
  };
#pragma unroll 1
  for (int i = 0; i < S::kAhead; ++i) fetch();
  uint32_t stage = ring;
#pragma unroll 1
  for (int b = 0; b < B; ++b) {
    if (b) rescale(b - 1);
    copy_async_wait<S::kAhead - 1>();  // this thread's copies of the block have landed
    {
      const uint4 lo = load_shared16(stage + 16 * tid), hi = load_shared16(stage + 2048 + 16 * tid);
      const uint32_t word[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      uint32_t v[32];
#pragma unroll
      for (int w = 0; w < 8; ++w)
#pragma unroll
        for (int m = 0; m < 4; ++m) v[4 * w + m] = codes_of(word[w], m);
      store_row(tmem_lane, v);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the digits
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int step = 0; step < 4; ++step)
        mma_i8(tmem + S::kSumsColumn, tmem + 8 * step,
               matrix_descriptor(stage + S::kCodeBytes + step * S::kDigitStep),
               instruction_descriptor(S::kColumns), step > 0);
      mma_commit(bar);
    }
    const __half* scales = reinterpret_cast<const __half*>(screen_shared + (stage - ring) +
                                                           S::kCodeBytes + 4 * S::kDigitStep);
    scale = __half2float(scales[tid]);
    variance = RISK ? __half2float(scales[kScreenThreads + tid]) : 0.0f;
    stage = stage + S::kStageBytes == ring + S::kRing ? ring : stage + S::kStageBytes;
    fetch();  // into the place of the block before this one, which nothing reads any more
  }
  rescale(B - 1);
  grid_dependency_release();  // the selection may be scheduled; it waits for this grid

  // Projections out, and across the CTA: a channel's gate and up rows are different threads.
  copy_async_wait<0>();
  __syncthreads();  // the ring has been read by every thread
#pragma unroll
  for (int t = 0; t < TOKENS; ++t)
    if (t < count) {
      exchange[t * S::kStride + tid] = run[t];
      if (RISK) exchange[(TOKENS + t) * S::kStride + tid] = spread[t];
      if (inside) {
        const size_t at = (static_cast<size_t>(s_token[t]) + (tid < 64 ? 0 : 1)) * L.N +
                          static_cast<size_t>(s_pair[t]) * I + channel;
        ws.partial[at] = run[t];
        if (RISK) ws.variances[at] = spread[t];
      }
    }
  __syncthreads();
  if (inside)
    for (int t = tid >> 6; t < count; t += 2) {
      const float* g = exchange + t * S::kStride + (tid & 63);
      finish_candidate(L, ws, s_pair[t], e, channel, g[0], g[64], RISK ? g[TOKENS * S::kStride] : 0.0f,
                       RISK ? g[TOKENS * S::kStride + 64] : 0.0f);
    }
  if (*abort && tid == 0) atomicExch(&ws.status[0], 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(S::kTmemColumns)
                 : "memory");
  }
}
