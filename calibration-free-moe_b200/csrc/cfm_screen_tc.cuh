// Expert-major screen on the 5th-generation tensor cores (sm_100a), for passes of many tokens.
//
// A CTA takes 128 channels of one expert and a pass of up to TOKENS tokens.  Per rotation block and
// tile (the channels' gate rows, then their up rows; one row per thread, the M of the instruction) the
// exact integer dots are one M128 x N x K128 product of bytes (cfm_screen.cuh).  Warps have roles:
//
//   * the threads of warps 0 to 3 hold a channel each.  They decode its row's 128 codes from 32 bytes
//     into 32 registers and store them straight into tensor memory, where the instruction takes its
//     first operand; a block later they read back the int32 sums of the row, combine the digits,
//     rescale, and add to the FP32 projections in block order.  A channel's gate and up rows are the
//     same thread's, so scores and features follow without an exchange;
//   * warp 4 brings the tokens' digits with cp.async, 16 bytes at a time, in the canonical K-major
//     layout of the second operand, and one of its threads issues the gate tile's product once the four
//     warps have arrived;
//   * one thread of warp 5 issues the up tile's, and brings codes and scales into a ring in shared
//     memory, contiguous runs that bulk copies take.
//
// So no thread waits for a product's latency (450 cycles alone, 1000 beside three other CTAs; a thread
// needs 54 cycles for each of its four instructions, whatever N up to 64), and the four warps never
// wait for one another.
// Bound by instruction issue and the latency between instructions: some 160 per warp and tile with four
// tokens, 56 of them the decode's, issued at 0.64 per scheduler and active cycle with five CTAs per SM (0.56
// with four and passes of eight); and by the last CTAs of a launch, alone on their SM.
// 64 tokens of the 128-expert layer (100 MB of codes: 15 us of HBM) 35 us, 32 tokens 24.5, 8 tokens
// 15, 256 tokens of hidden 4096 and width 1536 240, against 56, 44, 27 and 404 of 64 channels per CTA
// whose threads copied, waited for their product and met at a barrier once per block.  Persistent CTAs
// with units of 64 channels, whose two places in tensor memory alternate between blocks, took 59 us at 64
// tokens (140 instructions per block and warp for copies and waits that a pair of tiles shares here);
// one driver for all copies and products, 45.
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

// How long a wait goes on, how long, once one has run out, those for what is still in flight do, in
// nanoseconds, and how they ask.  (A build for tests has short waits run out.)
#ifndef CFM_SCREEN_WAIT_NS
#define CFM_SCREEN_WAIT_NS 1000000000u
#define CFM_SCREEN_DRAIN_NS 1000000000u
#define CFM_SCREEN_WAIT "try_wait"
#endif

constexpr int kScreenThreads = 192;
constexpr int kScreenChannels = 128;
constexpr int kScreenAhead = 4;  // blocks whose variances are on their way together (16: 83 us against 78 for 100
                                 // tokens of the 64-expert layer; the code outgrows its cache)

template <int TOKENS, bool RISK>
struct Screen {
  static constexpr int kColumns = TOKENS == 16 ? 48 : 4 * TOKENS;  // N: three digits per token, a multiple of 16
  static constexpr int kDigitStep = kColumns * 32;             // bytes of one K = 32 step
  static constexpr int kDigitBytes = 4 * kDigitStep;           // of a block
  static constexpr int kCodeBytes = kScreenChannels * 68;      // gate codes, up codes, gate scales, up scales
  static constexpr int kCodeRing = TOKENS == 16 ? 3 : 4;       // blocks
  static constexpr int kDigitRing = 3;                         // the next two are on their way
  // Tensor memory, for each tile 32 columns of its product's first operand and the sums, in two pieces:
  // four tokens 32 (sums) and 64, eight 128, sixteen 32 (first operand of the gate tile) and 128.
  static constexpr int kSumsStep = kColumns;
  static constexpr int kSmall = TOKENS == 8 ? 0 : 32, kLarge = TOKENS == 4 ? 64 : 128;
  static constexpr int kPerSm = TOKENS == 4 ? 5 : TOKENS == 8 ? 4 : 3;
  static constexpr int kStride = kScreenChannels * (RISK ? 4 : 2);  // floats per token of the end
  static constexpr size_t kCopies = static_cast<size_t>(kCodeRing) * kCodeBytes + kDigitRing * kDigitBytes;
  static constexpr size_t kEnd = static_cast<size_t>(TOKENS) * kStride * sizeof(float);
  static constexpr size_t kRing = kCopies > kEnd ? kCopies : kEnd;
  static size_t shared_bytes(int B) {
    return kRing + static_cast<size_t>(RISK ? 3 : 2) * TOKENS * B * sizeof(float);
  }
};

namespace tc {

// By the threads with `leader` set.
__device__ __forceinline__ void barrier_arrive(uint32_t bar, int leader) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.s32 p, %1, 0;\n\t"
      "@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
      "r"(leader)
      : "memory");
}

__device__ __forceinline__ void barrier_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

// `bytes` (a multiple of 16) from global to shared memory, both on 16-byte boundaries; arrives at
// the barrier.
__device__ __forceinline__ void copy_bulk(uint32_t shared, const void* global, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared),
               "l"(global), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void barrier_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Waits for the phase with the given parity, `limit` nanoseconds at most: then the word at `abort` is set.
// A thread that gives up, because its time ran out or another thread's has, clears `alive`; a phase that
// is complete counts all the same.  (One try suspends for up to 4 us.)
__device__ __forceinline__ void barrier_wait(uint32_t bar, uint32_t parity, uint32_t abort, int& alive,
                                             uint32_t limit = CFM_SCREEN_WAIT_NS) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .u32 start, now;\n\t"
      "mbarrier." CFM_SCREEN_WAIT ".parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra done;\n\t"
      "mov.u32 start, %%globaltimer_lo;\n"
      "again:\n\t"
      "ld.volatile.shared.u32 now, [%3];\n\t"
      "setp.ne.u32 p, now, 0;\n\t"
      "@p bra gone;\n\t"
      "mbarrier." CFM_SCREEN_WAIT ".parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra done;\n\t"
      "mov.u32 now, %%globaltimer_lo;\n\t"
      "sub.u32 now, now, start;\n\t"
      "setp.lt.u32 p, now, %4;\n\t"
      "@p bra again;\n\t"
      "st.volatile.shared.u32 [%3], 1;\n"
      "gone:\n\t"
      "mov.u32 %0, 0;\n"
      "done:\n\t}"
      : "+r"(alive)
      : "r"(bar), "r"(parity), "r"(abort), "r"(limit)
      : "memory");
}

// The same for the end of a product, whose rows and sums the thread is about to touch: having given up it
// goes on waiting, until the word at `late` is set or, after CFM_SCREEN_DRAIN_NS, sets that.  (By then no driver
// issues a product any more.  A vote of the warp before it goes on, instead, cost 2 us of 55.)
__device__ __forceinline__ void barrier_wait_product(uint32_t bar, uint32_t parity, uint32_t abort, uint32_t late,
                                                     int& alive) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .u32 start, now;\n\t"
      "mbarrier." CFM_SCREEN_WAIT ".parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra done;\n\t"
      "mov.u32 start, %%globaltimer_lo;\n"
      "again:\n\t"
      "ld.volatile.shared.u32 now, [%3];\n\t"
      "setp.ne.u32 p, now, 0;\n\t"
      "@p bra gone;\n\t"
      "mbarrier." CFM_SCREEN_WAIT ".parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra done;\n\t"
      "mov.u32 now, %%globaltimer_lo;\n\t"
      "sub.u32 now, now, start;\n\t"
      "setp.lt.u32 p, now, %5;\n\t"
      "@p bra again;\n\t"
      "st.volatile.shared.u32 [%3], 1;\n"
      "gone:\n\t"
      "mov.u32 %0, 0;\n\t"
      "mov.u32 start, %%globaltimer_lo;\n"
      "drain:\n\t"
      "mbarrier." CFM_SCREEN_WAIT ".parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra done;\n\t"
      "ld.volatile.shared.u32 now, [%4];\n\t"
      "setp.ne.u32 p, now, 0;\n\t"
      "@p bra done;\n\t"
      "mov.u32 now, %%globaltimer_lo;\n\t"
      "sub.u32 now, now, start;\n\t"
      "setp.lt.u32 p, now, %6;\n\t"
      "@p bra drain;\n\t"
      "st.volatile.shared.u32 [%4], 1;\n"
      "done:\n\t}"
      : "+r"(alive)
      : "r"(bar), "r"(parity), "r"(abort), "r"(late), "r"(static_cast<uint32_t>(CFM_SCREEN_WAIT_NS)),
        "r"(CFM_SCREEN_DRAIN_NS)
      : "memory");
}

// One lane of the warp, known to the compiler as one (instructions of a single thread then need no
// search for the active lane).
__device__ __forceinline__ bool elect_lane() {
  uint32_t one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(one));
  return one != 0;
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

// Sixteen columns of this thread's row.
__device__ __forceinline__ void store_columns16(uint32_t address, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(address),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

// Codes of four coordinates in the upper bits of their bytes, 64 times their value; m as in codes_of,
// counted from above.  (Shifts to the left, which the FMA pipe does as products, and so are the sums in
// combine(): the masks alone fill half of the integer pipe's time.)
__device__ __forceinline__ uint32_t codes_above(uint32_t word, int m) {
  return (word << (6 - 2 * m)) & 0xc0c0c0c0u;
}

// The dot product of a row from the three sums over its codes (64 times the digits' sums) and `base`,
// the negative sum of the values: code = trit + 1.
__device__ __forceinline__ int combine(const int* c, int base) {
  int dot;
  asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(dot) : "r"(c[1] * 256 + c[0]), "r"(1 << 26), "r"(c[2] * 1024 + base));
  return dot;  // the first part over 64: it is a multiple
}

// Accumulators of this thread's row, complete once load_wait() has returned.
__device__ __forceinline__ void load_columns16(uint32_t address, int* c) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]),
        "=r"(c[7]), "=r"(c[8]), "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]),
        "=r"(c[14]), "=r"(c[15])
      : "r"(address)
      : "memory");
}
__device__ __forceinline__ void load_columns8(uint32_t address, int* c) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]),
        "=r"(c[7])
      : "r"(address)
      : "memory");
}
__device__ __forceinline__ void load_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace tc

// grid (ceil(I / 128), most passes of TOKENS tokens), 192 threads; `dead_rows` more rows of CTAs
// clear the projections of the dead ones of the call's `pairs`.
template <int TOKENS, bool RISK>
__global__ void __launch_bounds__(kScreenThreads, Screen<TOKENS, RISK>::kPerSm)
    k_screen_tc(Layer L, Workspace ws, const uint8_t* padding, int pairs, int dead_rows) {
  using S = Screen<TOKENS, RISK>;
  using namespace tc;
  extern __shared__ __align__(1024) uint8_t screen_shared[];
  __shared__ uint64_t barriers[S::kCodeRing + 4 + 2 * S::kDigitRing];
  __shared__ uint32_t tmem_holder[2];
  __shared__ int abort_flag, late_flag, s_issued[2], s_fetched, s_pair[TOKENS], s_token[TOKENS];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(kFull, tid >> 5, 0);  // known to be the same in all lanes
  const uint32_t abort = shared_u32(&abort_flag), late = shared_u32(&late_flag);
  const int I = L.I, B = L.B, rows = 2 * I, c0 = blockIdx.x * kScreenChannels;
  const int channels = min(kScreenChannels, I - c0);
  const int busy_warps = (channels + 31) / 32;  // that hold channels
  // Barriers: a block's codes have landed (one per place of the ring); per tile, the rows of its
  // product are in place, and the product is complete; per place of their
  // ring, digits have landed and may be replaced.
  const uint32_t landed = shared_u32(barriers), ready = landed + 8 * S::kCodeRing, done = ready + 16, digits_landed = done + 16;
  const uint32_t digits_free = digits_landed + 8 * S::kDigitRing;
  if (warp == 5 && lane == 0) {
    abort_flag = late_flag = 0;
    for (int i = 0; i < S::kCodeRing; ++i) barrier_init(landed + 8 * i, 1);
    for (int i = 0; i < 2; ++i) {
      barrier_init(ready + 8 * i, busy_warps);
      barrier_init(done + 8 * i, 1);
    }
    for (int i = 0; i < 2 * S::kDigitRing; ++i) barrier_init(digits_landed + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();  // the warp's elected thread uses them before the CTA meets
  grid_dependency_wait();  // the digits and the passes are complete
  if (blockIdx.y + dead_rows >= gridDim.y) {
    clear_dead(L, ws, padding, pairs, dead_rows);
    return;
  }
  const int4 pass = *reinterpret_cast<const int4*>(ws.pass_work + blockIdx.y);
  if (static_cast<int>(blockIdx.y) >= ws.work_counts[kPassCount]) return;
  const int e = pass.x, first = pass.y, count = pass.z;
  const uint32_t codes = shared_u32(screen_shared), digits = codes + S::kCodeRing * S::kCodeBytes;

  // Of warp 5: codes and scales of the next block.
  const uint8_t* next_codes = reinterpret_cast<const uint8_t*>(L.sketch_grouped) +
                              (static_cast<size_t>(e) * B * rows + c0) * 32;
  const __half* next_scales = L.statistics + static_cast<size_t>(e) * B * 2 * rows + c0;
  const size_t up_codes = static_cast<size_t>(I) * 32, code_step = static_cast<size_t>(rows) * 32;
  auto fetch_codes = [&](uint32_t to, uint32_t bar) {
    barrier_expect(bar, channels * 68);
    copy_bulk(to, next_codes, channels * 32, bar);
    copy_bulk(to + kScreenChannels * 32, next_codes + up_codes, channels * 32, bar);
    copy_bulk(to + kScreenChannels * 64, next_scales, channels * 2, bar);
    copy_bulk(to + kScreenChannels * 66, next_scales + I, channels * 2, bar);
    next_codes += code_step;
    next_scales += 2 * rows;
  };
  int fetched = min(B, S::kCodeRing);
  if (warp == 5) {
    if (elect_lane())
      for (int b = 0; b < fetched; ++b) fetch_codes(codes + b * S::kCodeBytes, landed + 8 * b);
    __syncwarp();
  }
  // The small piece first: were the large ones held by CTAs that wait for a small one, none would end.
  if (warp == 4) {
    if (S::kSmall)
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(shared_u32(tmem_holder + 1))
                   : "memory");
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(shared_u32(tmem_holder)),
                 "n"(S::kLarge)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // First operands of the gate and the up tile, sums.
  const uint32_t tmem_rows[2] = {TOKENS == 16 ? tmem_holder[1] : tmem_holder[0], tmem_holder[0] + (TOKENS == 16 ? 0 : 32)};
  const uint32_t tmem_sums = TOKENS == 4 ? tmem_holder[1] : tmem_rows[1] + 32;
  // Per block and two tokens the scales of the fixed point and the sums of the values; energies.
  int4* factor = reinterpret_cast<int4*>(screen_shared + S::kRing);
  float* energy = reinterpret_cast<float*>(factor + TOKENS / 2 * B);

  // One thread issues the four steps of a tile's product; `second` is the low word of the digits'
  // descriptor.
  const uint64_t second_base = matrix_descriptor(digits);
  auto issue = [&](auto which, uint32_t second) {
    constexpr int tile = decltype(which)::value;
#pragma unroll
    for (int step = 0; step < 4; ++step)
      mma_i8(tmem_sums + tile * S::kSumsStep, tmem_rows[tile] + 8 * step,
             (second_base & 0xffffffff00000000ull) | (second + (step * S::kDigitStep >> 4)),
             instruction_descriptor(S::kColumns), step > 0);
    mma_commit(done + 8 * tile);
  };
  constexpr uint32_t kDigitPlaces = S::kDigitBytes >> 4;  // of the descriptor, from place to place
  constexpr std::integral_constant<int, 0> gate{};
  constexpr std::integral_constant<int, 1> up{};

  if (warp == 4) {
    // ---- digits, and the products of the gate tile ----
    const int token = ws.group_pairs[first + min(lane & (TOKENS - 1), count - 1)] / L.K;
    constexpr int kPieces = 3 * TOKENS * 8 / 32;  // of a block's digits, per lane
    const int8_t* from[kPieces];
    uint32_t to[kPieces];
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int piece = lane + 32 * i, column = piece >> 3, chunk = piece & 7, t = column / 3;
      const int of = __shfl_sync(kFull, token, t);
      from[i] = t < count ? ws.limbs + (static_cast<size_t>(of) * B * 3 + (column - 3 * t)) * kBlock + 16 * chunk
                          : nullptr;
      to[i] = digits + (chunk >> 1) * S::kDigitStep + (column >> 3) * 256 + (chunk & 1) * 128 + (column & 7) * 16;
    }
    auto fetch = [&](int place) {  // the next block
#pragma unroll
      for (int i = 0; i < kPieces; ++i)
        if (from[i]) {
          copy_async16(to[i] + place * S::kDigitBytes, from[i]);
          from[i] += 3 * kBlock;
        }
    };
#pragma unroll
    for (int b = 0; b < S::kDigitRing - 1; ++b) {
      if (b < B) fetch(b);
      copy_async_commit();
    }
    int place = 0, refill = S::kDigitRing - 1, turn = 0;
    uint32_t second = static_cast<uint32_t>(second_base);
    int alive = 1, issued = 0;
    for (int b = 0; b < B; ++b) {
      copy_async_wait<S::kDigitRing - 2>();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();  // the block's digits have landed, for all lanes
      barrier_arrive(digits_landed + 8 * place, lane == 0);
      barrier_wait(ready, b & 1, abort, alive);
      if (!__all_sync(kFull, alive)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_lane()) issue(gate, second);
      __syncwarp();
      ++issued;
      if (b + S::kDigitRing - 1 < B) {  // into the place of the block before this one
        if (b) barrier_wait(digits_free + 8 * refill, turn, abort, alive);
        if (!__all_sync(kFull, alive)) break;
        fetch(refill);
      }
      copy_async_commit();
      place = place + 1 == S::kDigitRing ? 0 : place + 1;
      second = place ? second + kDigitPlaces : static_cast<uint32_t>(second_base);
      refill = refill + 1 == S::kDigitRing ? 0 : refill + 1;
      if (refill == 0 && b) turn ^= 1;
    }
    copy_async_wait<0>();
    if (lane == 0) s_issued[0] = issued;
  } else if (warp == 5) {
    // ---- codes and scales, and the products of the up tile ----
    if (elect_lane()) {
      int alive = 1, issued = 0;
      uint32_t place = codes, bar = landed, free = digits_free + 8 * (S::kDigitRing - 1), turn = 0;
      uint32_t second = static_cast<uint32_t>(second_base), digit_bar = digits_landed;
      for (int b = 0; b < B; ++b) {
        barrier_wait(digit_bar, turn, abort, alive);
        barrier_wait(ready + 8, b & 1, abort, alive);
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue(up, second);
        ++issued;
        // The rows of this block came after the products of the one before, whose digits may go.
        if (b) barrier_arrive(free, 1);
        if (fetched < B) {  // the block's codes have been read
          fetch_codes(place, bar);
          ++fetched;
        }
        place += S::kCodeBytes;
        bar += 8;
        if (bar == ready) {
          place = codes;
          bar = landed;
        }
        free = digit_bar + 8 * S::kDigitRing;
        digit_bar += 8;
        second += kDigitPlaces;
        if (digit_bar == digits_free) {
          digit_bar = digits_landed;
          second = static_cast<uint32_t>(second_base);
          turn ^= 1;
        }
      }
      s_issued[1] = issued;
      s_fetched = fetched;
    }
    __syncwarp();
  } else {
    if (RISK)  // the variances, 128 bytes at a time, for the scores at the end (5 tokens: 17.0 us without, 16.3)
      for (int i = tid; i < 4 * B; i += kScreenChannels) {
        const int channel = c0 + 64 * (i & 1);
        if (channel < I)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(L.statistics + (static_cast<size_t>(e) * B * 2 + 2 * (i >> 2) + 1) * rows +
                                                         (i & 2 ? I : 0) + channel));
      }
    const int own = tid % TOKENS, own_pair = ws.group_pairs[first + min(own, count - 1)], own_token = own_pair / L.K;
    if (tid < TOKENS) {
      s_pair[tid] = own_pair;
      s_token[tid] = own_token;
    }
    const int2* factors_in = reinterpret_cast<const int2*>(ws.exponents) + static_cast<size_t>(own_token) * B;
    for (int b = tid / TOKENS; b < B; b += 128 / TOKENS) {
      const int2 f = factors_in[b];
      int* to = reinterpret_cast<int*>(factor + (b * TOKENS + own) / 2) + (own & 1);
      to[0] = __float_as_int(unscale_of(f.x));
      to[2] = -f.y;
      if (RISK) energy[b * TOKENS + own] = ws.norms[static_cast<size_t>(own_token) * B + b];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (warp < busy_warps) {
      const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;
      float run[2][TOKENS], scale[2] = {0.0f, 0.0f};
      // kLeads in the warp's leader, kFollows in its other threads, 0 once a wait has run out.  A leader that
      // has given up arrives no more, so a product is issued only while every warp's waits have ended in
      // time, and a thread that saw the last product's end knows that all copies have landed.
      constexpr int kFollows = 1, kLeads = 2;
      int state;
      asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\tselp.s32 %0, %2, %3, p;\n\t}"
                   : "=r"(state) : "r"(lane), "n"(kLeads), "n"(kFollows));
#pragma unroll
      for (int t = 0; t < TOKENS; ++t) run[0][t] = run[1][t] = 0.0f;
      // The sums of eight tokens of the tile's product before the next one; load_wait() completes them.
      auto load_sums = [&](int tile, int half, int (&c)[24]) {
        const uint32_t sums = tmem_sums + lanes + tile * S::kSumsStep + 24 * half;
        load_columns16(sums, c);
        if (TOKENS > 4 && count > 8 * half + 4) load_columns8(sums + 16, c + 16);
      };
      // Adds them, block b, to the projections, four tokens at a time.
      auto rescale = [&](auto which, int half, int b, const int (&c)[24]) {
        constexpr int tile = decltype(which)::value;
        const Pair scales = pair_of(scale[tile], scale[tile]);
        const int4* factors = factor + (b * TOKENS + 8 * half) / 2;
#pragma unroll
        for (int four = 0; four < (TOKENS > 4 ? 2 : 1); ++four) {
          if (TOKENS > 4 && 8 * half + 4 * four >= count) break;
#pragma unroll
          for (int two = 2 * four; two < 2 * four + 2; ++two) {
            const int4 f = factors[two];
            const int t = 8 * half + 2 * two, j = 6 * two;
            const Pair d = pair_mul(pair_of(__int2float_rn(combine(&c[j], f.z)), __int2float_rn(combine(&c[j + 3], f.w))),
                                    pair_of(__int_as_float(f.x), __int_as_float(f.y)));
            float p0, p1;
            pair_split(pair_mul(scales, d), p0, p1);
            run[tile][t] = __fadd_rn(run[tile][t], p0);
            run[tile][t + 1] = __fadd_rn(run[tile][t + 1], p1);
          }
        }
      };
      // Tile `which` of block b: its codes become the product's first operand while the sums of the
      // tile's product of the block before come in; then those are added.
      auto step = [&](auto which, auto begin, int b, uint32_t place) {
        constexpr int tile = decltype(which)::value;
        constexpr bool kFirst = decltype(begin)::value;  // block 0
        int c[24];
        if constexpr (!kFirst) {
          barrier_wait_product(done + 8 * tile, (b - 1) & 1, abort, late, state);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          load_sums(tile, 0, c);
        }
        const uint32_t at = place + tile * (kScreenChannels * 32) + 32 * tid;
        const uint4 lo = load_shared16(at), hi = load_shared16(at + 16);
        const float next_scale = __half2float(reinterpret_cast<const __half*>(
            screen_shared + (place - codes) + kScreenChannels * 64)[tile * kScreenChannels + tid]);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const uint4 word = part ? hi : lo;
          uint32_t v[16];
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            v[m] = codes_above(word.x, m);
            v[4 + m] = codes_above(word.y, m);
            v[8 + m] = codes_above(word.z, m);
            v[12 + m] = codes_above(word.w, m);
          }
          store_columns16(tmem_rows[tile] + lanes + 16 * part, v);
        }
        if constexpr (!kFirst) {
          load_wait();
          rescale(which, 0, b - 1, c);
          if (TOKENS == 16 && count > 8) {
            load_sums(tile, 1, c);
            load_wait();
            rescale(which, 1, b - 1, c);
          }
        }
        scale[tile] = next_scale;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        barrier_arrive(ready + 8 * tile, state == kLeads);  // the rows are in place, the sums read
      };
      auto finish = [&](auto which) {  // the last block's product
        constexpr int tile = decltype(which)::value;
        int c[24];
        barrier_wait_product(done + 8 * tile, (B - 1) & 1, abort, late, state);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int half = 0; half < (TOKENS + 7) / 8; ++half) {
          if (8 * half >= count) break;
          load_sums(tile, half, c);
          load_wait();
          rescale(which, half, B - 1, c);
        }
      };
      barrier_wait(landed, 0, abort, state);
      step(gate, std::true_type{}, 0, codes);
      step(up, std::true_type{}, 0, codes);
      uint32_t place = codes + S::kCodeBytes, bar = landed + 8, parity = 0;
#pragma unroll 1
      for (int b = 1; b < B; ++b) {
        barrier_wait(bar, parity, abort, state);
        step(gate, std::false_type{}, b, place);
        step(up, std::false_type{}, b, place);
        place += S::kCodeBytes;
        bar += 8;
        if (bar == ready) {
          place = codes;
          bar = landed;
          parity ^= 1;
        }
      }
      finish(gate);
      finish(up);
      grid_dependency_release();  // the selection may be scheduled; it waits for this grid

      // Projections out, scores and features of the pass's tokens in turn: the sums go through shared
      // memory, so that the code is there once.  The ring has been read by every warp.  A channel whose sums
      // did not come in time leaves nothing.
      const int channel = c0 + tid;
      if (tid < channels && state) {
        float* mine = reinterpret_cast<float*>(screen_shared) + tid;
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) {
          mine[t * S::kStride] = run[0][t];
          mine[t * S::kStride + kScreenChannels] = run[1][t];
        }
        if (RISK) {
          // Residual variances: per block, in block order, the row's times the energy of the token's
          // kept coordinates.
          float spread[2][TOKENS];
#pragma unroll
          for (int t = 0; t < TOKENS; ++t) spread[0][t] = spread[1][t] = 0.0f;
          const __half* plane = L.statistics + (static_cast<size_t>(e) * B * 2 + 1) * rows + channel;
          for (int b0 = 0; b0 < B; b0 += kScreenAhead) {
            __half v[2][kScreenAhead];
#pragma unroll
            for (int i = 0; i < kScreenAhead; ++i) {
              const __half* at = plane + static_cast<size_t>(min(b0 + i, B - 1)) * 2 * rows;
              v[0][i] = at[0];
              v[1][i] = at[I];
            }
#pragma unroll
            for (int i = 0; i < kScreenAhead; ++i) {
              if (b0 + i >= B) break;
              const float vg = __half2float(v[0][i]), vu = __half2float(v[1][i]);
              const float4* in = reinterpret_cast<const float4*>(energy + (b0 + i) * TOKENS);
#pragma unroll
              for (int four = 0; four < TOKENS / 4; ++four) {
                if (4 * four >= count) break;
                const float4 en = in[four];
                const Pair energies[2] = {pair_of(en.x, en.y), pair_of(en.z, en.w)};
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                  const int t = 4 * four + 2 * j;
                  float p0, p1;
                  pair_split(pair_mul(pair_of(vg, vg), energies[j]), p0, p1);
                  spread[0][t] = __fadd_rn(spread[0][t], p0);
                  spread[0][t + 1] = __fadd_rn(spread[0][t + 1], p1);
                  pair_split(pair_mul(pair_of(vu, vu), energies[j]), p0, p1);
                  spread[1][t] = __fadd_rn(spread[1][t], p0);
                  spread[1][t + 1] = __fadd_rn(spread[1][t + 1], p1);
                }
              }
            }
          }
#pragma unroll
          for (int t = 0; t < TOKENS; ++t) {
            mine[t * S::kStride + 2 * kScreenChannels] = spread[0][t];
            mine[t * S::kStride + 3 * kScreenChannels] = spread[1][t];
          }
        }
        const CandidateFactors factors = candidate_factors(L, e, channel);
#pragma unroll 1
        for (int t = 0; t < count; ++t) {
          const float* from = mine + t * S::kStride;
          const float g = from[0], u = from[kScreenChannels];
          const float vg = RISK ? from[2 * kScreenChannels] : 0.0f, vu = RISK ? from[3 * kScreenChannels] : 0.0f;
          const size_t at = static_cast<size_t>(s_token[t]) * L.N + static_cast<size_t>(s_pair[t]) * I + channel;
          ws.partial[at] = g;
          ws.partial[at + L.N] = u;
          if (RISK) {
            ws.variances[at] = vg;
            ws.variances[at + L.N] = vu;
          }
          finish_candidate(L, ws, s_pair[t], channel, factors, g, u, vg, vu);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 4) {
    if (abort_flag) {
      // Nothing may outlive the CTA: the last products, each place's last codes.  (Where no wait ran out, the
      // decoding warps have seen the end of all.)
      int alive = 1;
      for (int tile = 0; tile < 2; ++tile)
        if (s_issued[tile])
          barrier_wait(done + 8 * tile, (s_issued[tile] - 1) & 1, late, alive, CFM_SCREEN_DRAIN_NS);
      for (int p = 0; p < min(s_fetched, S::kCodeRing); ++p)
        barrier_wait(landed + 8 * p, ((s_fetched - p - 1) / S::kCodeRing) & 1, late, alive, CFM_SCREEN_DRAIN_NS);
      __syncwarp();
      if (lane == 0) atomicExch(&ws.status[0], 1);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_holder[0]), "n"(S::kLarge)
                 : "memory");
    if (S::kSmall)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem_holder[1]) : "memory");
  }
}
