// Construction-time kernel: the ternary sketch of the native gate/up rows,
// written straight into the two layouts the screen kernels read (sm_100a).
//
// Per expert, row and 128-coordinate rotation block (reference
// reader/sketch.py:84-150): rotate the row's block (signs, seven butterfly
// stages, 1/sqrt(128)); a coordinate keeps its sign when |v| > 0.7 mean|v|; the
// block's scale is the mean magnitude of the kept coordinates (over max(count,
// 1)), its residual variance mean((v - sign scale)^2); both stored FP16.
//
// The rotation is the reference's butterfly, bit for bit.  The three reductions over a
// block's 128 values (sum of magnitudes, sum of kept magnitudes, sum of squared
// residuals) are FP32 sums in a fixed order of their own (four consecutive values, then
// halves of the block, of the half, ...), which is not the order of a torch reduction: a
// coordinate whose magnitude sits within rounding of the threshold can come out
// differently from the reference builder's, and a scale can differ in its last FP16 bit.
// The readers take either sketch; parity tests use the reference builder's.
//
// What bounds it: 2 + 1/2 bytes per weight cross HBM, but every weight also takes seven
// butterfly stages, the threshold rule and two 2-bit codes, 0.75 warp instructions in all (24
// per weight and lane), of which the rotation is about a third.  They are issued at 0.62 per
// scheduler and cycle: four warps per scheduler, which 128 registers leave room for, do not
// cover what a warp waits for between two of its own, 5.2 cycles (fixed latencies 0.9, loads
// 0.75, shuffles 0.7, busy pipes 0.7; no pipe is more than 0.45 busy).  Hence the split: four lanes share a row's block,
// lane q holding the chunks 16 j + 4 q .. + 3 of it (j = 0 .. 7).  Five of the seven stages
// and all but two steps of every sum then stay inside a lane, where they run as packed
// pairs (chunks j and j + 4 of a lane in one f32x2 operation); a warp per row spent 42
// shuffles on a row's block, this spends 10.  The squares of the residual stay scalar: ptxas
// contracts a packed multiply and add in spite of the rounding modifiers, and that sum has
// to round twice.  Codes are packed by exact FP32 arithmetic (weights 1, 16, 256, 4096 on
// top of 1.5 * 2^23, whose low mantissa bits are the packed integer), and the
// coordinate-major words come from a 16 x 16 transpose of 2-bit fields over the sixteen
// rows of a warp.  128 experts of width 768, hidden size 2048: 1297 us with a warp per row,
// 428 us now (1.02 GB, 2.4 TB/s).
// Included by cfm_reader.cu inside namespace cfm.
#pragma once

constexpr int kBuildRows = 16;   // rows per warp = rows per coordinate-major word
constexpr int kBuildWarps = 8;   // 128 rows per CTA: a coordinate's words leave as 32-byte runs

// Sum of a value over the four lanes of a row, in the order of the block sums.
__device__ __forceinline__ float quad_sum(float x) {
  x = __fadd_rn(x, __shfl_xor_sync(kFull, x, 2));
  return __fadd_rn(x, __shfl_xor_sync(kFull, x, 1));
}

// Coordinate (0..15) of the 2-bit field p of a word of the row-major layout: four masked
// shifts of such a word give the byte-permute selectors of coordinates 0-3, 4-7, 8-11 and
// 12-15 (see decode_word).
__device__ __forceinline__ int field_coordinate(int p) {
  return (p & 8) + ((p & 1) << 2) + ((p & 7) >> 1);
}

// One row's block, a quarter of it per lane (`raw`: eight chunks of four BF16 values, `flip`:
// the sign bits the rotation turns over).  Returns this lane's two words of the row-major
// layout (words 2 q and 2 q + 1) and, in every lane, the block's scale and residual variance.
__device__ __forceinline__ uint2 build_row(const uint2 (&raw)[8], const uint2 (&flip)[8], int q,
                                           float& scale, float& residual) {
  Pair v[4][4];  // [j][i]: value i of chunks j and j + 4
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t ax = raw[j].x ^ flip[j].x, ay = raw[j].y ^ flip[j].y;
    const uint32_t bx = raw[j + 4].x ^ flip[j + 4].x, by = raw[j + 4].y ^ flip[j + 4].y;
    v[j][0] = pair_of(bf16_lo(ax), bf16_lo(bx));
    v[j][1] = pair_of(bf16_hi(ax), bf16_hi(bx));
    v[j][2] = pair_of(bf16_lo(ay), bf16_lo(by));
    v[j][3] = pair_of(bf16_hi(ay), bf16_hi(by));
    // Half-widths 1 and 2: the lower member takes the sum, the upper one the difference.
    const Pair a = pair_add(v[j][0], v[j][1]), d = pair_sub(v[j][0], v[j][1]);
    const Pair c = pair_add(v[j][2], v[j][3]), f = pair_sub(v[j][2], v[j][3]);
    v[j][0] = pair_add(a, c);
    v[j][2] = pair_sub(a, c);
    v[j][1] = pair_add(d, f);
    v[j][3] = pair_sub(d, f);
  }
#pragma unroll
  for (int w = 1; w <= 2; w <<= 1) {  // half-widths 4 and 8: the lanes of the row
    const float s = (q & w) ? -1.0f : 1.0f;
    const Pair own = pair_of(s, s);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[j][i] = pair_fma(v[j][i], own, __shfl_xor_sync(kFull, v[j][i], w));
  }
  float x[8][4];
  const Pair unit = pair_of(0.0883883461f, 0.0883883461f);  // float(1 / sqrt(128))
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // Half-widths 16, 32 (chunks j) and 64 (the halves of a pair).
    const Pair a = pair_add(v[0][i], v[1][i]), b = pair_sub(v[0][i], v[1][i]);
    const Pair c = pair_add(v[2][i], v[3][i]), d = pair_sub(v[2][i], v[3][i]);
    const Pair r[4] = {pair_add(a, c), pair_add(b, d), pair_sub(a, c), pair_sub(b, d)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      pair_split(r[j], lo, hi);
      v[j][i] = pair_mul(pair_of(__fadd_rn(lo, hi), __fsub_rn(lo, hi)), unit);
      pair_split(v[j][i], x[j][i], x[j + 4][i]);
    }
  }
  // Chunks pair up over the halves of the block, of the half, and so on down to the lanes.
  auto fold = [](const float (&s)[8]) {
    return quad_sum(__fadd_rn(__fadd_rn(__fadd_rn(s[0], s[4]), __fadd_rn(s[2], s[6])),
                              __fadd_rn(__fadd_rn(s[1], s[5]), __fadd_rn(s[3], s[7]))));
  };
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    s[j] = __fadd_rn(__fadd_rn(fabsf(x[j][0]), fabsf(x[j][1])),
                     __fadd_rn(fabsf(x[j][2]), fabsf(x[j][3])));
  const float cut = __fmul_rn(0.7f, __fmul_rn(fold(s), 0.0078125f));  // 0.7 * mean|v|

  // Members keep their sign; packed code + 1 of chunk j in the low half of packed[j].
  const float step = (q & 1) ? 4.0f : 1.0f;  // odd lanes' fields sit two bits higher
  const Pair weight[4] = {pair_of(step, step), pair_of(16.0f * step, 16.0f * step),
                          pair_of(256.0f * step, 256.0f * step),
                          pair_of(4096.0f * step, 4096.0f * step)};
  const float bias = 12582912.0f + 4369.0f * step;  // 1.5 * 2^23 + 0x1111 (a code of 1 each)
  Pair trit[4][4];
  uint32_t word[4];  // fields of chunk j (low half) and chunk j + 4 (high half)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    Pair packed = pair_of(bias, bias);
    s[j] = s[j + 4] = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float t[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float value = x[j + 4 * h][i];
        const bool member = fabsf(value) > cut;
        t[h] = member ? copysignf(1.0f, value) : 0.0f;
        if (member) s[j + 4 * h] = __fadd_rn(s[j + 4 * h], fabsf(value));
      }
      trit[j][i] = pair_of(t[0], t[1]);
      packed = pair_fma(trit[j][i], weight[i], packed);
    }
    float lo, hi;
    pair_split(packed, lo, hi);
    word[j] = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x5410);
  }
  const uint32_t zero_code = 0x11111111u << (q & 1 ? 2 : 0);  // set for a trit of zero
  int kept = 32;
#pragma unroll
  for (int j = 0; j < 4; ++j) kept -= __popc(word[j] & zero_code);
  kept += __shfl_xor_sync(kFull, kept, 2);
  kept += __shfl_xor_sync(kFull, kept, 1);
  scale = __fdiv_rn(fold(s), static_cast<float>(max(kept, 1)));
  const Pair minus = pair_of(-scale, -scale);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const Pair d = pair_fma(trit[j][i], minus, v[j][i]);  // the product is exact
      float lo, hi;
      pair_split(d, lo, hi);
      s[j] = i ? __fadd_rn(s[j], __fmul_rn(lo, lo)) : __fmul_rn(lo, lo);
      s[j + 4] = i ? __fadd_rn(s[j + 4], __fmul_rn(hi, hi)) : __fmul_rn(hi, hi);
    }
  }
  residual = __fmul_rn(fold(s), 0.0078125f);

  // Gather the four lanes' fields: odd and even lanes swap halves of the word list, then the
  // lower and upper pair of lanes swap the halves of the words.
  uint32_t mine[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t send = (q & 1) ? word[k] : word[k + 2];
    mine[k] = ((q & 1) ? word[k + 2] : word[k]) | __shfl_xor_sync(kFull, send, 1);
  }
  const uint32_t join = (q & 2) ? 0x3276u : 0x5410u;
  return make_uint2(__byte_perm(mine[0], __shfl_xor_sync(kFull, mine[0], 2), join),
                    __byte_perm(mine[1], __shfl_xor_sync(kFull, mine[1], 2), join));
}

// grid (B, ceil(2I / 128), E), 256 threads.  A warp takes sixteen rows of one block, eight at a
// time (lane = 4 row + q).
__global__ void __launch_bounds__(kBuildWarps * 32, 2)
    k_build_sketch(int H, int I, const __nv_bfloat16* gate_up, const int8_t* signs,
                   uint32_t* words, uint32_t* grouped, __half* statistics) {
  // Coordinate-major words of the CTA, [coordinate][warp]; the stride of 9 and the extra 8
  // per 32 coordinates put the 32 words a warp stores at a time into different banks.
  __shared__ uint32_t tile[kBlock * 9 + 3 * 8];
  const int b = blockIdx.x, e = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane & 3, r = lane >> 2;
  const int rows = 2 * I, B = H / kBlock, W = rows / kBuildRows;
  const int group0 = blockIdx.y * kBuildWarps, group = group0 + warp;
  if (group < W) {
    const int row0 = group * kBuildRows + r;
    const uint2* source = reinterpret_cast<const uint2*>(
        gate_up + (static_cast<size_t>(e) * rows + row0) * H + b * kBlock + 4 * q);
    uint2 raw[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        raw[h][j] = source[static_cast<size_t>(2 * h) * H + 4 * j];  // 8 rows of H / 4 pieces
    uint2 flip[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t s = *reinterpret_cast<const uint32_t*>(signs + b * kBlock + 16 * j + 4 * q);
      flip[j].x = ((s & 0x80u) << 8) | ((s & 0x8000u) << 16);
      flip[j].y = ((s >> 8) & 0x8000u) | (s & 0x80000000u);
    }
    uint2 own[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float scale, residual;
      own[h] = build_row(raw[h], flip, q, scale, residual);
      const int row = row0 + 8 * h;
      if (q == 0) {
        __half* plane = statistics + (static_cast<size_t>(e) * B + b) * 2 * rows + row;
        plane[0] = __float2half_rn(scale);
        plane[rows] = __float2half_rn(residual);
      }
      reinterpret_cast<uint2*>(grouped)[((static_cast<size_t>(e) * B + b) * rows + row) * 4 + q] =
          own[h];
    }
    // Transpose the 16 rows x 16 fields of each word: row bit 3 (the two halves), then row
    // bits 2, 1, 0 (lane bits 4, 3, 2) change places with the same bit of the field index.
    uint32_t t[2][2] = {{own[0].x, own[1].x}, {own[0].y, own[1].y}};
    const uint32_t bytes = (lane & 16) ? 0x3715u : 0x6240u;
    const int turn4 = (lane & 8) ? 28 : 4, turn2 = (lane & 4) ? 30 : 2;
    const uint32_t keep4 = (lane & 8) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
    const uint32_t keep2 = (lane & 4) ? 0xccccccccu : 0x33333333u;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t low = __byte_perm(t[k][0], t[k][1], 0x5410);
      t[k][1] = __byte_perm(t[k][0], t[k][1], 0x7632);
      t[k][0] = low;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t x = t[k][h];
        x = __byte_perm(x, __shfl_xor_sync(kFull, x, 16), bytes);
        uint32_t o = __shfl_xor_sync(kFull, x, 8);
        x = (x & keep4) | (__funnelshift_l(o, o, turn4) & ~keep4);
        o = __shfl_xor_sync(kFull, x, 4);
        x = (x & keep2) | (__funnelshift_l(o, o, turn2) & ~keep2);
        // Field 8 h + r of word 2 q + k, rows ascending from bit 0.
        const int c = 16 * (2 * q + k) + field_coordinate(8 * h + r);
        tile[c * 9 + (c >> 5) * 8 + warp] = x;
      }
    }
  }
  __syncthreads();
  // 32 bytes per coordinate; W is even, so a pair of words is in range or out of it.
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int c = (tid >> 2) + 64 * k, g = 2 * (tid & 3);
    if (group0 + g < W) {
      const uint32_t* in = tile + c * 9 + (c >> 5) * 8 + g;
      *reinterpret_cast<uint2*>(words + (static_cast<size_t>(e) * H + b * kBlock + c) * W + group0 +
                                g) = make_uint2(in[0], in[1]);
    }
  }
}
