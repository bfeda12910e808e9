// Device helpers of the sparse MoE decode reader (sm_100a).
//
// The arithmetic in this file is *pinned*: every operation is an IEEE-754
// single-precision add, multiply, divide or fused multiply-add issued through
// an explicit intrinsic, so the compiler can neither reassociate nor contract
// it, and a host restatement using the same operation sequence reproduces the
// results bit for bit.  Channel selection depends only on pinned arithmetic and
// on exact integer dot products.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cfm {

constexpr int kBlock = 128;          // coordinates per rotation block
constexpr int kWordRows = 16;        // sketch rows per 32-bit word
constexpr int kQuantBits = 21;       // block maximum maps into [2^21, 2^22]
constexpr int kDownTileRows = 64;    // kept rows per down tile
constexpr int kEncodeTileRows = 256; // channels per encoder tile
constexpr unsigned kFull = 0xffffffffu;

// Round an FP32 value to BF16 (nearest even) and widen it again.
__device__ __forceinline__ float bf16_round(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}

// exp(x) from Cody-Waite reduction and a degree-7 Horner polynomial.
// exp(x) = 2^n * p(r), n = rint(x * log2 e), r = x - n * ln 2 (two-term split).
// Saturates to +inf from 88 and to 0 below -87; NaN propagates.
// (Without branches, so that several go on at a time; outside of the range the result is replaced.)
__device__ __forceinline__ float pinned_exp(float x) {
  const float n = rintf(__fmul_rn(x, 1.44269502f));
  float r = __fmaf_rn(n, -0.693145752f, x);
  r = __fmaf_rn(n, -1.42860677e-06f, r);
  float p = 1.98412701e-04f;
  p = __fmaf_rn(p, r, 1.38888892e-03f);
  p = __fmaf_rn(p, r, 8.33333377e-03f);
  p = __fmaf_rn(p, r, 4.16666679e-02f);
  p = __fmaf_rn(p, r, 1.66666672e-01f);
  p = __fmaf_rn(p, r, 0.5f);
  p = __fmaf_rn(p, r, 1.0f);
  p = __fmaf_rn(p, r, 1.0f);
  const uint32_t e = static_cast<uint32_t>(static_cast<int>(n)) + 127u;  // in [1, 254]
  const float y = __fmul_rn(p, __uint_as_float(e << 23));
  return x >= 88.0f ? __int_as_float(0x7f800000) : x <= -87.0f ? 0.0f : x == x ? y : x;
}

// x / d, correctly rounded, from a value y within one unit in the last place of 1 / d: Markstein's
// division (IBM J. Res. Dev. 34, 1990), one step on the reciprocal and one on the quotient.  The step
// rounds the reciprocal correctly or leaves a quotient that the second one does, except where the
// significand of d is all ones: there 1 / d lies just above the middle of two values and the step ends
// on the lower one.  The upper one is (1/2 + 2^-24) 2^-k for d = (2 - 2^-23) 2^k.
// (Checked for every significand of d with both neighbours of 1 / d, and where the reciprocal does not
// round correctly, for every significand of x.)
__device__ __forceinline__ float divide_by_reciprocal(float x, float d, float y) {
  y = __fmaf_rn(__fmaf_rn(-d, y, 1.0f), y, y);
  const uint32_t bits = __float_as_uint(d);
  y = (~bits & 0x7fffffu) == 0 ? __uint_as_float(0x7f000000u - bits) : y;
  const float q = __fmul_rn(x, y);
  return __fmaf_rn(__fmaf_rn(-d, q, x), y, q);
}

// x / d, correctly rounded, for finite d from 1 on, |x| from 2^-60 on and quotients from 2^-126 on, the smallest
// normal one (SiLU comes down to 88 / e^88, 2^-120.5; GELU to 2 / (1 + e^88), just above 2^-126).  An infinite
// divisor gives NaN, which the activations replace.  Without branches, so that the five nodes of a risk score and
// several candidates go on at a time.  Large divisors are scaled for the reciprocal's sake.
__device__ __forceinline__ float divide_from_one(float x, float d) {
  const float scale = d > 1.8446744e19f ? 2.3283064e-10f : 1.0f;  // 2^64, 2^-32
  const float a = __fmul_rn(x, scale), b = __fmul_rn(d, scale);
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));  // within one unit in the last place
  return divide_by_reciprocal(a, b, y);
}

// SiLU: x / (1 + exp(-x)).  The divisor is 1 from 87 on, 2 about zero, and infinite from -88 down.
// GELU, tanh form: 0.5 x (1 + tanh(z)), z = sqrt(2/pi) (x + 0.044715 x^3), with
// tanh(z) = 1 - 2 / (exp(2 z) + 1).
// Both over one exponential and one division: the risk score has this five times over, and kernels
// that carried each form apart waited for instructions.  Every one of the 2^32 inputs gives the bits
// of the IEEE divisions.
__device__ __forceinline__ float pinned_activate(float x, int activation) {
  const bool gelu = activation == 1;
  const float infinity = __int_as_float(0x7f800000);
  float power = -x;
  if (gelu) {
    const float x3 = __fmul_rn(__fmul_rn(x, x), x);
    power = __fmul_rn(2.0f, __fmul_rn(0.797884583f, __fmaf_rn(0.044715f, x3, x)));
  }
  const float e = pinned_exp(power);
  const float q = divide_from_one(gelu ? 2.0f : x, __fadd_rn(1.0f, e));
  if (gelu) {
    const float th = __fsub_rn(1.0f, e < infinity ? q : e == e ? 0.0f : e);
    return __fmul_rn(__fmul_rn(0.5f, x), __fadd_rn(1.0f, th));
  }
  const float edge = x >= 87.0f ? x : x == -infinity ? __int_as_float(0x7fffffff) : -0.0f;
  return x >= 87.0f || x <= -88.0f ? edge : fabsf(x) < 8.6736174e-19f ? __fmul_rn(x, 0.5f) : q;  // 2^-60
}

// The gated feature with the reference's rounding points for an exactly
// computed channel: bf16(bf16(phi(bf16 g)) * bf16 u).
__device__ __forceinline__ float exact_feature(float g, float u, int activation) {
  const float gb = bf16_round(g), ub = bf16_round(u);
  return bf16_round(__fmul_rn(bf16_round(pinned_activate(gb, activation)), ub));
}

// The feature of a skipped channel from its sketch projections, `active` = phi(bf16 g): one rounding,
// bf16(phi(bf16 g) * bf16 u).
__device__ __forceinline__ float sketch_feature(float active, float u) {
  return bf16_round(__fmul_rn(active, bf16_round(u)));
}

// Point score: ((norm * phi(g)) * u)^2 * w^2 on BF16-rounded projections.
__device__ __forceinline__ float point_score(float active, float u, float norm, float w) {
  const float t = __fmul_rn(__fmul_rn(norm, active), bf16_round(u));
  return __fadd_rn(__fmul_rn(__fmul_rn(t, t), __fmul_rn(w, w)), 0.0f);
}

// Recovery-aware score: w^2 times the expected squared output error of skipping
// the channel, with the gate modelled as Gaussian around g (five Gauss-Hermite
// nodes), sketch residual variances vg and vu, down-column norm n and the
// recovery response split into alpha (along the down column) and beta (across):
//   n^2 max(E[a^2] - E[a]^2, 0) + ((n E[a] - alpha p)^2 + (beta p)^2),
// p = bf16(phi(g) u), `active` = phi(g), on BF16-rounded projections.
__device__ __forceinline__ float risk_score(float g, float active, float u, float vg, float vu, float norm,
                                            float alpha, float beta, float w, int activation) {
  const float gb = bf16_round(g), ub = bf16_round(u);
  const float sg = __fsqrt_rn(vg), su = __fsqrt_rn(vu);
  const float spread = __fadd_rn(__fmul_rn(ub, ub), __fmul_rn(su, su));
  float mu = 0.0f, second = 0.0f;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const float node = j == 0 ? -2.85697007f : j == 1 ? -1.35562618f : j == 2 ? 0.0f : j == 3 ? 1.35562618f : 2.85697007f;
    const float mass = j == 2 ? 0.533333333f : j == 1 || j == 3 ? 0.222075922f : 0.0112574113f;
    const float shift = __fmul_rn(node, sg);
    // The middle node is the gate itself (or NaN with sg).
    const float a = j == 2 ? __fadd_rn(active, shift) : pinned_activate(__fadd_rn(gb, shift), activation);
    mu = __fadd_rn(mu, __fmul_rn(__fmul_rn(mass, a), ub));
    second = __fadd_rn(second, __fmul_rn(__fmul_rn(mass, __fmul_rn(a, a)), spread));
  }
  const float p = bf16_round(__fmul_rn(active, ub));
  const float spread_error = fmaxf(__fsub_rn(second, __fmul_rn(mu, mu)), 0.0f);
  float risk = __fmul_rn(__fmul_rn(norm, norm), spread_error);
  const float along = __fsub_rn(__fmul_rn(norm, mu), __fmul_rn(alpha, p));
  const float across = __fmul_rn(beta, p);
  risk = __fadd_rn(risk, __fadd_rn(__fmul_rn(along, along), __fmul_rn(across, across)));
  return __fadd_rn(__fmul_rn(risk, __fmul_rn(w, w)), 0.0f);
}

// Two FP32 values in one 64-bit register and the packed operations on them; each half
// rounds exactly as the scalar operation does.
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair_of(float lo, float hi) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ void pair_split(Pair p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
  Pair d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// a - b: the product with -1 is exact, so the one rounding is that of the subtraction.
__device__ __forceinline__ Pair pair_sub(Pair a, Pair b) {
  return pair_fma(b, pair_of(-1.0f, -1.0f), a);
}

// 16-byte read-only load that does not allocate in L1 (streamed weights).
__device__ __forceinline__ uint4 load_stream16(const void* p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t load_stream4(const void* p) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Two BF16 values packed in a 32-bit word -> two floats (exact).
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) {
  return __uint_as_float(w & 0xffff0000u);
}

__device__ __forceinline__ uint32_t shared_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16 bytes global -> shared memory, past L1, in the thread's current cp.async group.
__device__ __forceinline__ void copy_async16(uint32_t shared, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(shared), "l"(global) : "memory");
}
__device__ __forceinline__ void copy_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int PENDING>
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

__device__ __forceinline__ uint4 load_shared16(uint32_t address) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(address)
               : "memory");
  return v;
}

// Programmatic dependent launch.  A kernel launched with programmatic stream
// serialisation may start while its predecessor in the stream is still running;
// grid_dependency_wait() returns once that predecessor has completed and its writes
// are visible, and must precede the first access to anything the predecessor wrote.
// grid_dependency_release() lets the successor of the calling grid be scheduled once
// every CTA of this grid has called it or exited.  Both do nothing in ordinary launches.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_dependency_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Exclusive scan of `value` over the CTA (blockDim.x a multiple of 32, at most
// 1024); `scratch` holds 33 ints.  Returns the sum of the earlier threads and
// writes the CTA total to `*total`.  Ends with a barrier.
__device__ __forceinline__ int block_exclusive_scan(int value, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int scan = value;
#pragma unroll
  for (int w = 1; w < 32; w <<= 1) {
    const int o = __shfl_up_sync(kFull, scan, w);
    if (lane >= w) scan += o;
  }
  __syncthreads();  // earlier users of the scratch are done
  if (lane == 31) scratch[warp] = scan;
  __syncthreads();
  if (warp == 0) {
    int t = lane < warps ? scratch[lane] : 0;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
      const int o = __shfl_up_sync(kFull, t, w);
      if (lane >= w) t += o;
    }
    scratch[lane] = t;  // inclusive scan of the warp totals
  }
  __syncthreads();
  *total = scratch[warps - 1];
  return scan - value + (warp ? scratch[warp - 1] : 0);
}

}  // namespace cfm
