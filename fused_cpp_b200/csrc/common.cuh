// Shared device helpers for the routed-expert MoE kernels (sm_100a).
//
// Arithmetic follows the reference CPU implementation statement by statement; every rounding step
// is spelled with a round-to-nearest intrinsic so that the compiler can neither fuse nor reorder it:
//   row quantiser      csrc/moe/arm/i8mm_w8a8/kernels.cpp:211-228 (NATIVE), tests/test_moe_w8a8.py:40-43 (TORCHREF)
//   exp(-gate)         csrc/moe/arm/i8mm_w8a8/kernels.cpp:200-209
//   clamped SwiGLU     csrc/moe/arm/i8mm_w8a8/kernels.cpp:230-246
//   bf16 store         csrc/moe/arm/i8mm_w8a8/kernels.cpp:194-198
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fused_moe_b200.h"

namespace fmoe {

// Layout of the status block at the start of every workspace (int32 words).
enum StatusWord : int {
  kStatusError = 0,      // first error code raised by a kernel (0 = none)
  kStatusDetail = 1,     // detail of that error (e.g. the offending flat route id)
  kStatusItems = 2,      // number of (expert, row-tile) work items of this call
  kStatusActive = 3,     // number of experts with at least one route
  kStatusWaitSite = 4,   // which bounded wait gave up (0 = none)
  kStatusItemsB = 5,     // work items of the second list (down GEMM)
  kStatusItemsC = 6,     // split mode: gate_up work items of the experts with many rows (two-SM kernel)
  kStatusItemsD = 7,     // split mode: down work items of those experts
  kStatusTallestC = 8,   // rows of the largest work item of lists C, D and (below) A, B
  kStatusTallestD = 9,
  kStatusMirror = 10,    // two words: address of page-locked host words that take the first error too (0 = none)
  kStatusTallestA = 12,
  kStatusTallestB = 13,
  kStatusWords = 16,
};

__device__ __forceinline__ void raise_error(int* status, int code, int detail, int wait_site = 0) {
  if (atomicCAS(status + kStatusError, 0, code) != 0) return;
  status[kStatusDetail] = detail;
  status[kStatusWaitSite] = wait_site;
  int* const mirror = *reinterpret_cast<int* volatile*>(status + kStatusMirror);
  if (mirror == nullptr) return;
  mirror[kStatusDetail] = detail;
  mirror[kStatusWaitSite] = wait_site;
  __threadfence_system();
  *reinterpret_cast<volatile int*>(mirror + kStatusError) = code;
}

// Word `index` of a cleared status block.
__device__ __forceinline__ int cleared_status_word(int index, const int* mirror) {
  const uint64_t address = reinterpret_cast<uint64_t>(mirror);
  return index == kStatusMirror ? static_cast<int>(address) : index == kStatusMirror + 1 ? static_cast<int>(address >> 32) : 0;
}

__device__ __forceinline__ float bf16_bits_to_f32(uint16_t bits) { return __uint_as_float(static_cast<uint32_t>(bits) << 16); }

// Nearest-even bf16 by adding 0x7fff + lsb, like the reference's store_bf16.
__device__ __forceinline__ uint16_t f32_to_bf16_bits(float value) {
  const uint32_t bits = __float_as_uint(value);
  const uint32_t lsb = (bits >> 16) & 1u;
  return static_cast<uint16_t>((bits + 0x7fffu + lsb) >> 16);
}

// fp32(2^(i/64)): the significand table of the FEXPA instruction.
__device__ __constant__ const uint32_t kExp2Table[64] = {
    0x3f800000u, 0x3f8164d2u, 0x3f82cd87u, 0x3f843a29u, 0x3f85aac3u, 0x3f871f62u, 0x3f88980fu, 0x3f8a14d5u,
    0x3f8b95c2u, 0x3f8d1adfu, 0x3f8ea43au, 0x3f9031dcu, 0x3f91c3d3u, 0x3f935a2bu, 0x3f94f4f0u, 0x3f96942du,
    0x3f9837f0u, 0x3f99e046u, 0x3f9b8d3au, 0x3f9d3edau, 0x3f9ef532u, 0x3fa0b051u, 0x3fa27043u, 0x3fa43516u,
    0x3fa5fed7u, 0x3fa7cd94u, 0x3fa9a15bu, 0x3fab7a3au, 0x3fad583fu, 0x3faf3b79u, 0x3fb123f6u, 0x3fb311c4u,
    0x3fb504f3u, 0x3fb6fd92u, 0x3fb8fbafu, 0x3fbaff5bu, 0x3fbd08a4u, 0x3fbf179au, 0x3fc12c4du, 0x3fc346cdu,
    0x3fc5672au, 0x3fc78d75u, 0x3fc9b9beu, 0x3fcbec15u, 0x3fce248cu, 0x3fd06334u, 0x3fd2a81eu, 0x3fd4f35bu,
    0x3fd744fdu, 0x3fd99d16u, 0x3fdbfbb8u, 0x3fde60f5u, 0x3fe0ccdfu, 0x3fe33f89u, 0x3fe5b907u, 0x3fe8396au,
    0x3feac0c7u, 0x3fed4f30u, 0x3fefe4bau, 0x3ff28177u, 0x3ff5257du, 0x3ff7d0dfu, 0x3ffa83b3u, 0x3ffd3e0cu,
};

// Approximate reciprocal (within one unit in the last place), the seed of quotient_fast.
__device__ __forceinline__ float reciprocal_seed(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}

// 1 / d rounded to nearest for d in [1, 2^40]: one Newton step on the seed.  (That it is the correctly rounded one is what
// quotient_fast rests on; with a seed one unit high the step would miss it at 32 mantissas.  tests/test_gpu_quotient.py compares it with
// __frcp_rn for every mantissa.)
__device__ __forceinline__ float reciprocal_fast(float d) {
  const float seed = reciprocal_seed(d);
  return __fmaf_rn(seed, __fmaf_rn(-d, seed, 1.0f), seed);
}

// n / d rounded to nearest for d in [1, 2^40] and |n| in [2^-60, 2^60]: by Markstein's theorem (P. W. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990) a quotient by the correctly rounded
// reciprocal that is corrected once by its exact remainder times that reciprocal is the correctly rounded one; in these ranges
// no step over- or underflows.  __fdiv_rn gives the same bits but tests its operands
// and branches, which keeps the compiler from overlapping the elements of an unrolled loop.
// (tests/test_gpu_quotient.py compares the two for every mantissa of d.)
__device__ __forceinline__ float quotient_fast(float n, float d) {
  const float r = reciprocal_fast(d);
  const float q = __fmul_rn(n, r);
  return __fmaf_rn(__fmaf_rn(-d, q, n), r, q);
}

// exp(-gate) with the reference's FEXPA evaluator: range reduction to multiples of 1/64 in the
// exponent, a table significand and a degree-2 correction.  `table` is kExp2Table or a copy of it in
// shared memory: lanes index it with different values, which the constant cache serialises (one
// address per pass) while shared memory serves 32 banks at once.
__device__ __forceinline__ float expneg_clamped(float x, const uint32_t* table) {
  const float encoded = __fmaf_rn(x, 1.4426950216293335f, 196735.0f);
  const float k = __fsub_rn(encoded, 196735.0f);
  float residual = __fmaf_rn(-k, 0.693145751953125f, x);
  residual = __fmaf_rn(-k, 1.428606765330187e-06f, residual);
  const uint32_t enc_bits = __float_as_uint(encoded);
  const uint32_t scale_bits = (((enc_bits >> 6) & 0xffu) << 23) | (table[enc_bits & 63u] & 0x007fffffu);
  const float scale = __uint_as_float(scale_bits);
  const float polynomial = __fmaf_rn(residual, 0.5000003576278687f, 1.000003695487976f);
  return __fmaf_rn(scale, __fmul_rn(polynomial, residual), scale);
}

__device__ __forceinline__ float expneg_with(float gate, const uint32_t* table) {
  float x = -gate;
  x = fminf(x, 87.0f);
  x = fmaxf(x, -87.0f);
  return expneg_clamped(x, table);
}

__device__ __forceinline__ float expneg(float gate) { return expneg_with(gate, kExp2Table); }

// (gate*up)/(exp(-gate)+1) -> bf16, with the optional +-limit clamp (limit <= 0: none).
__device__ __forceinline__ uint16_t swiglu_to_bf16_with(float gate, float up, float limit, const uint32_t* table) {
  if (limit > 0.0f) {
    gate = fminf(gate, limit);
    up = fmaxf(fminf(up, limit), -limit);
  }
  const float value = __fdiv_rn(__fmul_rn(gate, up), __fadd_rn(expneg_with(gate, table), 1.0f));
  return f32_to_bf16_bits(value);
}

// swiglu_to_bf16_with for N elements, the same bits.  Where every gate lies in [-27, 80] (no clamp of the exponent, and
// 1 + exp(-gate) below 2^40) and every product in the range of quotient_fast, no element has a branch and the N chains
// overlap; what lies outside, zeros, infinities and NaN among it, sends all N through the plain statement.
template <int N>
__device__ __forceinline__ void swiglu_group(const float (&gate)[N], const float (&up)[N], float limit, const uint32_t* table,
                                             uint16_t (&out)[N]) {
  constexpr uint32_t kSmallest = 0x21800000u;          // 2^-60
  constexpr uint32_t kRange = 0x5d800000u - kSmallest;  // up to 2^60
  const float clamp = limit > 0.0f ? limit : __int_as_float(0x7f800000);
  float product[N], denominator[N];
  uint32_t worst = 0;
  float lowest = 0.0f, highest = 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float g = fminf(gate[i], clamp);
    const float u = fmaxf(fminf(up[i], clamp), -clamp);
    product[i] = __fmul_rn(g, u);
    denominator[i] = __fadd_rn(expneg_clamped(-g, table), 1.0f);
    worst = max(worst, (__float_as_uint(product[i]) & 0x7fffffffu) - kSmallest);
    lowest = fminf(lowest, g);
    highest = fmaxf(highest, g);
  }
  if (worst <= kRange && lowest >= -27.0f && highest <= 80.0f) {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __bfloat16_as_ushort(__float2bfloat16_rn(quotient_fast(product[i], denominator[i])));
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = swiglu_to_bf16_with(gate[i], up[i], limit, table);
  }
}

// The other gated activations of the reference's BF16 op (csrc/moe/arm/common/fused_moe_bf16_tiled.cpp:1911-1936,
// arithmetic as in src/fused_cpp/moe/naive.py:28-54).
//   gelu:      0.5 * gate * (1 + erf(gate / sqrt(2))) * up
//   swigluoai: gate = min(gate, 7), up = clamp(up, +-7), (up + 1) * gate * sigmoid(1.702 * gate)
#define FMOE_ACT_SILU 0
#define FMOE_ACT_GELU 2
#define FMOE_ACT_SWIGLUOAI 3

// The activation as a type: the element loops are instances of it.  As a call inside the loop (a function kept out of line, one
// element at a time) the chain of an exponential and a division was paid in full for every element: 50 rows x 128 channels
// of swigluoai took an epilogue 10 us (200 tokens of the 16-expert layer 121.9 us, 113.3 with this and eight epilogue warps).
template <int kActivation>
struct ActivationTag {
  static constexpr int value = kActivation;
};

// Calls body(ActivationTag) with the gated activation of this launch; kSiluOnly: the path has no other.
template <bool kSiluOnly, typename Body>
__device__ __forceinline__ void with_activation(int activation, Body&& body) {
  if (kSiluOnly || activation == FMOE_ACT_SILU) {
    body(ActivationTag<FMOE_ACT_SILU>{});
  } else if (activation == FMOE_ACT_GELU) {
    body(ActivationTag<FMOE_ACT_GELU>{});
  } else {
    body(ActivationTag<FMOE_ACT_SWIGLUOAI>{});
  }
}

template <typename Tag>
__device__ __forceinline__ uint16_t gated_to_bf16(Tag, float gate, float up, float limit, const uint32_t* table) {
  if constexpr (Tag::value == FMOE_ACT_SILU) {
    return swiglu_to_bf16_with(gate, up, limit, table);
  } else if constexpr (Tag::value == FMOE_ACT_GELU) {
    return f32_to_bf16_bits(0.5f * gate * (1.0f + erff(gate * 0.70710678118654752440f)) * up);
  } else {
    gate = fminf(gate, 7.0f);
    up = fmaxf(fminf(up, 7.0f), -7.0f);
    const float glu = gate / (1.0f + expf(-1.702f * gate));
    return f32_to_bf16_bits((up + 1.0f) * glu);
  }
}

// N elements of either kind.
template <typename Tag, int N>
__device__ __forceinline__ void gated_group(Tag act, const float (&gate)[N], const float (&up)[N], float limit, const uint32_t* table,
                                            uint16_t (&out)[N]) {
  if constexpr (Tag::value == FMOE_ACT_SILU) {
    swiglu_group(gate, up, limit, table, out);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = gated_to_bf16(act, gate[i], up[i], limit, table);
  }
}

__device__ __forceinline__ uint16_t swiglu_to_bf16(float gate, float up, float limit) {
  return swiglu_to_bf16_with(gate, up, limit, kExp2Table);
}

// int32 accumulator -> fp32 with the activation and per-channel weight scale.
__device__ __forceinline__ float dequantize(int32_t accumulator, float activation_scale, float channel_scale, int numerics) {
  const float value = static_cast<float>(accumulator);  // cvt.rn.f32.s32
  if (numerics == FMOE_NUMERICS_NATIVE) return __fmul_rn(value, __fmul_rn(activation_scale, channel_scale));
  return __fmul_rn(__fmul_rn(value, activation_scale), channel_scale);
}

// Two-plane (16-bit fixed point) activations.  A row's values are X = rint(x / scale), scale = amax / kPlaneFullScale
// (1 for an all-zero row), |X| <= 32512 = 127 * 256, carried as X = 256 * high + low with low in [-128, 127] and high
// in [-127, 127].  The exact integer dot product with an int8 weight row is 256 * acc(high) + acc(low) (below 2^37 in
// magnitude); it is rounded to fp32 once, then scaled by the row scale and the channel scale in that order.
constexpr float kPlaneFullScale = 32512.0f;

__device__ __forceinline__ float plane_row_scale(float amax) { return amax > 0.0f ? __fdiv_rn(amax, kPlaneFullScale) : 1.0f; }

__device__ __forceinline__ int plane_fixed_point(float value, float scale) {
  const float rounded = rintf(__fdiv_rn(value, scale));  // ties to even
  return static_cast<int>(fmaxf(fminf(rounded, kPlaneFullScale), -kPlaneFullScale));
}

__device__ __forceinline__ float dequantize_planes(int32_t high, int32_t low, float activation_scale, float channel_scale) {
  const long long exact = static_cast<long long>(high) * 256 + static_cast<long long>(low);
  return __fmul_rn(__fmul_rn(__ll2float_rn(exact), activation_scale), channel_scale);
}

__device__ __forceinline__ float row_scale_from_amax(float amax, int numerics) {
  if (numerics == FMOE_NUMERICS_NATIVE) return amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
  const float scale = __fdiv_rn(amax, 127.0f);
  return scale < 1.0e-30f ? 1.0e-30f : scale;
}

// One activation value -> int8.  `scale_or_inverse` is 1/scale for NATIVE and scale for TORCHREF; clamp_low: -127, or -128
// for the single dense product.
__device__ __forceinline__ int quantize_value(float value, float scale_or_inverse, int numerics, float clamp_low = -127.0f) {
  if (numerics == FMOE_NUMERICS_NATIVE) {
    float scaled = __fmul_rn(value, scale_or_inverse);
    scaled = fmaxf(fminf(scaled, 127.0f), -127.0f);
    return static_cast<int>(roundf(scaled));  // ties away from zero
  }
  float rounded = rintf(__fdiv_rn(value, scale_or_inverse));  // ties to even
  rounded = fmaxf(fminf(rounded, 127.0f), clamp_low);
  return static_cast<int>(rounded);
}

__device__ __forceinline__ float max_or_nan(float a, float b) {
  float result;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(result) : "f"(a), "f"(b));
  return result;
}

// Four values by the exact statement.
__device__ __forceinline__ uint32_t quantize4_torchref_exact(float v0, float v1, float v2, float v3, float scale, float clamp_low) {
  const float values[4] = {v0, v1, v2, v3};
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    packed |= (static_cast<uint32_t>(quantize_value(values[i], scale, FMOE_NUMERICS_TORCHREF, clamp_low)) & 0xffu) << (8 * i);
  }
  return packed;
}

// The same out of line.  A row kernel runs for a few microseconds and fetches its instructions cold; four divisions at each of its
// unrolled groups, which it hardly ever enters, were most of its code (4072 rows of 2048 columns, a warp each, start to end
// behind the wait: 13.7 us with them, 6 to 7 us without; 509 Zipf tokens 430.7 -> 427.4 us).
static __device__ __noinline__ uint32_t quantize4_torchref_call(float v0, float v1, float v2, float v3, float scale, float clamp_low) {
  return quantize4_torchref_exact(v0, v1, v2, v3, scale, clamp_low);
}

// TORCHREF quantisation of four values of a row whose scale is that of the row's largest magnitude, with the division
// replaced by a multiplication wherever that cannot change the result.  value * (1/scale) differs from the correctly rounded
// value / scale by a few units in the last place (below 2e-5 in absolute terms for |quotient| <= 127.5), so the two round to
// the same integer unless the product lies within 1e-4 of a half-integer; only then the exact division decides.
// Bit-identical to quantize_value(TORCHREF).  Adding 1.5 * 2^23 rounds the product (exact inside the fused multiply-add)
// to the nearest integer, ties to even, in the low mantissa bits: the byte is read out of the sum's bit pattern and
// subtracting the constant again gives the integer for the boundary test, whose maximum keeps NaN.  No conversion
// instruction and no clamp: a quotient beyond +-127.5 needs a scale that is not the row's, or one of so few units of the
// smallest fp32 number that amax / 127 was rounded by 0.4 % (below 2^-141).  Such a scale's reciprocal overflows, and what is
// not finite (that, a NaN value, an infinite row) is a NaN or an infinity in the test and goes to the exact statement.
// One test per four values; the exact statement decides all four when any of them asks for it.  Four instructions
// per value: with the clamp, the product and its distance as separate operations (seven) 65536 rows of 2048 columns took
// 112 us, 105 us like this.
// kCall: the exact statement as a call, for kernels with many groups (the dense quantiser has two or four: 28.5 us for the op
// at 64 rows, 28.6 with a call).
template <bool kCall = true>
__device__ __forceinline__ uint32_t quantize4_torchref_fast(const float* values, float scale, float inverse, float clamp_low = -127.0f) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  uint32_t bits[4];
  float worst = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float shifted = __fmaf_rn(values[i], inverse, kMagic);
    const float nearest = __fsub_rn(shifted, kMagic);
    worst = max_or_nan(worst, fabsf(__fmaf_rn(values[i], inverse, -nearest)));
    bits[i] = __float_as_uint(shifted);
  }
  if (!(worst <= 0.4999f)) {
    if constexpr (kCall) return quantize4_torchref_call(values[0], values[1], values[2], values[3], scale, clamp_low);
    return quantize4_torchref_exact(values[0], values[1], values[2], values[3], scale, clamp_low);
  }
  // Low byte of each sum = the integer in two's complement.
  return __byte_perm(__byte_perm(bits[0], bits[1], 0x0040), __byte_perm(bits[2], bits[3], 0x0040), 0x5410);
}

__device__ __forceinline__ float quantize_operand(float scale, int numerics) {
  return numerics == FMOE_NUMERICS_NATIVE ? __fdiv_rn(1.0f, scale) : scale;
}

__device__ __forceinline__ float warp_max(float value) {
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) value = fmaxf(value, __shfl_xor_sync(0xffffffffu, value, offset));
  return value;
}

__device__ __forceinline__ int warp_sum(int value) {
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_xor_sync(0xffffffffu, value, offset);
  return value;
}

__device__ __forceinline__ float warp_sum(float value) {
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) value += __shfl_xor_sync(0xffffffffu, value, offset);
  return value;
}

}  // namespace fmoe
