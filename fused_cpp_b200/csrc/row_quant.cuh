// Pieces of the row kernels (quant.cu, front.cu): magnitudes, int8 packing and the two-plane split of bf16 rows.
#pragma once

#include "common.cuh"

namespace fmoe {

namespace {

__device__ __forceinline__ float block_max(float value, float* smem) {
  value = warp_max(value);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (lane == 0) smem[warp] = value;
  __syncthreads();
  float result = lane < (blockDim.x >> 5) ? smem[lane] : 0.0f;
  result = warp_max(result);
  __syncthreads();
  return result;
}

__device__ __forceinline__ void unpack8(const uint4& v, float* out) {
  const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[2 * i] = __uint_as_float(words[i] << 16);
    out[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t result;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(result) : "r"(a), "r"(b));
  return result;
}

// Largest magnitude of eight bf16 values, NaN left out: two values per instruction, exact like the fp32 form.
__device__ __forceinline__ float amax8(const uint4& v) {
  constexpr uint32_t kMagnitude = 0x7fff7fffu;
  uint32_t m = max_bf16x2(0u, v.x & kMagnitude);
  m = max_bf16x2(m, v.y & kMagnitude);
  m = max_bf16x2(m, v.z & kMagnitude);
  m = max_bf16x2(m, v.w & kMagnitude);
  return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u));
}

template <int kNumerics>
struct NumericsTag {
  static constexpr int value = kNumerics;
};

// Calls body(NumericsTag): one instance of a row loop per arithmetic statement, side by side instead of a choice per group.
template <typename Body>
__device__ __forceinline__ void with_numerics(int numerics, Body&& body) {
  if (numerics == FMOE_NUMERICS_TORCHREF) {
    body(NumericsTag<FMOE_NUMERICS_TORCHREF>{});
  } else {
    body(NumericsTag<FMOE_NUMERICS_NATIVE>{});
  }
}

// operand: 1/scale (NATIVE) or scale (TORCHREF); inverse: 1/scale, used by the TORCHREF fast path.
template <typename Tag>
__device__ __forceinline__ uint32_t pack4(Tag, const float* values, float operand, float inverse) {
  if constexpr (Tag::value == FMOE_NUMERICS_TORCHREF) return quantize4_torchref_fast(values, operand, inverse);
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    packed |= (static_cast<uint32_t>(quantize_value(values[i], operand, Tag::value)) & 0xffu) << (8 * i);
  }
  return packed;
}

template <typename Tag>
__device__ __forceinline__ uint4 pack16(Tag tag, const uint4& first, const uint4& second, float operand, float inverse) {
  float values[16];
  unpack8(first, values);
  unpack8(second, values + 8);
  return make_uint4(pack4(tag, values, operand, inverse), pack4(tag, values + 4, operand, inverse), pack4(tag, values + 8, operand, inverse),
                    pack4(tag, values + 12, operand, inverse));
}

// Eight values of a row -> eight bytes of its high and eight of its low plane (W8A16 in its fixed-point form).
__device__ __forceinline__ void split8_planes(const float* values, float scale, uint2* high_vector, uint2* low_vector) {
  uint32_t high[2] = {0, 0};
  uint32_t low[2] = {0, 0};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int fixed = plane_fixed_point(values[i], scale);
    const int low_part = ((fixed + 128) & 255) - 128;
    const int high_part = (fixed - low_part) >> 8;  // fixed - low_part is a multiple of 256
    high[i >> 2] |= (static_cast<uint32_t>(high_part) & 0xffu) << (8 * (i & 3));
    low[i >> 2] |= (static_cast<uint32_t>(low_part) & 0xffu) << (8 * (i & 3));
  }
  *high_vector = make_uint2(high[0], high[1]);
  *low_vector = make_uint2(low[0], low[1]);
}

// The same for 16 values.
__device__ __forceinline__ void split16_planes(const float* values, float scale, uint4* high_vector, uint4* low_vector) {
  uint2 high[2], low[2];
  split8_planes(values, scale, &high[0], &low[0]);
  split8_planes(values + 8, scale, &high[1], &low[1]);
  *high_vector = make_uint4(high[0].x, high[0].y, high[1].x, high[1].y);
  *low_vector = make_uint4(low[0].x, low[0].y, low[1].x, low[1].y);
}

}  // namespace

}  // namespace fmoe
