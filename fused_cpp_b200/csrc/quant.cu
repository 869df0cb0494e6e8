// Dynamic per-row symmetric int8 quantisation and the row gather of the BF16 path.
//
// The reference quantises x[token] once per route into the expert's private buffer
// (quantize_bf16_row, csrc/moe/arm/i8mm_w8a8/kernels.cpp:211-228, called at :639-644 and :655-656).
// One CTA handles one output row: pass 1 finds the row's absmax with 16-byte loads and a
// warp-shuffle/shared-memory reduction, pass 2 re-reads the row (L1/L2 resident) and stores 16 int8
// per thread as one 16-byte vector.  With `sorted_routes` the source row is the route's token, so
// the output is already in expert-sorted order for the grouped GEMM (gather and quantise fused).
#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"
#include "row_quant.cuh"

namespace fmoe {

namespace {

constexpr int kQuantThreads = 256;
constexpr int kFewRowsPerSm = 4;  // up to so many rows per SM latency counts, above it throughput

// cols % 16 == 0.  One CTA per output row.
__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_kernel(const uint16_t* x, int cols, const int* sorted_routes, int top_k,
                     const int* valid_rows, int numerics, int weight_mode, int8_t* __restrict__ q,
                     float* __restrict__ scale_out, bool chained) {
  __shared__ float smem[32];
  if (chained) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
  }
  const int64_t row = blockIdx.x;
  if (valid_rows && row >= __ldcg(valid_rows)) return;  // rows of dropped (out-of-range) routes
  const int64_t src_row = sorted_routes ? static_cast<int64_t>(__ldcg(sorted_routes + row) / top_k) : row;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * cols);
  const int vec16 = cols >> 4;
  float local = 0.0f;
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    local = fmaxf(local, amax8(src[2 * v]));
    local = fmaxf(local, amax8(src[2 * v + 1]));
  }
  const float amax = block_max(local, smem);
  float scale;
  int mode = numerics;
  if (weight_mode) {
    scale = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
    mode = FMOE_NUMERICS_TORCHREF;
  } else {
    scale = row_scale_from_amax(amax, numerics);
  }
  if (threadIdx.x == 0) scale_out[row] = scale;
  const float operand = quantize_operand(scale, mode);
  const float inverse = __fdiv_rn(1.0f, scale);
  uint4* dst = reinterpret_cast<uint4*>(q + row * cols);
  with_numerics(mode, [&](auto tag) {
    for (int v = threadIdx.x; v < vec16; v += kQuantThreads) dst[v] = pack16(tag, src[2 * v], src[2 * v + 1], operand, inverse);
  });
}

// Same work, one warp per output row, for rows of at most 32 * 16 * kVectors columns: the row is read once
// into registers (kVectors 32-byte pieces per lane), the absmax is a shuffle reduction, no block barrier.
// Rows of a few KB (the 2048-column intermediate of the W8A8 layer) are too short to keep a 256-thread CTA busy.
template <int kVectors>
__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_warp_kernel(const uint16_t* x, int64_t out_rows, int cols, const int* sorted_routes, int top_k,
                          const int* valid_rows, int numerics, int weight_mode, int8_t* __restrict__ q,
                          float* __restrict__ scale_out, bool chained) {
  if (chained) {
    ptx::launch_dependents();  // ahead of the wait, as in quantize_rows_held_kernel
    ptx::grid_dependency_wait();
  }
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (kQuantThreads / 32) + (threadIdx.x >> 5);
  if (row >= out_rows) return;
  if (valid_rows && row >= __ldcg(valid_rows)) return;
  const int64_t src_row = sorted_routes ? static_cast<int64_t>(__ldcg(sorted_routes + row) / top_k) : row;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * cols);
  const int vec16 = cols >> 4;
  uint4 held[kVectors][2];
  float local = 0.0f;
#pragma unroll
  for (int i = 0; i < kVectors; ++i) {
    const int v = lane + 32 * i;
    if (v < vec16) {
      held[i][0] = src[2 * v];
      held[i][1] = src[2 * v + 1];
      local = fmaxf(local, fmaxf(amax8(held[i][0]), amax8(held[i][1])));
    }
  }
  const float amax = warp_max(local);
  float scale;
  int mode = numerics;
  if (weight_mode) {
    scale = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
    mode = FMOE_NUMERICS_TORCHREF;
  } else {
    scale = row_scale_from_amax(amax, numerics);
  }
  if (lane == 0) scale_out[row] = scale;
  const float operand = quantize_operand(scale, mode);
  const float inverse = __fdiv_rn(1.0f, scale);
  uint4* dst = reinterpret_cast<uint4*>(q + row * cols);
  with_numerics(mode, [&](auto tag) {
#pragma unroll
    for (int i = 0; i < kVectors; ++i) {
      const int v = lane + 32 * i;
      if (v < vec16) dst[v] = pack16(tag, held[i][0], held[i][1], operand, inverse);
    }
  });
}

// The intermediate of a small batch, one CTA per row of at most 256 * 8 * kVectors columns (a multiple of 16): between two GEMMs
// nothing but this kernel's latency counts, so the row is read once, beside the row count, and held in registers, one barrier
// lies between the maximum and the store, and the GEMM behind it is let in before the wait: its CTAs take the SMs that
// gate_up leaves, and the first weights are on their way while the last rows are still computed.  One token of the 256-expert
// layer: down's first MMA 8.0 us after gate_up's end with the two-pass kernel and the launch behind the wait, 6.1 us like this
// (of 126 us; 16 tokens of the 16-expert one 71.5 -> 70.3).
// kPlanes: two int8 rows per route (split16_planes).
template <bool kPlanes, int kVectors>
__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_held_kernel(const uint16_t* x, int cols, const int* valid_rows, int numerics, int8_t* __restrict__ q, float* __restrict__ scale_out,
                          bool chained) {
  __shared__ float warp_amax[kQuantThreads / 32];
  if (chained) {
    ptx::launch_dependents();
    ptx::grid_dependency_wait();
  }
  const int64_t row = blockIdx.x;
  const int rows = __ldcg(valid_rows);
  const uint4* src = reinterpret_cast<const uint4*>(x + row * cols);
  const int vec8 = cols >> 3;
  uint4 held[kVectors];
  float local = 0.0f;
#pragma unroll
  for (int i = 0; i < kVectors; ++i) {
    const int v = threadIdx.x + i * kQuantThreads;
    held[i] = v < vec8 ? __ldcg(src + v) : make_uint4(0, 0, 0, 0);
  }
  if (row >= rows) return;  // rows of dropped (out-of-range) routes
#pragma unroll
  for (int i = 0; i < kVectors; ++i) local = fmaxf(local, amax8(held[i]));
  local = warp_max(local);
  const int lane = threadIdx.x & 31;
  if (lane == 0) warp_amax[threadIdx.x >> 5] = local;
  __syncthreads();
  const float amax = warp_max(warp_amax[lane & (kQuantThreads / 32 - 1)]);
  const float scale = kPlanes ? plane_row_scale(amax) : row_scale_from_amax(amax, numerics);
  if (threadIdx.x == 0) scale_out[row] = scale;
  const float operand = quantize_operand(scale, numerics);
  const float inverse = __fdiv_rn(1.0f, scale);
  with_numerics(numerics, [&](auto tag) {
#pragma unroll
    for (int i = 0; i < kVectors; ++i) {
      const int v = threadIdx.x + i * kQuantThreads;
      if (v >= vec8) break;
      float values[8];
      unpack8(held[i], values);
      if constexpr (kPlanes) {
        uint2 high, low;
        split8_planes(values, scale, &high, &low);
        reinterpret_cast<uint2*>(q + 2 * row * cols)[v] = high;
        reinterpret_cast<uint2*>(q + (2 * row + 1) * cols)[v] = low;
      } else {
        reinterpret_cast<uint2*>(q + row * cols)[v] = make_uint2(pack4(tag, values, operand, inverse), pack4(tag, values + 4, operand, inverse));
      }
    }
  });
}

constexpr int kHeldColumns = kQuantThreads * 8;  // per vector of a thread

template <bool kPlanes>
cudaError_t launch_held(const uint16_t* x, int64_t rows, int cols, const int* valid_rows, int numerics, int8_t* q, float* scale, cudaStream_t stream) {
  auto kernel = cols <= kHeldColumns ? quantize_rows_held_kernel<kPlanes, 1>
                : cols <= 2 * kHeldColumns ? quantize_rows_held_kernel<kPlanes, 2>
                                           : quantize_rows_held_kernel<kPlanes, 4>;
  return launch_streaming(kernel, dim3(static_cast<unsigned>(rows)), kQuantThreads, stream, true, x, cols, valid_rows, numerics, q, scale);
}

// cols % 16 == 0, top_k <= 32.  One CTA per token: the row is quantised once and stored to each of its routes'
// sorted positions (the reference re-quantises the token for every route, kernels.cpp:639-644; the bits are the same).
__global__ void __launch_bounds__(kQuantThreads)
quantize_tokens_scatter_kernel(const uint16_t* x, int cols, int top_k, const int* route_pos,
                               int numerics, int8_t* __restrict__ q, float* __restrict__ scale_out, bool chained) {
  __shared__ float smem[32];
  __shared__ int positions[32];
  const int64_t token = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(x + token * cols);
  const int vec16 = cols >> 4;
  float local = 0.0f;
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    local = fmaxf(local, amax8(__ldcg(src + 2 * v)));
    local = fmaxf(local, amax8(__ldcg(src + 2 * v + 1)));
  }
  if (chained) {
    ptx::grid_dependency_wait();  // the route build: x itself is older
    ptx::launch_dependents();
  }
  if (threadIdx.x < top_k) positions[threadIdx.x] = __ldcg(route_pos + token * top_k + threadIdx.x);
  const float amax = block_max(local, smem);  // its barriers also publish positions[]
  const float scale = row_scale_from_amax(amax, numerics);
  if (threadIdx.x < top_k && positions[threadIdx.x] >= 0) scale_out[positions[threadIdx.x]] = scale;
  const float operand = quantize_operand(scale, numerics);
  const float inverse = __fdiv_rn(1.0f, scale);
  with_numerics(numerics, [&](auto tag) {
    for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
      const uint4 out = pack16(tag, __ldcg(src + 2 * v), __ldcg(src + 2 * v + 1), operand, inverse);
      for (int slot = 0; slot < top_k; ++slot) {
        const int position = positions[slot];
        if (position >= 0) reinterpret_cast<uint4*>(q + static_cast<int64_t>(position) * cols)[v] = out;
      }
    }
  });
}

// W8A16 in its fixed-point form.  cols % 16 == 0.  One CTA per route row p (gathered by token when sorted_routes is
// given): the bf16 row becomes 16-bit fixed point (plane_fixed_point) and is stored as two int8 rows, the high plane at
// row 2p and the low plane at row 2p + 1 of `planes`; scale_out[p] is the row scale.
__global__ void __launch_bounds__(kQuantThreads)
split_rows_planes_kernel(const uint16_t* x, int cols, const int* sorted_routes, int top_k,
                         const int* valid_rows, int8_t* __restrict__ planes, float* __restrict__ scale_out, bool chained) {
  __shared__ float smem[32];
  if (chained) {
    ptx::launch_dependents();  // ahead of the wait, as in quantize_rows_held_kernel
    ptx::grid_dependency_wait();
  }
  const int64_t row = blockIdx.x;
  if (valid_rows && row >= __ldcg(valid_rows)) return;
  const int64_t src_row = sorted_routes ? static_cast<int64_t>(__ldcg(sorted_routes + row) / top_k) : row;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * cols);
  const int vec16 = cols >> 4;
  float local = 0.0f;
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    local = fmaxf(local, amax8(src[2 * v]));
    local = fmaxf(local, amax8(src[2 * v + 1]));
  }
  const float amax = block_max(local, smem);
  const float scale = plane_row_scale(amax);
  if (threadIdx.x == 0) scale_out[row] = scale;
  uint4* high_row = reinterpret_cast<uint4*>(planes + (2 * row) * cols);
  uint4* low_row = reinterpret_cast<uint4*>(planes + (2 * row + 1) * cols);
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    float values[16];
    unpack8(src[2 * v], values);
    unpack8(src[2 * v + 1], values + 8);
    split16_planes(values, scale, high_row + v, low_row + v);
  }
}

// The same split once per TOKEN, stored to the sorted positions of its top_k routes (route_pos, -1 = dropped): the bits
// every route would get from split_rows_planes_kernel, one read of x and one fixed-point conversion per token.
__global__ void __launch_bounds__(kQuantThreads)
split_tokens_scatter_planes_kernel(const uint16_t* x, int cols, int top_k, const int* route_pos,
                                   int8_t* __restrict__ planes, float* __restrict__ scale_out, bool chained) {
  __shared__ float smem[32];
  __shared__ int positions[32];
  const int64_t token = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(x + token * cols);
  const int vec16 = cols >> 4;
  float local = 0.0f;
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    local = fmaxf(local, amax8(__ldcg(src + 2 * v)));
    local = fmaxf(local, amax8(__ldcg(src + 2 * v + 1)));
  }
  if (chained) {
    ptx::grid_dependency_wait();  // the route build: x itself is older
    ptx::launch_dependents();
  }
  if (threadIdx.x < top_k) positions[threadIdx.x] = __ldcg(route_pos + token * top_k + threadIdx.x);
  const float amax = block_max(local, smem);  // its barriers also publish positions[]
  const float scale = plane_row_scale(amax);
  if (threadIdx.x < top_k && positions[threadIdx.x] >= 0) scale_out[positions[threadIdx.x]] = scale;
  for (int v = threadIdx.x; v < vec16; v += kQuantThreads) {
    float values[16];
    unpack8(__ldcg(src + 2 * v), values);
    unpack8(__ldcg(src + 2 * v + 1), values + 8);
    uint4 high_vector, low_vector;
    split16_planes(values, scale, &high_vector, &low_vector);
    for (int slot = 0; slot < top_k; ++slot) {
      const int64_t position = positions[slot];
      if (position >= 0) {
        reinterpret_cast<uint4*>(planes + (2 * position) * cols)[v] = high_vector;
        reinterpret_cast<uint4*>(planes + (2 * position + 1) * cols)[v] = low_vector;
      }
    }
  }
}

// Dense linear: arbitrary cols, fp32 or bf16 source, zero-padded to cols_padded, clamp to [-128,127]
// (single GEMM) or [-127,127] (paired GEMMs) with division and ties-to-even (csrc/i8gemm.cpp:384-399, :492-506).
// Status block and work items of the dense GEMM that follows (one "expert", row tiles of row_tile rows; the group key
// of a list entry in the fourth word), written by block 0 of the quantiser so that the op needs no launches of its own
// for them.  Every status word is written: the block starts out in an unknown state.
struct DenseItems {
  int64_t rows;
  int row_tile;
  int max_items;
  int* items;
  int* status;
};

__device__ __forceinline__ void write_dense_items(const DenseItems& d) {
  const int tiles = static_cast<int>((d.rows + d.row_tile - 1) / d.row_tile);
  const int count = tiles < d.max_items ? tiles : d.max_items;
  for (int t = threadIdx.x; t < count; t += blockDim.x) {
    d.items[4 * t + 0] = 0;
    d.items[4 * t + 1] = t * d.row_tile;
    d.items[4 * t + 2] = static_cast<int>(min(static_cast<int64_t>(d.row_tile), d.rows - static_cast<int64_t>(t) * d.row_tile));
    d.items[4 * t + 3] = count < 2048 ? (0 | (count << 20)) : (t | (1 << 20));
  }
  if (threadIdx.x < kStatusWords) {
    const int word = threadIdx.x;
    d.status[word] = (word == kStatusItems || word == kStatusItemsB) ? count : word == kStatusActive ? (d.rows > 0 ? 1 : 0) : 0;
  }
}

__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_dense_kernel(const void* __restrict__ x, int x_is_bf16, int cols, int cols_padded, float clamp_low,
                           int8_t* __restrict__ q, float* __restrict__ scale_out, DenseItems dense_items) {
  ptx::launch_dependents();
  if (blockIdx.x == 0) write_dense_items(dense_items);
  __shared__ float smem[32];
  const int64_t row = blockIdx.x;
  const float* xf = static_cast<const float*>(x) + row * cols;
  const uint16_t* xb = static_cast<const uint16_t*>(x) + row * cols;
  float local = 0.0f;
  for (int c = threadIdx.x; c < cols; c += kQuantThreads) {
    const float value = x_is_bf16 ? bf16_bits_to_f32(xb[c]) : xf[c];
    local = fmaxf(local, fabsf(value));
  }
  const float amax = block_max(local, smem);
  const float scale = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
  if (threadIdx.x == 0) scale_out[row] = scale;
  int8_t* dst = q + row * cols_padded;
  for (int c = threadIdx.x; c < cols_padded; c += kQuantThreads) {
    int value = 0;
    if (c < cols) {
      const float source = x_is_bf16 ? bf16_bits_to_f32(xb[c]) : xf[c];
      float rounded = rintf(__fdiv_rn(source, scale));
      rounded = fmaxf(fminf(rounded, 127.0f), clamp_low);
      value = static_cast<int>(rounded);
    }
    dst[c] = static_cast<int8_t>(value);
  }
}

constexpr int kGatherVectors = 4;  // 16-byte vectors a thread holds at a time: 8192 bf16 columns per CTA and round

// cols % 8 == 0.  out[p] = x[sorted_routes[p] / top_k].
__global__ void __launch_bounds__(kQuantThreads)
gather_rows_kernel(const uint16_t* x, int cols, const int* sorted_routes, int top_k,
                   const int* valid_rows, uint16_t* __restrict__ out, bool chained) {
  if (chained) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
  }
  const int64_t row = blockIdx.x;
  if (valid_rows && row >= __ldcg(valid_rows)) return;
  const int64_t src_row = __ldcg(sorted_routes + row) / top_k;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * cols);
  uint4* dst = reinterpret_cast<uint4*>(out + row * cols);
  const int vec8 = cols >> 3;
  for (int v0 = threadIdx.x; v0 < vec8; v0 += kGatherVectors * kQuantThreads) {
    uint4 held[kGatherVectors];
#pragma unroll
    for (int i = 0; i < kGatherVectors; ++i) {
      if (v0 + i * kQuantThreads < vec8) held[i] = src[v0 + i * kQuantThreads];
    }
#pragma unroll
    for (int i = 0; i < kGatherVectors; ++i) {
      if (v0 + i * kQuantThreads < vec8) dst[v0 + i * kQuantThreads] = held[i];
    }
  }
}

// cols % 8 == 0, top_k <= 32.  One CTA per token: its row is read once and stored to each of its routes' sorted positions
// (-1 = dropped).  Bound by the writes: a CTA per sorted row, which reads the row again for every route, took 127 us for
// 32760 rows of 14 KB; this one 86 us.
__global__ void __launch_bounds__(kQuantThreads)
gather_tokens_scatter_kernel(const uint16_t* x, int cols, int top_k, const int* route_pos, uint16_t* __restrict__ out, bool chained) {
  __shared__ int positions[32];
  const int64_t token = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(x + token * cols);
  const int vec8 = cols >> 3;
  for (int v0 = threadIdx.x; v0 < (vec8 + kQuantThreads - 1) / kQuantThreads * kQuantThreads; v0 += kGatherVectors * kQuantThreads) {
    uint4 held[kGatherVectors];
#pragma unroll
    for (int i = 0; i < kGatherVectors; ++i) {
      if (v0 + i * kQuantThreads < vec8) held[i] = __ldcg(src + v0 + i * kQuantThreads);
    }
    if (v0 == static_cast<int>(threadIdx.x)) {
      // The first round, which every thread takes part in.
      if (chained) {
        ptx::grid_dependency_wait();  // the route build: x itself is older
        ptx::launch_dependents();
      }
      if (threadIdx.x < top_k) positions[threadIdx.x] = __ldcg(route_pos + token * top_k + threadIdx.x);
      __syncthreads();
    }
    for (int slot = 0; slot < top_k; ++slot) {
      const int position = positions[slot];
      if (position < 0) continue;
      uint4* dst = reinterpret_cast<uint4*>(out + static_cast<int64_t>(position) * cols);
#pragma unroll
      for (int i = 0; i < kGatherVectors; ++i) {
        if (v0 + i * kQuantThreads < vec8) dst[v0 + i * kQuantThreads] = held[i];
      }
    }
  }
}

__global__ void gather_scalars_kernel(const float* in, int64_t n, const int* index,
                                      const int* valid_rows, float* __restrict__ out, bool chained) {
  if (chained) {
    ptx::grid_dependency_wait();
    ptx::launch_dependents();
  }
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n || (valid_rows && i >= __ldcg(valid_rows))) return;
  out[i] = in[index[i]];
}

}  // namespace

cudaError_t launch_gather_scalars(const float* in, int64_t n, const int* index, const int* valid_rows, float* out,
                                  cudaStream_t stream, bool chained) {
  if (n <= 0) return cudaSuccess;
  return launch_streaming(gather_scalars_kernel, dim3(static_cast<unsigned>((n + 255) / 256)), 256, stream, chained, in, n, index, valid_rows, out);
}

cudaError_t launch_quantize_rows(const uint16_t* x, int64_t out_rows, int cols, const int* sorted_routes, int top_k,
                                 const int* valid_rows, int numerics, int weight_mode, int8_t* q, float* scale,
                                 cudaStream_t stream, bool chained) {
  if (out_rows <= 0) return cudaSuccess;
  const int vec16 = cols >> 4;
  const unsigned warp_blocks = static_cast<unsigned>((out_rows + kQuantThreads / 32 - 1) / (kQuantThreads / 32));
  // A few rows (decode): one CTA per row spreads a row over 256 threads, where one warp per row would walk its 64
  // values per lane alone on an SM (10.7 us against the other kernel's ~5 us for 8 rows of 2048 columns).
  const bool few_rows = out_rows <= kFewRowsPerSm * threshold_sms;
  if (few_rows && chained && sorted_routes == nullptr && valid_rows != nullptr && weight_mode == 0 && cols <= 4 * kHeldColumns) {
    return launch_held<false>(x, out_rows, cols, valid_rows, numerics, q, scale, stream);
  }
  if (few_rows) {
    return launch_streaming(quantize_rows_kernel, dim3(static_cast<unsigned>(out_rows)), kQuantThreads, stream, chained, x, cols, sorted_routes,
                          top_k, valid_rows, numerics, weight_mode, q, scale);
  }
  if (vec16 <= 64) {
    return launch_streaming(quantize_rows_warp_kernel<2>, dim3(warp_blocks), kQuantThreads, stream, chained, x, out_rows, cols, sorted_routes, top_k,
                          valid_rows, numerics, weight_mode, q, scale);
  } else if (vec16 <= 128) {
    return launch_streaming(quantize_rows_warp_kernel<4>, dim3(warp_blocks), kQuantThreads, stream, chained, x, out_rows, cols, sorted_routes, top_k,
                          valid_rows, numerics, weight_mode, q, scale);
  }
  return launch_streaming(quantize_rows_kernel, dim3(static_cast<unsigned>(out_rows)), kQuantThreads, stream, chained, x, cols, sorted_routes, top_k,
                        valid_rows, numerics, weight_mode, q, scale);
}

cudaError_t launch_split_rows_planes(const uint16_t* x, int64_t out_rows, int cols, const int* sorted_routes, int top_k,
                                     const int* valid_rows, int8_t* planes, float* scale, cudaStream_t stream) {
  if (out_rows <= 0) return cudaSuccess;
  if (out_rows <= kFewRowsPerSm * threshold_sms && sorted_routes == nullptr && valid_rows != nullptr && cols <= 4 * kHeldColumns) {
    return launch_held<true>(x, out_rows, cols, valid_rows, FMOE_NUMERICS_TORCHREF, planes, scale, stream);
  }
  return launch_streaming(split_rows_planes_kernel, dim3(static_cast<unsigned>(out_rows)), kQuantThreads, stream, true, x, cols, sorted_routes,
                        top_k, valid_rows, planes, scale);
}

cudaError_t launch_split_tokens_scatter_planes(const uint16_t* x, int64_t tokens, int cols, int top_k, const int* route_pos, int8_t* planes,
                                               float* scale, cudaStream_t stream) {
  if (tokens <= 0) return cudaSuccess;
  return launch_streaming(split_tokens_scatter_planes_kernel, dim3(static_cast<unsigned>(tokens)), kQuantThreads, stream, true, x, cols, top_k,
                        route_pos, planes, scale);
}

cudaError_t launch_quantize_tokens_scatter(const uint16_t* x, int64_t tokens, int cols, int top_k, const int* route_pos,
                                           int numerics, int8_t* q, float* scale, cudaStream_t stream) {
  if (tokens <= 0) return cudaSuccess;
  return launch_streaming(quantize_tokens_scatter_kernel, dim3(static_cast<unsigned>(tokens)), kQuantThreads, stream, true, x, cols, top_k,
                        route_pos, numerics, q, scale);
}

// The same quantiser for rows whose length is a multiple of 8 and at most 16 * 1024: the row is read once, into registers
// (two groups of eight values per thread: a 512-thread CTA holds a 7168-column row), and the division is replaced as in
// quantize4_torchref_fast (the statement is the same clamp(rint(x / scale)); the lower clamp of -128 that the single product
// asks for binds only in its exact branch, in fp32 rows below 2.3e-41).  Latency-bound for a decode
// batch: one memory round trip instead of two, and the GEMM behind it fetches weights meanwhile (dense_gemm.cu has the
// figures of the op); HBM-bound above.
constexpr int kDenseVectors = 2;

template <bool kBf16>
__global__ void __launch_bounds__(1024)
quantize_rows_dense_vec8_kernel(const void* __restrict__ x, int cols, int cols_padded, float clamp_low, int8_t* __restrict__ q,
                                float* __restrict__ scale_out, DenseItems dense_items) {
  ptx::launch_dependents();  // the GEMM behind this kernel may start fetching its weights
  __shared__ float smem[32];
  if (blockIdx.x == 0) write_dense_items(dense_items);
  const int64_t row = blockIdx.x;
  const int vec8 = cols >> 3;
  float values[kDenseVectors][8];
  float local = 0.0f;
#pragma unroll
  for (int i = 0; i < kDenseVectors; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < vec8) {
      if constexpr (kBf16) {
        unpack8(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + row * cols)[v], values[i]);
      } else {
        const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(x) + row * cols) + 2 * v;
        *reinterpret_cast<float4*>(values[i]) = src[0];
        *reinterpret_cast<float4*>(values[i] + 4) = src[1];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) values[i][j] = 0.0f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) local = fmaxf(local, fabsf(values[i][j]));
  }
  const float amax = block_max(local, smem);
  const float scale = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
  if (threadIdx.x == 0) scale_out[row] = scale;
  const float inverse = __fdiv_rn(1.0f, scale);
  uint2* dst = reinterpret_cast<uint2*>(q + row * cols_padded);
#pragma unroll
  for (int i = 0; i < kDenseVectors; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < vec8) {
      dst[v] = make_uint2(quantize4_torchref_fast<false>(values[i], scale, inverse, clamp_low), quantize4_torchref_fast<false>(values[i] + 4, scale, inverse, clamp_low));
    }
  }
  // cols_padded is cols or cols + 8 (a multiple of 16).
  if (threadIdx.x == 0 && cols_padded > cols) dst[vec8] = make_uint2(0u, 0u);
}

// bf16 rows by the thousand, or longer than the registers of a CTA hold: a 256-thread CTA reads its row twice, the second
// time out of L1, and eight of them fit an SM (3000 rows of 7168 columns 19 us, 24 us with the row in registers; of the
// other kernel's shorter latency nothing is left from four rows per SM on).  The smallest bf16 number is 2^-133: no scale here
// is rounded enough for a quotient below -127.5, and the lower clamp does not matter.
__global__ void __launch_bounds__(kQuantThreads)
quantize_rows_dense_bf16x8_kernel(const uint16_t* __restrict__ x, int cols, int cols_padded, int8_t* __restrict__ q,
                                  float* __restrict__ scale_out, DenseItems dense_items) {
  ptx::launch_dependents();
  __shared__ float smem[32];
  if (blockIdx.x == 0) write_dense_items(dense_items);
  const int64_t row = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(x + row * cols);
  const int vec8 = cols >> 3;
  float local = 0.0f;
  for (int v = threadIdx.x; v < vec8; v += kQuantThreads) local = fmaxf(local, amax8(src[v]));
  const float amax = block_max(local, smem);
  const float scale = amax > 0.0f ? __fdiv_rn(amax, 127.0f) : 1.0f;
  if (threadIdx.x == 0) scale_out[row] = scale;
  const float inverse = __fdiv_rn(1.0f, scale);
  uint2* dst = reinterpret_cast<uint2*>(q + row * cols_padded);
  const int vec8_padded = cols_padded >> 3;
  for (int v = threadIdx.x; v < vec8_padded; v += kQuantThreads) {
    uint2 out = make_uint2(0u, 0u);
    if (v < vec8) {
      float values[8];
      unpack8(src[v], values);
      out.x = quantize4_torchref_fast<false>(values, scale, inverse);
      out.y = quantize4_torchref_fast<false>(values + 4, scale, inverse);
    }
    dst[v] = out;
  }
}

cudaError_t launch_quantize_rows_dense(const void* x, int x_is_bf16, int64_t rows, int cols, int cols_padded, int clamp_low,
                                       int8_t* q, float* scale, int row_tile, int max_items, int* items, int* status,
                                       cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  const DenseItems dense_items = {rows, row_tile, max_items, items, status};
  const int vec8 = cols >> 3;
  const bool aligned = cols % 8 == 0 && cols_padded - cols <= 8 && cols_padded % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
                       (reinterpret_cast<uintptr_t>(q) & 7u) == 0;
  const bool held = vec8 <= 1024 * kDenseVectors;  // a row fits the registers of one CTA
  if (aligned && x_is_bf16 && (rows > kFewRowsPerSm * threshold_sms || !held)) {
    quantize_rows_dense_bf16x8_kernel<<<static_cast<unsigned>(rows), kQuantThreads, 0, stream>>>(static_cast<const uint16_t*>(x), cols,
                                                                                                cols_padded, q, scale, dense_items);
  } else if (aligned && held) {
    int threads = 64;
    while (threads * kDenseVectors < vec8) threads *= 2;
    auto kernel = x_is_bf16 ? quantize_rows_dense_vec8_kernel<true> : quantize_rows_dense_vec8_kernel<false>;
    kernel<<<static_cast<unsigned>(rows), threads, 0, stream>>>(x, cols, cols_padded, static_cast<float>(clamp_low), q, scale, dense_items);
  } else {
    quantize_rows_dense_kernel<<<static_cast<unsigned>(rows), kQuantThreads, 0, stream>>>(
        x, x_is_bf16, cols, cols_padded, static_cast<float>(clamp_low), q, scale, dense_items);
  }
  return cudaGetLastError();
}

cudaError_t launch_gather_tokens_scatter(const uint16_t* x, int64_t tokens, int cols, int top_k, const int* route_pos, uint16_t* out,
                                         cudaStream_t stream) {
  if (tokens <= 0) return cudaSuccess;
  return launch_streaming(gather_tokens_scatter_kernel, dim3(static_cast<unsigned>(tokens)), kQuantThreads, stream, true, x, cols, top_k,
                          route_pos, out);
}

cudaError_t launch_gather_rows(const uint16_t* x, int64_t out_rows, int cols, const int* sorted_routes, int top_k,
                               const int* valid_rows, uint16_t* out, cudaStream_t stream, bool chained) {
  if (out_rows <= 0) return cudaSuccess;
  return launch_streaming(gather_rows_kernel, dim3(static_cast<unsigned>(out_rows)), kQuantThreads, stream, chained, x, cols, sorted_routes, top_k,
                        valid_rows, out);
}

}  // namespace fmoe
