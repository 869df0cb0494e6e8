// Route build and token rows of a small batch in one launch.
//
// A decode step's two first kernels - the route build (one CTA, 4 to 6 us) and the kernel that quantises or gathers each
// token's row into the sorted positions of its routes - are latency, not work, and the second one waits for the first only to
// learn those positions.  With at most kFrontMaxRoutes routes a token's CTA counts them itself: the sorted position of a
// route is the number of valid routes with a smaller expert id plus that of earlier routes with the same one, a few hundred
// comparisons per slot that hide behind the load of the row.  CTA 0 is the route build of route.cu, the others one token
// each; the GEMM behind it reads its work items behind its wait (GroupedGemmArgs::items_late).  Against the two launches, whole
// forwards with the status read, cold L2: one token of the 16-expert layer (int8) 49.7 -> 48.2 us, 16 tokens 62.8 -> 60.9, 100 and
// 200 tokens the same within the spread; bf16 52.1 -> 49.8, 77.6 -> 73.9, 89.6 -> 86.8, 93.9 -> 91.0; one token of the 256-expert layer
// 105.9 -> 104.8.  Most of that is a launch less for the host.  On the device alone (captured, no status read) it gains for the
// 256-expert layer (one token 87.3 -> 86.5) and W8A16 (16 tokens 38.5 -> 37.7), and costs small int8 layers the weights
// that gate_up fetched while the rows were quantised: 16 experts, 1 / 16 / 65 / 200 tokens 24.8 -> 26.9, 37.8 -> 38.8, 45.9 -> 49.7,
// 50.9 -> 52.8 us (bf16 65 tokens 65.7 -> 67.2).
// The reference's order of work is csrc/moe/arm/i8mm_w8a8/kernels.cpp:583-592 and :639-644.
#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"
#include "route_build.cuh"
#include "row_quant.cuh"

namespace fmoe {

namespace {

constexpr int kFrontThreads = 512;
constexpr int kFrontWarps = kFrontThreads / 32;
constexpr int kFrontMaxRoutes = 1024;   // two rounds of comparisons per thread, one CTA of route build
constexpr int kFrontMaxExperts = 512;   // histogram rows of kFrontWarps warps stay below the 48 KB every launch may have
// A CTA per token; two of them fit an SM (62 registers a thread), so from 2 * SMs tokens on they run in two waves.  That is still
// faster than two launches: device time of a captured forward with one route per token, int8, 512 experts of 2048 x 256, 443 tokens
// 120.4 -> 116.8 us, 592 tokens 138.3 -> 134.9; 16 experts of 2048 x 1024 47.7 -> 46.5 (300 tokens), 51.0 -> 50.9 (592).
constexpr int kFrontTokensPerSm = 4;
constexpr int kMaxTopK = 32;

struct RouteArgs {
  const int64_t* topk_ids;
  int64_t routes;
  int experts, warps;
  int64_t run;
  ItemLists lists;
  const int* mirror;
  int *status, *counts, *offsets, *sorted_routes, *row_expert, *route_pos;
};

// cols % 16 == 0, top_k <= 32.  The bits are those of route_build_kernel and of quantize_tokens_scatter_kernel,
// split_tokens_scatter_planes_kernel or gather_tokens_scatter_kernel.
template <FrontRows kRows>
__global__ void __launch_bounds__(kFrontThreads)
front_kernel(RouteArgs route, const uint16_t* x, int cols, int top_k, int numerics, void* rows_out, float* scale_out) {
  extern __shared__ int route_smem[];
  ptx::launch_dependents();  // an ordinary launch: everything before it has completed
  if (blockIdx.x == 0) {
    route_build<false>(route_smem, route.topk_ids, route.routes, route.experts, route.warps, route.run, route.lists, route.status, route.mirror,
                       route.counts, route.offsets, route.sorted_routes, route.row_expert, route.route_pos);
    return;
  }
  __shared__ float warp_amax[kFrontWarps];
  __shared__ int slot_ids[kMaxTopK];
  __shared__ int positions[kMaxTopK];
  const int token = static_cast<int>(blockIdx.x) - 1;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int routes = static_cast<int>(route.routes);

  // The row: 16 columns per thread and round, the first round held in registers.
  const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<int64_t>(token) * cols);
  const int vec16 = cols >> 4;
  uint4 held[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  if (static_cast<int>(threadIdx.x) < vec16) {
    held[0] = src[2 * threadIdx.x];
    held[1] = src[2 * threadIdx.x + 1];
  }
  constexpr int kRounds = kFrontMaxRoutes / kFrontThreads;
  int64_t ids[kRounds];
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    const int r = i * kFrontThreads + static_cast<int>(threadIdx.x);
    ids[i] = r < routes ? route.topk_ids[r] : -1;
  }
  if (threadIdx.x < top_k) {
    const int64_t id = route.topk_ids[token * top_k + threadIdx.x];
    slot_ids[threadIdx.x] = id >= 0 && id < route.experts ? static_cast<int>(id) : -1;
    positions[threadIdx.x] = 0;
  }
  __syncthreads();
  int before = 0;  // lane k: routes of this warp's share in front of slot k's
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    if (i * kFrontThreads + warp * 32 >= routes) break;  // warp-uniform
    const int r = i * kFrontThreads + static_cast<int>(threadIdx.x);
    const bool valid = ids[i] >= 0 && ids[i] < route.experts;
    for (int slot = 0; slot < top_k; ++slot) {
      const int mine = slot_ids[slot];
      const unsigned ahead = __ballot_sync(0xffffffffu, valid && (ids[i] < mine || (ids[i] == mine && r < token * top_k + slot)));
      if (lane == slot) before += __popc(ahead);
    }
  }
  if (before > 0) atomicAdd(&positions[lane], before);  // (lanes from top_k on counted nothing)

  float scale = 0.0f, operand = 0.0f, inverse = 0.0f;
  if constexpr (kRows != FrontRows::kBf16) {
    float local = fmaxf(amax8(held[0]), amax8(held[1]));
    for (int v = threadIdx.x + kFrontThreads; v < vec16; v += kFrontThreads) local = fmaxf(local, fmaxf(amax8(src[2 * v]), amax8(src[2 * v + 1])));
    local = warp_max(local);
    if (lane == 0) warp_amax[warp] = local;
  }
  __syncthreads();
  if constexpr (kRows != FrontRows::kBf16) {
    const float amax = warp_max(lane < kFrontWarps ? warp_amax[lane] : 0.0f);
    scale = kRows == FrontRows::kPlanes ? plane_row_scale(amax) : row_scale_from_amax(amax, numerics);
    operand = quantize_operand(scale, numerics);
    inverse = __fdiv_rn(1.0f, scale);
    if (threadIdx.x < top_k && slot_ids[threadIdx.x] >= 0) scale_out[positions[threadIdx.x]] = scale;
  }
  with_numerics(kRows == FrontRows::kInt8 ? numerics : FMOE_NUMERICS_TORCHREF, [&](auto tag) {
    for (int v = threadIdx.x; v < vec16; v += kFrontThreads) {
      if (v >= kFrontThreads) {
        held[0] = src[2 * v];
        held[1] = src[2 * v + 1];
      }
      uint4 first = held[0], second = held[1];  // bf16: the row as it is
      if constexpr (kRows == FrontRows::kPlanes) {
        float values[16];
        unpack8(held[0], values);
        unpack8(held[1], values + 8);
        split16_planes(values, scale, &first, &second);
      } else if constexpr (kRows == FrontRows::kInt8) {
        first = pack16(tag, held[0], held[1], operand, inverse);
      }
      for (int slot = 0; slot < top_k; ++slot) {
        if (slot_ids[slot] < 0) continue;  // dropped by the route build, which reports it
        const int64_t position = positions[slot];
        if constexpr (kRows == FrontRows::kInt8) {
          reinterpret_cast<uint4*>(static_cast<int8_t*>(rows_out) + position * cols)[v] = first;
        } else if constexpr (kRows == FrontRows::kPlanes) {
          reinterpret_cast<uint4*>(static_cast<int8_t*>(rows_out) + 2 * position * cols)[v] = first;
          reinterpret_cast<uint4*>(static_cast<int8_t*>(rows_out) + (2 * position + 1) * cols)[v] = second;
        } else {
          uint4* dst = reinterpret_cast<uint4*>(static_cast<uint16_t*>(rows_out) + position * cols) + 2 * v;
          dst[0] = first;
          dst[1] = second;
        }
      }
    }
  });
}

}  // namespace

bool front_pays(int64_t tokens, int top_k, int experts) {
  return tokens * top_k <= kFrontMaxRoutes && experts <= kFrontMaxExperts && tokens <= static_cast<int64_t>(kFrontTokensPerSm) * threshold_sms;
}

cudaError_t launch_front(FrontRows rows, const int64_t* topk_ids, int64_t tokens, int top_k, int experts, const ItemLists& lists, int* status,
                         int* counts, int* offsets, int* sorted_routes, int* row_expert, int* route_pos, const uint16_t* x, int cols,
                         int numerics, void* rows_out, float* scale_out, cudaStream_t stream, const int* mirror) {
  const int64_t routes = tokens * top_k;
  const int64_t used = (routes + 31) / 32;
  const int warps = static_cast<int>(used < kFrontWarps ? used : kFrontWarps);
  const int64_t run = 32 * ((used + warps - 1) / warps);
  const RouteArgs route = {topk_ids, routes, experts, warps, run, lists, mirror, status, counts, offsets, sorted_routes, row_expert, route_pos};
  const size_t smem = route_smem_bytes(warps, experts, false);
  auto kernel = rows == FrontRows::kInt8    ? front_kernel<FrontRows::kInt8>
                : rows == FrontRows::kBf16 ? front_kernel<FrontRows::kBf16>
                                           : front_kernel<FrontRows::kPlanes>;
  kernel<<<static_cast<unsigned>(tokens + 1), kFrontThreads, smem, stream>>>(route, x, cols, top_k, numerics, rows_out, scale_out);
  return cudaGetLastError();
}

}  // namespace fmoe
