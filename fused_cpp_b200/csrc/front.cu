// Route build and token rows of a small batch in one launch.
//
// A decode step's two first kernels - the route build (one CTA, 4 to 6 us) and the kernel that quantises or gathers each
// token's row into the sorted positions of its routes - are latency, not work, and the second one waits for the first only to
// learn those positions.  With at most kFrontMaxRoutes routes a token's CTA counts them itself: the sorted position of a
// route is the number of valid routes with a smaller expert id plus that of earlier routes with the same one, a few hundred
// comparisons per slot that hide behind the load of the row.  CTA 0 is the route build of route.cu, the others one token
// each; the GEMM behind it reads its work items behind its wait (GroupedGemmArgs::items_late).  Against the two launches, device time
// of a captured forward: 16 experts of 2048 x 1024, int8, 1 / 16 / 65 / 200 tokens 25.3 -> 23.2, 38.2 -> 37.0, 45.9 -> 44.1, 51.1 -> 48.7 us,
// bf16 200 tokens 72.7 -> 70.6, W8A16 16 tokens 37.9 -> 36.2; one token of the 256-expert layer 87.1 -> 84.3.  Eager with the status read, where a
// launch less for the host counts too: int8 1 and 16 tokens 50.2 -> 48.0, 63.4 -> 61.5, bf16 200 tokens 94.6 -> 91.2.
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
// A CTA per token; two of them fit an SM, so from 2 * SMs tokens on they run in two waves.  That is still faster than two launches (one
// route per token, captured: 512 experts of 2048 x 256, int8, 443 and 592 tokens 120.9 -> 117.8 us, 138.5 -> 136.0; 16 experts of
// 2048 x 1024 47.9 -> 46.2 at 300 tokens, 51.3 -> 50.9 at 592).
constexpr int kFrontTokensPerSm = 4;
constexpr int kFrontCtasPerSm = 2;
constexpr int kMaxTopK = 32;

struct RouteArgs {
  const int64_t* topk_ids;
  int64_t routes;
  int experts, warps;
  int64_t run;
  ItemLists lists;
  const int* mirror;
  int *status, *counts, *offsets, *sorted_routes, *row_expert, *route_pos;
  bool one_wave;  // every CTA of the launch is resident at once
};

// cols % 16 == 0, top_k <= 32.  The bits are those of route_build_kernel and of quantize_tokens_scatter_kernel,
// split_tokens_scatter_planes_kernel or gather_tokens_scatter_kernel.
template <FrontRows kRows>
__global__ void __launch_bounds__(kFrontThreads, kFrontCtasPerSm)
front_kernel(RouteArgs route, const uint16_t* x, int cols, int top_k, int numerics, void* rows_out, float* scale_out) {
  extern __shared__ int route_smem[];
  // (An ordinary launch: everything before it has completed.)  The GEMM behind may start once every CTA has let it in.  A CTA of a
  // single wave does so when its row is read and its positions are counted: with the GEMM's CTAs beside them from the start the 16-expert
  // int8 layer takes 49.2 instead of 44.1 us at 65 tokens, 26.7 instead of 23.2 at one.  With two waves the second one's start comes late by
  // itself, and it lets the GEMM in at once (500 tokens of two routes, bf16, 97.5 -> 91.3 us).
  if (!route.one_wave || blockIdx.x == 0) ptx::launch_dependents();
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
  ptx::launch_dependents();
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
  const RouteArgs route = {topk_ids, routes, experts, warps, run, lists, mirror, status, counts, offsets, sorted_routes, row_expert, route_pos,
                           tokens + 1 <= static_cast<int64_t>(kFrontCtasPerSm) * threshold_sms};
  const size_t smem = route_smem_bytes(warps, experts, false);
  auto kernel = rows == FrontRows::kInt8    ? front_kernel<FrontRows::kInt8>
                : rows == FrontRows::kBf16 ? front_kernel<FrontRows::kBf16>
                                           : front_kernel<FrontRows::kPlanes>;
  kernel<<<static_cast<unsigned>(tokens + 1), kFrontThreads, smem, stream>>>(route, x, cols, top_k, numerics, rows_out, scale_out);
  return cudaGetLastError();
}

}  // namespace fmoe
