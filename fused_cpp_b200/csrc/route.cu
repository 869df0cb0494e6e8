// Route build: per-expert route lists and the work-item lists of the grouped GEMMs.
//
// The reference walks topk_ids once on the calling thread and pushes each flat route id t*K+slot
// onto its expert's vector (csrc/moe/arm/i8mm_w8a8/kernels.cpp:583-592;
// csrc/moe/arm/common/fused_moe_bf16_tiled.cpp:6455-6469), i.e. a stable counting sort by expert.
// Here one launch of one thread-block cluster (1 to 8 CTAs) produces the same order:
//   1. every warp owns a run of consecutive routes and histograms it in its own shared-memory row;
//   2. the CTA turns the rows into exclusive counts over its warps, the cluster exchanges the CTA totals through
//      distributed shared memory, and every CTA scans the totals over the experts;
//   3. every warp replays its run in order; ballots rank equal ids inside a 32-route round, so positions are
//      assigned in ascending flat-id order.  Meanwhile one warp per list writes the (expert, row tile) work items.
// Ids outside [0, E) raise FMOE_ERR_EXPERT_ID_RANGE in the status block and are dropped.
//
// The work is a few KB per CTA: what bounds it is latency - launches, barriers and dependent loads - so the form that
// counts is the one with the fewest of them.  Back to back on one stream: 8 routes 6.2 us, 4072 routes 10.3 us, 65536
// routes 18.5 us, 147456 routes 31 us (256 experts).  The form before it (a memset of the status block and one block up
// to 1024 routes, three launches - histogram, one-block scan, scatter - above) took, by the stage timer, 14 / 35 / 60 /
// 105 us, where this one takes 9 / 13 / 28 / 54 us.
#include <cstdio>
#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"
#include "route_build.cuh"

namespace fmoe {

namespace {

constexpr int kRouteThreads = 1024;
constexpr int kRouteWarps = kRouteThreads / 32;
constexpr int kRoutesPerCta = 1024;         // one 32-route round per warp; more routes take more CTAs first, then more rounds
constexpr int kHistogramInts = 32 * 1024;   // shared-memory histogram rows: 32 warps up to 1024 experts, 16 up to 2048

template <bool kCluster>
__global__ void __launch_bounds__(kRouteThreads)
route_build_kernel(const int64_t* __restrict__ topk_ids, int64_t routes, int experts, int warps, int64_t run, ItemLists lists, int* status,
                   const int* mirror, int* counts, int* offsets, int* sorted_routes, int* row_expert, int* route_pos) {
  extern __shared__ int route_smem[];
  ptx::launch_dependents();  // an ordinary launch: everything before it has completed
  route_build<kCluster>(route_smem, topk_ids, routes, experts, warps, run, lists, status, mirror, counts, offsets, sorted_routes, row_expert,
                        route_pos);
}

// Work items from given per-expert counts and offsets (rows that already lie in expert order: nothing to sort).
__global__ void __launch_bounds__(128)
items_from_counts_kernel(int experts, const int* __restrict__ counts, const int* __restrict__ offsets, ItemLists lists, int* status) {
  build_item_list(threadIdx.x >> 5, experts, counts, offsets, lists, status, threadIdx.x & 31);
}

}  // namespace

// The status block is cleared by the build.
cudaError_t launch_route_build(const int64_t* topk_ids, int64_t routes, int experts, const ItemLists& lists, int* status, int* counts,
                               int* offsets, int* sorted_routes, int* row_expert, cudaStream_t stream, int* route_pos, const int* mirror) {
  static_assert(kMaxExperts * 16 <= kHistogramInts, "the histogram rows of kMaxExperts experts need at least 16 warps");
  int64_t ctas = 1;
  while (ctas < kMaxRouteCluster && ctas * kRoutesPerCta < routes) ctas *= 2;
  int warps = kHistogramInts / experts < kRouteWarps ? kHistogramInts / experts : kRouteWarps;
  const int64_t rounds = (routes + 32 * ctas * warps - 1) / (32 * ctas * warps);
  const int64_t run = 32 * (rounds > 0 ? rounds : 1);
  int threads = kRouteThreads;
  if (ctas == 1) {
    // A short list: fewer rows to clear and to scan, and no more warps than there is work for.
    const int64_t used = (routes + run - 1) / run;
    warps = static_cast<int>(used > 0 ? used : 1);
    const int wanted = warps * 32 > experts ? warps * 32 : experts;
    threads = wanted <= 128 ? 128 : wanted <= 256 ? 256 : wanted <= 512 ? 512 : kRouteThreads;
  }
  const size_t smem = route_smem_bytes(warps, experts, ctas > 1);
  static PerDeviceOnce configured;
  const int device = current_device_ordinal();
  if (configured.needed(device)) {
    constexpr int kMostBytes = static_cast<int>((kHistogramInts + 4 * kMaxExperts + 1 + kMaxExperts / 32) * sizeof(int));
    cudaError_t error = cudaFuncSetAttribute(route_build_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostBytes);
    if (error == cudaSuccess) error = cudaFuncSetAttribute(route_build_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostBytes);
    if (error != cudaSuccess) return error;
    configured.mark(device);
  }
  if (ctas == 1) {
    route_build_kernel<false><<<1, threads, smem, stream>>>(topk_ids, routes, experts, warps, run, lists, status, mirror, counts, offsets,
                                                            sorted_routes, row_expert, route_pos);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(ctas));
  config.blockDim = dim3(kRouteThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = static_cast<unsigned>(ctas);
  attribute.val.clusterDim.y = 1;
  attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, route_build_kernel<true>, topk_ids, routes, experts, warps, run, lists, status, mirror, counts, offsets,
                            sorted_routes, row_expert, route_pos);
}

cudaError_t launch_items_from_counts(int experts, const int* counts, const int* offsets, const ItemLists& lists, int* status,
                                     cudaStream_t stream) {
  items_from_counts_kernel<<<1, 128, 0, stream>>>(experts, counts, offsets, lists, status);
  return cudaGetLastError();
}


// ---- allocation-free route build ---------------------------------------------------------------
//
// Some hosts of this library must not allocate device memory once they are serving: an inference
// server that handed the whole HBM budget to its KV-cache pool at start-up has nothing left for a
// cudaMalloc to take, and a runtime whose memory plan is frozen after warm-up treats any later
// allocation as a bug.  For them the route build is also offered with its status block in a fixed array that
// lives in the library's device image (everything else the build needs is shared memory), so the call needs no
// workspace and performs no allocation of any kind.  The price is a fixed ceiling on the problem size and one
// status block shared by every call.

namespace {

constexpr int64_t kStaticMaxRoutes = 131072;  // tokens * top_k
constexpr int kStaticMaxExperts = 512;
constexpr int kStaticMaxDevices = 64;

// Held from the moment the library is loaded on a GPU until the process exits.
static __device__ __align__(256) int g_static_route_status[kStatusWords];

// In host code the array's name only stands for the symbol; the address a kernel can use has to be
// asked for, per device, with that device current.
int* static_status_for_current_device(cudaError_t* error) {
  static std::mutex guard;
  static int* address[kStaticMaxDevices] = {};
  int device = 0;
  *error = cudaGetDevice(&device);
  if (*error != cudaSuccess) return nullptr;
  if (device < 0 || device >= kStaticMaxDevices) {
    *error = cudaErrorInvalidDevice;
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(guard);
  if (address[device] == nullptr) {
    int* pointer = nullptr;
    *error = cudaGetSymbolAddress(reinterpret_cast<void**>(&pointer), g_static_route_status);
    if (*error != cudaSuccess) return nullptr;
    address[device] = pointer;
  }
  return address[device];
}

}  // namespace

}  // namespace fmoe

extern "C" int fmoe_route_build_noalloc(const int64_t* topk_ids, int64_t tokens, int32_t top_k, int32_t experts, int32_t* counts,
                                        int32_t* offsets, int32_t* sorted_routes, int32_t* row_expert, int32_t* status_out,
                                        void* stream_ptr) {
  char text[256];
  if (tokens < 0 || top_k <= 0 || experts <= 0) return fmoe::report_error(FMOE_ERR_INVALID_ARGUMENT, "invalid route-build shape");
  const int64_t routes = tokens * top_k;
  if (routes > fmoe::kStaticMaxRoutes || experts > fmoe::kStaticMaxExperts) {
    snprintf(text, sizeof(text),
             "fmoe_route_build_noalloc: %lld routes x %d experts exceeds the static scratch (at most %lld routes and %d experts); "
             "use fmoe_w8a8_forward / fmoe_bf16_forward with a caller workspace for larger problems",
             static_cast<long long>(routes), experts, static_cast<long long>(fmoe::kStaticMaxRoutes), fmoe::kStaticMaxExperts);
    return fmoe::report_error(FMOE_ERR_INVALID_ARGUMENT, text);
  }
  if (counts == nullptr || offsets == nullptr || status_out == nullptr ||
      (routes > 0 && (topk_ids == nullptr || sorted_routes == nullptr || row_expert == nullptr))) {
    return fmoe::report_error(FMOE_ERR_INVALID_ARGUMENT, "fmoe_route_build_noalloc: null pointer");
  }
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || !fmoe_device_supported(device)) {
    return fmoe::report_error(FMOE_ERR_UNSUPPORTED_DEVICE, "fmoe_route_build_noalloc: the current device is not a compute capability 10.x GPU");
  }
  cudaError_t error = cudaSuccess;
  int* status = fmoe::static_status_for_current_device(&error);
  if (status == nullptr) {
    snprintf(text, sizeof(text), "fmoe_route_build_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(error));
    return fmoe::report_error(FMOE_ERR_CUDA, text);
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  error = fmoe::launch_route_build(topk_ids, routes, experts, fmoe::no_item_lists(), status, counts, offsets, sorted_routes, row_expert, stream);
  if (error == cudaSuccess) error = cudaMemcpyAsync(status_out, status, 2 * sizeof(int), cudaMemcpyDeviceToDevice, stream);
  if (error != cudaSuccess) {
    snprintf(text, sizeof(text), "fmoe_route_build_noalloc: %s", cudaGetErrorString(error));
    return fmoe::report_error(FMOE_ERR_CUDA, text);
  }
  return FMOE_OK;
}
