// Route build, device side: the stable counting sort of flat route ids by expert and the work-item lists of the grouped
// GEMMs, by one CTA or one cluster of CTAs.  route.cu describes the steps and launches it by itself; front.cu runs it in one
// CTA of the kernel that prepares the token rows.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace fmoe {

namespace {

constexpr int kMaxRouteCluster = 8;         // portable cluster size

// The work items of one list: (expert, first sorted row, rows, group key) for every row tile of every expert that
// belongs to it.  Lists a and b (gate_up and down GEMM) have independent tile heights.  With split_rows > 0 they
// hold only the experts with at most split_rows rows, and lists c and d (tile big_tile) the experts with more: the
// batch's routing decides on the device, expert by expert, whether an expert's rows go to the weight-streaming kernel
// or to the two-SM kernel, with no host-side guess about the distribution.  Called by one whole warp.
__device__ void build_item_list(int list, int experts, const int* counts, const int* offsets, const ItemLists& lists, int* status, int lane) {
  const int split_rows = lists.split_rows;
  const int max_items = lists.max_items;
  const bool big = list >= 2;
  const int word = list == 0 ? kStatusItems : list == 1 ? kStatusItemsB : list == 2 ? kStatusItemsC : kStatusItemsD;
  if (big && split_rows <= 0) {
    if (lane == 0) status[word] = 0;
    return;
  }
  const int tile = list == 0 ? lists.tile_a : list == 1 ? lists.tile_b : lists.big_tile;
  int* items = list == 0 ? lists.items_a : list == 1 ? lists.items_b : list == 2 ? lists.items_c : lists.items_d;
  // Row tiles are powers of two but for the two-SM kernel's, 5/4 of one (320 token rows): its full height spares an expert a
  // second pass over its weights for a few rows; longer lists are cut at the power of two: two 256-row accumulators
  // fill tensor memory without sharing columns.  About 256 rows per expert (int8, 8192 tokens): 4228 -> 3877 us.  Lists of thousands of rows,
  // bf16, took 3312 us cut at 256 and 3367 us cut at 320; about 512 rows (int8, 16384 tokens) are the same either way.
  const bool tall = (tile & (tile - 1)) != 0;
  const int cut = tall ? tile / 5 * 4 : tile;
  const int shift = __ffs(cut) - 1;
  auto tiles_of = [&](int rows) { return tall && rows > cut && rows <= tile ? 1 : (rows + cut - 1) >> shift; };
  int carry = 0;
  int active = 0;
  int tallest = 0;
  constexpr int kBatch = 8;  // groups of 32 experts whose scans are interleaved: a scan is a chain of dependent shuffles
  for (int base = 0; base < experts; base += 32 * kBatch) {
    int count[kBatch], inclusive[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int e = base + 32 * i + lane;
      count[i] = e < experts ? counts[e] : 0;
      active += __popc(__ballot_sync(0xffffffffu, count[i] > 0));
      if (split_rows > 0 && big != (count[i] > split_rows)) count[i] = 0;  // belongs to the other list
      inclusive[i] = tiles_of(count[i]);
    }
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int other = __shfl_up_sync(0xffffffffu, inclusive[i], offset);
        if (lane >= offset) inclusive[i] += other;
      }
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int tiles = tiles_of(count[i]);
      const int first = carry + inclusive[i] - tiles;
      carry += __shfl_sync(0xffffffffu, inclusive[i], 31);
      if (tiles == 0) continue;
      const int e = base + 32 * i + lane;
      const int row0 = offsets[e];
      // The expert's rows are spread evenly over its tiles (in steps of 32 rows, the granularity of the MMA's N):
      // 330 rows become 192 + 138, not 256 + 74.
      int rows_per = tile;
      if (tiles > 1) {
        const int step = tile < 32 ? tile : 32;
        const int even = ((count[i] + tiles - 1) / tiles + step - 1) & ~(step - 1);
        if (even <= tile && (tiles - 1) * even < count[i]) rows_per = even;
      }
      tallest = max(tallest, min(rows_per, count[i]));
      for (int t = 0; t < tiles && first + t < max_items; ++t) {
        // Group key for the unit order of the grouped GEMM: first item of this expert and its tile count, so that the
        // row tiles of one (expert, channel block) are consecutive work units (see resolve_unit in umma_gemm.cu).
        reinterpret_cast<int4*>(items)[first + t] = make_int4(e, row0 + t * rows_per, min(rows_per, count[i] - t * rows_per),
                                                              tiles < 2048 ? (first | (tiles << 20)) : ((first + t) | (1 << 20)));
      }
    }
  }
  for (int offset = 16; offset > 0; offset >>= 1) tallest = max(tallest, __shfl_xor_sync(0xffffffffu, tallest, offset));
  if (lane == 0) {
    status[list == 0 ? kStatusTallestA : list == 1 ? kStatusTallestB : list == 2 ? kStatusTallestC : kStatusTallestD] = tallest;
    status[word] = carry < max_items ? carry : max_items;
    if (list == 0) status[kStatusActive] = active;
  }
}

// Exclusive scan of values[0..n) into out[0..n], out[n] = total.  Called by the whole block; chunk_sums has room for
// (n + 31) / 32 ints.  Every 32 values are scanned by one warp, the chunk totals by warp 0.
__device__ void block_exclusive_scan(const int* values, int* out, int n, int* chunk_sums) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int chunks = (n + 31) >> 5;
  for (int chunk = warp; chunk < chunks; chunk += static_cast<int>(blockDim.x >> 5)) {
    const int index = chunk * 32 + lane;
    const int value = index < n ? values[index] : 0;
    int inclusive = value;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, inclusive, offset);
      if (lane >= offset) inclusive += other;
    }
    if (index < n) out[index] = inclusive - value;
    if (lane == 31) chunk_sums[chunk] = inclusive;
  }
  __syncthreads();
  if (warp == 0) {
    int carry = 0;
    for (int base = 0; base < chunks; base += 32) {
      const int index = base + lane;
      const int value = index < chunks ? chunk_sums[index] : 0;
      int inclusive = value;
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, inclusive, offset);
        if (lane >= offset) inclusive += other;
      }
      if (index < chunks) chunk_sums[index] = carry + inclusive - value;
      carry += __shfl_sync(0xffffffffu, inclusive, 31);
    }
    if (lane == 0) out[n] = carry;
  }
  __syncthreads();
  for (int index = threadIdx.x; index < n; index += blockDim.x) out[index] += chunk_sums[index >> 5];
  __syncthreads();
}

// The lanes of the warp that hold the same `id` as this one.  One ballot per bit of the id: `__match_any_sync`, which
// answers the same, costs about 80 clocks of the SM per call (65536 routes: 22 us with it, 18.5 us with ballots).
__device__ __forceinline__ unsigned lanes_with_same(int id, int bits) {
  unsigned same = 0xffffffffu;
  for (int bit = 0; bit < bits; ++bit) {
    const bool set = (id >> bit) & 1;
    const unsigned with_bit = __ballot_sync(0xffffffffu, set);
    same &= set ? with_bit : ~with_bit;
  }
  return same;
}

// Shared memory: hist[warps][experts] | counts[experts] | offsets[experts + 1] | chunk sums | kCluster: totals[experts],
// base[experts].  `run` routes per warp (a multiple of 32); warp w of CTA c owns the run number c * warps + w.
// Called by every thread of the CTA (kCluster: of every CTA of the cluster).
template <bool kCluster>
__device__ __forceinline__ void route_build(int* route_smem, const int64_t* topk_ids, int64_t routes, int experts, int warps, int64_t run,
                                            const ItemLists& lists, int* status, const int* mirror, int* counts, int* offsets,
                                            int* sorted_routes, int* row_expert, int* route_pos) {
  namespace cg = cooperative_groups;
  int* hist = route_smem;
  int* s_counts = hist + warps * experts;  // routes per expert
  int* s_offsets = s_counts + experts;
  int* chunk_sums = s_offsets + experts + 1;
  int* totals = kCluster ? chunk_sums + (experts + 31) / 32 : s_counts;  // this CTA's routes per expert (read by the other CTAs)
  int* base = kCluster ? totals + experts : s_offsets;                   // first sorted position of this CTA's routes of an expert
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = kCluster ? static_cast<int>(cg::this_cluster().block_rank()) : 0;
  const int ctas = kCluster ? static_cast<int>(cg::this_cluster().num_blocks()) : 1;

  for (int i = threadIdx.x; i < warps * experts; i += blockDim.x) hist[i] = 0;
  if (rank == 0 && threadIdx.x < kStatusWords) status[threadIdx.x] = cleared_status_word(threadIdx.x, mirror);
  __syncthreads();

  const int64_t begin = (static_cast<int64_t>(rank) * warps + warp) * run;
  const int64_t end = warp < warps ? min(begin + run, routes) : begin;
  int* row = hist + warp * experts;
  int64_t bad_route = -1;  // reported below, once the status block is known to be clear
  constexpr int kBatch = kCluster ? 4 : 1;  // rounds whose loads are in flight together (one CTA: a warp has one round)
  for (int64_t r0 = begin; r0 < end; r0 += 32 * kBatch) {
    int64_t ids[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) ids[i] = r0 + 32 * i + lane < end ? topk_ids[r0 + 32 * i + lane] : -1;
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      if (r0 + 32 * i + lane >= end) continue;
      if (ids[i] >= 0 && ids[i] < experts) {
        atomicAdd(row + ids[i], 1);
      } else {
        bad_route = r0 + 32 * i + lane;
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < experts; e += blockDim.x) {
    int running = 0;
#pragma unroll 8
    for (int w = 0; w < warps; ++w) {
      const int value = hist[w * experts + e];
      hist[w * experts + e] = running;
      running += value;
    }
    totals[e] = running;
  }
  if constexpr (kCluster) {
    __syncwarp();
    cg::this_cluster().sync();  // totals of every CTA and the cleared status block are visible
    for (int e = threadIdx.x; e < experts; e += blockDim.x) {
      int values[kMaxRouteCluster];
#pragma unroll
      for (int c = 0; c < kMaxRouteCluster; ++c) values[c] = c < ctas ? cg::this_cluster().map_shared_rank(totals, c)[e] : 0;
      int before = 0, all = 0;
#pragma unroll
      for (int c = 0; c < kMaxRouteCluster; ++c) {
        if (c < rank) before += values[c];
        all += values[c];
      }
      base[e] = before;
      s_counts[e] = all;
    }
    // This CTA reads no other CTA's totals after this: the release orders the reads above before the arrival, which lets the
    // others leave.  (The loop's trip count differs inside a warp, and the barrier wants whole warps.)
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  __syncthreads();
  if (bad_route >= 0) raise_error(status, FMOE_ERR_EXPERT_ID_RANGE, static_cast<int>(bad_route));
  block_exclusive_scan(s_counts, s_offsets, experts, chunk_sums);
  for (int e = threadIdx.x; e < experts; e += blockDim.x) {
    const int offset = s_offsets[e];
    if (kCluster) base[e] += offset;
    if (rank == 0) {
      counts[e] = s_counts[e];
      offsets[e] = offset;
    }
  }
  if (rank == 0 && threadIdx.x == 0) offsets[experts] = s_offsets[experts];
  if (kCluster) __syncthreads();

  // One warp per work-item list, in different CTAs where there are several (the last warps: they have the shortest runs).
  const int list = (static_cast<int>(blockDim.x >> 5) - 1 - warp) * ctas + rank;
  if (list < 4) build_item_list(list, experts, s_counts, s_offsets, lists, status, lane);

  const unsigned lanes_below = (1u << lane) - 1u;
  const int bits = 32 - __clz(experts);  // of the ids 0 .. experts, where `experts` stands for a dropped route
  for (int64_t r0 = begin; r0 < end; r0 += 32 * kBatch) {
    int ids[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      ids[i] = experts;
      if (r0 + 32 * i + lane < end) {
        const int64_t value = topk_ids[r0 + 32 * i + lane];
        if (value >= 0 && value < experts) ids[i] = static_cast<int>(value);
      }
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      if (r0 + 32 * i >= end) break;  // warp-uniform
      const int64_t route = r0 + 32 * i + lane;
      const int id = ids[i];
      const bool valid = id < experts;
      const unsigned peers = lanes_with_same(id, bits);
      int position = -1;
      if (valid) position = base[id] + row[id] + __popc(peers & lanes_below);
      __syncwarp();
      if (valid && (peers & lanes_below) == 0) row[id] += __popc(peers);
      __syncwarp();
      if (valid) {
        sorted_routes[position] = static_cast<int>(route);
        if (!kCluster) row_expert[position] = id;
      }
      // Inverse permutation: sorted position of every flat route (-1 for a dropped route).
      if (route_pos != nullptr && route < end) route_pos[route] = position;
    }
  }
  if (kCluster) {
    // The expert of every sorted row, a run of consecutive positions per warp: a scattered store takes 32 clocks of the
    // SM, so with a longer list the rows are not written where their routes are found.  Each lane looks the expert of
    // its first position up and walks the offsets from there.
    const int64_t rows_end = min(end, static_cast<int64_t>(s_offsets[experts]));
    int low = 0;
    for (int high = experts; low < high;) {
      const int middle = (low + high) >> 1;
      if (s_offsets[middle + 1] > begin + lane) {
        high = middle;
      } else {
        low = middle + 1;
      }
    }
    for (int64_t p = begin + lane; p < rows_end; p += 32) {
      while (s_offsets[low + 1] <= p) ++low;
      row_expert[p] = low;
    }
  }
  if (kCluster) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // no CTA leaves while another may still read its totals
  }
}

// Bytes of shared memory behind `route_smem`.
inline size_t route_smem_bytes(int warps, int experts, bool cluster) {
  return (static_cast<size_t>(warps) * experts + 2 * static_cast<size_t>(experts) + 1 + (experts + 31) / 32 +
          (cluster ? 2 * static_cast<size_t>(experts) : 0)) * sizeof(int);
}

}  // namespace

}  // namespace fmoe
