// Grouped expert GEMM, two-SM form: a cluster of two CTAs drives `tcgen05.mma.cta_group::2` so that a
// 256 (channels) x 256 (tokens) tile costs each SM only 128 + 128 operand rows per K step.
//
// Same work as umma_gemm.cu (the reference's two run_stage sweeps and their epilogues,
// csrc/moe/arm/i8mm_w8a8/kernels.cpp:328-368, 230-257) for the prefill regime, where an expert has
// hundreds of rows.  Three things bound that regime and shape this kernel:
//   * one thread issues every MMA, and a dependent instruction costs it several clocks: a 128 x 128 x 32-byte
//     MMA runs 66 clocks, so anything beyond a dozen instructions per MMA starves the tensor pipe.  The pair
//     issues 256 x 256 MMAs (132 clocks each) from a loop that only adds constants to descriptor words;
//   * a 128 x 128 tile reads 8 KB of shared memory per 66 clocks, the full shared-memory bandwidth; here
//     each SM reads 4 + 4 KB per 132 clocks;
//   * the epilogue handles 128 x 256 accumulators per CTA per unit: eight warps, 32-column tensor-memory
//     loads, per-column metadata fetched one unit ahead, no block-wide barrier inside a unit.
//
// Pair layout.  CTA r of the pair (r = 0 leads) stages its own halves: 128 A rows (weight channels)
// and 128 B rows (tokens); the MMA reads A rows 0..127 from CTA 0 and 128..255 from CTA 1, B likewise,
// and leaves D rows 128r..128r+127 x 256 token columns in CTA r's tensor memory.
//   down:    A rows of CTA r = channels n0 + 128 r .. + 127.
//   gate_up: A rows of CTA r = channels c0 + 64 r .. + 63 as four groups of [16 gate rows | 16 up rows]
//            (one 5-D TMA box: {K bytes, 16 rows, gate/up, 4 groups, expert}), so lanes l and l + 16 of every
//            epilogue warp hold gate and up of the same channel and swap them with one shuffle.
// Work units.  Up to 256 token rows are one MMA per K step; an expert with 257 to 320 rows is one unit of two MMAs that share
// the weight tile, where two units of about 144 rows would each bring 32 KB of weights per K block for 20 KB of rows and
// wait for L2 (route.cu makes the items).  About 256 rows per expert, 8192 tokens of the 256-expert 7168 x 2048 int8 layer:
// gate_up 1969 -> 1770 us, down 1086 -> 1012 us.
// Barriers.  Both producers signal the leader's "full" barrier (TMA complete_tx through the cluster
// address), the leader's single MMA thread commits to the "empty" and "accumulator full" barriers of
// both CTAs, and the follower's epilogue warps arrive on the leader's "accumulator empty" barrier
// through its cluster address.  No load is a multicast load.  Every wait is bounded (see ptx.cuh).
#include <cuda.h>
#include <stdlib.h>

#include "acc_ring.cuh"
#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace fmoe {

namespace {

constexpr int kRowsPerCta = 128;    // A rows staged by one CTA
constexpr int kMmaTokens = 256;     // largest N of one MMA
constexpr int kMaxTokenRows = kPairItemRows;         // token rows of a work unit
constexpr int kTokensPerCta = kMaxTokenRows / 2;     // B rows staged by one CTA
constexpr int kBoxTokens = 16;                       // token rows of a block in one CTA, and of the smallest TMA box
constexpr int kMidBox = 4;                           // blocks of the middle box
constexpr int kFullBox = 8;                          // blocks of the largest
constexpr int kBlockKBytes = 128;
constexpr int kUmmaKBytes = 32;
#ifndef FMOE_PAIR_EPILOGUE_WARPS
#define FMOE_PAIR_EPILOGUE_WARPS 8
#endif
constexpr int kEpilogueWarps = FMOE_PAIR_EPILOGUE_WARPS;  // a multiple of 4: every TMEM lane quarter gets the same number
constexpr int kEpilogueThreads = kEpilogueWarps * 32;
constexpr int kThreads = 64 + kEpilogueThreads;
// Pipeline stages: a stage holds a CTA's weight rows and the token rows of the list's largest item.  Up to 128 rows per item (64
// per CTA) that is 24 KB instead of 36 and nine stages instead of six: with about a hundred rows per expert the weights'
// stream bounds the kernel, and half as many of their bytes again are on the way (256-expert layer, 2500 tokens int8 2266 ->
// 2203 us, 2048 tokens bf16 3888 -> 3835).  One longer item puts the whole list back on six stages: with uniform routing over 256
// experts a mean of a hundred rows has one about every second time, a mean of 110 nearly always.
constexpr int kStages = 6;
constexpr int kShortStages = 9;
constexpr int kShortTokens = 64;
constexpr int kWeightBytes = kRowsPerCta * kBlockKBytes;                // 16 KB
constexpr int kStageBytes = kWeightBytes + kTokensPerCta * kBlockKBytes;  // 36 KB
constexpr int kTmemColumns = 32 * kRingBlocks;                            // a ring of 32-column blocks (acc_ring.cuh)
static_assert(kMmaBlocks * 32 == kMmaTokens, "the ring's largest MMA");
constexpr size_t kControlBytes = 9216;
constexpr int kShortStageBytes = kWeightBytes + kShortTokens * kBlockKBytes;  // 24 KB
static_assert(kShortStages * kShortStageBytes <= kStages * kStageBytes, "both forms lie in the same shared memory");
constexpr size_t kSmemBytes = 1024 + static_cast<size_t>(kStages) * kStageBytes + kControlBytes;
static_assert(kSmemBytes <= 227 * 1024, "a CTA has 227 KB of shared memory");

// Per-column values of a work unit, staged one unit ahead so that the element loop reads shared memory.
struct ColumnMeta {
  float scale[kMaxTokenRows];      // activation scale of the row (int8)
  uint64_t rowptr[kMaxTokenRows];  // byte address of the output row (down / dense; may be peer memory)
};

struct PairControl {
  ColumnMeta meta[2];  // first: its arrays are read with 16-byte loads
  uint64_t full[kShortStages];
  uint64_t empty[kShortStages];
  uint64_t acc_full[2];
  uint64_t acc_part;      // the blocks of a unit that the next unit's accumulator takes over have been read (units that hand none over skip it)
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int abort_flag;
  uint32_t exp_table[64];  // copy of kExp2Table: divergent lookups are served by 32 banks
};
static_assert(sizeof(PairControl) <= kControlBytes, "control block exceeds its shared-memory reservation");

__device__ __forceinline__ uint32_t cluster_cta_rank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}

__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_address, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_address), "r"(cta));
  return remote;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrival on an mbarrier of either CTA.  It says that this warp's tensor-memory loads are done (they are: tcgen05.wait::ld
// stands in front of it) and publishes nothing that lies in memory, so it carries no cluster-wide release: that one waits
// until every store of the warp has reached L2, which in the epilogue are the result rows of the unit before (256-expert layer,
// 8192 tokens, int8, one pass after a pause: gate_up 1860 -> 1620 us, down 1015 -> 908, together with the release in front of
// the element loop; a steady loop is held by the power limit and gains 2 %, which is the spread of two runs; 2048 tokens of the
// 20-expert layer 374 -> 359).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_address) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}

// TMA tiled loads whose completion bytes go to an mbarrier given by its cluster address (the leader's).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster_address, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_address), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster_address, int c0, int c1,
                                                 int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      :
      : "r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_address), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(smem_result)), "r"(columns)
               : "memory");
}

__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t address, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}

// One arrival on the mbarrier at `cluster_address` once every MMA issued so far by this thread is done.
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t cluster_address) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_address) : "memory");
}

// D[tmem] (+)= A * B with the descriptors given as their 32-bit halves: the high word is the same for every
// operand tile of this kernel and the low word only ever has constants added to it, so the issuing thread
// spends one integer add per operand per MMA.
template <bool kInt8>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                          uint32_t accumulate) {
  if constexpr (kInt8) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], da, db, %4, p;\n\t"
        "}"
        :
        : "r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t"
        "}"
        :
        : "r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}

// 32 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld_x32(uint32_t address, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
      "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(address)
      : "memory");
}

__device__ __forceinline__ void epilogue_bar_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueThreads) : "memory"); }

// Work unit -> (work item, channel block), item-major: the units of one item (same token rows, successive
// channel blocks) are adjacent, and the same channel block of the next row tile of an expert is n_blocks
// units further, i.e. in flight on another pair at about the same time, so its weight tile comes from L2.
struct TrueTag {
  static constexpr bool value = true;
};
struct FalseTag {
  static constexpr bool value = false;
};

struct UnitInfo {
  int expert, row0, rows, block;
};

// rows_per_route: 2 in the two-plane form (first row and row count come back in token rows), else 1.
__device__ __forceinline__ UnitInfo load_unit(const int* items, int64_t unit, int64_t units, int n_blocks, int rows_per_route = 1) {
  UnitInfo info = {0, 0, 0, 0};
  if (unit < units) {
    const int item = static_cast<int>(unit / n_blocks);
    const int4 packed = __ldcg(reinterpret_cast<const int4*>(items) + item);
    info.expert = packed.x;
    info.row0 = packed.y * rows_per_route;
    info.rows = packed.z * rows_per_route;
    info.block = static_cast<int>(unit - static_cast<int64_t>(item) * n_blocks);
  }
  return info;
}

// The same unit with every field taken from lane 0 (all lanes hold the same values already).
__device__ __forceinline__ UnitInfo warp_uniform(UnitInfo info) {
  info.expert = __shfl_sync(0xffffffffu, info.expert, 0);
  info.row0 = __shfl_sync(0xffffffffu, info.row0, 0);
  info.rows = __shfl_sync(0xffffffffu, info.rows, 0);
  info.block = __shfl_sync(0xffffffffu, info.block, 0);
  return info;
}

// kPlanes (an instance of the int8 kernel; W8A16 in its fixed-point form): every route arrives as two int8 token rows,
// the high plane at row 2p and the low plane at row 2p + 1 of its 16-bit fixed-point activations, so a work item of r
// routes has 2r token rows (at most 160 routes) and accumulator columns (2j, 2j + 1) belong to route j: the exact
// integer dot product is 256 * column(2j) + column(2j + 1) (common.cuh: dequantize_planes).  Work items are given in
// routes; loads, the MMA's N and the epilogue count plane rows.
template <bool kInt8, bool kGateUp, bool kDense, bool kPlanes = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
umma_pair_grouped_gemm_kernel(const __grid_constant__ CUtensorMap weight_map, const __grid_constant__ CUtensorMap token_map,
                              const __grid_constant__ CUtensorMap token_map_mid, const __grid_constant__ CUtensorMap token_map_full,
                              GroupedGemmArgs args) {
  static_assert(!kPlanes || (kInt8 && !kDense), "the two-plane form is an instance of the int8 grouped kernel");
  constexpr int kElemBytes = kInt8 ? 1 : 2;
  constexpr int kBlockKElems = kBlockKBytes / kElemBytes;
  constexpr int kChannelsPerUnit = kGateUp ? 128 : 256;  // output channels one pair finishes per work unit
  constexpr int kRowsPerRoute = kPlanes ? 2 : 1;
  // The dense product's items hold at most 256 rows: two accumulators of 256 columns take turns, one MMA per K step, one
  // column of metadata per thread.  What larger items need is left out (3000 rows, 1536 -> 24576: 106.9 -> 105.9 us; 128 to 600 rows 0.1 to 0.5 us).
  constexpr bool kTall = !kDense;
  auto place = [](int start, int rows) {
    if constexpr (kTall) return place_unit(start, rows);
    return AccSlot{start, kMmaBlocks, (rows + 31) >> 5};  // a full half of the ring, whatever the unit takes of it
  };

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  PairControl* ctl = reinterpret_cast<PairControl*>(smem + static_cast<size_t>(kStages) * kStageBytes);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // the same value, known to be warp-uniform
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_cta_rank();
  const bool leader = cta == 0;
  int* status = args.status_rw;

  // (Values that come from global loads pass through a shuffle where the warps that feed TMA and the tensor pipe use
  // them: it changes nothing but lets the compiler treat them as warp-uniform.)
  auto count_items = [&]() { return __shfl_sync(0xffffffffu, min(__ldcg(args.status + args.item_count_word), args.max_items), 0); };
  if (args.items_late) ptx::grid_dependency_wait();
  int items = kDense ? 0 : count_items();
  const int n_blocks = (args.n_out + kChannelsPerUnit - 1) / kChannelsPerUnit;
  const int n_total = kGateUp ? 2 * args.n_out : args.n_out;
  int64_t units = static_cast<int64_t>(items) * n_blocks;
  const bool short_items =
      !kDense && __shfl_sync(0xffffffffu, __ldcg(args.status + args.tallest_word), 0) * kRowsPerRoute <= 2 * kShortTokens;
  const int stages = short_items ? kShortStages : kStages;
  const uint32_t stage_size = short_items ? kShortStageBytes : kStageBytes;
  const int k_blocks = (args.k + kBlockKElems - 1) / kBlockKElems;
  const int64_t first_unit = blockIdx.x >> 1;
  const int64_t unit_stride = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kShortStages; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&ctl->acc_full[b], 1);
      ptx::mbar_init(&ctl->acc_empty[b], 2 * kEpilogueWarps);  // the epilogue warps of both CTAs
    }
    ptx::mbar_init(&ctl->acc_part, 2 * kEpilogueWarps);
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
  }
  if (threadIdx.x >= 64 && threadIdx.x < 128) ctl->exp_table[threadIdx.x - 64] = kExp2Table[threadIdx.x - 64];
  if (warp == 1) {
    tmem_alloc_pair(&ctl->tmem_base, kTmemColumns);
    tmem_relinquish_pair();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // the peer's barriers are initialised before anything signals them
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort_flag;
  const uint32_t smem_base = ptx::smem_u32(smem);
  if constexpr (kDense) {
    // The work items come from the kernel right in front, the row quantiser: what overlaps it is the launch and the set-up above.
    // 129 / 600 / 3000 rows of 1536 -> 24576: 19.4 / 31.9 / 105.9 us as an ordinary launch, 17.8 / 30.5 / 104.8 us like this; 3000
    // rows of 7168 -> 1536 41.6 -> 39.9, of 16384 -> 1024 78.6 -> 79.4.
    ptx::grid_dependency_wait();
    items = count_items();
    units = static_cast<int64_t>(items) * n_blocks;
  }

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    // The whole warp walks the loop; one elected lane issues the loads (ptx::elect_one).
    {
      const bool issuer = ptx::elect_one();
      if (issuer) {
        ptx::prefetch_tensormap(&weight_map);
        ptx::prefetch_tensormap(&token_map);
        ptx::prefetch_tensormap(&token_map_mid);
        ptx::prefetch_tensormap(&token_map_full);
      }
      if (!args.beside) ptx::grid_dependency_wait();
      ptx::launch_dependents();
      const uint32_t full_leader0 = map_to_cta(ptx::smem_u32(&ctl->full[0]), 0);
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      UnitInfo cur = warp_uniform(load_unit(args.items, first_unit, units, n_blocks, kRowsPerRoute));
      int ring_end = 0;
      for (int64_t unit = first_unit; unit < units; unit += unit_stride) {
        const UnitInfo next = load_unit(args.items, unit + unit_stride, units, n_blocks, kRowsPerRoute);  // in flight during this unit
        // An MMA of N columns takes its first N/2 token rows from the leader's tile and the other N/2 from the follower's:
        // 16 rows per CTA and block.  One box brings the rows of a one-MMA unit, up to the next box size (a few
        // boxes of exactly its rows move less and take longer: about 512 rows per expert, 16384 tokens, 8087 -> 8216 us);
        // the two halves of a larger unit are laid out by boxes of 64 and 16 rows.
        const AccSlot slot = place(ring_end, cur.rows);
        ring_end = slot.start + slot.blocks;
        const int tail = kTall ? slot.blocks - slot.head : 0;
        const int head_row = cur.row0 + slot.head * kBoxTokens * static_cast<int>(cta);
        const int tail_row = cur.row0 + slot.head * 32 + tail * kBoxTokens * static_cast<int>(cta);
        const CUtensorMap* const one_box = slot.head <= kMidBox ? &token_map_mid : &token_map_full;
        const int loaded = tail > 0 ? slot.blocks : slot.head <= kMidBox ? kMidBox : kFullBox;
        const uint32_t stage_tx = 2u * (kWeightBytes + static_cast<uint32_t>(loaded) * kBoxTokens * kBlockKBytes);
        const int channel0 = cur.block * kChannelsPerUnit + (kChannelsPerUnit / 2) * static_cast<int>(cta);
        const int weight_row = cur.expert * n_total + channel0;  // down
        const int group = channel0 >> 4;                         // gate_up: 16-channel group
        for (int kb = 0; kb < k_blocks; ++kb) {
          ptx::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, status, 11);
          if (!issuer) {
            // the other lanes only keep step
          } else if (FMOE_DIAG_BIT(args, 2)) {
            if (leader) ptx::mbar_arrive(&ctl->full[stage]);
          } else {
            const uint32_t dst = smem_base + static_cast<uint32_t>(stage) * stage_size;
            const uint32_t bar = full_leader0 + 8u * static_cast<uint32_t>(stage);
            if (leader) ptx::mbar_arrive_expect_tx(&ctl->full[stage], stage_tx);
            const int x = kb * kBlockKElems;
            if constexpr (kGateUp) {
              if (args.gate_up_one_box) {
                // One 16 KB box of four groups of [16 gate rows | 16 up rows]: tensor dimensions
                // {K, row in group, gate/up, group, expert}.
                tma_load_5d_pair(dst, &weight_map, bar, x, 0, 0, group, cur.expert);
              } else {
                // The same rows as four 4 KB boxes: tensor dimensions {K, row in group, group, gate/up, expert}.
#pragma unroll
                for (int g = 0; g < 4; ++g) tma_load_5d_pair(dst + g * 32 * kBlockKBytes, &weight_map, bar, x, 0, group + g, 0, cur.expert);
              }
            } else {
              tma_load_2d_pair(dst, &weight_map, bar, x, weight_row);
            }
            const uint32_t tokens = dst + kWeightBytes;
            auto load_tokens = [&](uint32_t to, int blocks, int row) {
              int b = 0;
              for (; b + kMidBox <= blocks; b += kMidBox) {
                tma_load_2d_pair(to + b * kBoxTokens * kBlockKBytes, &token_map_mid, bar, x, row + b * kBoxTokens);
              }
              for (; b < blocks; ++b) tma_load_2d_pair(to + b * kBoxTokens * kBlockKBytes, &token_map, bar, x, row + b * kBoxTokens);
            };
            if (tail == 0) {
              tma_load_2d_pair(tokens, one_box, bar, x, head_row);
            } else {
              load_tokens(tokens, slot.head, head_row);
              load_tokens(tokens + slot.head * kBoxTokens * kBlockKBytes, tail, tail_row);
            }
          }
          ++issued;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        cur = warp_uniform(next);
      }
      if (leader) {
        // Drain: the leader's full barriers count both CTAs' bytes, so this also covers the follower's loads.
        const int pending = issued < stages ? issued : stages;
        for (int back = 0; back < pending; ++back) {
          int s = stage - 1 - back;
          uint32_t p = phase;
          if (s < 0) {
            s += stages;
            p ^= 1u;
          }
          const unsigned long long start = ptx::global_timer_ns();
          while (!ptx::mbar_try_wait(&ctl->full[s], p)) {
            if (ptx::global_timer_ns() - start > ptx::kWaitLimitNs) break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    // The whole warp walks the loop (waits included); one elected lane issues the MMAs and commits (ptx::elect_one).
    if (leader) {
      const bool issuer = ptx::elect_one();
      // Descriptor words (see ptx::make_smem_desc_sw128): the low word holds the start address >> 4 and the
      // ignored leading offset, the high word the 1024-byte group stride, version 1 and SWIZZLE_128B.
      const uint32_t desc_hi = static_cast<uint32_t>(1024 >> 4) | (1u << 14) | (2u << 29);
      const uint32_t a_lo_stage0 = ((smem_base & 0x3ffffu) >> 4) | (1u << 16);
      const uint32_t stage_step = stage_size >> 4;
      constexpr uint32_t kTokenStep = kWeightBytes >> 4;
      constexpr uint32_t kBlockStep = (kBoxTokens * kBlockKBytes) >> 4;  // one block's token rows in a CTA's tile
      const uint32_t empty_c0 = map_to_cta(ptx::smem_u32(&ctl->empty[0]), 0);
      const uint32_t empty_c1 = map_to_cta(ptx::smem_u32(&ctl->empty[0]), 1);
      const uint32_t accfull_c0 = map_to_cta(ptx::smem_u32(&ctl->acc_full[0]), 0);
      const uint32_t accfull_c1 = map_to_cta(ptx::smem_u32(&ctl->acc_full[0]), 1);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t a_lo = a_lo_stage0;
      int local = 0;
      UnitInfo cur = load_unit(args.items, first_unit, units, n_blocks, kRowsPerRoute);
      AccSlot before = {0, 0, 0};
      uint32_t handovers = 0;
      for (int64_t unit = first_unit; unit < units; unit += unit_stride, ++local) {
        const UnitInfo next = load_unit(args.items, unit + unit_stride, units, n_blocks, kRowsPerRoute);
        const uint32_t buffer = static_cast<uint32_t>(local) & 1u;
        const uint32_t use = static_cast<uint32_t>(local) >> 1;
        // N follows the rows this unit really has (a multiple of 32 for two-SM MMAs).  The row count comes from a global
        // load; the shuffle tells the compiler that every lane holds the same value.
        const int unit_rows = __shfl_sync(0xffffffffu, cur.rows, 0);
        const AccSlot slot = place(before.start + before.blocks, unit_rows);
        const int tail = kTall ? __shfl_sync(0xffffffffu, slot.blocks - slot.head, 0) : 0;
        const uint32_t idesc_head = __shfl_sync(0xffffffffu, ptx::make_instr_desc(kInt8, 2 * kRowsPerCta, 32 * slot.head), 0);
        const uint32_t idesc_tail = __shfl_sync(0xffffffffu, ptx::make_instr_desc(kInt8, 2 * kRowsPerCta, 32 * tail), 0);
        const uint32_t acc_head = __shfl_sync(0xffffffffu, tmem_base + 32u * static_cast<uint32_t>(slot.start & (kRingBlocks - 1)), 0);
        const uint32_t acc_tail =
            __shfl_sync(0xffffffffu, tmem_base + 32u * static_cast<uint32_t>((slot.start + slot.head) & (kRingBlocks - 1)), 0);
        const uint32_t tail_step = __shfl_sync(0xffffffffu, kTokenStep + kBlockStep * static_cast<uint32_t>(slot.head), 0);
        // The unit two before this one has left tensor memory, and the one before it the blocks that this one takes over.
        ptx::mbar_wait(&ctl->acc_empty[buffer], (use & 1u) ^ 1u, abort_flag, status, 12);
        if (kTall && blocks_shared(before, slot) > 0) {
          ptx::mbar_wait(&ctl->acc_part, handovers & 1u, abort_flag, status, 15);
          ++handovers;
        }
        before = slot;
        ptx::tcgen05_fence_after();
        // One loop per form: the usual one carries nothing of the other.
        auto main_loop = [&](auto tail_tag) {
          uint32_t accumulate = 0;
          for (int kb = 0; kb < k_blocks; ++kb) {
            ptx::mbar_wait(&ctl->full[stage], phase, abort_flag, status, 13);
            ptx::tcgen05_fence_after();
            if (issuer) {
              if (!FMOE_DIAG_BIT(args, 4)) {
#pragma unroll
                for (uint32_t ks = 0; ks < kBlockKBytes / kUmmaKBytes; ++ks) {
                  umma_pair<kInt8>(acc_head, a_lo + 2u * ks, a_lo + kTokenStep + 2u * ks, desc_hi, idesc_head, ks == 0 ? accumulate : 1u);
                }
                if constexpr (decltype(tail_tag)::value) {
#pragma unroll
                  for (uint32_t ks = 0; ks < kBlockKBytes / kUmmaKBytes; ++ks) {
                    umma_pair<kInt8>(acc_tail, a_lo + 2u * ks, a_lo + tail_step + 2u * ks, desc_hi, idesc_tail, ks == 0 ? accumulate : 1u);
                  }
                }
              }
              tcgen05_commit_pair(empty_c0 + 8u * static_cast<uint32_t>(stage));
              tcgen05_commit_pair(empty_c1 + 8u * static_cast<uint32_t>(stage));
            }
            accumulate = 1;
            a_lo += stage_step;
            if (++stage == stages) {
              stage = 0;
              phase ^= 1u;
              a_lo = a_lo_stage0;
            }
          }
        };
        if constexpr (kTall) {
          if (tail > 0) {
            main_loop(TrueTag{});
          } else {
            main_loop(FalseTag{});
          }
        } else {
          main_loop(FalseTag{});
        }
        if (issuer) {
          tcgen05_commit_pair(accfull_c0 + 8u * buffer);
          tcgen05_commit_pair(accfull_c1 + 8u * buffer);
        }
        cur = next;
      }
    }
  } else {
    // ---------------- epilogue (warps 2.. of both CTAs) ----------------
    if (!args.beside) ptx::grid_dependency_wait();
    const int quarter = warp & 3;                    // the TMEM lanes a warp may read are fixed by warp id % 4
    const int chunk_first = (warp - 2) >> 2;         // warps sharing a lane quarter take 32-column chunks round-robin
    constexpr int kChunkStep = kEpilogueWarps / 4;
    const int lane_in_tile = quarter * 32 + lane;    // TMEM lane = A row of this CTA
    const int tid = static_cast<int>(threadIdx.x) - 64;  // threads 0..255 stage the metadata of column tid and, below 64, of column 256 + tid
    const int n_out = args.n_out;
    const bool native = args.numerics == FMOE_NUMERICS_NATIVE;
    const float limit = args.swiglu_limit;
    const int activation = args.activation;
    uint32_t* const dump = kPlanes ? nullptr : static_cast<uint32_t*>(args.dump_acc);  // the dump holds one row per route
    const bool low = lane < 16;  // gate_up: lanes 0..15 hold gate rows, lanes 16..31 the up rows of the same channels
    // Output channel of this thread inside the unit's channel block.
    const int channel_in_unit = kGateUp ? 64 * static_cast<int>(cta) + 16 * quarter + (lane & 15)
                                        : kRowsPerCta * static_cast<int>(cta) + lane_in_tile;
    const uint32_t acc_part_leader = map_to_cta(ptx::smem_u32(&ctl->acc_part), 0);
    const uint32_t acc_empty_leader = map_to_cta(ptx::smem_u32(&ctl->acc_empty[0]), 0);
    const uint32_t acc_lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t* exp_table = ctl->exp_table;

    // Per-unit values: the column metadata in shared memory and this thread's weight scales in registers.  Both
    // are fetched while the previous unit is being finished.
    constexpr int kColumns = kTall ? 2 : 1;
    struct ThreadUnit {
      float column_scale[2];      // of columns `tid` and `tid` + 256 (the second with kTall)
      uint64_t column_rowptr[2];  // of the same columns: byte address of the output row (down / dense)
      float scale_gate, scale_up, bias;
    };
    auto fetch = [&](const UnitInfo& info, bool valid) {
      ThreadUnit t = {{0.0f, 0.0f}, {0ull, 0ull}, kInt8 ? 1.0f : 0.0f, kInt8 ? 1.0f : 0.0f, 0.0f};
      if (!valid) return t;
#pragma unroll
      for (int i = 0; i < kColumns; ++i) {
        const int column = tid + 256 * i;
        if (column >= info.rows) break;
        const int row = (info.row0 + column) / kRowsPerRoute;  // sorted position of the column's route
        if (kInt8) t.column_scale[i] = __ldcg(args.a_scale + row);
        if constexpr (kDense) {
          t.column_rowptr[i] = reinterpret_cast<uint64_t>(args.dense_out) + static_cast<uint64_t>(row) * n_out * (args.dense_out_bf16 ? 2 : 4);
        } else if constexpr (!kGateUp) {
          t.column_rowptr[i] = args.row_out_ptrs != nullptr
                                   ? __ldcg(args.row_out_ptrs + row)
                                   : reinterpret_cast<uint64_t>(args.route_out) +
                                         static_cast<uint64_t>(__ldcg(args.sorted_routes + row)) * n_out * (args.route_out_bf16 ? 2 : 4);
        }
      }
      const int n = info.block * kChannelsPerUnit + channel_in_unit;
      if (n < n_out) {
        if (kInt8) {
          const float* s = args.w_scale + static_cast<int64_t>(info.expert) * n_total;
          t.scale_gate = __ldcg(s + (kGateUp ? gate_channel(args, n) : n));
          if (kGateUp) t.scale_up = __ldcg(s + up_channel(args, n));
        }
        if (kDense && args.bias != nullptr) t.bias = args.bias[n];
        if (!kInt8 && !kDense && args.expert_bias != nullptr) {
          // BF16 path: the per-expert bias rides in the scale slots (unused without int8) and is ADDED.
          const int64_t first = static_cast<int64_t>(info.expert) * n_total;
          t.scale_gate = load_expert_bias(args, first + (kGateUp ? gate_channel(args, n) : n));
          if (kGateUp) t.scale_up = load_expert_bias(args, first + up_channel(args, n));
        }
      }
      return t;
    };

    // One accumulator value -> fp32 (int8: the reference's two multiplication orders, chosen at compile time).
    auto to_float = [&](auto native_tag, uint32_t bits, float a, float s) {
      if constexpr (kInt8) {
        const float value = static_cast<float>(static_cast<int>(bits));
        if constexpr (decltype(native_tag)::value) {
          return __fmul_rn(value, __fmul_rn(a, s));
        } else {
          return __fmul_rn(__fmul_rn(value, a), s);
        }
      } else {
        return __fadd_rn(__uint_as_float(bits), s);  // s = the channel's bias (0 without one)
      }
    };
    // Calls body(fast, native) with both flags turned into types: four instances of the element loop, one branch.
    auto dispatch = [&](bool fast, auto&& body) {
      if (fast) {
        if (native) {
          body(TrueTag{}, TrueTag{});
        } else {
          body(TrueTag{}, FalseTag{});
        }
      } else {
        if (native) {
          body(FalseTag{}, TrueTag{});
        } else {
          body(FalseTag{}, FalseTag{});
        }
      }
    };

    UnitInfo cur = load_unit(args.items, first_unit, units, n_blocks, kRowsPerRoute);
    UnitInfo next = load_unit(args.items, first_unit + unit_stride, units, n_blocks, kRowsPerRoute);
    ThreadUnit mine = fetch(cur, first_unit < units);
    auto publish = [&](ColumnMeta* meta, const ThreadUnit& t) {
#pragma unroll
      for (int i = 0; i < kColumns; ++i) {
        if (tid >= (i == 0 ? 256 : kMaxTokenRows - 256)) break;
        meta->scale[tid + 256 * i] = t.column_scale[i];
        meta->rowptr[tid + 256 * i] = t.column_rowptr[i];
      }
    };
    publish(&ctl->meta[0], mine);
    epilogue_bar_sync();

    int local = 0;
    AccSlot slot = place(0, cur.rows);
    for (int64_t unit = first_unit; unit < units; unit += unit_stride, ++local) {
      const uint32_t buffer = static_cast<uint32_t>(local) & 1u;
      const uint32_t use = static_cast<uint32_t>(local) >> 1;
      // Loads for the next unit (and the work item of the one after) are issued now and consumed after this unit.
      const ThreadUnit upcoming = fetch(next, unit + unit_stride < units);
      const UnitInfo after = load_unit(args.items, unit + 2 * unit_stride, units, n_blocks, kRowsPerRoute);

      const int rows = cur.rows;
      const int row0 = cur.row0;
      const int n = cur.block * kChannelsPerUnit + channel_in_unit;
      const bool channel_ok = n < n_out;
      const bool block_full = (cur.block + 1) * kChannelsPerUnit <= n_out;  // every thread's channel exists
      const ColumnMeta* meta = &ctl->meta[local & 1];
      const int chunks = FMOE_DIAG_BIT(args, 1) ? 0 : (rows + 31) >> 5;

      ptx::mbar_wait(&ctl->acc_full[buffer], use & 1u, abort_flag, status, 14);
      ptx::tcgen05_fence_after();
      // The next unit's accumulator may start on this one's first blocks: they are released as soon as they are read.
      const AccSlot next_slot = place(slot.start + slot.blocks, next.rows);
      const int handed_over = kTall ? blocks_shared(slot, next_slot) : 0;
      // A warp gives its share of them, and of the whole accumulator, back as soon as it holds the values of its last chunk
      // there in registers, before it works on them.
      bool part_held = handed_over > 0;
      bool all_held = true;
      auto release = [&](int next_chunk) {
        const bool part = part_held && handed_over_read(next_chunk, handed_over, chunks);
        const bool all = all_held && next_chunk >= chunks;
        if (!part && !all) return;
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (part) mbar_arrive_cluster(acc_part_leader);
          if (all) mbar_arrive_cluster(acc_empty_leader + 8u * buffer);
        }
        if (part) part_held = false;
        if (all) all_held = false;
      };
      release(chunk_first);
      for (int chunk = chunk_first; chunk < chunks; chunk += kChunkStep) {
        uint32_t v[32];
        tmem_ld_x32(acc_lane_base + 32u * static_cast<uint32_t>((slot.start + chunk) & (kRingBlocks - 1)), v);
        ptx::tmem_ld_wait();
        release(chunk + kChunkStep);
        const int col0 = chunk * 32;
        const bool fast = block_full && col0 + 32 <= rows && dump == nullptr;  // warp-uniform
        if constexpr (kGateUp && kPlanes) {
          // Columns 4q .. 4q + 3 are the (high, low) planes of two routes.  Lanes l (gate) and l + 16 (up) hold the same
          // channel: the gate lane finishes the first route of the four columns, the up lane the second, each receiving
          // the other's two plane values of that route.
          const float* scale = meta->scale + col0;
          with_activation<false>(activation, [&](auto act) {
            float gate[8], up[8];
            uint16_t result[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const uint32_t first = __shfl_xor_sync(0xffffffffu, low ? v[4 * q + 2] : v[4 * q], 16);
              const uint32_t second = __shfl_xor_sync(0xffffffffu, low ? v[4 * q + 3] : v[4 * q + 1], 16);
              const int column = 4 * q + (low ? 0 : 2);  // plane row of this lane's route inside the chunk
              const int gate_high = static_cast<int>(low ? v[4 * q] : first);
              const int gate_low = static_cast<int>(low ? v[4 * q + 1] : second);
              const int up_high = static_cast<int>(low ? first : v[4 * q + 2]);
              const int up_low = static_cast<int>(low ? second : v[4 * q + 3]);
              const float a = scale[column];
              gate[q] = dequantize_planes(gate_high, gate_low, a, mine.scale_gate);
              up[q] = dequantize_planes(up_high, up_low, a, mine.scale_up);
              if (col0 + column >= rows) gate[q] = up[q] = 1.0f;  // no row: nothing that could send the group to its slow branch
            }
            gated_group(act, gate, up, limit, exp_table, result);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int column = col0 + 4 * q + (low ? 0 : 2);
              if (column < rows && channel_ok) args.y[static_cast<int64_t>((row0 + column) >> 1) * n_out + n] = result[q];
            }
          });
        } else if constexpr (kPlanes) {
          // down: adjacent columns are the two planes of one route; the route's output row address is staged per column.
          const bool bf16_out = args.route_out_bf16 != 0;
          const uint64_t n_bytes = static_cast<uint64_t>(n) * (bf16_out ? 2 : 4);
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const int column = col0 + j;
            if (column >= rows || !channel_ok) continue;
            const float value = dequantize_planes(static_cast<int>(v[j]), static_cast<int>(v[j + 1]), meta->scale[column], mine.scale_gate);
            const uint64_t rowptr = meta->rowptr[column];
            if (bf16_out) {
              *reinterpret_cast<uint16_t*>(rowptr + n_bytes) = f32_to_bf16_bits(value);
            } else {
              *reinterpret_cast<float*>(rowptr + n_bytes) = value;
            }
          }
        } else if constexpr (kGateUp) {
          // Lanes l (gate) and l + 16 (up) hold the same channel: the gate lane finishes the even columns, the
          // up lane the odd ones, each receiving the other's value of that column.  Output rows are the sorted
          // rows themselves: row0 + column.
          uint16_t* const out0 = args.y + (static_cast<int64_t>(row0 + col0 + (low ? 0 : 1)) * n_out + n);
          const uint32_t pair_stride = 2u * static_cast<uint32_t>(n_out);
          const float4* scale4 = reinterpret_cast<const float4*>(meta->scale + col0);
          auto body = [&](auto fast_tag, auto native_tag) {
            constexpr bool kFast = decltype(fast_tag)::value;
            with_activation<kInt8>(activation, [&](auto act) {
#pragma unroll
              for (int group = 0; group < 2; ++group) {  // sixteen columns, eight elements of this thread
                float gate[8], up[8];
                uint16_t result[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const int p = 8 * group + i;
                  const float4 s4 = scale4[p >> 1];  // the scales of four columns (one broadcast load)
                  const uint32_t received = __shfl_xor_sync(0xffffffffu, low ? v[2 * p + 1] : v[2 * p], 16);
                  const uint32_t gate_bits = low ? v[2 * p] : received;
                  const uint32_t up_bits = low ? received : v[2 * p + 1];
                  const float a = (p & 1) == 0 ? (low ? s4.x : s4.y) : (low ? s4.z : s4.w);
                  gate[i] = to_float(native_tag, gate_bits, a, mine.scale_gate);
                  up[i] = to_float(native_tag, up_bits, a, mine.scale_up);
                  if constexpr (!kFast) {
                    const int column = col0 + 2 * p + (low ? 0 : 1);
                    if (column >= rows || !channel_ok) {
                      gate[i] = up[i] = 1.0f;  // no element: nothing that could send the group to its slow branch
                    } else if (dump != nullptr) {
                      uint32_t* out = dump + static_cast<int64_t>(row0 + column) * n_total;
                      out[n] = gate_bits;
                      out[n + n_out] = up_bits;
                    }
                  }
                }
                gated_group(act, gate, up, limit, exp_table, result);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  const int p = 8 * group + i;
                  if (kFast || (col0 + 2 * p + (low ? 0 : 1) < rows && channel_ok)) out0[static_cast<uint32_t>(p) * pair_stride] = result[i];
                }
              }
            });
          };
          dispatch(fast, body);
        } else {
          const float4* scale4 = reinterpret_cast<const float4*>(meta->scale + col0);
          const ulonglong2* rowptr2 = reinterpret_cast<const ulonglong2*>(meta->rowptr + col0);
          const bool bf16_out = kDense ? args.dense_out_bf16 != 0 : args.route_out_bf16 != 0;
          const uint64_t n_bytes = static_cast<uint64_t>(n) * (bf16_out ? 2 : 4);
          auto body = [&](auto fast_tag, auto native_tag) {
            constexpr bool kFast = decltype(fast_tag)::value;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 s4 = scale4[q];
              const ulonglong2 p01 = rowptr2[2 * q];
              const ulonglong2 p23 = rowptr2[2 * q + 1];
              const float scales[4] = {s4.x, s4.y, s4.z, s4.w};
              const uint64_t rowptrs[4] = {p01.x, p01.y, p23.x, p23.y};
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                const int j = 4 * q + h;
                if constexpr (!kFast) {
                  const int column = col0 + j;
                  if (column >= rows || !channel_ok) continue;
                  if (dump != nullptr) dump[static_cast<int64_t>(row0 + column) * n_total + n] = v[j];
                }
                float value = to_float(native_tag, v[j], scales[h], mine.scale_gate);
                if constexpr (kDense) {
                  value = __fadd_rn(value, mine.bias);
                  if (bf16_out) {
                    *reinterpret_cast<uint16_t*>(rowptrs[h] + n_bytes) = f32_to_bf16_bits(value);
                  } else {
                    *reinterpret_cast<float*>(rowptrs[h] + n_bytes) = value;
                  }
                } else if (bf16_out) {
                  *reinterpret_cast<uint16_t*>(rowptrs[h] + n_bytes) = f32_to_bf16_bits(value);
                } else {
                  *reinterpret_cast<float*>(rowptrs[h] + n_bytes) = value;
                }
              }
            }
          };
          dispatch(fast, body);
        }
      }

      // Publish the next unit's column metadata.  Nobody still reads that buffer: it belonged to the previous
      // unit, which every warp left before the barrier at the end of the previous iteration.
      publish(&ctl->meta[(local + 1) & 1], upcoming);
      epilogue_bar_sync();
      mine = upcoming;
      slot = next_slot;
      cur = next;
      next = after;
    }
  }

  if (args.beside && warp == 0) ptx::grid_dependency_wait();  // this kernel's end stands for the end of both
  ptx::tcgen05_fence_before();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while its peer may still signal its barriers or read its operands
  if (warp == 1) {
    __syncwarp();
    ptx::tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemColumns);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* symbol = nullptr;
    cudaDriverEntryPointQueryResult query;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &symbol, cudaEnableDefault, &query) == cudaSuccess &&
        query == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(symbol);
    }
  }
  return fn;
}

// gate_up weights [E, 2I, K] as a 5-D tensor whose boxes put the 16 gate rows of a channel group next to its 16
// up rows.  one_box: dimensions {K, 16 rows, gate|up, I/16 groups, E} and a box of four groups (16 KB, one TMA
// operation per stage; the gate|up stride is larger than the group stride that follows it).  Otherwise
// {K, 16 rows, I/16 groups, gate|up, E} with strides in ascending order and a box of one group (4 KB, four
// operations per stage): the fallback if the driver refuses the first encoding.
// The layout of w13 (gate rows then up rows, or alternating: args.interleaved) is in the strides of the first row
// dimension and of gate|up.
bool make_gate_up_map(CUtensorMap* map, const GroupedGemmArgs& args, bool int8, bool one_box) {
  EncodeTiledFn encode = encode_tiled_fn();
  if (encode == nullptr) return false;
  const uint64_t elem_bytes = int8 ? 1 : 2;
  const uint64_t k = static_cast<uint64_t>(args.k), inter = static_cast<uint64_t>(args.n_out), experts = static_cast<uint64_t>(args.experts);
  const uint64_t row_bytes = k * elem_bytes;
  const uint64_t channel_bytes = args.interleaved ? 2 * row_bytes : row_bytes;  // from a channel's row to the next channel's
  const uint64_t up_bytes = args.interleaved ? row_bytes : inter * row_bytes;   // from a channel's gate row to its up row
  void* const base = const_cast<void*>(args.weights);
  const cuuint32_t inner = static_cast<cuuint32_t>(kBlockKBytes / elem_bytes);
  const cuuint32_t elem_strides[5] = {1, 1, 1, 1, 1};
  const CUtensorMapDataType type = int8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  if (one_box) {
    const cuuint64_t dims[5] = {k, 16, 2, inter / 16, experts};
    const cuuint64_t strides[4] = {channel_bytes, up_bytes, 16 * channel_bytes, 2 * inter * row_bytes};
    const cuuint32_t box[5] = {inner, 16, 2, 4, 1};
    return encode(map, type, 5, base, dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  const cuuint64_t dims[5] = {k, 16, inter / 16, 2, experts};
  const cuuint64_t strides[4] = {channel_bytes, 16 * channel_bytes, up_bytes, 2 * inter * row_bytes};
  const cuuint32_t box[5] = {inner, 16, 1, 2, 1};
  return encode(map, type, 5, base, dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool kInt8, bool kGateUp, bool kDense, bool kPlanes = false>
cudaError_t launch_pair(const GroupedGemmArgs& args, cudaStream_t stream) {
  auto kernel = umma_pair_grouped_gemm_kernel<kInt8, kGateUp, kDense, kPlanes>;
  static PerDeviceOnce configured;
  const int device = current_device_ordinal();
  if (configured.needed(device)) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemBytes));
    if (err != cudaSuccess) return err;
    configured.mark(device);
  }
  CUtensorMap weight_map, token_map, token_map_mid, token_map_full;
  GroupedGemmArgs launch_args = args;
  bool weights_ok;
  if (kGateUp) {
    bool try_one = args.n_out % 64 == 0;
#ifdef FMOE_DIAG
    const char* forced = getenv("FUSED_CPP_MOE_GATE_UP_BOXES");  // diagnostic library only: "4" forces the four-box encoding
    if (forced != nullptr && forced[0] == '4') try_one = false;
#endif
    launch_args.gate_up_one_box = try_one && make_gate_up_map(&weight_map, args, kInt8, true);
    weights_ok = launch_args.gate_up_one_box || make_gate_up_map(&weight_map, args, kInt8, false);
  } else {
    weights_ok = make_sw128_map(&weight_map, args.weights, kInt8, static_cast<uint64_t>(args.experts) * args.n_out, args.k, kRowsPerCta);
  }
  const uint64_t token_rows = static_cast<uint64_t>(args.total_rows) * (kPlanes ? 2 : 1);
  if (!weights_ok || !make_sw128_map(&token_map, args.a_rows, kInt8, token_rows, args.k, kBoxTokens) ||
      !make_sw128_map(&token_map_mid, args.a_rows, kInt8, token_rows, args.k, kMidBox * kBoxTokens) ||
      !make_sw128_map(&token_map_full, args.a_rows, kInt8, token_rows, args.k, kFullBox * kBoxTokens)) {
    return cudaErrorInvalidValue;
  }
  const int sms = sm_count_of_current_device();
  const int channels_per_unit = kGateUp ? 128 : 256;
  const int n_blocks = (args.n_out + channels_per_unit - 1) / channels_per_unit;
  int64_t pairs = static_cast<int64_t>(args.max_items) * n_blocks;
  if (pairs > sms / 2) pairs = sms / 2;
  if (pairs <= 0) return cudaSuccess;
  return launch_chained(kernel, dim3(static_cast<unsigned>(2 * pairs)), kThreads, kSmemBytes, stream, true, weight_map, token_map,
                        token_map_mid, token_map_full, launch_args);
}

}  // namespace

cudaError_t launch_umma_pair_grouped_gemm(const GroupedGemmArgs& args, bool int8, bool gate_up, cudaStream_t stream) {
  if (args.max_items <= 0 || args.total_rows <= 0) return cudaSuccess;
  if (gate_up && args.n_out % 16 != 0) return cudaErrorInvalidValue;  // gate_up stages 16-channel groups
  if (args.w8a16 == 2) {
    // W8A16 in its fixed-point form: int8 kernel, two token rows per route, work items of at most 160 routes.
    if (!int8 || args.dense_out != nullptr || args.a_scale == nullptr) return cudaErrorInvalidValue;
    return gate_up ? launch_pair<true, true, false, true>(args, stream) : launch_pair<true, false, false, true>(args, stream);
  }
  if (args.dense_out != nullptr) {
    if (!int8 || gate_up) return cudaErrorInvalidValue;
    return launch_pair<true, false, true>(args, stream);
  }
  if (int8) return gate_up ? launch_pair<true, true, false>(args, stream) : launch_pair<true, false, false>(args, stream);
  return gate_up ? launch_pair<false, true, false>(args, stream) : launch_pair<false, false, false>(args, stream);
}

}  // namespace fmoe
