// Dense W8A8 linear over few rows, or few channels and a long K range: out[row, n] = (acc * row scale) * channel scale (+ bias[n]), acc = Xq * W^T
// (csrc/i8gemm.cpp:147-165), for one weight matrix or for two that share the quantised rows (csrc/i8gemm.cpp:454-570).
//
// Such a product streams its weights once and does almost nothing else, so what bounds it is HBM if enough SMs ask for
// weights, and latency before the first and after the last byte if not.  The kernel is built around that:
//   * A cluster of `parts` CTAs owns a block of 128 output channels and splits the K range: 7168 channels are 56 blocks,
//     which alone would leave two thirds of the SMs idle.  The parts' int32 accumulators meet through distributed
//     shared memory: every CTA leaves its own in shared memory and finishes every parts-th row from all of them
//     (integer sums: the order changes nothing).  No global table, nothing to clear, no atomics.
//   * The launch is a programmatic dependent of the row quantiser: barriers, tensor memory and the weight tiles of
//     every pipeline stage (up to 80 KB per CTA, two CTAs per SM) are fetched while the quantiser still runs; only the
//     token tiles and row scales wait for it.
//   * More than 128 rows are tiles of 128, a cluster each; the tiles of a channel block are neighbours and share its weights
//     in L2 (api.cu, dense_split_pays, says when that beats the two-SM kernel).
//   * Two weight matrices are one launch: the second one's channel blocks follow the first one's.
// Device time per op in a chain of ops (quantiser included; floor = weights at the copy bandwidth), against a persistent
// kernel without the cluster (a K split up to 16 rows over an int32 table with atomics) behind a finished quantiser:
//   16384 -> 7168    1 / 64 / 128 rows: 31.9 / 40.5 / 46.5 us -> 22.4 / 25.9 / 32.0 us (floor 18.2 / 18.7 / 19.1)
//   7168 -> 1536    16 / 64 / 128 rows: 14.4 / 22.2 / 25.6 us ->  8.0 /  9.5 / 12.8 us (floor 1.7 / 1.9 / 2.1)
//   1536 -> 24576    1 / 64 rows:       15.2 / 19.7 us        -> 10.4 / 12.9 us        (floor 5.9 / 6.4)
// What is left above the floor is launch and quantiser latency (about 5 us) and, with the rows, the exchange.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "ptx.cuh"

namespace fmoe {

namespace {

constexpr int kBlockM = 128;        // output channels per CTA (TMEM lanes)
constexpr int kBlockKBytes = 128;   // bytes of K per pipeline stage = one 128-byte swizzle row
constexpr int kUmmaKBytes = 32;     // bytes of K per tcgen05.mma
constexpr int kThreads = 192;       // warp 0: TMA, warp 1: tensor memory and MMA, warps 2..5: epilogue
constexpr int kWeightBytes = kBlockM * kBlockKBytes;
constexpr int kMaxStages = 10;
constexpr int kMaxParts = 8;        // portable cluster size
constexpr int kMinPartBlocks = 2;   // K blocks of a part, at least

// kDeep: one CTA per SM with all of its shared memory (few CTAs: the bytes in flight per CTA set the rate); otherwise
// two CTAs fit an SM.
template <int kRowTile, bool kDeep>
struct DenseConfig {
  static constexpr int kTokenBytes = kRowTile * kBlockKBytes;
  static constexpr int kStageBytes = kWeightBytes + kTokenBytes;
  static constexpr int kBudget = kDeep ? 200 * 1024 : 100 * 1024;
  static constexpr int kStages = kBudget / kStageBytes < kMaxStages ? kBudget / kStageBytes : kMaxStages;
  static constexpr int kTmemColumns = kRowTile < 32 ? 32 : kRowTile;
  static constexpr size_t kSmemBytes = 1024 /*alignment slack*/ + static_cast<size_t>(kStages) * kStageBytes + 2048 /*control block*/;
  static_assert(kStages * kStageBytes >= kRowTile * kBlockM * 4, "the accumulator exchange reuses the stages");
};

struct DenseControl {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  volatile int abort_flag;
  alignas(16) float row_scale[128];
  alignas(16) float channel_scale[kBlockM];
  alignas(16) float channel_bias[kBlockM];
};
static_assert(sizeof(DenseControl) <= 2048, "control block exceeds its shared-memory reservation");

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ int4 load_cluster_int4(uint32_t smem_address, int cta) {
  uint32_t remote;
  int4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_address), "r"(cta));
  asm volatile("ld.shared::cluster.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(remote) : "memory");
  return v;
}

// The matrix a CTA works on.
struct Side {
  const float* w_scale;
  void* out;
  int n;
  int out_bf16;
};

// Up to sixteen rows of one channel, from row `row` on (`count` of them, all sixteen with kAll): acc[j] belongs to row + j.
template <typename Out, bool kAll>
__device__ __forceinline__ void store_column(const Side& side, int row, int n, const uint32_t* acc, int count, const float* row_scale,
                                             float channel_scale, float bias) {
  Out* out = static_cast<Out*>(side.out) + static_cast<int64_t>(row) * side.n + n;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (!kAll && j >= count) break;
    const float value = __fadd_rn(dequantize(static_cast<int>(acc[j]), row_scale[j], channel_scale, FMOE_NUMERICS_TORCHREF), bias);
    if constexpr (sizeof(Out) == 2) {
      out[static_cast<int64_t>(j) * side.n] = f32_to_bf16_bits(value);
    } else {
      out[static_cast<int64_t>(j) * side.n] = value;
    }
  }
}

// Four channels of a row, of which `columns` exist; vector_store: dense_vector_store holds (then all four do).
__device__ __forceinline__ void store_row4(const Side& side, int row, int n, int4 acc, float row_scale, float4 scale, float4 bias,
                                           int columns, bool vector_store) {
  const int sums[4] = {acc.x, acc.y, acc.z, acc.w};
  const float scales[4] = {scale.x, scale.y, scale.z, scale.w};
  const float biases[4] = {bias.x, bias.y, bias.z, bias.w};
  float out[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) out[j] = __fadd_rn(dequantize(sums[j], row_scale, scales[j], FMOE_NUMERICS_TORCHREF), biases[j]);
  const int64_t index = static_cast<int64_t>(row) * side.n + n;
  if (vector_store && side.out_bf16) {
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(side.out) + index) =
        make_uint2(static_cast<uint32_t>(f32_to_bf16_bits(out[0])) | (static_cast<uint32_t>(f32_to_bf16_bits(out[1])) << 16),
                   static_cast<uint32_t>(f32_to_bf16_bits(out[2])) | (static_cast<uint32_t>(f32_to_bf16_bits(out[3])) << 16));
  } else if (vector_store) {
    *reinterpret_cast<float4*>(static_cast<float*>(side.out) + index) = make_float4(out[0], out[1], out[2], out[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j >= columns) break;
      if (side.out_bf16) {
        static_cast<uint16_t*>(side.out)[index + j] = f32_to_bf16_bits(out[j]);
      } else {
        static_cast<float*>(side.out)[index + j] = out[j];
      }
    }
  }
}

template <int kRowTile, bool kDeep>
__global__ void __launch_bounds__(kThreads)
dense_gemm_kernel(const __grid_constant__ CUtensorMap first_map, const __grid_constant__ CUtensorMap second_map,
                  const __grid_constant__ CUtensorMap token_map, DenseGemmArgs args) {
  using Cfg = DenseConfig<kRowTile, kDeep>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  DenseControl* ctl = reinterpret_cast<DenseControl*>(smem + static_cast<size_t>(Cfg::kStages) * Cfg::kStageBytes);
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);  // known to the compiler as warp-uniform
  const int lane = threadIdx.x & 31;
  int* status = args.status;
  const int parts = args.parts;
  const int part = static_cast<int>(blockIdx.x) % parts;  // = rank in the cluster
  const int unit = static_cast<int>(blockIdx.x) / parts;  // row tiles of a channel block side by side: they share its weights
  const int all_blocks = unit / args.row_tiles;
  const int row0 = (unit - all_blocks * args.row_tiles) * kRowTile;
  const int rows = min(kRowTile, args.rows - row0);  // of this CTA's tile
  const bool second = all_blocks >= args.first_blocks;
  const Side side = {second ? args.w_scale[1] : args.w_scale[0], second ? args.out[1] : args.out[0], second ? args.n[1] : args.n[0], args.out_bf16};
  const int n0 = (all_blocks - (second ? args.first_blocks : 0)) * kBlockM;
  const int kb_begin = part * args.k_blocks / parts;
  const int count = (part + 1) * args.k_blocks / parts - kb_begin;  // K blocks of this CTA, at least one

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    ptx::mbar_init(&ctl->acc_full, 1);
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&ctl->tmem_base, Cfg::kTmemColumns);
    ptx::tmem_relinquish();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    // ---------------- TMA producer (the whole warp walks the loops, one elected lane issues) ----------------
    const bool issuer = ptx::elect_one();
    const CUtensorMap* weight_map = second ? &second_map : &first_map;
    const int ahead = count < Cfg::kStages ? count : Cfg::kStages;
    // Weights of the first stages: they do not depend on the quantiser that may still be running.
    for (int i = 0; i < ahead; ++i) {
      if (issuer) {
        ptx::mbar_arrive_expect_tx(&ctl->full[i], Cfg::kStageBytes);
        ptx::tma_load_2d(smem + static_cast<size_t>(i) * Cfg::kStageBytes, weight_map, &ctl->full[i], (kb_begin + i) * kBlockKBytes, n0);
      }
    }
    ptx::grid_dependency_wait();
    for (int i = 0; i < ahead; ++i) {
      if (issuer) {
        ptx::tma_load_2d(smem + static_cast<size_t>(i) * Cfg::kStageBytes + kWeightBytes, &token_map, &ctl->full[i], (kb_begin + i) * kBlockKBytes, row0);
      }
    }
    int stage = ahead == Cfg::kStages ? 0 : ahead;
    uint32_t phase = ahead == Cfg::kStages ? 1u : 0u;
    for (int i = ahead; i < count; ++i) {
      ptx::mbar_wait(&ctl->empty[stage], phase ^ 1u, abort_flag, status, 21);
      if (issuer) {
        uint8_t* stage_base = smem + static_cast<size_t>(stage) * Cfg::kStageBytes;
        ptx::mbar_arrive_expect_tx(&ctl->full[stage], Cfg::kStageBytes);
        ptx::tma_load_2d(stage_base, weight_map, &ctl->full[stage], (kb_begin + i) * kBlockKBytes, n0);
        ptx::tma_load_2d(stage_base + kWeightBytes, &token_map, &ctl->full[stage], (kb_begin + i) * kBlockKBytes, row0);
      }
      if (++stage == Cfg::kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    // Drain: every load must have landed before the CTA may exit (the MMA warp has consumed them unless it gave up).
    for (int back = 0; back < ahead; ++back) {
      int s = stage - 1 - back;
      uint32_t p = phase;
      if (s < 0) {
        s += Cfg::kStages;
        p ^= 1u;
      }
      const unsigned long long start = ptx::global_timer_ns();
      while (!ptx::mbar_try_wait(&ctl->full[s], p)) {
        if (ptx::global_timer_ns() - start > ptx::kWaitLimitNs) break;
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool issuer = ptx::elect_one();
    const uint32_t idesc = ptx::make_instr_desc(true, kBlockM, (rows + 15) & ~15);
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < count; ++i) {
      ptx::mbar_wait(&ctl->full[stage], phase, abort_flag, status, 22);
      ptx::tcgen05_fence_after();
      const uint32_t stage_addr = ptx::smem_u32(smem + static_cast<size_t>(stage) * Cfg::kStageBytes);
      if (issuer) {
#pragma unroll
        for (int ks = 0; ks < kBlockKBytes / kUmmaKBytes; ++ks) {
          ptx::umma_ss<true>(tmem_base, ptx::make_smem_desc_sw128(stage_addr + ks * kUmmaKBytes),
                             ptx::make_smem_desc_sw128(stage_addr + kWeightBytes + ks * kUmmaKBytes), idesc, (i > 0 || ks > 0) ? 1u : 0u);
        }
        ptx::tcgen05_commit(&ctl->empty[stage]);
      }
      if (++stage == Cfg::kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (issuer) ptx::tcgen05_commit(&ctl->acc_full);
  }

  // ---------------- epilogue (warps 2..5): one thread per channel ----------------
  const int quarter = warp & 3;  // the TMEM lanes a warp may read are fixed by warp id % 4
  const int channel = quarter * 32 + lane;
  const int n = n0 + channel;
  const bool channel_ok = n < side.n;
  float channel_scale = 1.0f, bias = 0.0f;
  int* exchange = reinterpret_cast<int*>(smem);  // [rows][128 channels], once the stages are done with
  if (warp >= 2) {
    const int thread = static_cast<int>(threadIdx.x) - 64;
    // Before the wait, hence through L2: a scale or bias that an earlier call read at this address may still lie in L1.
    if (channel_ok) {
      channel_scale = __ldcg(side.w_scale + n);
      if (!second && args.bias != nullptr) bias = __ldcg(args.bias + n);
    }
    ctl->channel_scale[channel] = channel_scale;
    ctl->channel_bias[channel] = bias;
    ptx::grid_dependency_wait();  // the row scales come from the quantiser
    if (thread < rows) ctl->row_scale[thread] = args.a_scale[row0 + thread];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    ptx::mbar_wait(&ctl->acc_full, 0, abort_flag, status, 23);
    ptx::tcgen05_fence_after();
    const uint32_t acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    // Sixteen rows at a time, which form they take decided outside the value loop: with the checks inside it every value waited for
    // the one before it (128 rows, 64 -> 64: 14.2 -> 9.0 us per op; 7168 -> 129280: 193 -> 172 us; 7168 -> 1536: 17.6 -> 12.8 us).
    for (int c0 = 0; c0 < rows; c0 += 16) {
      uint32_t bits[16];
      ptx::tmem_ld_x8(acc + c0, bits);
      ptx::tmem_ld_x8(acc + c0 + 8, bits + 8);
      ptx::tmem_ld_wait();
      const int count = rows - c0;
      const float* const row_scale = ctl->row_scale + c0;
      if (parts > 1) {
        // (Rows of the last sixteen that do not exist have room in the stages too.)
#pragma unroll
        for (int j = 0; j < 16; ++j) exchange[(c0 + j) * kBlockM + channel] = static_cast<int>(bits[j]);
      } else if (channel_ok && side.out_bf16) {
        if (count >= 16) {
          store_column<uint16_t, true>(side, row0 + c0, n, bits, 16, row_scale, channel_scale, bias);
        } else {
          store_column<uint16_t, false>(side, row0 + c0, n, bits, count, row_scale, channel_scale, bias);
        }
      } else if (channel_ok) {
        if (count >= 16) {
          store_column<float, true>(side, row0 + c0, n, bits, 16, row_scale, channel_scale, bias);
        } else {
          store_column<float, false>(side, row0 + c0, n, bits, count, row_scale, channel_scale, bias);
        }
      }
      __syncwarp();  // the next tensor-memory load wants the whole warp
    }
  }
  if (parts > 1) {
    __syncwarp();
    cluster_sync();  // every part's accumulators lie in its shared memory
    if (warp >= 2) {
      // A warp finishes a row at a time, four channels per lane: 16-byte loads, all parts' in flight together.
      const int c4 = 4 * lane;
      const uint32_t mine = ptx::smem_u32(exchange) + 4u * static_cast<uint32_t>(c4);
      const int columns = side.n - (n0 + c4);  // channels of this lane that exist, if below four
      const float4 scales = *reinterpret_cast<const float4*>(ctl->channel_scale + c4);
      const float4 biases = *reinterpret_cast<const float4*>(ctl->channel_bias + c4);
      const bool vector_store = (second ? args.vector_store[1] : args.vector_store[0]) != 0;  // a lane's four channels all exist or none does
      constexpr int kBatch = 2;  // rows of a warp whose loads are in flight together (a remote load takes most of a microsecond)
      for (int first = part + parts * (warp - 2); first < rows; first += 4 * parts * kBatch) {
        int4 values[kBatch][kMaxParts];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int row = first + 4 * parts * b;
#pragma unroll
          for (int c = 0; c < kMaxParts; ++c) {
            values[b][c] = make_int4(0, 0, 0, 0);
            if (c < parts && row < rows) values[b][c] = load_cluster_int4(mine + static_cast<uint32_t>(row) * (kBlockM * 4), c);
          }
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int row = first + 4 * parts * b;
          if (row >= rows || columns <= 0) continue;
          int4 sum = values[b][0];
#pragma unroll
          for (int c = 1; c < kMaxParts; ++c) {
            sum.x += values[b][c].x;
            sum.y += values[b][c].y;
            sum.z += values[b][c].z;
            sum.w += values[b][c].w;
          }
          store_row4(side, row0 + row, n0 + c4, sum, ctl->row_scale[row], scales, biases, columns, vector_store);
        }
      }
    }
    __syncwarp();
    cluster_sync();  // no part leaves while another may still read its accumulators
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    ptx::tcgen05_fence_after();
    ptx::tmem_dealloc(tmem_base, Cfg::kTmemColumns);
  }
}

// How many clusters of 1 .. kMaxParts CTAs can be resident at once with one CTA per SM (asked once per device: a cluster
// lives inside a GPC, so this is less than SMs / cluster size).  Also sets the kernels' shared-memory attributes.
struct Residency {
  int clusters[kMaxParts + 1] = {};
};

template <int kRowTile, bool kDeep>
cudaError_t configure() {
  auto kernel = dense_gemm_kernel<kRowTile, kDeep>;
  const cudaError_t error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(DenseConfig<kRowTile, kDeep>::kSmemBytes));
  return error != cudaSuccess ? error
                              : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

template <int kRowTile>
cudaError_t residency(Residency* out) {
  static std::mutex guard;  // a thread that finds the flag set has to find the table too
  static PerDeviceOnce configured;
  static Residency known[kMaxDevices];
  const std::lock_guard<std::mutex> lock(guard);
  const int device = current_device_ordinal();
  if (!configured.needed(device)) {
    *out = known[device];
    return cudaSuccess;
  }
  cudaError_t error = configure<kRowTile, true>();
  if (error == cudaSuccess) error = configure<kRowTile, false>();
  for (int parts = 1; parts <= kMaxParts && error == cudaSuccess; ++parts) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(parts));
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = DenseConfig<kRowTile, true>::kSmemBytes;
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = static_cast<unsigned>(parts);
    attribute.val.clusterDim.y = 1;
    attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    error = cudaOccupancyMaxActiveClusters(&out->clusters[parts], dense_gemm_kernel<kRowTile, true>, &config);
  }
  if (error != cudaSuccess) return error;
  if (device >= 0 && device < kMaxDevices) known[device] = *out;
  configured.mark(device);
  return cudaSuccess;
}

template <int kRowTile, bool kDeep>
cudaError_t launch_kernel(const DenseGemmArgs& args, int blocks, const CUtensorMap* maps, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(blocks * args.parts));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = DenseConfig<kRowTile, kDeep>::kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = static_cast<unsigned>(args.parts);
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, dense_gemm_kernel<kRowTile, kDeep>, maps[0], maps[1], maps[2], args);
}

template <int kRowTile>
cudaError_t launch_dense(DenseGemmArgs args, const void* a_rows, const int8_t* const* weights, bool split, cudaStream_t stream) {
  const uint64_t k = static_cast<uint64_t>(args.k_padded);
  CUtensorMap maps[3];
  if (!make_sw128_map(&maps[0], weights[0], true, args.n[0], k, kBlockM) ||
      !make_sw128_map(&maps[1], args.n[1] > 0 ? weights[1] : weights[0], true, args.n[1] > 0 ? args.n[1] : args.n[0], k, kBlockM) ||
      !make_sw128_map(&maps[2], a_rows, true, args.rows, k, kRowTile)) {
    return cudaErrorInvalidValue;
  }
  Residency one_per_sm;
  const cudaError_t error = residency<kRowTile>(&one_per_sm);
  if (error != cudaSuccess) return error;
  const int blocks = (args.first_blocks + (args.n[1] + kBlockM - 1) / kBlockM) * args.row_tiles;
  // As many parts as leave all clusters resident at once, two CTAs per SM if need be, every part at least two K blocks.
  // Device time per op of a chain of ops, parts 1 / 2 / 3 / 4 / 5 / 8, 64 rows: 16384 -> 7168 (56 blocks; clusters of five
  // and more take a second wave) 35 / 28 / 28 / 27 / 29 / 33 us; 7168 -> 1536 (12 blocks) 18.5 / 13.5 / 11.4 / 10.4 / 10.3 / 9.6 us;
  // 1536 -> 24576 (192 blocks, 12 K blocks) 13 / 19 / 22 / 23 / 27 us.  One CTA per SM with deep stages where that holds them
  // all: 7168 -> 1536 12.2 -> 11.5 us.
  args.parts = 1;
  for (int parts = kMaxParts; split && parts > 1; --parts) {
    if (blocks <= 2 * one_per_sm.clusters[parts] && parts * kMinPartBlocks <= args.k_blocks) {
      args.parts = parts;
      break;
    }
  }
  if (blocks <= one_per_sm.clusters[args.parts]) return launch_kernel<kRowTile, true>(args, blocks, maps, stream);
  return launch_kernel<kRowTile, false>(args, blocks, maps, stream);
}

}  // namespace

cudaError_t launch_dense_gemm(const DenseGemmArgs& caller_args, const void* a_rows, const int8_t* const* weights, bool split, cudaStream_t stream) {
  DenseGemmArgs args = caller_args;
  if (args.rows <= 0 || args.n[0] <= 0 || args.k_padded % 16 != 0) return cudaErrorInvalidValue;
  args.row_tiles = (args.rows + kDenseMaxRows - 1) / kDenseMaxRows;
  args.first_blocks = (args.n[0] + kBlockM - 1) / kBlockM;
  args.k_blocks = (args.k_padded + kBlockKBytes - 1) / kBlockKBytes;
  for (int i = 0; i < 2; ++i) args.vector_store[i] = dense_vector_store(args.out[i], args.n[i], args.out_bf16 != 0) ? 1 : 0;
  if (args.rows <= 16) return launch_dense<16>(args, a_rows, weights, split, stream);
  if (args.rows <= 32) return launch_dense<32>(args, a_rows, weights, split, stream);
  if (args.rows <= 64) return launch_dense<64>(args, a_rows, weights, split, stream);
  return launch_dense<128>(args, a_rows, weights, split, stream);
}

}  // namespace fmoe
