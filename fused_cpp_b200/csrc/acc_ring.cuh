// Placement of the two-SM grouped GEMM's accumulators in tensor memory (plain integer rules, also compiled for the host).
#pragma once

#ifdef __CUDACC__
#define FMOE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FMOE_HOST_DEVICE inline
#endif

namespace fmoe {

constexpr int kRingBlocks = 16;  // 32-column blocks of tensor memory
constexpr int kMmaBlocks = 8;    // largest N of one MMA, in blocks

// Where a unit's accumulator lies.  Tensor memory is a ring of sixteen 32-column blocks; a unit of up to 320 rows takes
// one block per 32 rows, behind the unit before it, so that its main loop runs while that unit's accumulator is still
// being read.  A unit whose one MMA would run over the ring's end starts behind it instead.  Where that gap and the two
// units come to more than sixteen blocks the second takes over leading blocks of the first, at most seven of them if both
// have up to 256 rows (rows 32, 256, 256 do it, as any sequence of mixed sizes can; units of 256 rows never do), and waits
// for those (blocks_shared, barrier acc_part), not for the whole accumulator.
// Up to 256 rows are one MMA over consecutive columns; above that two MMAs share the staged weight tile, the first over
// `head` blocks.  Where the ring ends inside the accumulator the split lies there, and each MMA gets at least 64
// columns (a 32-column MMA takes as long as a 64-column one: it reads the same weight rows).
struct AccSlot {
  int start;   // running block number; its place in the ring is start mod 16
  int blocks;
  int head;
};

FMOE_HOST_DEVICE AccSlot place_unit(int start, int rows) {
  AccSlot slot = {start, (rows + 31) >> 5, 0};
  const int place = start & (kRingBlocks - 1);
  const int room = kRingBlocks - place;
  if (slot.blocks <= kMmaBlocks) {
    if (slot.blocks > room) slot.start += room;
    slot.head = slot.blocks;
  } else if (slot.blocks <= room || room < 2) {
    if (room < 2) slot.start += room;
    slot.head = (slot.blocks + 1) >> 1;
  } else {
    const int most = slot.blocks - 2 < kMmaBlocks ? slot.blocks - 2 : kMmaBlocks;
    slot.head = room < most ? room : most;
    slot.start += room - slot.head;
  }
  return slot;
}

// Leading blocks of `before` that lie where `slot`, the unit after it, has its accumulator.
FMOE_HOST_DEVICE int blocks_shared(const AccSlot& before, const AccSlot& slot) {
  const int shared = slot.start + slot.blocks - kRingBlocks - before.start;
  return shared > 0 ? shared : 0;
}

// A warp of the epilogue reads every other chunk (block) of a unit, `chunks` of them in all; its next one is `next_chunk`.  Whether
// it is past the blocks that the next unit takes over, and so owes their barrier its arrival.  A unit's chunks are its blocks, and
// blocks_shared is never more than those; but a unit whose accumulator is not read at all (the diagnostic library's switch,
// chunks = 0) hands its blocks over too, and the barrier counts every warp once a handover.
FMOE_HOST_DEVICE bool handed_over_read(int next_chunk, int handed_over, int chunks) {
  return next_chunk >= handed_over || next_chunk >= chunks;
}

}  // namespace fmoe
