// Host-side rules of the CUDA sources, compiled for the CPU tests.
#include "acc_ring.cuh"
#include "kernels.h"

extern "C" int dense_vector_store(uintptr_t out, int n, int bf16) {
  return fmoe::dense_vector_store(reinterpret_cast<const void*>(out), n, bf16 != 0) ? 1 : 0;
}

// slots: start, blocks, head of every unit of a sequence; shared: blocks handed over by the unit before it.
extern "C" void place_units(const int* rows, int count, int* slots, int* shared) {
  fmoe::AccSlot before = {0, 0, 0};
  for (int i = 0; i < count; ++i) {
    const fmoe::AccSlot slot = fmoe::place_unit(before.start + before.blocks, rows[i]);
    slots[3 * i] = slot.start;
    slots[3 * i + 1] = slot.blocks;
    slots[3 * i + 2] = slot.head;
    shared[i] = fmoe::blocks_shared(before, slot);
    before = slot;
  }
}

// Arrivals of one epilogue warp (chunks first, first + step, ...) on the handover barrier of a unit, in the order of the kernel's
// epilogue; *early counts those in front of a load of a handed-over block.
extern "C" int handover_arrivals(int first, int step, int handed_over, int chunks, int* early) {
  bool held = handed_over > 0;
  int arrivals = 0;
  auto release = [&](int next_chunk) {
    if (!held || !fmoe::handed_over_read(next_chunk, handed_over, chunks)) return;
    held = false;
    ++arrivals;
  };
  release(first);
  for (int chunk = first; chunk < chunks; chunk += step) {
    if (!held && chunk < handed_over) ++*early;
    release(chunk + step);
  }
  return arrivals;
}
