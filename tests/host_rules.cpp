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
