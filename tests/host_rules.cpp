// Host-side rules of the CUDA sources, compiled for the CPU tests.
#include "kernels.h"

extern "C" int dense_vector_store(uintptr_t out, int n, int bf16) {
  return fmoe::dense_vector_store(reinterpret_cast<const void*>(out), n, bf16 != 0) ? 1 : 0;
}
