// Host build of the grid barrier's test (csrc/evp_kernels.cuh).  Test code only.
#include "evp_kernels.cuh"

extern "C" int barrier_complete(unsigned count, unsigned need) {
  return evp::barrier_complete(count, need);
}
