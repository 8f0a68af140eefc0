// branch_memory_4.cu -- branch kernels over a theta in memory, blocks of 4 states.
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_memory_4(int e2) {
  if (e2 == 1) return memory_fns<1>();
  return memory_fns<2>();
}

}  // namespace gems
