// branch_memory_wide.cu -- branch kernels over a theta in memory, large blocks of 61 states.
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_memory_wide(int e2) {
  if (e2 == 8) return memory_fns<8>();
  if (e2 == 12) return memory_fns<12>();
  return memory_fns<16>();
}

}  // namespace gems
