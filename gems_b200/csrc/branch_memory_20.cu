// branch_memory_20.cu -- branch kernels over a theta in memory, blocks of 20 states and small ones of 61.
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_memory_20(int e2) {
  if (e2 == 3) return memory_fns<3>();
  if (e2 == 4) return memory_fns<4>();
  return memory_fns<5>();
}

}  // namespace gems
