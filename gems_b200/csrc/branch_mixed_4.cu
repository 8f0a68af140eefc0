// branch_mixed_4.cu -- branch kernels over FP32 partials of 4 states.
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_mixed_4(bool safe, int e2) {
  if (e2 == 1) return safe ? branch_fns<kM4, true, 1>() : branch_fns<kM4, false, 1>();
  return safe ? branch_fns<kM4, true, 2>() : branch_fns<kM4, false, 2>();
}

}  // namespace gems
