// branch_f64_61_wide.cu -- branch kernels over FP64 partials of 61 states (more categories).
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_f64_61_wide(bool safe, int e2) {
  if (e2 == 8) return safe ? branch_fns<kR61, true, 8>() : branch_fns<kR61, false, 8>();
  if (e2 == 12) return safe ? branch_fns<kR61, true, 12>() : branch_fns<kR61, false, 12>();
  return safe ? branch_fns<kR61, true, 16>() : branch_fns<kR61, false, 16>();
}

}  // namespace gems
