// branch_f64_61.cu -- branch kernels over FP64 partials of 61 states (up to five categories).
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_f64_61(bool safe, int e2) {
  if (e2 == 3) return safe ? branch_fns<kR61, true, 3>() : branch_fns<kR61, false, 3>();
  if (e2 == 4) return safe ? branch_fns<kR61, true, 4>() : branch_fns<kR61, false, 4>();
  return safe ? branch_fns<kR61, true, 5>() : branch_fns<kR61, false, 5>();
}

}  // namespace gems
