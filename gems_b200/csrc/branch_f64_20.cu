// branch_f64_20.cu -- branch kernels over FP64 partials of 20 states.
#include "branch_kernels.cuh"

namespace gems {

BranchFns branch_f64_20(bool safe, int e2) {
  if (e2 == 3) return safe ? branch_fns<kR20, true, 3>() : branch_fns<kR20, false, 3>();
  if (e2 == 4) return safe ? branch_fns<kR20, true, 4>() : branch_fns<kR20, false, 4>();
  return safe ? branch_fns<kR20, true, 5>() : branch_fns<kR20, false, 5>();
}

}  // namespace gems
