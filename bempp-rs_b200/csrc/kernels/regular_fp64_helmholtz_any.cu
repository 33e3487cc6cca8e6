// Regular quadrature, FP64, Helmholtz, any rule, phases of any size (see regular_fp64.cuh).
#include "regular_fp64.cuh"

namespace bempp_b200 {

cudaError_t launch_fp64_helmholtz_any(const CellSet& test, const SpaceTiles& tt,
            const CellSet& trial, const SpaceTiles& st,
            const RegularRule& rule, const RegularArgs& a,
            cudaStream_t stream, bool direct) {
  return fp64::launch_op<false, kHelmholtz, fp64::kAnyPhase>(test, tt, trial, st, rule, a, stream, direct);
}

}  // namespace bempp_b200
