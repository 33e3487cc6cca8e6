// Regular quadrature, FP64, Helmholtz, the 6-point rule, phases referenced to the pair and at most 0.42 (see regular_fp64.cuh).
#include "regular_fp64.cuh"

namespace bempp_b200 {

cudaError_t launch_fp64_helmholtz6_short(const CellSet& test, const SpaceTiles& tt,
            const CellSet& trial, const SpaceTiles& st,
            const RegularRule& rule, const RegularArgs& a,
            cudaStream_t stream, bool direct) {
  return fp64::launch_op<true, kHelmholtz, fp64::kShort>(test, tt, trial, st, rule, a, stream, direct);
}

}  // namespace bempp_b200
