// Regular quadrature, FP64: which of the instantiations of regular_fp64.cuh a launch takes.
//   * rules made of two S21 orbits (the 6-point rule): the register-resident form, 3.5
//     operations per squared distance against 3.1 + loads for the general form;
//   * Helmholtz: phases referenced to the pair where the launch's bound k (rad_x + rad_y)
//     <= 0.8 holds (14 operations for sine and cosine), else reduced by pi/2 (18).  The
//     6-point rule's points lie within 0.725 circumradii, which the bound takes in; at
//     most 0.42 takes 12 operations.
#include "regular_fp64.cuh"

namespace bempp_b200 {

using Launch = cudaError_t(const CellSet&, const SpaceTiles&, const CellSet&, const SpaceTiles&,
                           const RegularRule&, const RegularArgs&, cudaStream_t, bool);
Launch launch_fp64_laplace6, launch_fp64_laplace, launch_fp64_helmholtz6, launch_fp64_helmholtz6_short,
    launch_fp64_helmholtz6_any, launch_fp64_helmholtz, launch_fp64_helmholtz_any;

cudaError_t launch_regular_fp64(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                                const SpaceTiles& st, const RegularRule& rule,
                                const RegularArgs& a, cudaStream_t stream, bool direct) {
  const bool orbits = fp64::has_orbit_form(rule);
  const double phase = orbits ? fp64::orbit_reach(rule) * a.phase_bound : a.phase_bound;
  Launch* fn;
  if (a.kernel == kLaplace)
    fn = orbits ? launch_fp64_laplace6 : launch_fp64_laplace;
  else if (orbits && phase <= 0.42)
    fn = launch_fp64_helmholtz6_short;
  else if (phase <= 0.8)
    fn = orbits ? launch_fp64_helmholtz6 : launch_fp64_helmholtz;
  else
    fn = orbits ? launch_fp64_helmholtz6_any : launch_fp64_helmholtz_any;
  return fn(test, tt, trial, st, rule, a, stream, direct);
}

}  // namespace bempp_b200
