// Regular quadrature, FP64: which of the instantiations of regular_fp64.cuh a launch takes.
//   * rules made of two S21 orbits (the 6-point rule): the register-resident form, 3.5
//     operations per squared distance against 3.1 + loads for the general form;
//   * Helmholtz: phases referenced to the pair where the launch's bound k (rad_x + rad_y)
//     <= 0.8 holds (14 operations for sine and cosine), else reduced by pi/2 (18).  The
//     6-point rule's points lie within 0.725 circumradii, which the bound takes in; at
//     most 0.42 takes 12 operations.
//   * an operator of one space on a mesh in a poor order, its matrix beyond L2: every tile pair
//     instead of the lower half.  Blocks too large for the accumulators are added directly, and
//     direct adds to the transposed entries scatter over as many columns as the warp has test
//     cells.  Lower half -> all pairs, P1, shuffled cells: 20,480 triangles Laplace single layer
//     89.8 -> 17.8 ms, double 89.8 -> 18.1, hypersingular 93.6 -> 17.4, Helmholtz double 123.2 -> 46.8;
//     8,192 triangles (134 and 269 MB) 4.6 -> 2.9 and 12.7 -> 8.0; 5,120 (52 and 105 MB) 1.12 -> 1.21 and
//     2.90 -> 3.18.  A mesher's order (45 DOFs per tile), 20,480 triangles: Laplace 16.4 -> 14.8, 16.6 ->
//     16.2, 16.1 -> 14.1; Helmholtz, whose kernel values cost more than the adds, 36.5 -> 52.9
//     (hypersingular): there only where a tile's cells share next to no DOF.  Rules of more
//     points, whose kernel values cost more than the adds: the lower half always.
#include "regular_fp64.cuh"

namespace bempp_b200 {

using Launch = cudaError_t(const CellSet&, const SpaceTiles&, const CellSet&, const SpaceTiles&,
                           const RegularRule&, const RegularArgs&, cudaStream_t, bool);
Launch launch_fp64_laplace6, launch_fp64_laplace, launch_fp64_helmholtz6, launch_fp64_helmholtz6_short,
    launch_fp64_helmholtz6_any, launch_fp64_helmholtz, launch_fp64_helmholtz_any;

cudaError_t launch_regular_fp64(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                                const SpaceTiles& st, const RegularRule& rule,
                                const RegularArgs& a, cudaStream_t stream, bool direct) {
  if (a.symmetric && !direct && rule.npts <= 6) {
    constexpr int64_t kL2 = 126 << 20;
    const int64_t bytes = a.ld * a.ld * (a.kernel == kHelmholtz ? 16 : 8);
    const bool poor_order = a.kernel == kHelmholtz
                                ? tt.mean_tile_dofs > 2 * tt.tile_cells
                                : tt.max_tile_dofs * tt.most_dofs[0] * 8 > fp64::kAccumulatorBytes;
    // (not discontinuous P1, whose pairs own their entries)
    if (poor_order && bytes > kL2 && a.ld < 2 * static_cast<int64_t>(test.ncells)) {
      RegularArgs all = a;
      all.symmetric = 0;
      return launch_regular_fp64(test, tt, trial, st, rule, all, stream, direct);
    }
  }
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
