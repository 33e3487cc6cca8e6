// Off-surface potential operators of the boundary kernels, FP64:
//   P[i, j] = sum_{cells c with DOF j} jdet_c sum_q w_q psi_b(xi_q) K(x_i, y_c(xi_q)),
// single layer K = G(x, y), double layer K = n_y . grad_y G(x, y), with
//   Laplace     G = 1 / (4 pi r),         n_y . grad_y G = (x - y).n_y / (4 pi r^3),
//   Helmholtz   G = e^{ikr} / (4 pi r),   n_y . grad_y G = e^{ikr} (1 - ikr) (x - y).n_y / (4 pi r^3),
// r = |x - y|, for evaluation points x_i off the surface (regular quadrature only).  The
// reference declares src/boundary_evaluators.rs (empty) and keeps bempp-cl values for these
// four operators in commented tests (tests/compare_to_bempp_cl.rs:208-320); the kernel
// conventions are those of its boundary operators (src/boundary_assemblers/helpers.rs:7-40,
// integrands/single_layer.rs, integrands/double_layer.rs).
//
// The FP64 pipe bounds the kernel: a Helmholtz double layer costs about 40 operations per
// (point, rule point), 18 of them the sine and cosine.  So the distances come from the
// cell's centroid c and offsets g_0, g_1 (regular_fp64.cuh): with dc = x - c,
//   |x - y_q|^2 = (|dc|^2 + |y_q - c|^2) + alpha_q W0 + beta_q W1,  W = -2 dc.g,
// three operations instead of six, (x - y_q).n = dc.n is formed once per cell, and the rule
// points go through the kernel values six at a time.  Where those terms cancel (a point whose
// distance from the centroid is below 1.14 times the rule points' largest: see
// fp64::close_pair) the components of x - y_q are taken instead, after the other cells.
//
// Mapping.  A CTA stages one tile of 32 trial cells; each of its four warps has 32 points
// (lane = point) and walks the tile's cells, or a chunk of them where the points are few.
// DP0: every (point, cell) pair owns its entry (coalesced stores).  Other spaces: each lane
// sums into its own column of the tile's DOFs in shared memory, added to the zeroed output
// once per tile (27 coalesced adds per 32 cells instead of 96); spaces whose columns do not
// fit (degree 2) add every cell's values directly.
//
// B200, differences of coordinates and a global add per cell, basis and point -> this form:
// Helmholtz double layer P1, 5,120 cells x 2,000 points, 6-point rule: 0.351 -> 0.294 ms; single
// layer DP0 0.285 -> 0.206; Laplace double layer P1, 8,000 cells x 3,000 points: 0.382 -> 0.271;
// 16-point rule, Helmholtz double layer P1, 3,000 x 2,000: 0.497 -> 0.393, 300 cells x 60 points:
// 0.059 -> 0.032 (the chunks).  Telling the close points apart takes 2 % of these times (the call
// at 5,120 cells x 2,000 points: 0.277 -> 0.283 ms; with the test by FP64 operations and a branch 0.296).
#include "regular_fp64.cuh"

namespace bempp_b200 {
namespace {

using namespace tiles;

constexpr int kGroup = 6;  // rule points per kernel evaluation (their chains hide the FP64 latency)

struct PotentialRule {
  int npts;
  double reach;                     // see fp64::rule_reach
  double ab[kMaxRegularPoints][2];  // coordinates along g_0, g_1
  double w[kMaxRegularPoints][6];   // weight times basis values
};

// Shared memory: trial tile, |y_q - c|^2 and weights per rule point, DOF columns.
template <int NB>
__host__ __device__ inline size_t potential_smem(int q, int cap, int parts, size_t* columns) {
  size_t o = sizeof(double) * fp64::kRows * kTile;
  o += sizeof(double) * kTile * q;          // squared lengths
  o += sizeof(double) * q * (2 + NB);       // (alpha, beta), weights
  o += sizeof(int) * NB * kTile;            // the cells' columns, or their DOFs
  o = (o + 15) & ~size_t(15);
  *columns = o;
  o += sizeof(double) * static_cast<size_t>(kWarps) * cap * kTile * parts + sizeof(int) * cap;
  return o;
}

template <int KER, int OP, int NB>
__global__ void __launch_bounds__(kThreads, 4)
    potential_tiles(const double* __restrict__ points, int npoints, CellSet trial, SpaceTiles st,
                    const __grid_constant__ PotentialRule rule, double k,
                    double* __restrict__ out, int64_t ld, int ns, int cap) {
  constexpr int NP = KER == kHelmholtz ? 2 : 1;
  const int Q = rule.npts;
  const int cpt = kTile / ns;
  const int tile = blockIdx.y / cpt, c0 = tile * kTile;
  const int j0 = (blockIdx.y % cpt) * ns, j1 = min(j0 + ns, min(kTile, trial.ncells - c0));
  if (j0 >= j1) return;
  extern __shared__ __align__(16) unsigned char smem[];
  size_t columns;
  potential_smem<NB>(Q, cap, NP, &columns);
  Tile S;
  S.pts = nullptr;
  S.rel = nullptr;
  S.vid = S.ldof = nullptr;
  S.geo = reinterpret_cast<double*>(smem);
  double* len = S.geo + fp64::kRows * kTile;  // [q * kTile + cell]
  double* ab = len + kTile * Q;               // [2 * q]
  double* wt = ab + 2 * Q;                    // [q * NB + b]
  int* dof = reinterpret_cast<int*>(wt + NB * Q);  // [cell * NB + b]
  for (int i = threadIdx.x; i < kNumGeomFields * kTile; i += kThreads)
    S.geo[i] = __ldg(trial.geom + static_cast<int64_t>(i / kTile) * trial.stride + c0 + i % kTile);
  for (int i = threadIdx.x; i < Q; i += kThreads) {
    ab[2 * i] = rule.ab[i][0];
    ab[2 * i + 1] = rule.ab[i][1];
#pragma unroll
    for (int b = 0; b < NB; ++b) wt[i * NB + b] = rule.w[i][b];
  }
  for (int i = threadIdx.x; i < NB * kTile; i += kThreads) {
    const int64_t e = static_cast<int64_t>(c0) * NB + i;
    dof[i] = c0 + i / NB >= trial.ncells ? 0
             : NB > 1 && cap > 0         ? __ldg(st.cell_ldof + e) * kTile * NP
                                         : __ldg(st.cell_dofs + e);
  }
  __syncthreads();
  if (threadIdx.x < kTile) fp64::geometry_to_offsets(S, threadIdx.x, rule.reach);
  __syncthreads();
  if (threadIdx.x < kTile)  // squared: compared with |x - c|^2
    S.geo[fp64::rR * kTile + threadIdx.x] *= S.G(fp64::rR, threadIdx.x);
  for (int i = threadIdx.x; i < kTile * Q; i += kThreads) {
    const int c = i % kTile, q = i / kTile;
    const double al = ab[2 * q], be = ab[2 * q + 1];
    const double e0 = S.G(fp64::rE, c), e1 = S.G(fp64::rE + 1, c), h = S.G(fp64::rE + 2, c) - e0 - e1;
    len[i] = fma(al * al, e0, fma(al * be, h, be * be * e1));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * kWarps + warp) * kTile, i = i0 + lane;
  if (i0 >= npoints) return;  // no block barrier follows
  const bool valid = i < npoints;
  const int64_t at = 3 * static_cast<int64_t>(valid ? i : i0);
  const double x0 = points[at], x1 = points[at + 1], x2 = points[at + 2];
  double* col = reinterpret_cast<double*>(smem + columns) + static_cast<size_t>(warp) * cap * kTile * NP;
  int nds = 0, so = 0;
  if (NB > 1 && cap > 0) {
    so = __ldg(st.tile_dof_off + tile);
    nds = __ldg(st.tile_dof_off + tile + 1) - so;
    for (int s = lane; s < nds * kTile * NP; s += 32) col[s] = 0.0;
    __syncwarp();
  }
  // the cell's sums u, times sc, to the lane's entries
  auto put = [&](int js, double (&u)[NP][NB], double sc) {
    if (NB == 1) {
      if (valid) {
        const int64_t o = i + ld * dof[js];
        if (NP == 2)
          reinterpret_cast<double2*>(out)[o] = make_double2(u[0][0] * sc, u[NP - 1][0] * sc);
        else
          out[o] = u[0][0] * sc;
      }
    } else if (cap > 0) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        double* c = col + dof[js * NB + b] + lane;
#pragma unroll
        for (int part = 0; part < NP; ++part) c[part * kTile] = fma(u[part][b], sc, c[part * kTile]);
      }
    } else if (valid) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int64_t o = i + ld * dof[js * NB + b];
#pragma unroll
        for (int part = 0; part < NP; ++part) atomicAdd(out + NP * o + part, u[part][b] * sc);
      }
    }
  };
  unsigned close = 0u;  // the lane's cells left for the second loop
  for (int js = j0; js < j1; ++js) {
    const double dx = (x0 - S.G(fp64::rC, js)) - S.G(fp64::rL, js),
                 dy = (x1 - S.G(fp64::rC + 1, js)) - S.G(fp64::rL + 1, js),
                 dz = (x2 - S.G(fp64::rC + 2, js)) - S.G(fp64::rL + 2, js);
    const double r0 = fma(dz, dz, fma(dy, dy, dx * dx));
    auto dot = [&](int row) { return fma(dz, S.G(row + 2, js), fma(dy, S.G(row + 1, js), dx * S.G(row, js))); };
    const double W0 = -2.0 * dot(fp64::rG0), W1 = -2.0 * dot(fp64::rG1);
    double u[NP][NB];
#pragma unroll
    for (int part = 0; part < NP; ++part)
#pragma unroll
      for (int b = 0; b < NB; ++b) u[part][b] = 0.0;
    auto some = [&](int q, auto count) {
      constexpr int N = decltype(count)::value;
      double r2[N], K[2][N];
#pragma unroll
      for (int n = 0; n < N; ++n) r2[n] = r0 + len[(q + n) * kTile + js];
#pragma unroll
      for (int n = 0; n < N; ++n) r2[n] = fma(ab[2 * (q + n)], W0, r2[n]);
#pragma unroll
      for (int n = 0; n < N; ++n) r2[n] = fma(ab[2 * (q + n) + 1], W1, r2[n]);
      fp64::kernel_values<KER, OP, fp64::kAnyPhase, N>(r2, k, 0.0, K[0], K[1]);
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double w = wt[(q + n) * NB + b];
#pragma unroll
          for (int part = 0; part < NP; ++part) u[part][b] = fma(K[part][n], w, u[part][b]);
        }
    };
    int q = 0;
    for (; q + kGroup <= Q; q += kGroup) some(q, std::integral_constant<int, kGroup>{});
    for (; q + 2 <= Q; q += 2) some(q, std::integral_constant<int, 2>{});
    if (q < Q) some(q, std::integral_constant<int, 1>{});
    double sc = S.G(fp64::rJ, js) * kInv4Pi;
    if (OP == kDL) sc *= dot(fp64::rN);
    // high words: no operation of the FP64 pipe, no branch before the kernel values
    const bool near_cell = __double2hiint(r0) <= __double2hiint(S.G(fp64::rR, js));
    close |= near_cell ? 1u << js : 0u;
    if (!near_cell) put(js, u, sc);
  }
  if (!valid) close = 0u;
  for (; close; close &= close - 1) {
    const int js = __ffs(close) - 1;
    const double dx = (x0 - S.G(fp64::rC, js)) - S.G(fp64::rL, js),
                 dy = (x1 - S.G(fp64::rC + 1, js)) - S.G(fp64::rL + 1, js),
                 dz = (x2 - S.G(fp64::rC + 2, js)) - S.G(fp64::rL + 2, js);
    double u[NP][NB];
#pragma unroll
    for (int part = 0; part < NP; ++part)
#pragma unroll
      for (int b = 0; b < NB; ++b) u[part][b] = 0.0;
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const double al = ab[2 * q], be = ab[2 * q + 1];
      const double ex = dx - fma(al, S.G(fp64::rG0, js), be * S.G(fp64::rG1, js)),
                   ey = dy - fma(al, S.G(fp64::rG0 + 1, js), be * S.G(fp64::rG1 + 1, js)),
                   ez = dz - fma(al, S.G(fp64::rG0 + 2, js), be * S.G(fp64::rG1 + 2, js));
      const double r2 = fma(ez, ez, fma(ey, ey, ex * ex));
      double K[2];
      fp64::kernel_values<KER, OP, fp64::kAnyPhase, 1>(&r2, k, 0.0, K, K + 1);
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int part = 0; part < NP; ++part) u[part][b] = fma(K[part], wt[q * NB + b], u[part][b]);
    }
    double sc = S.G(fp64::rJ, js) * kInv4Pi;
    if (OP == kDL)
      sc *= fma(dz, S.G(fp64::rN + 2, js), fma(dy, S.G(fp64::rN + 1, js), dx * S.G(fp64::rN, js)));
    put(js, u, sc);
  }
  if (NB > 1 && cap > 0 && valid) {
    // columns of DOFs that the chunk's cells do not touch stay zero
#pragma unroll 4
    for (int s = 0; s < nds; ++s) {
      const int64_t o = i + ld * __ldg(st.tile_dofs + so + s);
#pragma unroll
      for (int part = 0; part < NP; ++part) {
        const double v = col[(s * NP + part) * kTile + lane];
        if (v != 0.0) atomicAdd(out + NP * o + part, v);
      }
    }
  }
}

template <int KER, int OP, int NB>
cudaError_t launch_nb(const double* points, int npoints, const CellSet& trial,
                      const SpaceTiles& st, const RegularRule& rule, double k, double* out,
                      int64_t ld, cudaStream_t stream) {
  constexpr int NP = KER == kHelmholtz ? 2 : 1;
  PotentialRule r{};
  r.npts = rule.npts;
  r.reach = fp64::rule_reach(rule);
  for (int q = 0; q < rule.npts; ++q) {
    r.ab[q][0] = rule.phi[0][q] - rule.phi[2][q];
    r.ab[q][1] = rule.phi[1][q] - rule.phi[2][q];
    for (int b = 0; b < NB; ++b)
      r.w[q][b] = NB == 1 ? rule.w[q] : NB == 3 ? rule.wphi[b][q] : rule.wphi2[b][q];
  }
  // DOF columns of up to 16 KB per warp; larger ones are left out
  int cap = 0;
  if (NB > 1 && sizeof(double) * st.max_tile_dofs * kTile * NP <= (size_t(16) << 10))
    cap = st.max_tile_dofs;
  size_t columns;
  const size_t smem = potential_smem<NB>(rule.npts, cap, NP, &columns);
  auto fn = potential_tiles<KER, OP, NB>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  const int gx = (npoints + kWarps * kTile - 1) / (kWarps * kTile);
  const int tiles = (trial.ncells + kTile - 1) / kTile;
  // whole tiles, or chunks of their cells until the chip has two waves of CTAs
  int ns = kTile;
  while (ns > 1 && static_cast<long long>(gx) * tiles * (kTile / ns) < 8 * fp64::kSMs) ns /= 2;
  const long long gy = static_cast<long long>(tiles) * (kTile / ns);
  if (gy > 65535) ns = kTile;
  const dim3 grid(gx, tiles * (kTile / ns));
  fn<<<grid, kThreads, smem, stream>>>(points, npoints, trial, st, r, k, out, ld, ns, cap);
  return cudaGetLastError();
}

template <int KER, int OP>
cudaError_t launch_op(const double* points, int npoints, const CellSet& trial,
                      const SpaceTiles& st, const RegularRule& rule, double k, double* out,
                      int64_t ld, cudaStream_t stream) {
  switch (st.nbasis) {
    case 1: return launch_nb<KER, OP, 1>(points, npoints, trial, st, rule, k, out, ld, stream);
    case 3: return launch_nb<KER, OP, 3>(points, npoints, trial, st, rule, k, out, ld, stream);
    case 6: return launch_nb<KER, OP, 6>(points, npoints, trial, st, rule, k, out, ld, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_potential(int kernel, int op, const double* points, int npoints,
                             const CellSet& trial, const SpaceTiles& st, const RegularRule& rule,
                             double k, double* out, int64_t ld, cudaStream_t stream) {
  if (npoints <= 0 || trial.ncells <= 0) return cudaSuccess;
  if (op != kSL && op != kDL) return cudaErrorInvalidValue;
  if (kernel == kLaplace)
    return op == kSL ? launch_op<kLaplace, kSL>(points, npoints, trial, st, rule, k, out, ld, stream)
                     : launch_op<kLaplace, kDL>(points, npoints, trial, st, rule, k, out, ld, stream);
  return op == kSL ? launch_op<kHelmholtz, kSL>(points, npoints, trial, st, rule, k, out, ld, stream)
                   : launch_op<kHelmholtz, kDL>(points, npoints, trial, st, rule, k, out, ld, stream);
}

}  // namespace bempp_b200
