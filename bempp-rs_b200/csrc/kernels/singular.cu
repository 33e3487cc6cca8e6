// Singular quadrature for cell pairs that share a vertex, an edge or the whole cell.
//
// Replaces bempp-rs assemble_batch_singular (src/boundary_assemblers.rs:608-685) with
// SingularCellPairAssembler (src/boundary_assemblers/cell_pair_assemblers.rs:109-152):
// entry[a][b] = sum_i f(x(xi_i), y(eta_i)) w_i jdet_x jdet_y over the Duffy rule of the
// pair's adjacency configuration.  The reference emits COO triplets per pair and adds them
// into the dense matrix serially (src/boundary_assemblers.rs:206-213); here they are
// stored (DP0 x DP0, where every pair owns its entry) or added with atomics, or stored per
// pair for the CSR singular path.
//
// Directions.  On flat cells every coordinate of a Duffy region is a multiple of xi, so
// x - y = rho d with rho = xi (common vertex), xi eta1 (common edge) or xi eta1 eta2 (one
// cell) and d depending on the other 3, 2 or 1 coordinates only.  The rule's 512 / 1280 /
// 1536 points (order 4) are the products of 128 / 80 / 24 directions d and 4 / 16 / 64
// values of rho:
//   * Laplace kernels are homogeneous, K(rho d) = rho^-1 K(d) or rho^-2 K(d): the sum over
//     rho of the weights and basis values is a number of the rule (SingularRules::weights)
//     and the kernel is evaluated once per direction;
//   * Helmholtz: rho, the weights of the inner coordinates and the products of the basis
//     functions are polynomials in xi and rho with few coefficients per direction, so the
//     sum over the radii at theta = k |d| is a combination of a few functions
//     P_q(theta) = sum_j v_j mu_q(j) rho_j^-1 e^{i theta rho_j}, mu one of 1, xi, xi^2 (common
//     vertex) or 1, xi, rho, xi^2, xi rho, rho^2 (edge): power series in theta whose
//     coefficients depend on the rule alone (SeriesRules, kernel constants).  Per
//     direction: N terms of 3 or 6 series and 9 or 15 updates, in place of a sine, a cosine
//     and a block update at each of 4 or 16 radii.  One cell (24 directions): the block's
//     series per direction, from a table;
//   * phases beyond the series' range (|theta| > 3.4) take |d| and 1/|d| once per direction
//     and the phase at every point.
// The sums are those of the rule, in another order; forming d without the cancelling
// common vertex is also more accurate than x - y from two maps.
//
// Mapping.  2^lanes threads per pair share its directions (a power of two that fills the
// chip: one thread per pair on large meshes, a warp on small ones), each with the pair's
// tangents in registers; pairs are grouped by configuration, so that a warp's threads read
// the same rule entries.  One warp per pair over all points spent its time on 42
// operations per point and on shuffling nine sums through five steps.
// 266,180 pairs (20,480 triangles), order 4, B200, one warp per pair over all points -> now:
// Laplace single layer DP0 0.55 -> 0.08 ms, double layer P1 0.93 -> 0.18, hypersingular P1
// 0.54 -> 0.09; Helmholtz k = 8 single layer DP0 0.90 -> 0.12, double layer P1 1.54 -> 0.48,
// hypersingular P1 1.50 -> 0.37.  (The block's series per direction from a table for every
// configuration was slower, 2.0 ms for the Helmholtz double layer: the broadcast loads of 90
// coefficients per term filled the L1 return path; hence constants for the vertex and edge
// pairs.)
#include <type_traits>

#include "launch.h"

namespace bempp_b200 {
namespace {

constexpr int kThreads = 128;

struct CellData {
  double t0[3], t1[3], n[3], jdet, diam;
};

__device__ __forceinline__ void load_cell(const CellSet& cs, int c, CellData& d) {
  const int n = cs.stride;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d.t0[k] = g(cs.geom, kT0x + k, n, c);
    d.t1[k] = g(cs.geom, kT1x + k, n, c);
    d.n[k] = g(cs.geom, kNx + k, n, c);
  }
  d.jdet = g(cs.geom, kJdet, n, c);
  d.diam = g(cs.geom, kDiam, n, c);
}

// Weights of one direction for NBT x NBS blocks, w[a][b] (or w[0][0]: their sum).
template <int NBT, int NBS>
__device__ __forceinline__ void direction_weights(const double* w, double out[NBT][NBS]) {
  if constexpr (NBT == 1 && NBS == 1) {
    out[0][0] = __ldg(w);
  } else {
    constexpr int kN = NBT * NBS;
    double v[kN + 1];
    const double2* p = reinterpret_cast<const double2*>(w);
#pragma unroll
    for (int i = 0; i < (kN + 1) / 2; ++i) {
      const double2 x = __ldg(p + i);
      v[2 * i] = x.x;
      v[2 * i + 1] = x.y;
    }
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) out[a][b] = v[a * NBS + b];
  }
}

// Series sums of one pair's share of the directions, N terms.  Common vertex and edge:
// blk[i][j] collects the products of {1, x1, x2} and {1, y1, y2} (see DirectionRule; only
// the constant on a piecewise constant side); one cell: the basis functions themselves.
template <int N, int OP, int NBT, int NBS, class Direction>
__device__ __forceinline__ void series_sums(int kind, int sub, int step, int ndir, int first,
                                            double k, const SingularRules& rules,
                                            const SeriesRules& series, const Direction& direction,
                                            double blk_re[NBT][NBS], double blk_im[NBT][NBS],
                                            double& S_re, double& S_im) {
  constexpr bool kGrad = OP == kDL || OP == kADL;
  constexpr bool kScalar = NBT == 1 && NBS == 1;
  // P_q: real and imaginary part at theta, z = theta^2, times the factors f and f theta
  auto value = [&](int q, double z, double fr, double fi, double& re, double& im) {
    re = series.c[q][2 * N - 2];
    im = series.c[q][2 * N - 1];
#pragma unroll
    for (int n = N - 2; n >= 0; --n) {
      re = fma(re, z, series.c[q][2 * n]);
      im = fma(im, z, series.c[q][2 * n + 1]);
    }
    re *= fr;
    im *= fi;
  };
  auto at = [&](int i, double& z, double& fr, double& fi) {
    double r2, dn;
    direction(i, r2, dn);
    const double rinv = rsqrt_refined(r2), theta = k * (r2 * rinv);
    z = theta * theta;
    fr = __ldg(rules.share + first + i) * (kGrad ? dn * rinv * rinv * rinv : rinv);
    fi = fr * theta;
  };
  auto add = [&](int i, int j, double c, double re, double im) {
    blk_re[i][j] = fma(c, re, blk_re[i][j]);
    blk_im[i][j] = fma(c, im, blk_im[i][j]);
  };
  if (kScalar || (kind == 2 && OP == kHS)) {
    const int q = kind == 0 ? 0 : kind == 1 ? 3 : 9;
    double c[2 * N];
#pragma unroll
    for (int n = 0; n < 2 * N; ++n) c[n] = series.c[q][n];
    for (int i = sub; i < ndir; i += step) {
      double z, fr, fi;
      at(i, z, fr, fi);
      double re = c[2 * N - 2], im = c[2 * N - 1];
#pragma unroll
      for (int n = N - 2; n >= 0; --n) {
        re = fma(re, z, c[2 * n]);
        im = fma(im, z, c[2 * n + 1]);
      }
      S_re = fma(fr, re, S_re);
      S_im = fma(fi, im, S_im);
    }
    if constexpr (kScalar) {
      blk_re[0][0] = S_re;
      blk_im[0][0] = S_im;
    }
  }
  if constexpr (!kScalar) {
    const double2* raw = reinterpret_cast<const double2*>(rules.raw) + 2 * first;
    if (kind == 0) {
      for (int i = sub; i < ndir; i += step) {
        double z, fr, fi, p0r, p0i, p1r, p1i, p2r, p2i;
        at(i, z, fr, fi);
        const double2 X = __ldg(raw + 2 * i), Y = __ldg(raw + 2 * i + 1);
        value(0, z, fr, fi, p0r, p0i);
        value(1, z, fr, fi, p1r, p1i);
        if (OP == kHS) {
          S_re += p0r;
          S_im += p0i;
        }
        add(0, 0, 1.0, p0r, p0i);
        if constexpr (NBS == 3) {
          add(0, 1, Y.x, p1r, p1i);
          add(0, 2, Y.y, p1r, p1i);
        }
        if constexpr (NBT == 3) {
          add(1, 0, X.x, p1r, p1i);
          add(2, 0, X.y, p1r, p1i);
        }
        if constexpr (NBT == 3 && NBS == 3) {
          value(2, z, fr, fi, p2r, p2i);
          add(1, 1, X.x * Y.x, p2r, p2i);
          add(1, 2, X.x * Y.y, p2r, p2i);
          add(2, 1, X.y * Y.x, p2r, p2i);
          add(2, 2, X.y * Y.y, p2r, p2i);
        }
      }
    } else if (kind == 1) {
      // x1 = xi - X1 rho, x2 = X2 rho, the same for y
      for (int i = sub; i < ndir; i += step) {
        double z, fr, fi, ar, ai, br, bi, cr, ci;
        at(i, z, fr, fi);
        const double2 X = __ldg(raw + 2 * i), Y = __ldg(raw + 2 * i + 1);
        value(3, z, fr, fi, ar, ai);  // 1
        value(4, z, fr, fi, br, bi);  // xi
        value(5, z, fr, fi, cr, ci);  // rho
        if (OP == kHS) {
          S_re += ar;
          S_im += ai;
        }
        add(0, 0, 1.0, ar, ai);
        if constexpr (NBS == 3) {
          add(0, 1, 1.0, br, bi);
          add(0, 1, -Y.x, cr, ci);
          add(0, 2, Y.y, cr, ci);
        }
        if constexpr (NBT == 3) {
          add(1, 0, 1.0, br, bi);
          add(1, 0, -X.x, cr, ci);
          add(2, 0, X.y, cr, ci);
        }
        if constexpr (NBT == 3 && NBS == 3) {
          value(6, z, fr, fi, ar, ai);  // xi^2
          value(7, z, fr, fi, br, bi);  // xi rho
          value(8, z, fr, fi, cr, ci);  // rho^2
          add(1, 1, 1.0, ar, ai);
          add(1, 1, -(X.x + Y.x), br, bi);
          add(1, 1, X.x * Y.x, cr, ci);
          add(1, 2, Y.y, br, bi);
          add(1, 2, -X.x * Y.y, cr, ci);
          add(2, 1, X.y, br, bi);
          add(2, 1, -X.y * Y.x, cr, ci);
          add(2, 2, X.y * Y.y, cr, ci);
        }
      }
    } else {
      // one cell: rows of the block's series per direction (even row, odd row; 9 of 10 values)
      const double2* table = reinterpret_cast<const double2*>(rules.cell_series[kGrad ? 1 : 0]);
      for (int i = sub; i < ndir; i += step) {
        double z, fr, fi, re[9], im[9];
        at(i, z, fr, fi);
        const double share = __ldg(rules.share + first + i);
        fr /= share;  // the table holds the whole weights
        fi /= share;
        const double2* row = table + static_cast<int64_t>(i) * (kSeriesTerms * 10);
#pragma unroll
        for (int e = 0; e < 9; ++e) re[e] = im[e] = 0.0;
#pragma unroll 1
        for (int n = N - 1; n >= 0; --n) {
          double v[20];
#pragma unroll
          for (int e = 0; e < 10; ++e) {
            const double2 w = __ldg(row + n * 10 + e);
            v[2 * e] = w.x;
            v[2 * e + 1] = w.y;
          }
#pragma unroll
          for (int e = 0; e < 9; ++e) {
            re[e] = fma(re[e], z, v[e]);
            im[e] = fma(im[e], z, v[10 + e]);
          }
        }
#pragma unroll
        for (int e = 0; e < 9; ++e)
          add(NBT == 3 ? e / 3 : 0, NBS == 3 ? e % 3 : 0, 1.0, fr * re[e], fi * im[e]);
      }
    }
  }
}

// Products of {1, x1, x2} and {1, y1, y2} -> of the basis functions 1 - x1, x1 - x2, x2 of
// the cells' vertices in the roles P0, P1, P2, moved to the local vertices that play them
// (roles: two bits each, test cell first).
template <int NBT, int NBS>
__device__ __forceinline__ void to_basis(double b[NBT][NBS], int roles) {
  if constexpr (NBT == 3) {
#pragma unroll
    for (int j = 0; j < NBS; ++j) {
      const double r[3] = {b[0][j] - b[1][j], b[1][j] - b[2][j], b[2][j]};
      const int p0 = roles & 3, p1 = (roles >> 2) & 3;
#pragma unroll
      for (int a = 0; a < 3; ++a) b[a][j] = p0 == a ? r[0] : p1 == a ? r[1] : r[2];
    }
  }
  if constexpr (NBS == 3) {
#pragma unroll
    for (int i = 0; i < NBT; ++i) {
      const double r[3] = {b[i][0] - b[i][1], b[i][1] - b[i][2], b[i][2]};
      const int p0 = (roles >> 6) & 3, p1 = (roles >> 8) & 3;
#pragma unroll
      for (int a = 0; a < 3; ++a) b[i][a] = p0 == a ? r[0] : p1 == a ? r[1] : r[2];
    }
  }
}

template <int KER, int OP, int NBT, int NBS>
__global__ void __launch_bounds__(kThreads)
    singular_fp64(CellSet test, const int* __restrict__ tdofs, CellSet trial,
                  const int* __restrict__ sdofs, SingularRules rules, SingularPairs pairs,
                  double k, double* __restrict__ out, int64_t ld, int unique_entries,
                  double* __restrict__ pair_values, int trial_lo, int trial_hi, int lanes,
                  const __grid_constant__ SeriesRules series) {
  constexpr bool kCplx = KER == kHelmholtz;
  constexpr bool kGrad = OP == kDL || OP == kADL;
  const int64_t thread = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const int64_t index = thread >> lanes;
  const int sub = static_cast<int>(thread) & ((1 << lanes) - 1);
  bool valid = index < pairs.npairs;
  const int pair = valid ? static_cast<int>(index) : 0;
  const int tc = __ldg(pairs.test_cell + pair), sc = __ldg(pairs.trial_cell + pair);
  valid = valid && sc >= trial_lo && sc < trial_hi;
  const int cfg = __ldg(pairs.config + pair);
  CellData x, y;
  load_cell(test, tc, x);
  load_cell(trial, sc, y);
  const int first = __ldg(rules.dir_offset + cfg);
  const int ndir = valid ? __ldg(rules.dir_offset + cfg + 1) - first : 0;

  double blk_re[NBT][NBS], blk_im[NBT][NBS];
  double S_re = 0.0, S_im = 0.0;
#pragma unroll
  for (int a = 0; a < NBT; ++a)
#pragma unroll
    for (int b = 0; b < NBS; ++b) blk_re[a][b] = blk_im[a][b] = 0.0;

  // every phase of the pair is at most k (diam_x + diam_y)
  const double bound = kCplx ? fabs(k) * (x.diam + y.diam) : 0.0;
  const bool in_series = bound <= 3.4;
  const double2* coef = reinterpret_cast<const double2*>(rules.coef) + 2 * first;
  // the direction's offset, its square, and (DL / ADL) its component along the normal
  auto direction = [&](int i, double& r2, double& dn) {
    const double2 cx = __ldg(coef + 2 * i), cy = __ldg(coef + 2 * i + 1);
    double d[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
      d[c] = fma(cx.x, x.t0[c], fma(cx.y, x.t1[c], fma(-cy.x, y.t0[c], -cy.y * y.t1[c])));
    r2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
    dn = OP == kDL   ? fma(d[2], y.n[2], fma(d[1], y.n[1], d[0] * y.n[0]))
         : OP == kADL ? -fma(d[2], x.n[2], fma(d[1], x.n[1], d[0] * x.n[0]))
                      : 0.0;
  };
  constexpr int kVariant = (NBT == 3 ? 2 : 0) + (NBS == 3 ? 1 : 0);
  if constexpr (KER == kLaplace) {
    constexpr bool kSum = OP == kHS || (NBT == 1 && NBS == 1);  // the weights' sum suffices
    constexpr int kStride = kSum ? 1 : NBT * NBS == 9 ? 10 : 4;
    const double* w = rules.weights[kGrad ? 1 : 0][kSum ? 0 : kVariant] +
                      static_cast<int64_t>(first) * kStride;
#pragma unroll 2
    for (int i = sub; i < ndir; i += 1 << lanes) {
      double r2, dn;
      direction(i, r2, dn);
      const double K = kGrad ? dn * rinv3_refined(r2) : rsqrt_refined(r2);
      if constexpr (kSum) {
        S_re = fma(K, __ldg(w + i), S_re);
      } else {
        double v[NBT][NBS];
        direction_weights<NBT, NBS>(w + static_cast<int64_t>(i) * kStride, v);
#pragma unroll
        for (int a = 0; a < NBT; ++a)
#pragma unroll
          for (int b = 0; b < NBS; ++b) blk_re[a][b] = fma(K, v[a][b], blk_re[a][b]);
      }
    }
    if constexpr (kSum && OP != kHS) blk_re[0][0] = S_re;
  } else {
    const int n = rules.order, n2 = n * n, n3 = n2 * n;
    const int kind = cfg < 9 ? 0 : cfg < 27 ? 1 : 2;   // common vertex, edge, one cell
    const int per = kind == 0 ? n3 : kind == 1 ? n2 : n;     // directions per region
    const int inner = kind == 0 ? n : kind == 1 ? n2 : n3;   // values of rho
    const double2* rho = reinterpret_cast<const double2*>(rules.rho) +
                         (kind == 0 ? 0 : kind == 1 ? n : n + n2);
    const int off = __ldg(rules.offset + cfg);
    const double2* txi = reinterpret_cast<const double2*>(rules.test_xi);
    const double2* sxi = reinterpret_cast<const double2*>(rules.trial_xi);
    const bool small_phase = bound <= 0.8;
    if (in_series) {
      auto by_series = [&](auto count) {
        series_sums<decltype(count)::value, OP, NBT, NBS>(kind, sub, 1 << lanes, ndir, first, k, rules,
                                                          series, direction, blk_re, blk_im, S_re, S_im);
      };
      // terms: the first left out is below 2e-17 at the bound
      if (bound <= 0.1745)
        by_series(std::integral_constant<int, 6>{});
      else if (bound <= 0.5171)
        by_series(std::integral_constant<int, 8>{});
      else if (bound <= 1.3702)
        by_series(std::integral_constant<int, 11>{});
      else
        by_series(std::integral_constant<int, kSeriesTerms>{});
    } else {
    auto points = [&](auto small) {
      for (int i = sub; i < ndir; i += 1 << lanes) {
        double r2, dn;
        direction(i, r2, dn);
        const double rinv = rsqrt_refined(r2), kr = k * (r2 * rinv);
        const double f0 = kGrad ? dn * rinv * rinv * rinv : rinv;
        double s_re = 0.0, s_im = 0.0;  // DP0 and the plain sum: scaled by f0 at the end
        int at = off + (i / per) * n2 * n2 + i % per;
        auto some = [&](int j, auto count) {
          constexpr int N = decltype(count)::value;
          double t[N], w0[N], sn[N], cs[N];
#pragma unroll
          for (int m = 0; m < N; ++m) {
            const double2 rh = __ldg(rho + j + m);  // rho, 1 / rho
            t[m] = kr * rh.x;
            w0[m] = __ldg(rules.w + at + m * per) * (kGrad ? rh.y * rh.y : rh.y);
          }
          if constexpr (decltype(small)::value)
            sincos_small_n<N>(t, sn, cs);
          else
            sincos_any_n<N>(t, sn, cs);
#pragma unroll
          for (int m = 0; m < N; ++m) {
            double re = cs[m], im = sn[m];
            if constexpr (kGrad) {
              re = fma(t[m], sn[m], cs[m]);
              im = fma(-t[m], cs[m], sn[m]);
            }
            if constexpr (OP == kHS || (NBT == 1 && NBS == 1)) {
              s_re = fma(w0[m], re, s_re);
              s_im = fma(w0[m], im, s_im);
            }
            if constexpr (NBT != 1 || NBS != 1) {
              const double f = w0[m] * f0;
              const double kre = f * re, kim = f * im;
              const double2 xi = __ldg(txi + at + m * per), et = __ldg(sxi + at + m * per);
              const double psi[3] = {1.0 - et.x - et.y, et.x, et.y};
              const double phi[3] = {1.0 - xi.x - xi.y, xi.x, xi.y};
#pragma unroll
              for (int a = 0; a < NBT; ++a) {
                const double vr = NBT == 1 ? kre : kre * phi[a], vi = NBT == 1 ? kim : kim * phi[a];
#pragma unroll
                for (int b = 0; b < NBS; ++b) {
                  blk_re[a][b] = NBS == 1 ? blk_re[a][b] + vr : fma(vr, psi[b], blk_re[a][b]);
                  blk_im[a][b] = NBS == 1 ? blk_im[a][b] + vi : fma(vi, psi[b], blk_im[a][b]);
                }
              }
            }
          }
          at += N * per;
        };
        int j = 0;
        for (; j + 4 <= inner; j += 4) some(j, std::integral_constant<int, 4>{});
        for (; j < inner; ++j) some(j, std::integral_constant<int, 1>{});
        S_re = fma(f0, s_re, S_re);
        S_im = fma(f0, s_im, S_im);
      }
    };
    if (small_phase)
      points(std::true_type{});
    else
      points(std::false_type{});
    if constexpr (NBT == 1 && NBS == 1) {
      blk_re[0][0] = S_re;
      blk_im[0][0] = S_im;
    }
    }
  }
  // sums over the pair's threads (every thread of the warp takes part)
  for (int s = (1 << lanes) >> 1; s > 0; s >>= 1) {
    if (OP == kHS) {
      S_re += __shfl_xor_sync(0xffffffffu, S_re, s);
      if (kCplx) S_im += __shfl_xor_sync(0xffffffffu, S_im, s);
    }
    if (OP != kHS || kCplx) {
#pragma unroll
      for (int a = 0; a < NBT; ++a)
#pragma unroll
        for (int b = 0; b < NBS; ++b) {
          blk_re[a][b] += __shfl_xor_sync(0xffffffffu, blk_re[a][b], s);
          if (kCplx) blk_im[a][b] += __shfl_xor_sync(0xffffffffu, blk_im[a][b], s);
        }
    }
  }
  if (sub != 0 || !valid) return;
  if constexpr (kCplx && (NBT == 3 || NBS == 3)) {
    // series sums of vertex and edge pairs: from products of {1, x1, x2} to basis functions
    if (cfg < 27 && in_series) {
      const int roles = __ldg(rules.roles + cfg);
      to_basis<NBT, NBS>(blk_re, roles);
      to_basis<NBT, NBS>(blk_im, roles);
    }
  }

  const double jj = x.jdet * y.jdet;
  double o_re[NBT][NBS], o_im[NBT][NBS];
  if (OP != kHS) {
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        o_re[a][b] = blk_re[a][b] * jj * kInv4Pi;
        o_im[a][b] = blk_im[a][b] * jj * kInv4Pi;
      }
  } else {
    double ct[NBT][3], cs[NBS][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (NBT == 3) {
        ct[0][d] = x.t0[d] - x.t1[d];
        ct[1][d] = x.t1[d];
        ct[2][d] = -x.t0[d];
      } else {
        ct[0][d] = 0.0;
      }
      if (NBS == 3) {
        cs[0][d] = y.t0[d] - y.t1[d];
        cs[1][d] = y.t1[d];
        cs[2][d] = -y.t0[d];
      } else {
        cs[0][d] = 0.0;
      }
    }
    const double nn = x.n[0] * y.n[0] + x.n[1] * y.n[1] + x.n[2] * y.n[2];
    const double nnsc = -k * k * nn * jj;
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        const double cc = ct[a][0] * cs[b][0] + ct[a][1] * cs[b][1] + ct[a][2] * cs[b][2];
        double re = S_re * cc, im = S_im * cc;
        if (kCplx) {
          re = fma(nnsc, blk_re[a][b], re);
          im = fma(nnsc, blk_im[a][b], im);
        }
        o_re[a][b] = re * kInv4Pi;
        o_im[a][b] = im * kInv4Pi;
      }
  }
  if (pair_values) {
    double* pv = pair_values + static_cast<int64_t>(pair) * NBT * NBS * (kCplx ? 2 : 1);
#pragma unroll
    for (int b = 0; b < NBS; ++b)
#pragma unroll
      for (int a = 0; a < NBT; ++a) {
        const int e = a + NBT * b;
        if (kCplx) {
          pv[2 * e] = o_re[a][b];
          pv[2 * e + 1] = o_im[a][b];
        } else {
          pv[e] = o_re[a][b];
        }
      }
  }
  if (out) {
#pragma unroll
    for (int b = 0; b < NBS; ++b) {
      const int64_t col = static_cast<int64_t>(__ldg(sdofs + sc * NBS + b)) * ld;
#pragma unroll
      for (int a = 0; a < NBT; ++a) {
        const int64_t o = col + __ldg(tdofs + tc * NBT + a);
        if (unique_entries) {  // DP0 x DP0: this pair owns the entry
          if (kCplx) {
            reinterpret_cast<double2*>(out)[o] = make_double2(o_re[a][b], o_im[a][b]);
          } else {
            out[o] = o_re[a][b];
          }
        } else {
          if (kCplx) {
            atomicAdd(out + 2 * o, o_re[a][b]);
            atomicAdd(out + 2 * o + 1, o_im[a][b]);
          } else {
            atomicAdd(out + o, o_re[a][b]);
          }
        }
      }
    }
  }
}

template <int KER, int OP, int NBT, int NBS>
cudaError_t launch_one(const CellSet& test, const int* tdofs, const CellSet& trial,
                       const int* sdofs, const SingularRules& rules, const SingularPairs& pairs,
                       const SingularArgs& a, cudaStream_t stream) {
  // threads per pair: four warps per scheduler of the chip, at most a warp per pair
  int lanes = 0;
  while (lanes < 5 && (static_cast<int64_t>(pairs.npairs) << lanes) < 148 * 4 * 4 * 32) ++lanes;
  const int64_t blocks = ((static_cast<int64_t>(pairs.npairs) << lanes) + kThreads - 1) / kThreads;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  singular_fp64<KER, OP, NBT, NBS><<<static_cast<unsigned>(blocks), kThreads, 0, stream>>>(
      test, tdofs, trial, sdofs, rules, pairs, a.k, static_cast<double*>(a.out), a.ld,
      a.unique_entries, a.pair_values, a.trial_lo, a.trial_hi, lanes,
      rules.host_series ? rules.host_series[OP == kDL || OP == kADL ? 1 : 0] : SeriesRules{});
  return cudaGetLastError();
}

template <int KER, int OP>
cudaError_t launch_nb(const CellSet& test, const int* tdofs, int nbt, const CellSet& trial,
                      const int* sdofs, int nbs, const SingularRules& rules,
                      const SingularPairs& pairs, const SingularArgs& a, cudaStream_t stream) {
  if (nbt == 1 && nbs == 1)
    return launch_one<KER, OP, 1, 1>(test, tdofs, trial, sdofs, rules, pairs, a, stream);
  if (nbt == 1 && nbs == 3)
    return launch_one<KER, OP, 1, 3>(test, tdofs, trial, sdofs, rules, pairs, a, stream);
  if (nbt == 3 && nbs == 1)
    return launch_one<KER, OP, 3, 1>(test, tdofs, trial, sdofs, rules, pairs, a, stream);
  if (nbt == 3 && nbs == 3)
    return launch_one<KER, OP, 3, 3>(test, tdofs, trial, sdofs, rules, pairs, a, stream);
  return cudaErrorInvalidValue;
}

template <int KER>
cudaError_t launch_op(const CellSet& test, const int* tdofs, int nbt, const CellSet& trial,
                      const int* sdofs, int nbs, const SingularRules& rules,
                      const SingularPairs& pairs, const SingularArgs& a, cudaStream_t stream) {
  switch (a.op) {
    case kSL: return launch_nb<KER, kSL>(test, tdofs, nbt, trial, sdofs, nbs, rules, pairs, a, stream);
    case kDL: return launch_nb<KER, kDL>(test, tdofs, nbt, trial, sdofs, nbs, rules, pairs, a, stream);
    case kADL: return launch_nb<KER, kADL>(test, tdofs, nbt, trial, sdofs, nbs, rules, pairs, a, stream);
    case kHS: return launch_nb<KER, kHS>(test, tdofs, nbt, trial, sdofs, nbs, rules, pairs, a, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_singular(const CellSet& test, const int* test_dofs, int nbt,
                            const CellSet& trial, const int* trial_dofs, int nbs,
                            const SingularRules& rules, const SingularPairs& pairs,
                            const SingularArgs& a, cudaStream_t stream) {
  if (pairs.npairs <= 0) return cudaSuccess;
  if (nbt > 3 || nbs > 3) {  // degree-2 spaces: the generic warp-per-pair kernel
    GenericPairArgs g;
    g.kernel = a.kernel;
    g.op = a.op;
    g.k = a.k;
    g.nbt = nbt;
    g.nbs = nbs;
    g.test = test;
    g.trial = trial;
    g.test_dofs = test_dofs;
    g.trial_dofs = trial_dofs;
    g.rule = RegularRule{};
    g.rules = rules;
    g.pairs = pairs;
    g.singular = true;
    g.same_grid = 1;
    g.out = a.out;
    g.ld = a.ld;
    g.trial_lo = a.trial_lo;
    g.trial_hi = a.trial_hi;
    g.pair_values = a.pair_values;
    return launch_generic_pairs(g, stream);
  }
  return a.kernel == kLaplace
             ? launch_op<kLaplace>(test, test_dofs, nbt, trial, trial_dofs, nbs, rules, pairs, a, stream)
             : launch_op<kHelmholtz>(test, test_dofs, nbt, trial, trial_dofs, nbs, rules, pairs, a, stream);
}

}  // namespace bempp_b200
