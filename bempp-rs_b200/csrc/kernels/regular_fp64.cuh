// Regular (non-singular) quadrature of all operators on DP0 / P1 / DP1 spaces, FP64.
//
// The sums of regular.cu's file comment (src/boundary_assemblers.rs:396-521,689-773 and
// src/boundary_assemblers/cell_pair_assemblers.rs:283-339 of bempp-rs), in a form that
// needs few FP64 operations per point pair: the FP64 pipe (64 lanes per SM and cycle)
// bounds every kernel of this file, and every instruction of it counts.
//
// Distances.  With c the centroid, g_a = V_a - c (g_0 + g_1 + g_2 = 0) and dc = c_x - c_y,
// a rule point is c + sum_a lambda_a g_a, so |x_p - y_q|^2 is a bilinear form in the rule's
// constants whose coefficients are formed once per cell pair:
//   * a rule made of two S21 orbits (the 6-point rule: three points c + gamma g_a per
//     orbit): |x - y|^2 = (|dc|^2 + gamma^2 |g_a|^2 + 2 gamma dc.g_a)
//     + (gamma'^2 |g'_b|^2 - 2 gamma' dc.g'_b) - 2 gamma gamma' g_a.g'_b, two operations
//     per point pair (an addition and an FMA) from 21 numbers kept in registers, where
//     differences of coordinates cost six and three shared-memory loads (pair_orbits);
//   * any other rule: A_p + |y_q - c_y|^2 + alpha_q W0_p + beta_q W1_p, (alpha, beta) the
//     coordinates of the point along g_0, g_1: three operations, the rule's constants
//     loaded once for four test points (point_block).
// The centroids' rounding, which would shift every point of a cell alike, is kept beside
// the offsets and enters dc.  The terms are as large as H^2, H = |dc| and both cells' extents
// together, so the sum is off by eps H^2 and 1/r by eps (H/r)^2, where differences of
// coordinates lose eps |x| / r.  Pairs whose rule points may be closer than H / 16 (nearly in
// contact without a shared vertex; see close_pair) are therefore integrated from the
// components of x - y (pair_by_components).
// P1 basis functions on an S21 orbit take two values, so U_b = sum_q w_q phi_b(q) K_q is
// c S + d K_b with S the orbit's sum: 12 operations per 6 points instead of 18.
//
// Mapping.  A CTA has four warps; each warp owns a tile of 32 test cells (lane = cell) and
// walks a chunk of up to 16 cells of one trial tile (the same for the four warps, staged
// with the test tiles by TMA bulk copies).  DP0 x DP0 blocks are stored; other blocks are
// summed per test DOF (the tile's DOF incidence, lane = DOF) into the warp's own
// accumulator of the DOF block, which is added to the output once, so that no two warps
// share an accumulator and the loop has no block-wide barrier.  A chunk's trial DOFs are
// renumbered on the device, so that 16 cells need about 15 columns.  Accumulators too
// large for shared memory (discontinuous P1: 96 test DOFs per tile) are left out: each
// lane then adds its entries to the output directly.
// Small meshes take shorter chunks (down to one trial cell), and the general rule's kernel
// can split the test points over the four warps (SPLIT).
//
// Regular part on a B200, coordinate differences in 32 x 32 tiles per CTA -> this form:
//   20,480 triangles, 6-point rule: Laplace single layer DP0 6.55 -> 5.05 ms, double layer P1
//   (both orders of a pair at once) 17.7 -> 13.3, hypersingular P1 9.5 -> 7.3; Helmholtz
//   k = 8 single layer DP0 15.8 -> 12.5, double layer P1 39.8 -> 35.9, hypersingular P1
//   28.0 -> 21.4; 5,120 triangles, k = 8 (phases beyond 0.8): single layer 1.61 -> 1.18;
//   2,048 triangles, 37-point rule: double layer P1 10.7 -> 4.0 (both orders at once);
//   80 triangles, 37-point rule: single layer DP0 0.374 -> 0.021.
// In FP64 issue slots the double layer needs about 19 per point pair for both orders (26
// before), the hypersingular operator 11 (15), the Helmholtz single layer 27 to 29 (33).
#pragma once

#include <algorithm>

#include "launch.h"
#include "tiles.cuh"

namespace bempp_b200 {
namespace fp64 {

using namespace tiles;

constexpr int kChunk = 16;   // most trial cells per CTA
constexpr int kBand = 16;    // trial tiles per band of a tx >= sy launch (see tile_order.h)

// Phases of Helmholtz kernels: referenced to the pair, |k (r - r0)| <= 0.8 for every pair
// of the launch (checked on the host), or any phase k r reduced by multiples of pi/2; kShort:
// referenced and at most 0.42, two terms less (20,480 triangles, k = 8, 0.41 at most, B200:
// whole single layer DP0 13.5 -> 12.7 ms).
enum Phase : int { kReferenced = 0, kAnyPhase = 1, kShort = 2 };

// Rows of a staged tile (every row of the grid's geometry) after geometry_to_offsets: vertex
// 0 becomes what the rounded centroid lacks, the tangents become g_0, g_1 and the last
// three rows |g_0|^2, |g_1|^2, |g_2|^2.  One more row: the cell's part of the distance of the
// centroids within which close_pair looks at a pair.
enum Row : int { rL = kV0x, rG0 = kT0x, rG1 = kT1x, rN = kNx, rJ = kJdet, rC = kCx, rE = kDiam,
                 rR = kNumGeomFields };
static_assert(kV0x == 0 && kRad == kDiam + 1 && kH == kDiam + 2, "three rows for the squared lengths");
constexpr int kRows = kNumGeomFields + 1;

// reach: every rule point of a cell lies in the triangle c + reach (g_0, g_1, g_2).
struct OrbitRule {
  double reach;
  double g[2], g2[2];  // gamma, gamma^2
  double w[2];         // weight of each point
  double c[2], d[2];   // w (1 - gamma) / 3, w gamma: w phi_b(q) = c + d [b = q]
  double m[2][2];      // -2 gamma gamma'
};

// Rule constants of the general kernel, per point: alpha = l0 - l2, beta = l1 - l2, w,
// w phi_0, w phi_1, w phi_2 (l the barycentric coordinates).
constexpr int kPointFields = 6;
struct PointRule {
  int npts;
  double reach;
  double p[kMaxRegularPoints][kPointFields];
};

struct Shape {
  int ns;         // trial cells per chunk (a power of two, at most kChunk)
  int ntt;        // test tiles
  int nsup;       // groups of test tiles (four, or one with SPLIT)
  int ty0, ty1;   // trial tiles of this launch
  int gather;     // the accumulators fit: sum in shared memory, else add directly
  int cap;        // doubles per accumulator
};

// Blocks of a tx >= sy launch: bands of kBand trial tiles, within a band the groups of
// test tiles from the band's first row on, the band's rows fastest (groups partly above
// the diagonal leave those warps idle).
__host__ __device__ inline long long band_prefix(long long k, int n0, int step) {
  return kBand * (n0 * k - step * (k * (k - 1) / 2));
}
__host__ __device__ inline long long lower_group_count(int nsup, int per, int ty0, int ty1) {
  const int n0 = nsup - ty0 / per, step = kBand / per;
  const int nb = (ty1 - ty0 + kBand - 1) / kBand;
  if (nb <= 0) return 0;
  return band_prefix(nb - 1, n0, step) +
         static_cast<long long>(ty1 - ty0 - (nb - 1) * kBand) * (n0 - step * (nb - 1));
}
__host__ __device__ inline void lower_group(long long b, int nsup, int per, int ty0, int ty1,
                                            int& group, int& sy) {
  const int n0 = nsup - ty0 / per, step = kBand / per;
  int lo = 0, hi = (ty1 - ty0 + kBand - 1) / kBand - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (band_prefix(mid, n0, step) <= b)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int r0 = ty0 + lo * kBand, h = min(kBand, ty1 - r0);
  const int l = static_cast<int>(b - band_prefix(lo, n0, step));
  group = ty0 / per + lo * step + l / h;
  sy = r0 + l % h;
}

// Kernel values of N points from r^2: 1/r, 1/r^3 or, Helmholtz, e^{i(kr - kr0)} / r and
// e^{i(kr - kr0)} (1 - ikr) / r^3 (kr0 = 0 unless the phase is referenced).  Each step runs
// over the N points before the next, so that their dependence chains interleave: with three
// or four warps per scheduler the FP64 latency is hidden by nothing else.
template <int KER, int OP, int PH, int N>
__device__ __forceinline__ void kernel_values(const double r2[N], double k, double kr0,
                                              double re[N], double im[N]) {
  constexpr bool kGrad = OP == kDL || OP == kADL;
  double y[N], e[N];
#pragma unroll
  for (int i = 0; i < N; ++i) asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[i]) : "d"(r2[i]));
  if constexpr (KER == kLaplace && kGrad) {
    // rinv3_refined
    double y2[N], t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) y2[i] = y[i] * y[i];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = fma(-r2[i], y2[i], 1.0);
#pragma unroll
    for (int i = 0; i < N; ++i) y2[i] *= y[i];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = fma(e[i], 1.875, 1.5);
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = fma(e[i], t[i], 1.0);
#pragma unroll
    for (int i = 0; i < N; ++i) re[i] = y2[i] * t[i];
    return;
  }
  // rsqrt_refined
  double rinv[N];
  {
    double t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = r2[i] * y[i];
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = fma(-t[i], y[i], 1.0);
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = fma(e[i], 0.375, 0.5);
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = fma(e[i], t[i], 1.0);
#pragma unroll
    for (int i = 0; i < N; ++i) rinv[i] = y[i] * t[i];
  }
  if constexpr (KER == kLaplace) {
#pragma unroll
    for (int i = 0; i < N; ++i) re[i] = rinv[i];
    return;
  }
  double kr[N], sn[N], cs[N];
#pragma unroll
  for (int i = 0; i < N; ++i) kr[i] = r2[i] * rinv[i];  // r, times k below
  if constexpr (PH != kAnyPhase) {
    double t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (kGrad) kr[i] *= k;
      t[i] = kGrad ? kr[i] - kr0 : fma(k, kr[i], -kr0);
    }
    sincos_small_n<N, PH == kShort>(t, sn, cs);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) kr[i] *= k;
    sincos_any_n<N>(kr, sn, cs);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if constexpr (kGrad) {
      const double f = rinv[i] * rinv[i] * rinv[i];
      re[i] = f * fma(kr[i], sn[i], cs[i]);
      im[i] = f * fma(-kr[i], cs[i], sn[i]);
    } else {
      re[i] = rinv[i] * cs[i];
      im[i] = rinv[i] * sn[i];
    }
  }
}

// What a cell pair's quadrature leaves: the block, PAIRED the block of the reverse order
// (indexed [test-tile basis][trial-tile basis] too), and for the hypersingular operator
// the plain sum s.
template <int NP, int NBT, int NBS, bool PAIRED>
struct Blocks {
  double f[NP][NBT][NBS];
  double t[PAIRED ? NP : 1][PAIRED ? NBT : 1][PAIRED ? NBS : 1];
  double s[NP];
};

template <int NP, int NBT, int NBS, bool PAIRED>
__device__ __forceinline__ void clear(Blocks<NP, NBT, NBS, PAIRED>& blk) {
#pragma unroll
  for (int part = 0; part < NP; ++part) {
    blk.s[part] = 0.0;
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        blk.f[part][a][b] = 0.0;
        if constexpr (PAIRED) blk.t[part][a][b] = 0.0;
      }
  }
}

template <int KER, int OP, int NBT, int NBS, bool PAIRED>
struct Traits {
  static constexpr int kParts = KER == kHelmholtz ? 2 : 1;
  static constexpr bool kHSSum = OP == kHS;                        // s is needed
  static constexpr bool kBlock = OP != kHS || KER == kHelmholtz;   // f is needed
  static constexpr bool kTestFactor = OP == kDL || PAIRED;         // (x_p - y).n_y
  static constexpr bool kTrialFactor = OP == kADL || PAIRED;       // (y_q - x).n_x
  // the normal factors carry jdet_x jdet_y / (4 pi) where no phase is left to multiply with
  template <int PH>
  static constexpr bool kScaledFactors = (kTestFactor || kTrialFactor) && (KER == kLaplace || PH == kAnyPhase);
  // test points of a point_block: enough chains to fill the pipe within the registers
  static constexpr int kPoints =
      KER == kHelmholtz && (PAIRED || (NBS == 3 && OP != kSL)) ? 2 : 4;
  // trial points per turn of its loop: two where the registers hold both (37-point rule, 2,048
  // triangles, one -> two: Laplace single layer DP0 2.35 -> 2.23 ms, double layer P1 4.26 -> 4.03,
  // hypersingular 2.40 -> 2.24; Helmholtz single layer DP0 8.98 -> 8.43), one where they spill or
  // cost a CTA (16-point rule, two bodies of 1,500 and 1,200: double layer P1 0.60 -> 0.67;
  // Helmholtz single layer P1 1.77 -> 2.26, hypersingular 2.22 -> 2.36)
  static constexpr int kTrialUnroll =
      KER == kLaplace ? (OP == kDL && !PAIRED && NBT * NBS == 9 ? 1 : 2) : (NBT * NBS == 1 ? 2 : 1);
};

// Scalars of one cell pair (test cell = the lane's, trial cell js).
struct PairGeometry {
  double r0;                     // |dc|^2
  double dgx0, dgx1, dgy0, dgy1; // dc.g_0, dc.g_1 of the test cell, of the trial cell
  double m00, m01, m10, m11;     // g_a.g'_b
  double fx, fx0, fx1;           // (x - y).n_y = fx + l.g terms (kTestFactor)
  double fy, fy0, fy1;           // (y - x).n_x
};

template <int KER, int OP, int NBT, int NBS, bool PAIRED>
__device__ __forceinline__ void pair_geometry(const Tile& T, int it, const Tile& S, int js,
                                              double scale, PairGeometry& p) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  const double dx = (T.G(rC, it) - S.G(rC, js)) + (T.G(rL, it) - S.G(rL, js)),
               dy = (T.G(rC + 1, it) - S.G(rC + 1, js)) + (T.G(rL + 1, it) - S.G(rL + 1, js)),
               dz = (T.G(rC + 2, it) - S.G(rC + 2, js)) + (T.G(rL + 2, it) - S.G(rL + 2, js));
  p.r0 = fma(dz, dz, fma(dy, dy, dx * dx));
  auto dot = [](double ax, double ay, double az, double bx, double by, double bz) {
    return fma(az, bz, fma(ay, by, ax * bx));
  };
  const double ax = T.G(rG0, it), ay = T.G(rG0 + 1, it), az = T.G(rG0 + 2, it);
  const double bx = T.G(rG1, it), by = T.G(rG1 + 1, it), bz = T.G(rG1 + 2, it);
  const double ux = S.G(rG0, js), uy = S.G(rG0 + 1, js), uz = S.G(rG0 + 2, js);
  const double vx = S.G(rG1, js), vy = S.G(rG1 + 1, js), vz = S.G(rG1 + 2, js);
  p.dgx0 = dot(dx, dy, dz, ax, ay, az);
  p.dgx1 = dot(dx, dy, dz, bx, by, bz);
  p.dgy0 = dot(dx, dy, dz, ux, uy, uz);
  p.dgy1 = dot(dx, dy, dz, vx, vy, vz);
  p.m00 = dot(ax, ay, az, ux, uy, uz);
  p.m01 = dot(ax, ay, az, vx, vy, vz);
  p.m10 = dot(bx, by, bz, ux, uy, uz);
  p.m11 = dot(bx, by, bz, vx, vy, vz);
  if constexpr (Tr::kTestFactor) {
    const double nx = scale * S.G(rN, js), ny = scale * S.G(rN + 1, js), nz = scale * S.G(rN + 2, js);
    p.fx = dot(dx, dy, dz, nx, ny, nz);
    p.fx0 = dot(ax, ay, az, nx, ny, nz);
    p.fx1 = dot(bx, by, bz, nx, ny, nz);
  }
  if constexpr (Tr::kTrialFactor) {
    const double nx = scale * T.G(rN, it), ny = scale * T.G(rN + 1, it), nz = scale * T.G(rN + 2, it);
    p.fy = -dot(dx, dy, dz, nx, ny, nz);
    p.fy0 = dot(ux, uy, uz, nx, ny, nz);
    p.fy1 = dot(vx, vy, vz, nx, ny, nz);
  }
}

// Whether rule points of a pair may be closer than kSeparation times `limit`, the sum of the
// cells' rR rows.  Not where |dc| reaches the limit; nearer pairs are looked at along dc, where
// the points of a cell lie within reach times its vertices.  An ordinary mesh has no such
// pair with the 6-point rule; with 37 points and anisotropic cells about one cell in ten has one.
constexpr double kSeparation = 0.125;
__device__ __forceinline__ bool separated(double r0, double along, double limit) {
  return along > 0.0 && along * along > kSeparation * kSeparation * limit * limit * r0;
}
__device__ __forceinline__ bool close_pair(const PairGeometry& p, double limit, double reach) {
  if (p.r0 >= limit * limit) return false;
  const double x = fmin(fmin(p.dgx0, p.dgx1), -(p.dgx0 + p.dgx1)),
               y = fmax(fmax(p.dgy0, p.dgy1), -(p.dgy0 + p.dgy1));
  return !separated(p.r0, fma(reach, x - y, p.r0), limit);
}

// Box of a cell's centroid and rR: the high words of its bounds, as integers of the same order
// (two that compare equal may still meet).
struct Box {
  int lo[3], hi[3];
};
__device__ __forceinline__ Box cell_box(const Tile& t, int c) {
  auto key = [](double x) {
    const int b = __double2hiint(x);
    return b ^ ((b >> 31) & 0x7fffffff);
  };
  const double r = t.G(rR, c);
  Box b;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = t.G(rC + d, c);
    b.lo[d] = key(x - r);
    b.hi[d] = key(x + r);
  }
  return b;
}
// Box of a warp's tile of n cells.
__device__ __forceinline__ Box tile_box(const Tile& t, int it, int n) {
  Box b = cell_box(t, it);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    b.lo[d] = __reduce_min_sync(0xffffffffu, it < n ? b.lo[d] : 0x7fffffff);
    b.hi[d] = __reduce_max_sync(0xffffffffu, it < n ? b.hi[d] : static_cast<int>(0x80000000));
  }
  return b;
}
// Trial cells (bit j) of [j0, j1) whose box meets that of the test tile: those that close_pair
// has to look at.  Far tiles have none.
__device__ __forceinline__ unsigned cells_in_reach(const Box& test, const Tile& S, int it, int j0,
                                                   int j1) {
  const Box b = cell_box(S, it);
  bool meets = it >= j0 && it < j1;
#pragma unroll
  for (int d = 0; d < 3; ++d) meets = meets && b.lo[d] <= test.hi[d] && b.hi[d] >= test.lo[d];
  return __ballot_sync(0xffffffffu, meets);
}

// The 6-point rule: two orbits of three points on each cell.  The loop over the test
// cell's orbits stays rolled (18 point pairs of straight code), everything else is in
// registers.
template <int KER, int OP, int NBT, int NBS, bool PAIRED, int PH>
__device__ __forceinline__ void pair_orbits(const PairGeometry& p, const Tile& T, int it,
                                            const Tile& S, int js, const OrbitRule& rule,
                                            double k, double kr0,
                                            Blocks<Traits<KER, OP, NBT, NBS, PAIRED>::kParts,
                                                   NBT, NBS, PAIRED>& out) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
  // M[a][b] = g_a.g'_b, rows and columns summing to zero
  double M[3][3];
  M[0][0] = p.m00;
  M[0][1] = p.m01;
  M[1][0] = p.m10;
  M[1][1] = p.m11;
  M[0][2] = -(p.m00 + p.m01);
  M[1][2] = -(p.m10 + p.m11);
  M[2][0] = -(p.m00 + p.m10);
  M[2][1] = -(p.m01 + p.m11);
  M[2][2] = -(M[2][0] + M[2][1]);
  const double dgx[3] = {p.dgx0, p.dgx1, -(p.dgx0 + p.dgx1)};
  double Y[2][3], by[2][3];  // trial terms of |x - y|^2, trial normal factors
  {
    const double dgy[3] = {p.dgy0, p.dgy1, -(p.dgy0 + p.dgy1)};
    const double fb[3] = {p.fy0, p.fy1, -(p.fy0 + p.fy1)};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double e = S.G(rE + b, js);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        Y[o][b] = fma(rule.g2[o], e, -2.0 * rule.g[o] * dgy[b]);
        if constexpr (Tr::kTrialFactor) by[o][b] = fma(rule.g[o], fb[b], p.fy);
      }
    }
  }
  clear(out);
  // c-terms of the test basis (w phi_a = c + d [a = point]), added to every row at the end
  double cf[NP][NBS], ct[PAIRED ? NP : 1][NBS];
#pragma unroll
  for (int part = 0; part < NP; ++part)
#pragma unroll
    for (int b = 0; b < NBS; ++b) {
      cf[part][b] = 0.0;
      if constexpr (PAIRED) ct[part][b] = 0.0;
    }
  const double ex[3] = {T.G(rE, it), T.G(rE + 1, it), T.G(rE + 2, it)};
#pragma unroll(PH == kAnyPhase && !PAIRED ? 1 : 2)
  for (int op = 0; op < 2; ++op) {
    const double gp = rule.g[op], g2 = rule.g2[op];
    const double m0 = rule.m[op][0], m1 = rule.m[op][1];
    double sumF[NP][NBS], sumT[PAIRED ? NP : 1][NBS], tot[NP][2];
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      tot[part][0] = tot[part][1] = 0.0;
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        sumF[part][b] = 0.0;
        if constexpr (PAIRED) sumT[part][b] = 0.0;
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double X = fma(g2, ex[a], fma(2.0 * gp, dgx[a], p.r0));
      double U[NP][NBS], V[PAIRED ? NP : 1][NBS];
      double r2[6], K6[2][6];
#pragma unroll
      for (int i = 0; i < 6; ++i) r2[i] = X + Y[i / 3][i % 3];
#pragma unroll
      for (int i = 0; i < 6; ++i) r2[i] = fma(i < 3 ? m0 : m1, M[a][i % 3], r2[i]);
      kernel_values<KER, OP, PH, 6>(r2, k, kr0, K6[0], K6[1]);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        double K[NP][3];
#pragma unroll
        for (int part = 0; part < NP; ++part)
#pragma unroll
          for (int b = 0; b < 3; ++b) K[part][b] = K6[part][3 * o + b];
#pragma unroll
        for (int part = 0; part < NP; ++part) {
          const double sum = (K[part][0] + K[part][1]) + K[part][2];
          if constexpr (Tr::kHSSum) tot[part][o] += sum;
          if constexpr (Tr::kBlock) {
            if constexpr (OP == kADL) {
              // the trial factor inside the sum
              double q[3];
#pragma unroll
              for (int b = 0; b < 3; ++b) q[b] = K[part][b] * by[o][b];
              const double qs = (q[0] + q[1]) + q[2];
              if constexpr (NBS == 1) {
                U[part][0] = o == 0 ? rule.w[0] * qs : fma(rule.w[1], qs, U[part][0]);
              } else {
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                  const double prev = o == 0 ? rule.c[0] * qs : fma(rule.c[1], qs, U[part][b]);
                  U[part][b] = fma(rule.d[o], q[b], prev);
                }
              }
            } else if constexpr (NBS == 1) {
              U[part][0] = o == 0 ? rule.w[0] * sum : fma(rule.w[1], sum, U[part][0]);
            } else {
              // U_b = sum_o (c_o sum + d_o K_b)
#pragma unroll
              for (int b = 0; b < 3; ++b) {
                const double prev = o == 0 ? rule.c[0] * sum : fma(rule.c[1], sum, U[part][b]);
                U[part][b] = fma(rule.d[o], K[part][b], prev);
              }
            }
            if constexpr (PAIRED) {
              double q[3];
#pragma unroll
              for (int b = 0; b < 3; ++b) q[b] = K[part][b] * by[o][b];
              const double qs = (q[0] + q[1]) + q[2];
#pragma unroll
              for (int b = 0; b < 3; ++b) {
                const double prev = o == 0 ? rule.c[0] * qs : fma(rule.c[1], qs, V[part][b]);
                V[part][b] = fma(rule.d[o], q[b], prev);
              }
            }
          }
        }
      }
      if constexpr (Tr::kBlock) {
        if constexpr (Tr::kTestFactor) {
          const double fa = a == 0 ? p.fx0 : a == 1 ? p.fx1 : -(p.fx0 + p.fx1);
          const double ap = fma(gp, fa, p.fx);
#pragma unroll
          for (int part = 0; part < NP; ++part)
#pragma unroll
            for (int b = 0; b < NBS; ++b) U[part][b] *= ap;
        }
#pragma unroll
        for (int part = 0; part < NP; ++part)
#pragma unroll
          for (int b = 0; b < NBS; ++b) {
            sumF[part][b] += U[part][b];
            if constexpr (NBT == 3) out.f[part][a][b] = fma(rule.d[op], U[part][b], out.f[part][a][b]);
            if constexpr (PAIRED) {
              sumT[part][b] += V[part][b];
              out.t[part][a][b] = fma(rule.d[op], V[part][b], out.t[part][a][b]);
            }
          }
      }
    }
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      if constexpr (Tr::kHSSum)
        out.s[part] = fma(rule.w[op], fma(rule.w[1], tot[part][1], rule.w[0] * tot[part][0]),
                          out.s[part]);
      if constexpr (Tr::kBlock) {
#pragma unroll
        for (int b = 0; b < NBS; ++b) {
          cf[part][b] = fma(NBT == 3 ? rule.c[op] : rule.w[op], sumF[part][b], cf[part][b]);
          if constexpr (PAIRED) ct[part][b] = fma(rule.c[op], sumT[part][b], ct[part][b]);
        }
      }
    }
  }
  if constexpr (Tr::kBlock) {
#pragma unroll
    for (int part = 0; part < NP; ++part)
#pragma unroll
      for (int a = 0; a < NBT; ++a)
#pragma unroll
        for (int b = 0; b < NBS; ++b) {
          out.f[part][a][b] += cf[part][b];
          if constexpr (PAIRED) out.t[part][a][b] += ct[part][b];
        }
  }
}

// PB test points (from p0 on) of the general rule against every trial point; rt: the rule
// table in shared memory (kRuleStride doubles per point), Yq: |y_q - c_y|^2 of the trial
// cell.  p: with dgx doubled, dgy and m times -2.
constexpr int kRuleStride = 8;
template <int KER, int OP, int NBT, int NBS, bool PAIRED, int PH, int PB>
__device__ __forceinline__ void point_block(const PairGeometry& p, double ex0, double hx,
                                            double ex1, const double* rt, const double* Yq, int Q,
                                            int p0, double k, double kr0,
                                            Blocks<Traits<KER, OP, NBT, NBS, PAIRED>::kParts,
                                                   NBT, NBS, PAIRED>& out) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
  double A[PB], W0[PB], W1[PB];
#pragma unroll
  for (int i = 0; i < PB; ++i) {
    const double2 ab = *reinterpret_cast<const double2*>(rt + kRuleStride * (p0 + i));
    A[i] = fma(ab.x, fma(ab.x, ex0, fma(ab.y, hx, p.dgx0)), fma(ab.y, fma(ab.y, ex1, p.dgx1), p.r0));
    W0[i] = fma(ab.x, p.m00, fma(ab.y, p.m10, p.dgy0));
    W1[i] = fma(ab.x, p.m01, fma(ab.y, p.m11, p.dgy1));
  }
  double U[NP][PB][NBS], V[PAIRED ? NP : 1][PB][NBS], G[NP][PB];
#pragma unroll
  for (int part = 0; part < NP; ++part)
#pragma unroll
    for (int i = 0; i < PB; ++i) {
      G[part][i] = 0.0;
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        U[part][i][b] = 0.0;
        if constexpr (PAIRED) V[part][i][b] = 0.0;
      }
    }
#pragma unroll(Tr::kTrialUnroll)
  for (int q = 0; q < Q; ++q) {
    const double2* e = reinterpret_cast<const double2*>(rt + kRuleStride * q);
    const double2 ab = e[0], wp = e[1], pp = NBS == 3 ? e[2] : make_double2(0.0, 0.0);
    const double y = Yq[q], w = wp.x;
    double u[NBS], v[NBS];  // weights of U and V
    double fq = 1.0;
    if constexpr (Tr::kTrialFactor) fq = fma(ab.x, p.fy0, fma(ab.y, p.fy1, p.fy));
    if constexpr (NBS == 3) {
      u[0] = wp.y;
      u[1] = pp.x;
      u[2] = pp.y;
    } else {
      u[0] = w;
    }
#pragma unroll
    for (int b = 0; b < NBS; ++b) {
      v[b] = Tr::kTrialFactor ? u[b] * fq : 0.0;
      if (OP == kADL && !PAIRED) u[b] = v[b];
    }
    double r2[PB], K[2][PB];
#pragma unroll
    for (int i = 0; i < PB; ++i) r2[i] = A[i] + y;
#pragma unroll
    for (int i = 0; i < PB; ++i) r2[i] = fma(ab.x, W0[i], r2[i]);
#pragma unroll
    for (int i = 0; i < PB; ++i) r2[i] = fma(ab.y, W1[i], r2[i]);
    kernel_values<KER, OP, PH, PB>(r2, k, kr0, K[0], K[1]);
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      if constexpr (Tr::kHSSum) {
#pragma unroll
        for (int i = 0; i < PB; ++i) G[part][i] = fma(K[part][i], w, G[part][i]);
      }
      if constexpr (Tr::kBlock) {
#pragma unroll
        for (int b = 0; b < NBS; ++b)
#pragma unroll
          for (int i = 0; i < PB; ++i) {
            U[part][i][b] = fma(K[part][i], u[b], U[part][i][b]);
          }
        if constexpr (PAIRED) {
#pragma unroll
          for (int b = 0; b < NBS; ++b)
#pragma unroll
            for (int i = 0; i < PB; ++i) V[part][i][b] = fma(K[part][i], v[b], V[part][i][b]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < PB; ++i) {
    const double2* e = reinterpret_cast<const double2*>(rt + kRuleStride * (p0 + i));
    const double2 ab = e[0], wp = e[1], pp = NBT == 3 ? e[2] : make_double2(0.0, 0.0);
    const double ap = Tr::kTestFactor ? fma(ab.x, p.fx0, fma(ab.y, p.fx1, p.fx)) : 1.0;
    const double c[3] = {NBT == 3 ? wp.y : wp.x, pp.x, pp.y};
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      if constexpr (Tr::kHSSum) out.s[part] = fma(wp.x, G[part][i], out.s[part]);
      if constexpr (Tr::kBlock) {
#pragma unroll
        for (int b = 0; b < NBS; ++b) {
          const double f = Tr::kTestFactor ? ap * U[part][i][b] : U[part][i][b];
#pragma unroll
          for (int a = 0; a < NBT; ++a) {
            out.f[part][a][b] = fma(c[a], f, out.f[part][a][b]);
            if constexpr (PAIRED) out.t[part][a][b] = fma(c[a], V[part][i][b], out.t[part][a][b]);
          }
        }
      }
    }
  }
}

// A close pair: the squared distances from the components of
// x_p - y_q = dc + alpha_p g_0 + beta_p g_1 - (alpha_q g'_0 + beta_q g'_1), test points first,
// first + step, ...; phases not referenced to the pair (dc may be zero).  Adds to out.  Rolled
// loops: these pairs are few.
template <int KER, int OP, int NBT, int NBS, bool PAIRED>
__device__ __forceinline__ void pair_by_components(
    const PairGeometry& p, const Tile& T, int it, const Tile& S, int js, const double* rt, int Q,
    int first, int step, double k,
    Blocks<Traits<KER, OP, NBT, NBS, PAIRED>::kParts, NBT, NBS, PAIRED>& out) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
#pragma unroll 1
  for (int i = first; i < Q; i += step) {
    const double* x = rt + kRuleStride * i;  // alpha, beta, w, w phi_0, w phi_1, w phi_2
    double dx[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      dx[d] = ((T.G(rC + d, it) - S.G(rC + d, js)) + (T.G(rL + d, it) - S.G(rL + d, js))) +
              fma(x[0], T.G(rG0 + d, it), x[1] * T.G(rG1 + d, it));
    double U[NP][NBS], V[PAIRED ? NP : 1][NBS], G[NP];
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      G[part] = 0.0;
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        U[part][b] = 0.0;
        if constexpr (PAIRED) V[part][b] = 0.0;
      }
    }
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const double* y = rt + kRuleStride * q;
      double r2 = 0.0, K[2];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double e = dx[d] - fma(y[0], S.G(rG0 + d, js), y[1] * S.G(rG1 + d, js));
        r2 = fma(e, e, r2);
      }
      kernel_values<KER, OP, kAnyPhase, 1>(&r2, k, 0.0, K, K + 1);
      const double fq = Tr::kTrialFactor ? fma(y[0], p.fy0, fma(y[1], p.fy1, p.fy)) : 1.0;
#pragma unroll
      for (int part = 0; part < NP; ++part) {
        if constexpr (Tr::kHSSum) G[part] = fma(K[part], y[2], G[part]);
        if constexpr (Tr::kBlock) {
#pragma unroll
          for (int b = 0; b < NBS; ++b) {
            const double u = NBS == 3 ? y[3 + b] : y[2];
            U[part][b] = fma(K[part], OP == kADL && !PAIRED ? u * fq : u, U[part][b]);
            if constexpr (PAIRED) V[part][b] = fma(K[part], u * fq, V[part][b]);
          }
        }
      }
    }
    const double ap = Tr::kTestFactor ? fma(x[0], p.fx0, fma(x[1], p.fx1, p.fx)) : 1.0;
#pragma unroll
    for (int part = 0; part < NP; ++part) {
      if constexpr (Tr::kHSSum) out.s[part] = fma(x[2], G[part], out.s[part]);
      if constexpr (Tr::kBlock) {
#pragma unroll
        for (int a = 0; a < NBT; ++a) {
          const double c = NBT == 3 ? x[3 + a] : x[2];
#pragma unroll
          for (int b = 0; b < NBS; ++b) {
            out.f[part][a][b] = fma(c, Tr::kTestFactor ? ap * U[part][b] : U[part][b], out.f[part][a][b]);
            if constexpr (PAIRED) out.t[part][a][b] = fma(c, V[part][b], out.t[part][a][b]);
          }
        }
      }
    }
  }
}

// CTAs per SM the register allocation must allow.  (Helmholtz DP0 x DP0: three; with four, 128
// registers, the values that the close pairs need after the loop cost 3 %: 20,480 triangles,
// k = 8, 13.12 ms against 12.76.)
template <bool ORBITS, int KER, int OP, int NBT, int NBS, bool PAIRED>
constexpr int min_ctas() {
  if (KER == kHelmholtz) return PAIRED ? 2 : 3;
  return PAIRED ? (ORBITS ? 3 : 2) : OP == kHS && ORBITS ? 4 : OP == kHS || NBT * NBS == 9 ? 3 : 4;
}

// Staged blocks of a warp: entry ab = a * kTile + lane has NBS values, entry 3 * kTile is
// zero (what a lane with fewer incident cells than another reads).  Values of one entry side
// by side: 64-bit accesses of consecutive lanes are free of bank conflicts for NBS = 1, 3.
template <int NBS>
__host__ __device__ constexpr int stage_row() {
  return (3 * kTile + 1) * NBS + 1;
}
// Blocks staged at a time: real and imaginary parts of one order, or both orders of a real
// kernel (paired Helmholtz blocks take two passes, so that two CTAs per SM fit).
template <int NP, bool PAIRED>
__host__ __device__ constexpr int stage_blocks() {
  return NP == 2 || PAIRED ? 2 : 1;
}
// Laplace hypersingular: trial cells whose sums are staged before one pass over the DOFs.
constexpr int kSumBatch = 2;
// Incident cells of a DOF that its lane keeps in registers.
constexpr int kIncident = 8;

template <bool ORBITS>
struct RuleOf {
  using type = OrbitRule;
};
template <>
struct RuleOf<false> {
  using type = PointRule;
};

// Shared memory: mbarrier, rule table and squared lengths (general rule), trial tile, then
// per warp: test tile, stage and accumulators or the transposed block.
struct Layout {
  size_t rule, lengths, trial, curls, warp0, per_warp;
  size_t tile_t, stage, acc, inc, mirror;  // offsets within a warp's part
  size_t total;
};
template <bool ORBITS, int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED, bool SPLIT>
__host__ __device__ inline Layout layout(int Q, int ns, int gather, int cap, int mirror) {
  constexpr int NP = KER == kHelmholtz ? 2 : 1;
  constexpr bool kSumOnly = KER == kLaplace && OP == kHS;
  Layout l{};
  size_t o = 16;
  l.rule = o;
  o += sizeof(double) * kRuleStride * Q;
  l.lengths = o;
  if (!ORBITS) o += sizeof(double) * static_cast<size_t>(ns) * ((Q + 1) & ~1);
  l.trial = o;
  o += sizeof(double) * kRows * kTile + sizeof(int) * 9 * kTile;
  l.curls = o;
  if (kSumOnly && gather) o += sizeof(double) * 9 * kTile;
  o = (o + 15) & ~size_t(15);
  l.warp0 = o;
  size_t w = 0;
  l.tile_t = w;
  w += sizeof(double) * kRows * kTile + sizeof(int) * 3 * kTile;
  l.stage = w;
  if (!DIRECT && NBT == 3 && gather)
    w += sizeof(double) * (kSumOnly ? kSumBatch * kTile + 9 * kTile  // and the test cells' curls
                                    : stage_blocks<NP, PAIRED>() * stage_row<NBS>());
  l.acc = w;
  if (!DIRECT && gather) w += sizeof(double) * static_cast<size_t>(cap) * NP * (PAIRED ? 2 : 1);
  l.inc = w;
  if (!DIRECT && NBT == 3 && gather) w += 6 * kTile + 16;
  w = (w + 15) & ~size_t(15);
  l.mirror = w;
  if (DIRECT && SPLIT)
    w += sizeof(double) * NP * ns * (kTile + 1);
  else if (DIRECT && mirror)
    w += sizeof(double) * NP * 8 * (kTile + 1);
  w = (w + 15) & ~size_t(15);
  l.per_warp = w;
  l.total = o + kWarps * w;
  return l;
}

__device__ __forceinline__ Tile tile_at(unsigned char* at) {
  Tile t;
  t.pts = nullptr;
  t.rel = nullptr;
  t.geo = reinterpret_cast<double*>(at);
  t.vid = reinterpret_cast<int*>(at + sizeof(double) * kRows * kTile);
  t.ldof = t.vid + 3 * kTile;
  return t;
}

// Issues the bulk copies of one tile (one thread): all geometry rows and the vertex ids.
constexpr size_t kTileStride = sizeof(double) * kRows * kTile + sizeof(int) * 3 * kTile;  // in memory
constexpr unsigned kStagedBytes = sizeof(double) * kNumGeomFields * kTile + sizeof(int) * 3 * kTile;
__device__ inline void stage_geometry(const Tile& t, const CellSet& cs, int c0, uint64_t* m) {
  const int64_t S = cs.stride;
  for (int f = 0; f < kNumGeomFields; ++f)
    bulk_copy(t.geo + f * kTile, cs.geom + f * S + c0, sizeof(double) * kTile, m);
  for (int v = 0; v < 3; ++v) bulk_copy(t.vid + v * kTile, cs.vids + v * S + c0, sizeof(int) * kTile, m);
}

// The rows of column c as Row describes them, for a rule of that reach (rR to about 20 bits).
__device__ __forceinline__ void geometry_to_offsets(const Tile& t, int c, double reach) {
  double g0[3], g1[3], g2[3], e[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double t0 = t.G(kT0x + d, c), t1 = t.G(kT1x + d, c), third = (t0 + t1) * (1.0 / 3.0);
    t.geo[(rL + d) * kTile + c] = (t.G(kV0x + d, c) - t.G(kCx + d, c)) + third;
    g0[d] = -third;
    g1[d] = t0 + g0[d];
    g2[d] = t1 + g0[d];
    e[0] = fma(g0[d], g0[d], e[0]);
    e[1] = fma(g1[d], g1[d], e[1]);
    e[2] = fma(g2[d], g2[d], e[2]);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    t.geo[(rG0 + d) * kTile + c] = g0[d];
    t.geo[(rG1 + d) * kTile + c] = g1[d];
    t.geo[(rE + d) * kTile + c] = e[d];
  }
  const double most = fmax(fmax(e[0], e[1]), e[2]);
  double root;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(root) : "d"(most));
  t.geo[rR * kTile + c] = most > 0.0 ? reach * (1.0 / (1.0 - kSeparation)) * (most * root) : 0.0;
}

// Curl of basis function a of a flat cell from its offsets: t0 - t1, t1, -t0.
__device__ __forceinline__ double curl_of(const Tile& t, int c, int a, int d) {
  const double g0 = t.G(rG0 + d, c), g1 = t.G(rG1 + d, c);
  return a == 0 ? fma(2.0, g1, g0) : a == 1 ? -(fma(2.0, g0, g1)) : g0 - g1;
}

// A pair's block from its sums: reference phase, jdet_x jdet_y / (4 pi), curls (Laplace
// hypersingular: the sum s stays, the curls enter where it is added).
template <int KER, int OP, int NBT, int NBS, bool PAIRED, int PH>
__device__ __forceinline__ void finish_block(
    const Tile& T, int it, const Tile& S, int js, double k, double kr0, double sc,
    Blocks<Traits<KER, OP, NBT, NBS, PAIRED>::kParts, NBT, NBS, PAIRED>& blk) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
  constexpr bool kC = NP == 2;
  if constexpr (kC && PH != kAnyPhase) {
    double ps, pc;
    sincos_any(kr0, ps, pc);
    if constexpr (Tr::kHSSum) {
      const double re = blk.s[0] * pc - blk.s[1] * ps, im = blk.s[0] * ps + blk.s[1] * pc;
      blk.s[0] = re;
      blk.s[1] = im;
    }
    const double f = OP == kHS ? 1.0 : sc;
    const double cr = pc * f, ci = ps * f;
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        const double re = blk.f[0][a][b] * cr - blk.f[1][a][b] * ci;
        blk.f[1][a][b] = blk.f[0][a][b] * ci + blk.f[1][a][b] * cr;
        blk.f[0][a][b] = re;
        if constexpr (PAIRED) {
          const double tr = blk.t[0][a][b] * cr - blk.t[1][a][b] * ci;
          blk.t[1][a][b] = blk.t[0][a][b] * ci + blk.t[1][a][b] * cr;
          blk.t[0][a][b] = tr;
        }
      }
  } else if constexpr (OP == kSL) {
#pragma unroll
    for (int part = 0; part < NP; ++part)
#pragma unroll
      for (int a = 0; a < NBT; ++a)
#pragma unroll
        for (int b = 0; b < NBS; ++b) blk.f[part][a][b] *= sc;
  }
  if constexpr (OP == kHS && kC) {
    // curl-curl - k^2 normal-normal
    const double nn = T.G(rN, it) * S.G(rN, js) + T.G(rN + 1, it) * S.G(rN + 1, js) +
                      T.G(rN + 2, it) * S.G(rN + 2, js);
    const double nnsc = -k * k * nn * sc;
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        double cc = 0.0;
        if constexpr (NBT == 3 && NBS == 3)
#pragma unroll
          for (int d = 0; d < 3; ++d) cc = fma(curl_of(T, it, a, d), curl_of(S, js, b, d), cc);
        cc *= kInv4Pi;
#pragma unroll
        for (int part = 0; part < NP; ++part)
          blk.f[part][a][b] = fma(nnsc, blk.f[part][a][b], blk.s[part] * cc);
      }
  }
}

// Adds a pair's block to the output (rows, cols: its global DOFs), and the transposed one
// where the launch covers both orders of a pair.
template <int KER, int OP, int NBT, int NBS, bool PAIRED>
__device__ __forceinline__ void add_block(
    const Tile& T, int it, const Tile& S, int js, const int* rows, const int* cols, double* out,
    int64_t ld, bool mirror, int swapped,
    Blocks<Traits<KER, OP, NBT, NBS, PAIRED>::kParts, NBT, NBS, PAIRED>& blk) {
  constexpr int NP = Traits<KER, OP, NBT, NBS, PAIRED>::kParts;
  if constexpr (KER == kLaplace && OP == kHS && NBT == 3 && NBS == 3) {
#pragma unroll
    for (int a = 0; a < NBT; ++a)
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        double cc = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) cc = fma(curl_of(T, it, a, d), curl_of(S, js, b, d), cc);
        blk.f[0][a][b] = blk.s[0] * cc * kInv4Pi;
      }
  }
#pragma unroll
  for (int b = 0; b < NBS; ++b) {
    const int col = cols[b];
#pragma unroll
    for (int a = 0; a < NBT; ++a) {
      const int64_t o = static_cast<int64_t>(col) * ld + rows[a];
      const int64_t om = static_cast<int64_t>(rows[a]) * ld + col;
#pragma unroll
      for (int part = 0; part < NP; ++part) {
        double v = blk.f[part][a][b], m = v;
        if constexpr (PAIRED) {
          m = swapped ? v : blk.t[part][a][b];
          v = swapped ? blk.t[part][a][b] : v;
        }
        atomicAdd(out + NP * o + part, v);
        if (mirror) atomicAdd(out + NP * om + part, m);
      }
    }
  }
}

// The close pairs of a warp, after its other pairs: bit js of `todo` is the lane's pair with
// trial cell js.  They are found before the loop over the pairs and added after it, directly:
// with a branch for them in the loop everything was slower (20,480 triangles, Laplace
// hypersingular P1 7.5 -> 8.0 ms, Helmholtz single layer DP0 12.7 -> 13.2; 80 triangles, 37-point
// rule 21 -> 33 us); apart from it they cost 0 to 2 %.  tdofs, sdofs: DOFs of the tiles' cells.
// DIRECT: the entries (and their transposes) were stored as zeros; SPLIT: sums[part][trial cell
// of the chunk][lane] instead.
template <int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED, bool SPLIT>
__device__ __noinline__ void add_close_pairs(const Tile T, int it, const Tile S, unsigned todo,
                                             const double* rt, int Q, int warp,
                                             double k, const int* tdofs, const int* sdofs, int ti0,
                                             int sj0, double* out, int64_t ld, bool mirror, int swapped,
                                             double* sums, int ns, int j0) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
  for (; todo; todo &= todo - 1) {
    const int js = __ffs(todo) - 1;
    const double sc = T.G(rJ, it) * S.G(rJ, js) * kInv4Pi;
    PairGeometry p;
    pair_geometry<KER, OP, NBT, NBS, PAIRED>(T, it, S, js, Tr::template kScaledFactors<kAnyPhase> ? sc : 1.0, p);
    Blocks<NP, NBT, NBS, PAIRED> blk;
    clear(blk);
    pair_by_components<KER, OP, NBT, NBS, PAIRED>(p, T, it, S, js, rt, Q, SPLIT ? warp : 0,
                                                  SPLIT ? kWarps : 1, k, blk);
    finish_block<KER, OP, NBT, NBS, PAIRED, kAnyPhase>(T, it, S, js, k, 0.0, sc, blk);
    if constexpr (DIRECT) {
#pragma unroll
      for (int part = 0; part < NP; ++part) {
        const double v = blk.f[part][0][0];
        if constexpr (SPLIT) {
          sums[(part * ns + js - j0) * (kTile + 1) + it] = v;
        } else {
          out[NP * (static_cast<int64_t>(sj0 + js) * ld + ti0 + it) + part] = v;
          if (mirror) out[NP * (static_cast<int64_t>(ti0 + it) * ld + sj0 + js) + part] = v;
        }
      }
    } else {
      add_block<KER, OP, NBT, NBS, PAIRED>(T, it, S, js, tdofs + it * NBT, sdofs + js * NBS, out, ld,
                                           mirror, swapped, blk);
    }
  }
}

template <bool ORBITS, int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED, int PH,
          bool SPLIT>
__global__ void __launch_bounds__(kThreads, min_ctas<ORBITS, KER, OP, NBT, NBS, PAIRED>())
    regular_fp64(CellSet test, SpaceTiles tt, CellSet trial, SpaceTiles st,
                 const __grid_constant__ typename RuleOf<ORBITS>::type rule, double k, int same_grid,
                 double* __restrict__ out, int64_t ld, Shape sh, int symmetric, int swapped,
                 unsigned* __restrict__ timeouts, int polls) {
  using Tr = Traits<KER, OP, NBT, NBS, PAIRED>;
  constexpr int NP = Tr::kParts;
  constexpr bool kC = NP == 2;
  // Laplace hypersingular: one sum per cell pair is staged, the curls enter per DOF
  constexpr bool kSumOnly = KER == kLaplace && OP == kHS;
  constexpr int kPer = SPLIT ? 1 : kWarps;  // test tiles per CTA
  const int warp = threadIdx.x >> 5, it = threadIdx.x & 31;
  int Q = 6;
  if constexpr (!ORBITS) Q = rule.npts;
  const int cpt = kTile / sh.ns;
  const long long unit = blockIdx.x / cpt;
  const int chunk = blockIdx.x % cpt;
  int group, sy;
  if (symmetric) {
    lower_group(unit, sh.nsup, kPer, sh.ty0, sh.ty1, group, sy);
  } else {
    group = static_cast<int>(unit % sh.nsup);
    sy = sh.ty0 + static_cast<int>(unit / sh.nsup);
  }
  const int tx = group * kPer + (SPLIT ? 0 : warp);
  const int sj0 = sy * kTile;
  const int j0 = chunk * sh.ns;                              // first cell of the chunk
  const int j1 = min(j0 + sh.ns, min(kTile, trial.ncells - sj0));
  // nothing to do for the whole CTA: past the mesh's end, or above the diagonal
  if (j0 >= j1 || (symmetric && group * kPer + kPer - 1 < sy)) return;
  const bool mine = tx < sh.ntt && !(symmetric && tx < sy);
  const bool mirror = symmetric && tx > sy;
  const int ti0 = tx * kTile;
  const int nti = mine ? min(kTile, test.ncells - ti0) : 0;

  extern __shared__ __align__(16) unsigned char smem[];
  const Layout L = layout<ORBITS, KER, OP, NBT, NBS, DIRECT, PAIRED, SPLIT>(
      Q, sh.ns, sh.gather, sh.cap, symmetric);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);
  double* rt = reinterpret_cast<double*>(smem + L.rule);
  double* lengths = reinterpret_cast<double*>(smem + L.lengths);
  const int Qp = (Q + 1) & ~1;
  const Tile S = tile_at(smem + L.trial);
  int* sdof = S.ldof + 3 * kTile;  // global DOFs of the chunk's columns (at most 96)
  unsigned char* wbase = smem + L.warp0 + warp * L.per_warp;
  // SPLIT: the four warps read one test tile (the first warp's)
  const Tile T = tile_at(SPLIT ? smem + L.warp0 + L.tile_t : wbase + L.tile_t);
  double* stage = reinterpret_cast<double*>(wbase + L.stage);
  double* acc = reinterpret_cast<double*>(wbase + L.acc);
  uint8_t* inc_off = wbase + L.inc;
  uint8_t* inc_ent = inc_off + 3 * kTile + 1;
  double* mir = reinterpret_cast<double*>(wbase + L.mirror);

  // ---- staging: the trial tile and each warp's test tile, one transaction barrier
  if (threadIdx.x == 0) mbar_init(mbar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    int tiles_here = 1;
    for (int w = 0; w < kPer; ++w) {
      const int t = group * kPer + w;
      tiles_here += (t < sh.ntt && !(symmetric && t < sy)) ? 1 : 0;
    }
    mbar_expect_tx(mbar, tiles_here * kStagedBytes);
    stage_geometry(S, trial, sj0, mbar);
    for (int w = 0; w < kPer; ++w) {
      const int t = group * kPer + w;
      if (t < sh.ntt && !(symmetric && t < sy))
        stage_geometry(tile_at(smem + L.warp0 + w * L.per_warp + L.tile_t), test, t * kTile, mbar);
    }
  }
  int ndt = 0, nds = 0;
  const int* tdofs = nullptr;
  if constexpr (!DIRECT) {
    if (mine) {
      const int o = __ldg(tt.tile_dof_off + tx);
      ndt = __ldg(tt.tile_dof_off + tx + 1) - o;
      tdofs = tt.tile_dofs + o;
    }
    if (sh.gather) {
      // the chunk's trial DOFs, renumbered: bit l of used = the tile's DOF l occurs
      const int so = __ldg(st.tile_dof_off + sy);
      unsigned used[3] = {0u, 0u, 0u};
      int l[NBS];
#pragma unroll
      for (int b = 0; b < NBS; ++b) {
        const bool in = it >= j0 && it < j1;
        l[b] = in ? __ldg(st.cell_ldof + static_cast<int64_t>(sj0 + it) * NBS + b) : 0;
        if (in) {
          const unsigned bit = 1u << (l[b] & 31);
          used[0] |= l[b] < 32 ? bit : 0u;
          used[1] |= (l[b] >> 5) == 1 ? bit : 0u;
          used[2] |= (l[b] >> 5) == 2 ? bit : 0u;
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) used[i] = __reduce_or_sync(0xffffffffu, used[i]);
      const int n0 = __popc(used[0]), n1 = __popc(used[1]);
      nds = n0 + n1 + __popc(used[2]);
      if (warp == 0) {
        auto place = [&](int v) {
          const unsigned below = (1u << (v & 31)) - 1u;
          return v < 32 ? __popc(used[0] & below)
                        : v < 64 ? n0 + __popc(used[1] & below) : n0 + n1 + __popc(used[2] & below);
        };
#pragma unroll
        for (int b = 0; b < NBS; ++b) S.ldof[b * kTile + it] = place(l[b]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if ((used[i] >> it) & 1u) sdof[place(32 * i + it)] = __ldg(st.tile_dofs + so + 32 * i + it);
      }
      if (mine) {
        for (int i = it; i < ndt * nds; i += 32)
#pragma unroll
          for (int x = 0; x < NP * (PAIRED ? 2 : 1); ++x) acc[x * sh.cap + i] = 0.0;
        if constexpr (NBT == 3)
          for (int i = it; i < 6 * kTile + 1; i += 32)
            inc_off[i] = i <= 3 * kTile
                             ? __ldg(tt.inc_off + static_cast<int64_t>(tx) * (3 * kTile + 1) + i)
                             : __ldg(tt.inc_ent + static_cast<int64_t>(tx) * 3 * kTile + i - (3 * kTile + 1));
      }
    } else {
      for (int i = threadIdx.x; i < NBS * kTile; i += kThreads) {
        const int c = i % kTile, b = i / kTile;
        S.ldof[i] = c >= j0 && c < j1
                        ? __ldg(st.cell_dofs + static_cast<int64_t>(sj0 + c) * NBS + b) : 0;
      }
    }
  }
  if constexpr (ORBITS) {  // point a of orbit o is c + gamma_o g_a; constant indexes only
    if (threadIdx.x < 6) {
      const int a = threadIdx.x % 3;
      const bool o = threadIdx.x >= 3;
      const double g = o ? rule.g[1] : rule.g[0], c = o ? rule.c[1] : rule.c[0], d = o ? rule.d[1] : rule.d[0];
      double* e = rt + threadIdx.x * kRuleStride;
      e[0] = a == 0 ? g : a == 2 ? -g : 0.0;
      e[1] = a == 1 ? g : a == 2 ? -g : 0.0;
      e[2] = o ? rule.w[1] : rule.w[0];
#pragma unroll
      for (int b = 0; b < 3; ++b) e[3 + b] = a == b ? c + d : c;
    }
  } else {
    for (int i = threadIdx.x; i < Q; i += kThreads)
#pragma unroll
      for (int f = 0; f < kPointFields; ++f) rt[i * kRuleStride + f] = rule.p[i][f];
  }
  const bool staged = mbar_wait_bounded(mbar, 0, polls);
  if (__syncthreads_or(!staged)) {
    // the copies did not complete in time: record it, give them a last bounded wait and
    // leave this block's entries unwritten (the host reports the failure)
    if (threadIdx.x == 0) atomicAdd(timeouts, 1u);
    mbar_wait_bounded(mbar, 0);
    return;
  }
  if (warp == 0) geometry_to_offsets(S, it, rule.reach);
  if constexpr (SPLIT) {
    if (warp == 1) geometry_to_offsets(T, it, rule.reach);
  } else {
    if (mine) geometry_to_offsets(T, it, rule.reach);
  }
  Box box;
  if (!SPLIT && mine) box = tile_box(T, it, nti);
  __syncthreads();
  if (SPLIT) box = tile_box(T, it, nti);
  double* scurl = reinterpret_cast<double*>(smem + L.curls);  // [(b * 3 + d) * kTile + c]
  double* tcurl = stage + kSumBatch * kTile;                  // [(a * kTile + c) * 3 + d]
  if constexpr (kSumOnly && !DIRECT) {
    if (sh.gather) {
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (warp == 0) scurl[(a * 3 + d) * kTile + it] = curl_of(S, it, a, d) * kInv4Pi;
          if (mine) tcurl[(a * kTile + it) * 3 + d] = curl_of(T, it, a, d);
        }
      __syncthreads();
    }
  }
  if constexpr (!ORBITS) {
    // |y_q - c_y|^2 of the chunk's cells: alpha^2 e0 + alpha beta (e2 - e0 - e1) + beta^2 e1
    for (int i = threadIdx.x; i < (j1 - j0) * Q; i += kThreads) {
      const int j = i / Q, q = i - j * Q;
      const double al = rt[q * kRuleStride], be = rt[q * kRuleStride + 1];
      const double e0 = S.G(rE, j0 + j), e1 = S.G(rE + 1, j0 + j), h = S.G(rE + 2, j0 + j) - e0 - e1;
      lengths[j * Qp + q] = fma(al * al, e0, fma(al * be, h, be * be * e1));
    }
    __syncthreads();
  }
  if (!mine && !SPLIT) return;  // SPLIT: the tile is the same for every warp

  const bool lane_cell = it < nti;
  // the lane's pairs that the loop leaves out, bit js: vertex-sharing ones and close ones
  unsigned skip = lane_cell ? 0u : ~0u, close = 0u;
  if (same_grid && lane_cell) {
    const int a0 = T.vid[it], a1 = T.vid[kTile + it], a2 = T.vid[2 * kTile + it];
#pragma unroll 4
    for (int js = j0; js < j1; ++js)
      if (share_vertex(a0, a1, a2, S.vid[js], S.vid[kTile + js], S.vid[2 * kTile + js])) skip |= 1u << js;
  }
  for (unsigned at = cells_in_reach(box, S, it, j0, j1); at; at &= at - 1) {
    const int js = __ffs(at) - 1;
    PairGeometry p;
    pair_geometry<KER, kSL, 1, 1, false>(T, it, S, js, 1.0, p);
    if (!((skip >> js) & 1u) && close_pair(p, T.G(rR, it) + S.G(rR, js), rule.reach)) close |= 1u << js;
  }
  skip |= close;
  // not in a register through the loop (20,480 triangles, double layer P1: 13.76 -> 13.61 ms): in the
  // lane's own rR, which nothing reads from here on (SPLIT: the warps share the tile)
  if constexpr (!SPLIT) reinterpret_cast<unsigned*>(T.geo + rR * kTile)[2 * it] = close;
  int rows[NBT];  // direct adds: the lane's test DOFs
  if constexpr (!DIRECT) {
    if (!sh.gather)
#pragma unroll
      for (int a = 0; a < NBT; ++a)
        rows[a] = lane_cell ? __ldg(tt.cell_dofs + static_cast<int64_t>(ti0 + it) * NBT + a) : 0;
  }

  // the incident (basis, cell) entries of DOF `it`, a byte each, and the warp's largest number
  // of them; tiles with more than 32 DOFs or kIncident cells at one take the plain loop
  unsigned ent[2] = {0u, 0u};
  int count = 0, most = 0;
  bool in_registers = false;
  if constexpr (!DIRECT && NBT == 3) {
    if (sh.gather) {
      __syncwarp();
      const int first = it < ndt ? inc_off[it] : 0;
      count = it < ndt ? inc_off[it + 1] - first : 0;
      most = __reduce_max_sync(0xffffffffu, count);
      in_registers = ndt <= kTile && most <= kIncident;
#pragma unroll
      for (int e = 0; e < kIncident; ++e) {
        const unsigned v = e < count ? inc_ent[first + e] : 3u * kTile;
        ent[e / 4] |= v << (8 * (e % 4));
      }
      if constexpr (!kSumOnly) {
        if (it < stage_blocks<NP, PAIRED>())
#pragma unroll
          for (int b = 0; b < NBS; ++b) stage[it * stage_row<NBS>() + 3 * kTile * NBS + b] = 0.0;
      }
      __syncwarp();
    }
  }

#pragma unroll 1
  for (int js = j0; js < j1; ++js) {
    const bool have = !((skip >> js) & 1u);
    const double sc = T.G(rJ, it) * S.G(rJ, js) * kInv4Pi;  // jdet_x jdet_y / (4 pi)
    PairGeometry p;
    pair_geometry<KER, OP, NBT, NBS, PAIRED>(T, it, S, js, Tr::template kScaledFactors<PH> ? sc : 1.0, p);
    double kr0 = 0.0;
    if constexpr (kC && PH != kAnyPhase) kr0 = k * (p.r0 * rsqrt_refined(p.r0));
    Blocks<NP, NBT, NBS, PAIRED> blk;
    if constexpr (ORBITS) {
      pair_orbits<KER, OP, NBT, NBS, PAIRED, PH>(p, T, it, S, js, rule, k, kr0, blk);
    } else {
      clear(blk);
      p.dgx0 *= 2.0;
      p.dgx1 *= 2.0;
      p.dgy0 *= -2.0;
      p.dgy1 *= -2.0;
      p.m00 *= -2.0;
      p.m01 *= -2.0;
      p.m10 *= -2.0;
      p.m11 *= -2.0;
      const double ex0 = T.G(rE, it), ex1 = T.G(rE + 1, it), hx = T.G(rE + 2, it) - ex0 - ex1;
      constexpr int PB = Tr::kPoints;
      const double* Yq = lengths + (js - j0) * Qp;
      int q0 = SPLIT ? warp * PB : 0;
#pragma unroll 1
      for (; q0 + PB <= Q; q0 += SPLIT ? kWarps * PB : PB)
        point_block<KER, OP, NBT, NBS, PAIRED, PH, PB>(p, ex0, hx, ex1, rt, Yq, Q, q0, k, kr0, blk);
      // the remainder of the rule, one point at a time (SPLIT: one warp each)
      int rest = Q - Q % PB;
      if (SPLIT) rest += (warp + kWarps - (Q / PB) % kWarps) % kWarps;
#pragma unroll 1
      for (; rest < Q; rest += SPLIT ? kWarps : 1)
        point_block<KER, OP, NBT, NBS, PAIRED, PH, 1>(p, ex0, hx, ex1, rt, Yq, Q, rest, k, kr0, blk);
    }
    finish_block<KER, OP, NBT, NBS, PAIRED, PH>(T, it, S, js, k, kr0, sc, blk);
    // ---- where it goes
    if constexpr (DIRECT) {
      double v[2] = {have ? blk.f[0][0][0] : 0.0, kC && have ? blk.f[NP - 1][0][0] : 0.0};
      if constexpr (SPLIT) {
#pragma unroll
        for (int part = 0; part < NP; ++part)
          mir[(part * sh.ns + js - j0) * (kTile + 1) + it] = v[part];
      } else {
        const int64_t o = static_cast<int64_t>(sj0 + js) * ld + ti0 + it;
        if (lane_cell) {
          if (kC)
            reinterpret_cast<double2*>(out)[o] = make_double2(v[0], v[1]);
          else
            out[o] = v[0];
        }
        if (mirror) {
          // the transposed entries, up to eight columns j at a time: (row sj0 + j, column
          // ti0 + i), j fastest
          const int jj = (js - j0) & 7;
#pragma unroll
          for (int part = 0; part < NP; ++part) mir[(part * 8 + jj) * (kTile + 1) + it] = v[part];
          if (jj == 7 || js == j1 - 1) {
            __syncwarp();
            const int first = js - jj, n = jj + 1;
            for (int e = it; e < 8 * kTile; e += 32) {
              const int i = e >> 3, j = e & 7;
              if (j < n && i < nti) {
                const int64_t om = static_cast<int64_t>(ti0 + i) * ld + sj0 + first + j;
                if (kC)
                  reinterpret_cast<double2*>(out)[om] =
                      make_double2(mir[j * (kTile + 1) + i], mir[(8 + j) * (kTile + 1) + i]);
                else
                  out[om] = mir[j * (kTile + 1) + i];
              }
            }
            __syncwarp();
          }
        }
      }
    } else if (!sh.gather) {
      // no accumulator: every lane adds its entries
      if (have) {
        int cols[NBS];
#pragma unroll
        for (int b = 0; b < NBS; ++b) cols[b] = S.ldof[b * kTile + js];
        add_block<KER, OP, NBT, NBS, PAIRED>(T, it, S, js, rows, cols, out, ld, mirror, swapped, blk);
      }
    } else if constexpr (NBT == 1) {
      // one DOF per test cell: lanes own their rows
      if (lane_cell) {
        const int d = __ldg(tt.cell_ldof + ti0 + it);
#pragma unroll
        for (int b = 0; b < NBS; ++b) {
          const int i = d + ndt * S.ldof[b * kTile + js];
#pragma unroll
          for (int part = 0; part < NP; ++part)
            acc[part * sh.cap + i] += have ? blk.f[part][0][b] : 0.0;
        }
      }
    } else if constexpr (kSumOnly) {
      // lane d: vector sums over the test cells of DOF d of s curl_a, for up to kSumBatch trial
      // cells at once, then their products with the trial cells' curls
      const int jj = (js - j0) % kSumBatch;
      stage[jj * kTile + it] = have ? blk.s[0] : 0.0;
      if (jj == kSumBatch - 1 || js == j1 - 1) {
        __syncwarp();
        for (int d = it; d < ndt; d += kTile) {
          double z[kSumBatch][3];
#pragma unroll
          for (int j = 0; j < kSumBatch; ++j) z[j][0] = z[j][1] = z[j][2] = 0.0;
          auto add = [&](int ab, bool on) {
            const double* cu = tcurl + (on ? ab : 0) * 3;
            const double c0 = cu[0], c1 = cu[1], c2 = cu[2];
#pragma unroll
            for (int j = 0; j < kSumBatch; ++j) {
              double v = stage[j * kTile + (ab & (kTile - 1))];
              v = on && j <= jj ? v : 0.0;
              z[j][0] = fma(v, c0, z[j][0]);
              z[j][1] = fma(v, c1, z[j][1]);
              z[j][2] = fma(v, c2, z[j][2]);
            }
          };
          if (in_registers) {
#pragma unroll
            for (int e = 0; e < kIncident; ++e)
              if (e < most) add((ent[e / 4] >> (8 * (e % 4))) & 0xffu, e < count);
          } else {
            for (int e = inc_off[d]; e < inc_off[d + 1]; ++e) add(inc_ent[e], true);
          }
#pragma unroll
          for (int j = 0; j < kSumBatch; ++j) {
            if (j > jj) break;
            // the curls of a cell's basis sum to zero
            const int c = js - jj + j;
            const double* cs = scurl + c;
            const double v0 = fma(z[j][2], cs[2 * kTile], fma(z[j][1], cs[kTile], z[j][0] * cs[0]));
            const double v1 = fma(z[j][2], cs[5 * kTile], fma(z[j][1], cs[4 * kTile], z[j][0] * cs[3 * kTile]));
            acc[d + ndt * S.ldof[c]] += v0;
            acc[d + ndt * S.ldof[kTile + c]] += v1;
            acc[d + ndt * S.ldof[2 * kTile + c]] -= v0 + v1;
          }
        }
        __syncwarp();
      }
    } else {
      constexpr int NX = NP * (PAIRED ? 2 : 1), GX = stage_blocks<NP, PAIRED>();
      constexpr int kRow = stage_row<NBS>();
#pragma unroll
      for (int x0 = 0; x0 < NX; x0 += GX) {
        if (PAIRED && !mirror && x0 >= NP) break;  // a diagonal tile pair: one order only
#pragma unroll
        for (int x = 0; x < GX; ++x)
#pragma unroll
          for (int a = 0; a < NBT; ++a)
#pragma unroll
            for (int b = 0; b < NBS; ++b) {
              double v = blk.f[(x0 + x) % NP][a][b];
              if constexpr (PAIRED)
                v = ((x0 + x >= NP) != (swapped != 0)) ? blk.t[(x0 + x) % NP][a][b] : v;
              stage[x * kRow + (a * kTile + it) * NBS + b] = have ? v : 0.0;
            }
        __syncwarp();
        for (int d = it; d < ndt; d += kTile) {
          double g[GX][NBS];
#pragma unroll
          for (int x = 0; x < GX; ++x)
#pragma unroll
            for (int b = 0; b < NBS; ++b) g[x][b] = 0.0;
          auto add = [&](int ab) {
#pragma unroll
            for (int x = 0; x < GX; ++x)
#pragma unroll
              for (int b = 0; b < NBS; ++b) g[x][b] += stage[x * kRow + ab * NBS + b];
          };
          if (in_registers) {
#pragma unroll
            for (int e = 0; e < kIncident; ++e)
              if (e < most) add((ent[e / 4] >> (8 * (e % 4))) & 0xffu);
          } else {
            for (int e = inc_off[d]; e < inc_off[d + 1]; ++e) add(inc_ent[e]);
          }
#pragma unroll
          for (int b = 0; b < NBS; ++b) {
            double* dst = acc + x0 * sh.cap + d + ndt * S.ldof[b * kTile + js];
#pragma unroll
            for (int x = 0; x < GX; ++x) dst[x * sh.cap] += g[x][b];
          }
        }
        __syncwarp();
      }
    }
  }
  if constexpr (!SPLIT) close = reinterpret_cast<volatile unsigned*>(T.geo + rR * kTile)[2 * it];
  if (__any_sync(0xffffffffu, close != 0u))
    add_close_pairs<KER, OP, NBT, NBS, DIRECT, PAIRED, SPLIT>(
        T, it, S, close, rt, Q, warp, k, DIRECT ? nullptr : tt.cell_dofs + static_cast<int64_t>(ti0) * NBT,
        DIRECT ? nullptr : st.cell_dofs + static_cast<int64_t>(sj0) * NBS, ti0, sj0, out, ld, mirror,
        swapped, mir, sh.ns, j0);
  // ---- flush
  if constexpr (DIRECT && SPLIT) {
    __syncthreads();
    auto sum = [&](int part, int j, int i) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w)
        v += reinterpret_cast<const double*>(smem + L.warp0 + w * L.per_warp + L.mirror)
            [(part * sh.ns + j) * (kTile + 1) + i];
      return v;
    };
    const int n = j1 - j0;
    for (int e = threadIdx.x; e < n * kTile; e += kThreads) {
      const int i = e % kTile, j = e / kTile;
      if (i >= nti) continue;
      const int64_t o = static_cast<int64_t>(sj0 + j0 + j) * ld + ti0 + i;
      const int64_t om = static_cast<int64_t>(ti0 + i) * ld + sj0 + j0 + j;
      const double re = sum(0, j, i);
      if constexpr (kC) {
        const double2 v = make_double2(re, sum(1, j, i));
        reinterpret_cast<double2*>(out)[o] = v;
        if (mirror) reinterpret_cast<double2*>(out)[om] = v;
      } else {
        out[o] = re;
        if (mirror) out[om] = re;
      }
    }
  }
  if constexpr (!DIRECT) {
    if (sh.gather) {
      __syncwarp();
      auto put = [&](const double* src, int d, int s, int64_t o) {
#pragma unroll
        for (int part = 0; part < NP; ++part) {
          const double v = src[part * sh.cap + d + ndt * s];
          if (v != 0.0) atomicAdd(out + NP * o + part, v);
        }
      };
      for (int d = it; d < ndt; d += 32) {
        const int row = __ldg(tdofs + d);
#pragma unroll 4
        for (int s = 0; s < nds; ++s) put(acc, d, s, static_cast<int64_t>(sdof[s]) * ld + row);
      }
      if (mirror) {
        // the transposed entries, trial DOFs fastest, two columns at a time when they fit
        const double* src = acc + (PAIRED ? NP : 0) * sh.cap;
        const int w = nds <= 16 ? 16 : 32, s0 = it & (w - 1);
        for (int s = s0; s < nds; s += w) {
          const int row = sdof[s];
#pragma unroll 4
          for (int d = it / w; d < ndt; d += 32 / w)
            put(src, d, s, static_cast<int64_t>(__ldg(tdofs + d)) * ld + row);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------- launches ---
// The reach of a rule: with m the least barycentric coordinate of a point, the point is
// c + sum_a (lambda_a - m) g_a, factors >= 0 whose sum is 1 - 3 m.
inline double rule_reach(const RegularRule& r) {
  double reach = 0.0;
  for (int q = 0; q < r.npts; ++q)
    reach = fmax(reach, 1.0 - 3.0 * fmin(fmin(r.phi[0][q], r.phi[1][q]), r.phi[2][q]));
  return reach;
}

inline OrbitRule orbit_rule(const RegularRule& r) {
  OrbitRule o{};
  o.reach = rule_reach(r);
  for (int i = 0; i < 2; ++i) {
    const double l0 = r.phi[0][3 * i];  // the orbit's first point is c + gamma g_0
    o.g[i] = (l0 - 1.0 / 3.0) * 1.5;
    o.g2[i] = o.g[i] * o.g[i];
    o.w[i] = r.w[3 * i];
    o.c[i] = r.w[3 * i] * (1.0 - o.g[i]) / 3.0;
    o.d[i] = r.w[3 * i] * o.g[i];
  }
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) o.m[i][j] = -2.0 * o.g[i] * o.g[j];
  return o;
}

inline PointRule point_rule(const RegularRule& r) {
  PointRule p{};
  p.npts = r.npts;
  p.reach = rule_reach(r);
  for (int q = 0; q < r.npts; ++q) {
    const double l0 = r.phi[0][q], l1 = r.phi[1][q], l2 = r.phi[2][q];
    const double f[kPointFields] = {l0 - l2, l1 - l2, r.w[q], r.wphi[0][q], r.wphi[1][q], r.wphi[2][q]};
    for (int i = 0; i < kPointFields; ++i) p.p[q][i] = f[i];
  }
  return p;
}

// The largest offset of a point of such a rule from the centroid, in circumradii.
inline double orbit_reach(const RegularRule& r) {
  double g = 0.0;
  for (int o = 0; o < 2; ++o) g = fmax(g, fabs((r.phi[0][3 * o] - 1.0 / 3.0) * 1.5));
  return g;
}

// Two S21 orbits, points in vertex order (point b of an orbit has its largest or smallest
// barycentric coordinate at vertex b), as pair_orbits needs.
inline bool has_orbit_form(const RegularRule& r) {
  if (r.npts != 6) return false;
  for (int o = 0; o < 2; ++o) {
    const double big = r.phi[0][3 * o], small = r.phi[1][3 * o];
    for (int b = 0; b < 3; ++b) {
      if (r.w[3 * o + b] != r.w[3 * o]) return false;
      for (int v = 0; v < 3; ++v)
        if (!(fabs(r.phi[v][3 * o + b] - (v == b ? big : small)) <= 1e-15)) return false;
    }
  }
  return true;
}

constexpr int kSMs = 148;
constexpr int kAccumulatorBytes = 20 << 10;  // per warp, at most (see set_accumulator)

template <int KER, int NBS, bool DIRECT, bool PAIRED>
inline void set_accumulator(Shape& sh, const SpaceTiles& tt, const SpaceTiles& st) {
  // accumulators of up to 20 KB per warp (the other arrays take 7 to 11 KB of a warp: two CTAs of
  // four warps stay resident with 17 KB, one with more); larger ones (discontinuous P1, meshes whose
  // tiles touch many DOFs) are replaced by direct adds, which cost less than the flushes of
  // shorter chunks (20,480 triangles in a mesher's order, 45 DOFs per tile on average and 77 at most,
  // Laplace double layer P1: 16.3 ms with direct adds, 23.2 with accumulators for eight cells)
  sh.cap = 0;
  sh.gather = 0;
  if (!DIRECT) {
    // (a shorter chunk lies within one of eight or sixteen cells)
    sh.cap = tt.max_tile_dofs * std::min(sh.ns * NBS, st.most_dofs[sh.ns > 8 ? 0 : 1]);
    const size_t bytes = sizeof(double) * static_cast<size_t>(sh.cap) * (KER == kHelmholtz ? 2 : 1) *
                         (PAIRED ? 2 : 1);
    sh.gather = bytes <= kAccumulatorBytes ? 1 : 0;
    if (!sh.gather) sh.cap = 0;
  }
}

template <bool ORBITS, int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED, int PH,
          bool SPLIT>
cudaError_t launch_shape(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                         const SpaceTiles& st, const RegularRule& rule, const RegularArgs& a,
                         Shape sh, cudaStream_t stream) {
  constexpr int kPer = SPLIT ? 1 : kWarps;
  sh.nsup = (sh.ntt + kPer - 1) / kPer;
  const long long units = a.symmetric
                              ? lower_group_count(sh.nsup, kPer, sh.ty0, sh.ty1)
                              : static_cast<long long>(sh.nsup) * (sh.ty1 - sh.ty0);
  const long long blocks = units * (kTile / sh.ns);
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  if (blocks <= 0) return cudaSuccess;
  set_accumulator<KER, NBS, DIRECT, PAIRED>(sh, tt, st);
  const Layout L = layout<ORBITS, KER, OP, NBT, NBS, DIRECT, PAIRED, SPLIT>(
      rule.npts, sh.ns, sh.gather, sh.cap, a.symmetric);
  auto fn = regular_fp64<ORBITS, KER, OP, NBT, NBS, DIRECT, PAIRED, PH, SPLIT>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(L.total));
  if (e != cudaSuccess) {
    cudaGetLastError();  // not sticky: clear it, so that it is not reported by a later launch
    return e;
  }
  unsigned* timeouts = nullptr;
  int polls = 0;
  if ((e = stage_wait_state(&timeouts, &polls)) != cudaSuccess) return e;
  typename RuleOf<ORBITS>::type r;
  if constexpr (ORBITS)
    r = orbit_rule(rule);
  else
    r = point_rule(rule);
  fn<<<static_cast<unsigned>(blocks), kThreads, L.total, stream>>>(
      test, tt, trial, st, r, a.k, a.same_grid, static_cast<double*>(a.out), a.ld, sh, a.symmetric,
      PAIRED && a.op == kADL ? 1 : 0, timeouts, polls);
  return cudaGetLastError();
}

// Trial cells per CTA of the 6-point rule's kernels (`tiles`: CTAs that whole tiles would take).
// A CTA costs its staging, incidence and flush (about `fixed` trial cells' time per wave of
// the CTAs that an SM holds, and the adds of its block); a trial cell costs one unit per CTA
// on the SM, but not less than four (one warp's latency), a fifth more where it adds directly, and
// two thirds more where one CTA fills the SM's shared memory (a torus of 20,480 triangles in rows,
// 34 DOFs per tile, Helmholtz double layer P1, k = 8: chunks of sixteen 63.9 ms, of eight 42.7).
// The least estimate, longer chunks on ties.  B200, shorter chunks until 888 CTAs -> this: 640 triangles, one space, Laplace double
// layer P1 53 -> 35 us, single layer DP0 27 -> 19; 1,280: double layer 91 -> 77; two bodies of
// 800 and 700, hypersingular 46 -> 41; Helmholtz, k = 10: 1,280 hypersingular 168 -> 142, two
// bodies double layer 156 -> 123.
template <int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED>
inline int orbit_chunk(long long tiles, Shape sh, const SpaceTiles& tt, const SpaceTiles& st,
                       int npts, int symmetric) {
  constexpr bool kC = KER == kHelmholtz;
  const long long fixed = (DIRECT ? 5 : 10) / (kC ? 2 : 1), adds = DIRECT ? 0 : kC ? 1 : 2;
  int best = kChunk;
  long long least = 0;
  for (int ns = kChunk; ns >= 1; ns /= 2) {
    sh.ns = ns;
    set_accumulator<KER, NBS, DIRECT, PAIRED>(sh, tt, st);
    const size_t smem = layout<true, KER, OP, NBT, NBS, DIRECT, PAIRED, false>(
                            npts, ns, sh.gather, sh.cap, symmetric).total + 1024;
    const long long resident = std::max<long long>(
        1, std::min<long long>(min_ctas<true, KER, OP, NBT, NBS, PAIRED>(), (size_t(227) << 10) / smem));
    const long long n = (tiles * (kTile / ns) + kSMs - 1) / kSMs;  // CTAs of the fullest SM
    const bool direct_adds = !DIRECT && !sh.gather;
    const long long cells = ns * std::max(4LL, n) * (direct_adds ? 6 : 5) / 5 * (resident == 1 && n > 1 ? 5 : 3) / 3;
    const long long cost = (n + resident - 1) / resident * fixed + (direct_adds ? 0 : n * adds) + cells;
    if (ns == kChunk || cost < least) {
      least = cost;
      best = ns;
    }
  }
  return best;
}

template <bool ORBITS, int KER, int OP, int NBT, int NBS, bool DIRECT, bool PAIRED, int PH>
cudaError_t launch_one(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                       const SpaceTiles& st, const RegularRule& rule, const RegularArgs& a,
                       cudaStream_t stream) {
  const int trial_tiles = (trial.ncells + kTile - 1) / kTile;
  if (a.trial_tile0 < 0 || a.trial_tile0 > trial_tiles || a.trial_tiles < 0)
    return cudaErrorInvalidValue;
  const int ny = a.trial_tiles > 0 ? std::min(a.trial_tiles, trial_tiles - a.trial_tile0)
                                   : trial_tiles - a.trial_tile0;
  if (ny <= 0) return cudaSuccess;
  Shape sh{};
  sh.ntt = (test.ncells + kTile - 1) / kTile;
  sh.ty0 = a.trial_tile0;
  sh.ty1 = a.trial_tile0 + ny;
  long long tiles = static_cast<long long>((sh.ntt + kWarps - 1) / kWarps) * ny;
  if (a.symmetric) tiles = (tiles + 1) / 2;
  sh.ns = kChunk;
  if constexpr (ORBITS)
    sh.ns = orbit_chunk<KER, OP, NBT, NBS, DIRECT, PAIRED>(tiles, sh, tt, st, rule.npts, a.symmetric);
  else  // shorter chunks until the chip has about three CTAs per SM twice over
    while (sh.ns > 1 && tiles * (kTile / sh.ns) < 6 * kSMs) sh.ns /= 2;
  if constexpr (!ORBITS) {
    // still too few warps: the rule's test points over the four warps of a CTA
    if (tiles * (kTile / sh.ns) < 2 * kSMs && rule.npts >= 12) {
      return launch_shape<ORBITS, KER, OP, NBT, NBS, DIRECT, PAIRED, PH, true>(
          test, tt, trial, st, rule, a, sh, stream);
    }
  }
  return launch_shape<ORBITS, KER, OP, NBT, NBS, DIRECT, PAIRED, PH, false>(
      test, tt, trial, st, rule, a, sh, stream);
}

template <bool ORBITS, int KER, int OP, int PH>
cudaError_t launch_spaces(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                          const SpaceTiles& st, const RegularRule& rule, const RegularArgs& a,
                          cudaStream_t stream, bool direct) {
  if (a.symmetric == 2) {
    if constexpr (OP == kDL) {
      if (direct || tt.nbasis != 3 || st.nbasis != 3) return cudaErrorInvalidValue;
      return launch_one<ORBITS, KER, OP, 3, 3, false, true, PH>(test, tt, trial, st, rule, a, stream);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  if constexpr (OP != kHS) {
    if (direct)
      return launch_one<ORBITS, KER, OP, 1, 1, true, false, PH>(test, tt, trial, st, rule, a, stream);
  }
  if (direct) return cudaErrorInvalidValue;
  if (tt.nbasis == 3 && st.nbasis == 3)
    return launch_one<ORBITS, KER, OP, 3, 3, false, false, PH>(test, tt, trial, st, rule, a, stream);
  if constexpr (OP == kHS && KER == kLaplace) {
    // piecewise constants have no curl: nothing to add to the zeroed output
    return tt.nbasis <= 3 && st.nbasis <= 3 ? cudaSuccess : cudaErrorInvalidValue;
  } else {
    if (tt.nbasis == 1 && st.nbasis == 1)
      return launch_one<ORBITS, KER, OP, 1, 1, false, false, PH>(test, tt, trial, st, rule, a, stream);
    if (tt.nbasis == 1 && st.nbasis == 3)
      return launch_one<ORBITS, KER, OP, 1, 3, false, false, PH>(test, tt, trial, st, rule, a, stream);
    if (tt.nbasis == 3 && st.nbasis == 1)
      return launch_one<ORBITS, KER, OP, 3, 1, false, false, PH>(test, tt, trial, st, rule, a, stream);
    return cudaErrorInvalidValue;
  }
}

template <bool ORBITS, int KER, int PH>
cudaError_t launch_op(const CellSet& test, const SpaceTiles& tt, const CellSet& trial,
                      const SpaceTiles& st, const RegularRule& rule, const RegularArgs& a,
                      cudaStream_t stream, bool direct) {
  if (a.symmetric == 2 && (a.op == kDL || a.op == kADL))  // one kernel, its blocks swapped
    return launch_spaces<ORBITS, KER, kDL, PH>(test, tt, trial, st, rule, a, stream, direct);
  switch (a.op) {
    case kSL: return launch_spaces<ORBITS, KER, kSL, PH>(test, tt, trial, st, rule, a, stream, direct);
    case kDL: return launch_spaces<ORBITS, KER, kDL, PH>(test, tt, trial, st, rule, a, stream, direct);
    case kADL: return launch_spaces<ORBITS, KER, kADL, PH>(test, tt, trial, st, rule, a, stream, direct);
    case kHS: return launch_spaces<ORBITS, KER, kHS, PH>(test, tt, trial, st, rule, a, stream, direct);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fp64
}  // namespace bempp_b200
