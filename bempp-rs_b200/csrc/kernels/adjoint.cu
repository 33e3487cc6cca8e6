// Adjoint gradient of J = Re(lambda^H A(x, k) mu) for the Helmholtz single-layer operator
// on DP0 x DP0, with respect to every vertex coordinate and the wavenumber, without
// forming dA.
//
// A_ij = (1/4pi) jdet_i jdet_j sum_n w_n e^{ik r_n} / r_n over the rule of the pair
// (regular tensor rule, or the Duffy rule of an adjacent pair), r_n = |x_n - y_n| with
// x_n = sum_a phi_a(xi_n) V_{i,a} and y_n = sum_b phi_b(eta_n) V_{j,b} (phi the P1
// barycentric weights, V the cell vertices).  The discrete sum is differentiated
// exactly:
//   dA_ij/dV_{i,a} = (1/4pi) [ djdet_i/dV_a jdet_j sum_n w_n G_n
//                              + jdet_i jdet_j sum_n w_n phi_a(xi_n) grad_x G_n ],
//   grad_x (e^{ikr}/r) = e^{ikr} (ikr - 1) (x - y) / r^3,  grad_y = -grad_x,
//   djdet/dV1 = t1 x n, djdet/dV2 = n x t0, djdet/dV0 = -(t1 x n + n x t0),
//   dA_ij/dk = (1/4pi) jdet_i jdet_j sum_n w_n i e^{ikr_n}.
// Each pair contributes Re(conj(lambda_i) mu_j dA_ij) to 9 + 9 vertex coordinates of
// its two cells and to dJ/dk; contributions are reduced per CTA (test side in
// registers and shared memory, trial side by warp shuffles) and added per cell, then a
// last kernel scatters the per-cell-vertex gradients to the vertices.
//
// Regular pairs use 32 x 32 cell tiles (lane = test cell, both tiles staged in shared memory
// by TMA bulk copies on an mbarrier with the regular kernels' bounded wait and timeout
// counter); adjacent pairs use eight threads per pair over their Duffy rule.  FP64 with the
// 6-point rule: adjoint_sl_orbits.  Other rules in FP64: adjoint_sl_regular.  Mixed:
// far pairs (centroid distance >= 2 diameters) in FP32 with centroid-relative points and
// the reference phase e^{ik r0} folded into the pair weight, as in regular.cu.
#include <type_traits>

#include "regular_fp64.cuh"

namespace bempp_b200 {
namespace {

using namespace tiles;

// d jdet / d V_a of a flat cell, a = 0, 1, 2 (3-vectors)
__device__ __forceinline__ void jdet_gradient(const double t0[3], const double t1[3],
                                              const double n[3], double g[3][3]) {
  const double a[3] = {t1[1] * n[2] - t1[2] * n[1], t1[2] * n[0] - t1[0] * n[2],
                       t1[0] * n[1] - t1[1] * n[0]};  // t1 x n
  const double b[3] = {n[1] * t0[2] - n[2] * t0[1], n[2] * t0[0] - n[0] * t0[2],
                       n[0] * t0[1] - n[1] * t0[0]};  // n x t0
  for (int d = 0; d < 3; ++d) {
    g[1][d] = a[d];
    g[2][d] = b[d];
    g[0][d] = -(a[d] + b[d]);
  }
}

template <int QT, bool MIXED>
__global__ void __launch_bounds__(kThreads, 3)
    adjoint_sl_regular(CellSet cs, RegularRule rule, double k, const double2* __restrict__ lam,
                       const double2* __restrict__ mu, double* __restrict__ grad_cell,
                       double* __restrict__ totals, unsigned* __restrict__ stage_timeouts,
                       int stage_polls) {
  const int Q = QT > 0 ? QT : rule.npts;
  // A_ij = A_ji on far pairs (one cell set and one rule on both sides), so only tile pairs
  // tx >= sy are visited; an off-diagonal tile takes c_ij + c_ji for both orders of its pairs
  int tx, sy;
  const int ntt = (cs.ncells + kTile - 1) / kTile;
  lower_tile_pair(blockIdx.x, ntt, 0, ntt, tx, sy);
  const bool both = tx > sy;
  const int ti0 = tx * kTile, sj0 = sy * kTile;
  const int nti = min(kTile, cs.ncells - ti0), nsj = min(kTile, cs.ncells - sj0);
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);  // completion of the tile copies
  unsigned char* cursor = smem + 16;
  const Tile T = carve_tile(cursor, Q, MIXED, 1);
  const Tile S = carve_tile(cursor, Q, MIXED, 1);
  double* s_test = reinterpret_cast<double*>(cursor);  // [kTile][9] test-cell gradients
  double* s_trial = s_test + kTile * 9;                // [kTile][9] trial-cell gradients
  double* s_tot = s_trial + kTile * 9;                 // J, dJ/dk
  // both tiles by bulk (TMA) copies on one mbarrier, issued by one thread, while the
  // others clear the gradient accumulators
  if (threadIdx.x == 0) mbar_init(mbar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(mbar, 2 * bulk_tile_bytes(Q, MIXED));
    stage_tile_bulk(T, cs, ti0, Q, MIXED, mbar);
    stage_tile_bulk(S, cs, sj0, Q, MIXED, mbar);
  }
  for (int e = threadIdx.x; e < 2 * kTile * 9 + 2; e += kThreads) s_test[e] = 0.0;
  const bool staged = mbar_wait_bounded(mbar, 0, stage_polls);
  if (__syncthreads_or(!staged)) {
    // the copies did not complete in time: record it, give them a last bounded wait and
    // add nothing (the host reports the failure)
    if (threadIdx.x == 0) atomicAdd(stage_timeouts, 1u);
    mbar_wait_bounded(mbar, 0);
    return;
  }

  const int it = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool valid = it < nti;
  const double2 li = valid ? lam[ti0 + it] : make_double2(0.0, 0.0);
  const double2 mi = valid && both ? mu[ti0 + it] : make_double2(0.0, 0.0);
  const int a0 = T.vid[it], a1 = T.vid[kTile + it], a2 = T.vid[2 * kTile + it];
  const double jdet_i = T.G(fJdet, it);

  double gt[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};  // test-cell vertex gradients
  double jval = 0.0, dk = 0.0;
  for (int js = warp; js < nsj; js += kWarps) {
    const bool adjacent = share_vertex(a0, a1, a2, S.vid[js], S.vid[kTile + js],
                                       S.vid[2 * kTile + js]);
    const bool active = valid && !adjacent;
    // c = conj(lambda_i) mu_j (+ conj(lambda_j) mu_i off the diagonal)
    const double2 mj = mu[sj0 + js];
    double c_re = li.x * mj.x + li.y * mj.y, c_im = li.x * mj.y - li.y * mj.x;
    if (both) {
      const double2 lj = lam[sj0 + js];
      c_re += lj.x * mi.x + lj.y * mi.y;
      c_im += lj.x * mi.y - lj.y * mi.x;
    }
    double S0_re = 0.0, S0_im = 0.0, Sk_re = 0.0, Sk_im = 0.0;
    double uq[QT > 0 ? QT : kMaxRegularPoints][3];
#pragma unroll
    for (int q = 0; q < Q; ++q) uq[q][0] = uq[q][1] = uq[q][2] = 0.0;
    double vt[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    bool far = false;
    if (MIXED && active) {
      const double dcx = T.G(fCx, it) - S.G(fCx, js), dcy = T.G(fCy, it) - S.G(fCy, js),
                   dcz = T.G(fCz, it) - S.G(fCz, js);
      const double dist2 = dcx * dcx + dcy * dcy + dcz * dcz;
      const double lim = 2.0 * fmax(T.G(fDiam, it), S.G(fDiam, js));
      far = dist2 >= lim * lim;
      if (far) {
        // FP32 far pair: centroid-relative points, reference phase folded into the weight
        // c' = c e^{ik r0}, e^{ik r} = e^{ik r0} e^{ik (r - r0)}, r - r0 = s / (r + r0).
        const float fdx = static_cast<float>(dcx), fdy = static_cast<float>(dcy),
                    fdz = static_cast<float>(dcz);
        const double r0 = sqrt(dist2);
        const float r0f = static_cast<float>(r0), r0sq = r0f * r0f, kf = static_cast<float>(k);
        float pc, ps;
        phase_cos_sin(k * r0, pc, ps);
        const float cr = static_cast<float>(c_re * pc - c_im * ps);
        const float ci = static_cast<float>(c_re * ps + c_im * pc);
        const bool taylor = fabs(k) * (T.G(fRad, it) + S.G(fRad, js)) <= 0.8;
        float fS0r = 0.f, fS0i = 0.f, fSkr = 0.f, fSki = 0.f;
        float fuq[QT > 0 ? QT : kMaxRegularPoints][3];
        float fvt[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
        for (int q = 0; q < Q; ++q) fuq[q][0] = fuq[q][1] = fuq[q][2] = 0.f;
#pragma unroll 1
        for (int p = 0; p < Q; ++p) {
          const float ax = T.R(p, 0, it), ay = T.R(p, 1, it), az = T.R(p, 2, it);
          const float alpha = 2.f * fmaf(fdx, ax, fmaf(fdy, ay, fdz * az));
          const float px = fdx + ax, py = fdy + ay, pz = fdz + az;
          float vp0 = 0.f, vp1 = 0.f, vp2 = 0.f, gr = 0.f, gi = 0.f, er = 0.f, ei = 0.f;
          const float wp = rule.wf[p];
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const float yx = S.R(q, 0, js), yy = S.R(q, 1, js), yz = S.R(q, 2, js);
            const float Dx = ax - yx, Dy = ay - yy, Dz = az - yz;
            const float beta = 2.f * fmaf(fdx, yx, fmaf(fdy, yy, fdz * yz));
            const float sq = (alpha - beta) + fmaf(Dx, Dx, fmaf(Dy, Dy, Dz * Dz));
            const float r2 = r0sq + sq;
            const float rinv = rsqrt_approx(r2);
            const float r = r2 * rinv, kr = kf * r;
            const float t = kf * sq * rcp_approx(r + r0f);
            float csn, sn;
            if (taylor)
              poly_cos_sin(t, csn, sn);
            else
              reduced_cos_sin(t, csn, sn);
            const float wq = rule.wf[q];
            gr = fmaf(wq * rinv, csn, gr);
            gi = fmaf(wq * rinv, sn, gi);
            er = fmaf(wq, csn, er);
            ei = fmaf(wq, sn, ei);
            const float f_re = -csn - kr * sn, f_im = kr * csn - sn;
            const float gs = wq * (cr * f_re - ci * f_im) * (rinv * rinv * rinv);
            const float dx = px - yx, dy = py - yy, dz = pz - yz;
            vp0 = fmaf(gs, dx, vp0);
            vp1 = fmaf(gs, dy, vp1);
            vp2 = fmaf(gs, dz, vp2);
            const float wgs = wp * gs;
            fuq[q][0] = fmaf(wgs, dx, fuq[q][0]);
            fuq[q][1] = fmaf(wgs, dy, fuq[q][1]);
            fuq[q][2] = fmaf(wgs, dz, fuq[q][2]);
          }
          fS0r = fmaf(wp, gr, fS0r);
          fS0i = fmaf(wp, gi, fS0i);
          fSkr = fmaf(wp, er, fSkr);
          fSki = fmaf(wp, ei, fSki);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const float f = wp * rule.phif[a][p];
            fvt[a][0] = fmaf(f, vp0, fvt[a][0]);
            fvt[a][1] = fmaf(f, vp1, fvt[a][1]);
            fvt[a][2] = fmaf(f, vp2, fvt[a][2]);
          }
        }
        // back to FP64; S0 and Sk pick up e^{ik r0} through c' in R0 and dk below, so
        // express them relative to the original c by rotating: S = e^{ik r0} S'.
        S0_re = static_cast<double>(fS0r) * pc - static_cast<double>(fS0i) * ps;
        S0_im = static_cast<double>(fS0r) * ps + static_cast<double>(fS0i) * pc;
        Sk_re = static_cast<double>(fSkr) * pc - static_cast<double>(fSki) * ps;
        Sk_im = static_cast<double>(fSkr) * ps + static_cast<double>(fSki) * pc;
#pragma unroll
        for (int q = 0; q < Q; ++q)
          for (int d = 0; d < 3; ++d) uq[q][d] = fuq[q][d];
        for (int a = 0; a < 3; ++a)
          for (int d = 0; d < 3; ++d) vt[a][d] = fvt[a][d];
      }
    }
    if (active && !far) {
      // e^{ikr} referenced to the pair (e^{ik r0} e^{ik (r - r0)}, r0 = |c_x - c_y|) when
      // k (rad_x + rad_y) <= 0.8 bounds every phase k (r - r0): c is rotated by e^{ik r0}
      // for the gradient terms and the sums S0, Sk are rotated back after the loop
      const bool ref = fabs(k) * (T.G(fRad, it) + S.G(fRad, js)) <= 0.8;
      double kr0 = 0.0, pc = 1.0, ps = 0.0, cq_re = c_re, cq_im = c_im;
      if (ref) {
        const double dcx = T.G(fCx, it) - S.G(fCx, js), dcy = T.G(fCy, it) - S.G(fCy, js),
                     dcz = T.G(fCz, it) - S.G(fCz, js);
        const double r0sq = dcx * dcx + dcy * dcy + dcz * dcz;
        kr0 = k * (r0sq * rsqrt_refined(r0sq));
        sincos_cw(kr0, ps, pc);
        cq_re = c_re * pc - c_im * ps;
        cq_im = c_re * ps + c_im * pc;
      }
#pragma unroll 1
      for (int p = 0; p < Q; ++p) {
        const double x0 = T.P(p, 0, it), x1 = T.P(p, 1, it), x2 = T.P(p, 2, it);
        double vp[3] = {0.0, 0.0, 0.0};
        double g_re = 0.0, g_im = 0.0, e_re = 0.0, e_im = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const double dx = x0 - S.P(q, 0, js), dy = x1 - S.P(q, 1, js), dz = x2 - S.P(q, 2, js);
          const double r2 = dx * dx + dy * dy + dz * dz;
          const double rinv = rsqrt_refined(r2);
          const double r = r2 * rinv, kr = k * r;
          double sn, csn;
          if (ref)
            sincos_small(fma(k, r, -kr0), sn, csn);
          else
            sincos(kr, &sn, &csn);
          const double wq = rule.w[q];
          g_re = fma(wq * rinv, csn, g_re);
          g_im = fma(wq * rinv, sn, g_im);
          e_re = fma(wq, csn, e_re);
          e_im = fma(wq, sn, e_im);
          // Re(c e^{ikr} (ikr - 1)) / r^3
          const double f_re = -csn - kr * sn, f_im = kr * csn - sn;
          const double gs = wq * (cq_re * f_re - cq_im * f_im) * rinv * rinv * rinv;
          vp[0] = fma(gs, dx, vp[0]);
          vp[1] = fma(gs, dy, vp[1]);
          vp[2] = fma(gs, dz, vp[2]);
          const double wgs = rule.w[p] * gs;
          uq[q][0] = fma(wgs, dx, uq[q][0]);
          uq[q][1] = fma(wgs, dy, uq[q][1]);
          uq[q][2] = fma(wgs, dz, uq[q][2]);
        }
        const double wp = rule.w[p];
        S0_re = fma(wp, g_re, S0_re);
        S0_im = fma(wp, g_im, S0_im);
        Sk_re = fma(wp, e_re, Sk_re);
        Sk_im = fma(wp, e_im, Sk_im);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double f = wp * rule.phi[a][p];
          vt[a][0] = fma(f, vp[0], vt[a][0]);
          vt[a][1] = fma(f, vp[1], vt[a][1]);
          vt[a][2] = fma(f, vp[2], vt[a][2]);
        }
      }
      if (ref) {
        const double s0r = S0_re * pc - S0_im * ps, s0i = S0_re * ps + S0_im * pc;
        const double skr = Sk_re * pc - Sk_im * ps, ski = Sk_re * ps + Sk_im * pc;
        S0_re = s0r;
        S0_im = s0i;
        Sk_re = skr;
        Sk_im = ski;
      }
    }
    const double jdet_j = S.G(fJdet, js);
    const double jj = jdet_i * jdet_j * kInv4Pi;
    const double R0 = c_re * S0_re - c_im * S0_im;  // Re(c S0)
    // trial-side contributions of this lane, then a warp reduction over the test cells
    double gs_[3][3];
    {
      double tj_t0[3], tj_t1[3], tj_n[3], djj[3][3];
      for (int d = 0; d < 3; ++d) {
        tj_t0[d] = S.G(fT0x + d, js);
        tj_t1[d] = S.G(fT1x + d, js);
      }
      tj_n[0] = S.G(fNx, js);
      tj_n[1] = S.G(fNy, js);
      tj_n[2] = S.G(fNz, js);
      jdet_gradient(tj_t0, tj_t1, tj_n, djj);
      const double rj = R0 * jdet_i * kInv4Pi;
#pragma unroll
      for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double acc = 0.0;
#pragma unroll
          for (int q = 0; q < Q; ++q) acc = fma(rule.phi[b][q], uq[q][d], acc);
          gs_[b][d] = active ? (-jj * acc + rj * djj[b][d]) : 0.0;
        }
    }
#pragma unroll
    for (int e = 0; e < 9; ++e) {
      double v = gs_[e / 3][e % 3];
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
      if (it == 0) s_trial[js * 9 + e] += v;  // each js belongs to one warp
    }
    if (active) {
      double ti_t0[3], ti_t1[3], ti_n[3], dji[3][3];
      for (int d = 0; d < 3; ++d) {
        ti_t0[d] = T.G(fT0x + d, it);
        ti_t1[d] = T.G(fT1x + d, it);
      }
      ti_n[0] = T.G(fNx, it);
      ti_n[1] = T.G(fNy, it);
      ti_n[2] = T.G(fNz, it);
      jdet_gradient(ti_t0, ti_t1, ti_n, dji);
      const double ri = R0 * jdet_j * kInv4Pi;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int d = 0; d < 3; ++d) gt[a][d] += jj * vt[a][d] + ri * dji[a][d];
      jval += R0 * jj;
      dk += (c_re * (-Sk_im) - c_im * Sk_re) * jj;  // Re(c i Sk)
    }
  }
  if (valid) {
#pragma unroll
    for (int e = 0; e < 9; ++e) atomicAdd(s_test + it * 9 + e, gt[e / 3][e % 3]);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    jval += __shfl_xor_sync(0xffffffffu, jval, s);
    dk += __shfl_xor_sync(0xffffffffu, dk, s);
  }
  if (it == 0) {
    atomicAdd(s_tot, jval);
    atomicAdd(s_tot + 1, dk);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kTile * 9; e += kThreads) {
    const int c = e / 9;
    if (c < nti) atomicAdd(grad_cell + static_cast<int64_t>(ti0 + c) * 9 + (e % 9), s_test[e]);
    if (c < nsj) atomicAdd(grad_cell + static_cast<int64_t>(sj0 + c) * 9 + (e % 9), s_trial[e]);
  }
  if (threadIdx.x == 0) {
    atomicAdd(totals, s_tot[0]);
    atomicAdd(totals + 1, s_tot[1]);
  }
}

// The regular pairs in FP64 with the 6-point rule, on the distances and kernel values of
// regular_fp64.cuh (registers only, two operations per squared distance).  With
// x_p = c + gamma_p g_a, y_q = c' + gamma_q g'_b and the scalars
//   h_pq = Re(c e^{ikr} (ikr - 1)) / r^3,
// every vector sum of h_pq (x_p - y_q) is a combination of dc and the g's with scalar
// coefficients: row sums R_p = sum_q w_q h_pq, column sums, and G_pb = sum over the trial
// orbits of w gamma h.  So the loop over point pairs keeps scalars (about 5 operations per
// pair for all sums, where accumulating the vectors per test and per trial point took 8 and
// the differences 3 more) and the vectors are formed once per cell pair.  Pairs nearly in
// contact (close_pair; the combinations above lose eps H / r there, as differences of
// coordinates do) are left to a second pass, CLOSE, that takes the squared distances from the
// components of x_p - y_q: in one loop with the others they cost 200 bytes of spills.
// Returns whether the lane has such pairs.
// The largest circumradii of the two tiles decide between the phase referenced to the pair and
// the reduced phase.  5,120 triangles, k = 5, B200: 3.3 ms with coordinate differences,
// 1.97 in this form.
template <int PH, bool CLOSE>
__device__ __forceinline__ bool adjoint_orbit_pairs(
    const Tile& T, const Tile& S, int it, int warp, int ti0, int sj0, int nti, int nsj, bool both,
    const fp64::OrbitRule& rule, double k, const double2* __restrict__ lam,
    const double2* __restrict__ mu, const double* jx, const double* jy, double* s_test,
    double* s_trial, double& jval, double& dk) {
  using namespace fp64;
  const bool valid = it < nti;
  const double2 li = valid ? lam[ti0 + it] : make_double2(0.0, 0.0);
  const double2 mi = valid && both ? mu[ti0 + it] : make_double2(0.0, 0.0);
  const int a0 = T.vid[it], a1 = T.vid[kTile + it], a2 = T.vid[2 * kTile + it];
  double* mine = s_test + warp * 9 * kTile + it;
  bool found = false;
#pragma unroll 1
  for (int js = warp; js < nsj; js += kWarps) {
    const bool regular = valid && !share_vertex(a0, a1, a2, S.vid[js], S.vid[kTile + js],
                                                S.vid[2 * kTile + js]);
    PairGeometry p;
    pair_geometry<kHelmholtz, kSL, 1, 1, false>(T, it, S, js, 1.0, p);
    const bool close = regular && close_pair(p, T.G(rR, it) + S.G(rR, js), rule.reach);
    const bool active = CLOSE ? close : regular && !close;
    found = found || close;
    if (CLOSE && !__any_sync(0xffffffffu, active)) continue;
    // c = conj(lambda_i) mu_j (+ conj(lambda_j) mu_i off the diagonal)
    const double2 mj = mu[sj0 + js];
    double c_re = li.x * mj.x + li.y * mj.y, c_im = li.x * mj.y - li.y * mj.x;
    if (both) {
      const double2 lj = lam[sj0 + js];
      c_re += lj.x * mi.x + lj.y * mi.y;
      c_im += lj.x * mi.y - lj.y * mi.x;
    }
    // phase referenced to the pair: c is rotated by e^{ik r0} for the gradient terms, the
    // sums S0, Sk after the loop
    double kr0 = 0.0, pc = 1.0, ps = 0.0, q_re = c_re, q_im = c_im;
    if (PH == kReferenced) {
      kr0 = k * (p.r0 * rsqrt_refined(p.r0));
      sincos_any(kr0, ps, pc);
      q_re = c_re * pc - c_im * ps;
      q_im = c_re * ps + c_im * pc;
    }
    double M[3][3], Y[2][3];
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
    const double dgy[3] = {p.dgy0, p.dgy1, -(p.dgy0 + p.dgy1)};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double e = S.G(rE + b, js);
#pragma unroll
      for (int o = 0; o < 2; ++o) Y[o][b] = fma(rule.g2[o], e, -2.0 * rule.g[o] * dgy[b]);
    }
    double S0_re = 0.0, S0_im = 0.0, Sk_re = 0.0, Sk_im = 0.0;
    // sums of h: columns (times the test weight), w phi_a w gamma by (test, trial vertex),
    // and the row sums' combinations
    double col[2][3] = {{0, 0, 0}, {0, 0, 0}}, Cd[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double cC[3] = {0, 0, 0}, Db[3] = {0, 0, 0}, Ad[3] = {0, 0, 0}, cA = 0.0;
    double BR[3] = {0, 0, 0}, BD[3] = {0, 0, 0};
#pragma unroll 1
    for (int op = 0; op < 2; ++op) {
      const double gp = rule.g[op], g2 = rule.g2[op], wp = rule.w[op], cp = rule.c[op],
                   dp = rule.d[op], m0 = rule.m[op][0], m1 = rule.m[op][1];
      double s0r[2] = {0, 0}, s0i[2] = {0, 0}, skr[2] = {0, 0}, ski[2] = {0, 0};
      double sumG[3] = {0, 0, 0}, sumR = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double X = fma(g2, T.G(rE + a, it), fma(2.0 * gp, dgx[a], p.r0));
        double h[6];
        {
          double r2[6], y[6], t[6], kr[6], sn[6], csn[6];
#pragma unroll
          for (int i = 0; i < 6; ++i) r2[i] = X + Y[i / 3][i % 3];
#pragma unroll
          for (int i = 0; i < 6; ++i) r2[i] = fma(i < 3 ? m0 : m1, M[a][i % 3], r2[i]);
          if (CLOSE) {
#pragma unroll
            for (int i = 0; i < 6; ++i) r2[i] = 0.0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const double g0 = T.G(rG0 + d, it), g1 = T.G(rG1 + d, it), u0 = S.G(rG0 + d, js), u1 = S.G(rG1 + d, js);
              const double x = fma(gp, a == 0 ? g0 : a == 1 ? g1 : -(g0 + g1),
                                   (T.G(rC + d, it) - S.G(rC + d, js)) + (T.G(rL + d, it) - S.G(rL + d, js)));
#pragma unroll
              for (int i = 0; i < 6; ++i) {
                const double e = fma(-rule.g[i / 3], i % 3 == 0 ? u0 : i % 3 == 1 ? u1 : -(u0 + u1), x);
                r2[i] = fma(e, e, r2[i]);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 6; ++i) y[i] = rsqrt_refined(r2[i]);
#pragma unroll
          for (int i = 0; i < 6; ++i) kr[i] = k * (r2[i] * y[i]);
          if (PH == kReferenced) {
#pragma unroll
            for (int i = 0; i < 6; ++i) t[i] = kr[i] - kr0;
            sincos_small_n<6>(t, sn, csn);
          } else {
            sincos_any_n<6>(kr, sn, csn);
          }
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            s0r[i / 3] = fma(y[i], csn[i], s0r[i / 3]);
            s0i[i / 3] = fma(y[i], sn[i], s0i[i / 3]);
            skr[i / 3] += csn[i];
            ski[i / 3] += sn[i];
          }
          // Re(q e^{ikr} (ikr - 1)) / r^3
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            const double fr = fma(kr[i], sn[i], csn[i]), fi = fma(kr[i], csn[i], -sn[i]);
            h[i] = -(fma(q_im, fi, q_re * fr)) * (y[i] * y[i] * y[i]);
          }
        }
        const double sum0 = (h[0] + h[1]) + h[2], sum1 = (h[3] + h[4]) + h[5];
        const double R = fma(rule.w[1], sum1, rule.w[0] * sum0);
        const double base = fma(rule.c[1], sum1, rule.c[0] * sum0);
        sumR += R;
        Ad[a] = fma(dp, R, Ad[a]);
        BR[a] = fma(gp * cp, R, BR[a]);
        BD[a] = fma(gp * dp, R, BD[a]);
        Db[a] = fma(dp, base, Db[a]);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const double G = fma(rule.d[1], h[3 + b], rule.d[0] * h[b]);
          Cd[a][b] = fma(dp, G, Cd[a][b]);
          sumG[b] += G;
          col[0][b] = fma(wp, h[b], col[0][b]);
          col[1][b] = fma(wp, h[3 + b], col[1][b]);
        }
      }
      cA = fma(cp, sumR, cA);
#pragma unroll
      for (int b = 0; b < 3; ++b) cC[b] = fma(cp, sumG[b], cC[b]);
      S0_re = fma(wp, fma(rule.w[1], s0r[1], rule.w[0] * s0r[0]), S0_re);
      S0_im = fma(wp, fma(rule.w[1], s0i[1], rule.w[0] * s0i[0]), S0_im);
      Sk_re = fma(wp, fma(rule.w[1], skr[1], rule.w[0] * skr[0]), Sk_re);
      Sk_im = fma(wp, fma(rule.w[1], ski[1], rule.w[0] * ski[0]), Sk_im);
    }
    if (PH == kReferenced) {
      const double s0r = S0_re * pc - S0_im * ps, s0i = S0_re * ps + S0_im * pc;
      const double skr = Sk_re * pc - Sk_im * ps, ski = Sk_re * ps + Sk_im * pc;
      S0_re = s0r;
      S0_im = s0i;
      Sk_re = skr;
      Sk_im = ski;
    }
    const double jdet_i = T.G(rJ, it), jdet_j = S.G(rJ, js);
    const double jj = jdet_i * jdet_j * kInv4Pi;
    const double R0 = c_re * S0_re - c_im * S0_im;  // Re(c S0)
    const double ri = R0 * jdet_j * kInv4Pi, rj = R0 * jdet_i * kInv4Pi;
    // column combinations of the trial side: w phi_b and w phi_b gamma
    const double k0 = (col[0][0] + col[0][1]) + col[0][2], k1 = (col[1][0] + col[1][1]) + col[1][2];
    const double cB = fma(rule.c[1], k1, rule.c[0] * k0);
    double Bd[3], Tb[3], Td[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      Bd[b] = cB + fma(rule.d[1], col[1][b], rule.d[0] * col[0][b]);
      Tb[b] = fma(rule.g[1] * rule.c[1], col[1][b], rule.g[0] * rule.c[0] * col[0][b]);
      Td[b] = fma(rule.g[1] * rule.d[1], col[1][b], rule.g[0] * rule.d[0] * col[0][b]);
    }
    double gs[9];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double dc = (T.G(rC + d, it) - S.G(rC + d, js)) + (T.G(rL + d, it) - S.G(rL + d, js));
      const double gx0 = T.G(rG0 + d, it), gx1 = T.G(rG1 + d, it), gy0 = S.G(rG0 + d, js), gy1 = S.G(rG1 + d, js);
      const double gx[3] = {gx0, gx1, -(gx0 + gx1)}, gy[3] = {gy0, gy1, -(gy0 + gy1)};
      const double vx = fma(gx0, BR[0] - BR[2], gx1 * (BR[1] - BR[2]));
      const double vy = fma(gy0, Tb[0] - Tb[2], gy1 * (Tb[1] - Tb[2]));
      // sum over q of the trial offsets with the c-part of the test basis
      const double wc = fma(gy0, cC[0] - cC[2], gy1 * (cC[1] - cC[2]));
      const double wb = fma(gx0, Db[0] - Db[2], gx1 * (Db[1] - Db[2]));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double C = fma(gy0, Cd[a][0] - Cd[a][2], gy1 * (Cd[a][1] - Cd[a][2]));
        const double vt = fma(dc, cA + Ad[a], vx) + fma(gx[a], BD[a], -(wc + C));
        if (active) mine[(3 * a + d) * kTile] += fma(jj, vt, ri * jx[(3 * a + d) * kTile + it]);
        const double D = fma(gx0, Cd[0][a] - Cd[2][a], gx1 * (Cd[1][a] - Cd[2][a]));
        const double ut = fma(dc, Bd[a], wb + D) - fma(gy[a], Td[a], vy);
        gs[3 * a + d] = active ? fma(-jj, ut, rj * jy[(3 * a + d) * kTile + js]) : 0.0;
      }
    }
    if (active) {
      jval = fma(R0, jj, jval);
      dk += (c_re * (-Sk_im) - c_im * Sk_re) * jj;  // Re(c i Sk)
    }
    // trial side: nine sums over the lanes; eight of them by halves (lane l ends with value
    // l / 4), 14 exchanges in place of 45
    double v4[4], v2[2], v1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool hi = it & 16;
      v4[i] = (hi ? gs[i + 4] : gs[i]) + __shfl_xor_sync(0xffffffffu, hi ? gs[i] : gs[i + 4], 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool hi = it & 8;
      v2[i] = (hi ? v4[i + 2] : v4[i]) + __shfl_xor_sync(0xffffffffu, hi ? v4[i] : v4[i + 2], 8);
    }
    {
      const bool hi = it & 4;
      v1 = (hi ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, hi ? v2[0] : v2[1], 4);
    }
    v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
    v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
    double v8 = gs[8];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v8 += __shfl_xor_sync(0xffffffffu, v8, s);
    if ((it & 3) == 0) s_trial[js * 9 + (it >> 2)] += v1;  // each js belongs to one warp
    if (it == 1) s_trial[js * 9 + 8] += v8;
  }
  return found;
}

__global__ void __launch_bounds__(kThreads, 2)
    adjoint_sl_orbits(CellSet cs, const __grid_constant__ fp64::OrbitRule rule, double k,
                      const double2* __restrict__ lam, const double2* __restrict__ mu,
                      double* __restrict__ grad_cell, double* __restrict__ totals,
                      unsigned* __restrict__ stage_timeouts, int stage_polls) {
  using namespace fp64;
  int tx, sy;
  const int ntt = (cs.ncells + kTile - 1) / kTile;
  lower_tile_pair(blockIdx.x, ntt, 0, ntt, tx, sy);
  const bool both = tx > sy;
  const int ti0 = tx * kTile, sj0 = sy * kTile;
  const int nti = min(kTile, cs.ncells - ti0), nsj = min(kTile, cs.ncells - sj0);
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);  // completion of the tile copies
  const Tile T = tile_at(smem + 16), S = tile_at(smem + 16 + kTileStride);
  double* jx = reinterpret_cast<double*>(smem + 16 + 2 * kTileStride);  // d jdet / d V, [e * kTile + c]
  double* jy = jx + 9 * kTile;
  double* s_test = jy + 9 * kTile;                   // [warp][9][kTile] test-cell gradients
  double* s_trial = s_test + kWarps * 9 * kTile;     // [kTile][9] trial-cell gradients
  double* s_tot = s_trial + kTile * 9;               // J, dJ/dk
  if (threadIdx.x == 0) mbar_init(mbar, 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(mbar, 2 * kStagedBytes);
    stage_geometry(T, cs, ti0, mbar);
    stage_geometry(S, cs, sj0, mbar);
  }
  for (int e = threadIdx.x; e < (kWarps + 1) * kTile * 9 + 2; e += kThreads) s_test[e] = 0.0;
  const bool staged = mbar_wait_bounded(mbar, 0, stage_polls);
  if (__syncthreads_or(!staged)) {
    // the copies did not complete in time: record it, give them a last bounded wait and
    // add nothing (the host reports the failure)
    if (threadIdx.x == 0) atomicAdd(stage_timeouts, 1u);
    mbar_wait_bounded(mbar, 0);
    return;
  }
  const int it = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // every phase k (r - r0) of the tile pair is at most k (largest rad_x + largest rad_y)
  bool referenced;
  {
    double rx = it < nti ? T.G(kRad, it) : 0.0, ry = it < nsj ? S.G(kRad, it) : 0.0;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      rx = fmax(rx, __shfl_xor_sync(0xffffffffu, rx, s));
      ry = fmax(ry, __shfl_xor_sync(0xffffffffu, ry, s));
    }
    referenced = fabs(k) * (rx + ry) <= 0.8;
  }
  __syncthreads();  // the rows of kRad change meaning below
  if (warp < 2) {
    const Tile& t = warp == 0 ? T : S;
    double t0[3], t1[3], n[3], dj[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      t0[d] = t.G(kT0x + d, it);
      t1[d] = t.G(kT1x + d, it);
      n[d] = t.G(kNx + d, it);
    }
    jdet_gradient(t0, t1, n, dj);
#pragma unroll
    for (int e = 0; e < 9; ++e) (warp == 0 ? jx : jy)[e * kTile + it] = dj[e / 3][e % 3];
    geometry_to_offsets(t, it, rule.reach);
  }
  __syncthreads();

  double jval = 0.0, dk = 0.0;
  const bool found =
      referenced ? adjoint_orbit_pairs<kReferenced, false>(T, S, it, warp, ti0, sj0, nti, nsj, both, rule, k,
                                                           lam, mu, jx, jy, s_test, s_trial, jval, dk)
                 : adjoint_orbit_pairs<kAnyPhase, false>(T, S, it, warp, ti0, sj0, nti, nsj, both, rule, k,
                                                         lam, mu, jx, jy, s_test, s_trial, jval, dk);
  if (__any_sync(0xffffffffu, found))
    adjoint_orbit_pairs<kAnyPhase, true>(T, S, it, warp, ti0, sj0, nti, nsj, both, rule, k, lam, mu, jx,
                                         jy, s_test, s_trial, jval, dk);
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    jval += __shfl_xor_sync(0xffffffffu, jval, s);
    dk += __shfl_xor_sync(0xffffffffu, dk, s);
  }
  if (it == 0) {
    atomicAdd(s_tot, jval);
    atomicAdd(s_tot + 1, dk);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kTile * 9; e += kThreads) {
    const int c = e / 9, f = e % 9;
    if (c < nti) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += s_test[(w * 9 + f) * kTile + c];
      atomicAdd(grad_cell + static_cast<int64_t>(ti0 + c) * 9 + f, v);
    }
    if (c < nsj) atomicAdd(grad_cell + static_cast<int64_t>(sj0 + c) * 9 + f, s_trial[e]);
  }
  if (threadIdx.x == 0) {
    atomicAdd(totals, s_tot[0]);
    atomicAdd(totals + 1, s_tot[1]);
  }
}

// Adjacent pairs over their Duffy rules, kPairLanes threads per pair (pairs are grouped by
// configuration, so a warp's pairs read the same points).  phi and psi are affine in the
// points' coordinates, so the 18 vertex sums are combinations of five vector sums of
// h (x - y), h = Re(c e^{ikr} (ikr - 1)) w / r^3, with factors 1, xi_0, xi_1, eta_0, eta_1: 17 sums per
// pair to reduce over eight lanes, where a warp per pair reduced 22 over 32.
// 66,500 pairs (5,120 triangles, order 4), k = 5, B200: 0.77 -> 0.47 ms.
constexpr int kPairLanes = 8;
__global__ void __launch_bounds__(256)
    adjoint_sl_singular(CellSet cs, SingularRules rules, SingularPairs pairs, double k,
                        const double2* __restrict__ lam, const double2* __restrict__ mu,
                        double* __restrict__ grad_cell, double* __restrict__ totals) {
  const int64_t index = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / kPairLanes;
  const int sub = threadIdx.x % kPairLanes;
  const bool valid = index < pairs.npairs;
  const int pair = valid ? static_cast<int>(index) : 0;
  const int tc = __ldg(pairs.test_cell + pair), sc = __ldg(pairs.trial_cell + pair),
            cfg = __ldg(pairs.config + pair);
  double tx[2][3], ty[2][3], dv[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    tx[0][d] = g(cs.geom, kT0x + d, cs.stride, tc);
    tx[1][d] = g(cs.geom, kT1x + d, cs.stride, tc);
    ty[0][d] = g(cs.geom, kT0x + d, cs.stride, sc);
    ty[1][d] = g(cs.geom, kT1x + d, cs.stride, sc);
    dv[d] = g(cs.geom, kV0x + d, cs.stride, tc) - g(cs.geom, kV0x + d, cs.stride, sc);
  }
  const double2 li = lam[tc], mj = mu[sc];
  const double c_re = li.x * mj.x + li.y * mj.y, c_im = li.x * mj.y - li.y * mj.x;
  const int off = __ldg(rules.offset + cfg), npts = valid ? __ldg(rules.offset + cfg + 1) - off : 0;
  // |k r| <= k (diam_x + diam_y) for a pair sharing a vertex: no phase reduction needed
  // when that is below pi/4
  const bool small_phase =
      fabs(k) * (g(cs.geom, kDiam, cs.stride, tc) + g(cs.geom, kDiam, cs.stride, sc)) <= 0.78;
  const double2* txi = reinterpret_cast<const double2*>(rules.test_xi);
  const double2* sxi = reinterpret_cast<const double2*>(rules.trial_xi);
  double R0 = 0.0, dk = 0.0, v[5][3];
#pragma unroll
  for (int e = 0; e < 5; ++e)
#pragma unroll
    for (int d = 0; d < 3; ++d) v[e][d] = 0.0;
  auto points = [&](auto small) {
#pragma unroll 1
    for (int i = off + sub; i < off + npts; i += kPairLanes) {
      const double2 xi = __ldg(txi + i), et = __ldg(sxi + i);
      const double w = __ldg(rules.w + i);
      double d[3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
        d[c] = fma(xi.x, tx[0][c], fma(xi.y, tx[1][c], fma(-et.x, ty[0][c], fma(-et.y, ty[1][c], dv[c]))));
      const double r2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
      const double rinv = rsqrt_refined(r2), kr = k * (r2 * rinv);
      double sn, csn;
      if constexpr (decltype(small)::value)
        sincos_taylor(kr, sn, csn);
      else
        sincos_any(kr, sn, csn);
      // Re(c e^{ikr}), Re(i c e^{ikr})
      const double a = fma(c_re, csn, -c_im * sn), b = -fma(c_re, sn, c_im * csn);
      const double wr = w * rinv;
      R0 = fma(wr, a, R0);
      dk = fma(w, b, dk);
      const double h = wr * (rinv * rinv) * fma(kr, b, -a);
      const double f[5] = {h, h * xi.x, h * xi.y, h * et.x, h * et.y};
#pragma unroll
      for (int e = 0; e < 5; ++e)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[e][c] = fma(f[e], d[c], v[e][c]);
    }
  };
  if (small_phase)
    points(std::true_type{});
  else
    points(std::false_type{});
#pragma unroll
  for (int s = kPairLanes / 2; s > 0; s >>= 1) {
    R0 += __shfl_xor_sync(0xffffffffu, R0, s);
    dk += __shfl_xor_sync(0xffffffffu, dk, s);
#pragma unroll
    for (int e = 0; e < 5; ++e)
#pragma unroll
      for (int c = 0; c < 3; ++c) v[e][c] += __shfl_xor_sync(0xffffffffu, v[e][c], s);
  }
  const double jx = g(cs.geom, kJdet, cs.stride, tc), jy = g(cs.geom, kJdet, cs.stride, sc);
  const double jj = jx * jy * kInv4Pi;
  // J and dJ/dk: one addition per CTA (one per pair queued at the two addresses)
  double J = sub == 0 && valid ? R0 * jj : 0.0, K = sub == 0 && valid ? dk * jj : 0.0;
#pragma unroll
  for (int s = kPairLanes; s < 32; s <<= 1) {
    J += __shfl_xor_sync(0xffffffffu, J, s);
    K += __shfl_xor_sync(0xffffffffu, K, s);
  }
  __shared__ double part[2][8];
  if ((threadIdx.x & 31) == 0) {
    part[0][threadIdx.x >> 5] = J;
    part[1][threadIdx.x >> 5] = K;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += part[threadIdx.x][w];
    atomicAdd(totals + threadIdx.x, sum);
  }
  // one thread per side of the pair
  if (sub > 1 || !valid) return;
  const int cell = sub == 0 ? tc : sc;
  double t0[3], t1[3], n[3], dj[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    t0[d] = sub == 0 ? tx[0][d] : ty[0][d];
    t1[d] = sub == 0 ? tx[1][d] : ty[1][d];
    n[d] = g(cs.geom, kNx + d, cs.stride, cell);
  }
  jdet_gradient(t0, t1, n, dj);
  const double rj = R0 * (sub == 0 ? jy : jx) * kInv4Pi, sj = sub == 0 ? jj : -jj;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double p1 = sub == 0 ? v[1][c] : v[3][c], p2 = sub == 0 ? v[2][c] : v[4][c];
    const double p[3] = {(v[0][c] - p1) - p2, p1, p2};
#pragma unroll
    for (int a = 0; a < 3; ++a)
      atomicAdd(grad_cell + static_cast<int64_t>(cell) * 9 + a * 3 + c, fma(sj, p[a], rj * dj[a][c]));
  }
}

// Per-cell-vertex gradients -> per-point gradients (npoints x 3).
__global__ void cell_to_point_gradient(CellSet cs, const double* __restrict__ grad_cell,
                                       double* __restrict__ grad_points) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cs.ncells) return;
  for (int a = 0; a < 3; ++a) {
    const int v = cs.vids[a * cs.stride + c];
    for (int d = 0; d < 3; ++d)
      atomicAdd(grad_points + 3 * static_cast<int64_t>(v) + d,
                grad_cell[static_cast<int64_t>(c) * 9 + a * 3 + d]);
  }
}

}  // namespace

cudaError_t launch_adjoint_sl(const CellSet& cs, const RegularRule& rule,
                              const SingularRules& rules, const SingularPairs& pairs, double k,
                              const double* lam, const double* mu, double* grad_cell,
                              double* grad_points, int npoints, double* totals, bool mixed,
                              cudaStream_t stream) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(grad_cell, 0, sizeof(double) * 9 * cs.ncells, stream)) != cudaSuccess)
    return e;
  if ((e = cudaMemsetAsync(grad_points, 0, sizeof(double) * 3 * npoints, stream)) != cudaSuccess)
    return e;
  if ((e = cudaMemsetAsync(totals, 0, sizeof(double) * 2, stream)) != cudaSuccess) return e;
  if (cs.ncells <= 0) return cudaSuccess;
  const size_t smem = 16 /* mbarrier */ +
                      2 * (sizeof(double) * tile_doubles(rule.npts) +
                           sizeof(float) * tile_floats(rule.npts, mixed) + sizeof(int) * tile_ints(1) + 16) +
                      sizeof(double) * (2 * kTile * 9 + 2) + 16;
  unsigned* timeouts = nullptr;
  int polls = 0;
  if ((e = stage_wait_state(&timeouts, &polls)) != cudaSuccess) return e;
  const long long ntt = (cs.ncells + kTile - 1) / kTile;
  if (ntt * (ntt + 1) / 2 > 0x7fffffffLL) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(ntt * (ntt + 1) / 2));  // tile pairs tx >= sy
  const double2* l2 = reinterpret_cast<const double2*>(lam);
  const double2* m2 = reinterpret_cast<const double2*>(mu);
  if (!mixed && fp64::has_orbit_form(rule)) {
    const size_t bytes = 16 + 2 * fp64::kTileStride +
                         sizeof(double) * ((2 * 9 + (kWarps + 1) * 9) * kTile + 2);
    e = cudaFuncSetAttribute(adjoint_sl_orbits, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    adjoint_sl_orbits<<<grid, kThreads, bytes, stream>>>(cs, fp64::orbit_rule(rule), k, l2, m2,
                                                         grad_cell, totals, timeouts, polls);
  } else {
    auto fn = !mixed           ? adjoint_sl_regular<0, false>
              : rule.npts == 6 ? adjoint_sl_regular<6, true>
                               : adjoint_sl_regular<0, true>;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    fn<<<grid, kThreads, smem, stream>>>(cs, rule, k, l2, m2, grad_cell, totals, timeouts, polls);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (pairs.npairs > 0) {
    const int per = 256 / kPairLanes;
    adjoint_sl_singular<<<(pairs.npairs + per - 1) / per, 256, 0, stream>>>(cs, rules, pairs, k, l2,
                                                                           m2, grad_cell, totals);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  cell_to_point_gradient<<<(cs.ncells + 255) / 256, 256, 0, stream>>>(cs, grad_cell, grad_points);
  return cudaGetLastError();
}

}  // namespace bempp_b200
