// Batched Helmholtz single-layer DP0 sweep over many wavenumbers and meshes.
//
// One persistent launch for the far pairs: every CTA repeatedly takes the next work item
// (mesh, chunk of wavenumbers, super-tile pair) from a global counter (items of the
// largest mesh first), stages the tiles once, and writes the far-pair entries of its
// 32 x 32 blocks for the wavenumbers of its chunk, complex64.  The pairs the mesh's near
// field marks (centroid distance below twice the larger diameter, or a shared vertex: the
// same masks as the one-off mixed assembly) are left to two FP64 launches that run beside
// it (forked in the same captured graph): near pairs by the 6-point rule with the
// pair-referenced phase, vertex-sharing pairs by their Duffy rules.
// The single layer is symmetric on one mesh, so only tile pairs (test tile >= trial tile)
// are items: an off-diagonal block is also written transposed (through shared memory,
// whole 32-byte sectors).  No two launches or items write the same entry, so nothing
// orders them; the only shared state is the item counter (reset before every launch).
//
// Far pairs.  With r0 the centroid distance, t = K (r - r0) (K the largest wavenumber of
// the pass) and f = w w' / r, the sum for k = x K is e^{ikr0} sum f e^{ixt}.  The
// polynomials of the cosine and sine turn it into sum_n C_n(x) M_n with the moments
// M_n = sum f t^n, which do not depend on k: per cell pair 36 inverse distances and the
// moments (9 for |t| <= 0.8, 12 for |t| <= 2), per wavenumber as many products, one phase
// k r0 and a rotation, where every wavenumber took the 36 distances, square roots,
// reciprocals, cosines and sines anew.  Wavenumbers whose |x t| may exceed 2 keep t and f in
// registers and reduce the phases by pi/2 in packed arithmetic.  Distances in FP32 in the
// orbit form of regular_fp64.cuh, two trial points (one of each orbit) per packed
// instruction; products of wavenumber and r0 in FP64 as before.
//
// Three ellipsoids of 5,120, 1,280 and 320 triangles, 8 wavenumbers up to 20, B200, each
// wavenumber by itself -> this form: far pairs 6.6 -> 1.7 ms, vertex-sharing pairs 2.3 -> 0.8, the
// whole call 8.1 to 8.5 -> 2.7 to 3.1; error against FP64 4.2e-8 -> 3.9e-8 (the phase k r0 and its rotation are
// FP64 here).  The far pairs issue in 60% of the cycles (16 warps per SM at 128 registers).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "regular_fp64.cuh"

namespace bempp_b200 {
namespace {

using namespace tiles;

constexpr int kPass = 8;          // wavenumbers per pass over a tile pair
constexpr int kMoments = 12;      // at most: 9 for |t| <= 0.8, 12 for |t| <= 2
constexpr float kWide = 2.0f;     // the moments' largest |x t|
// The moments' largest |t|: t^11 <= 7e19 stays within FP32, and where x^11 underflows, (x t)^11
// is below rounding.  A pass with a wavenumber beyond it takes the phases of each on its own, so
// that no wavenumber spoils another's matrix.
constexpr float kMomentRange = 64.0f;
constexpr int kMirrorRow = 36;    // padded row of the transposing buffer: no bank conflicts
constexpr int kMirrorGroup = 4;   // trial cells per group of the transposing buffer
constexpr int kSingularGroup = 4; // wavenumbers per thread of the vertex-sharing pairs

struct OrbitSweepRule {
  float kappa, kappa2;  // the second orbit's offsets are kappa times the first's
  float m[2][2];        // -2 kappa_o kappa_o'
  float w[2];           // weight of a point of each orbit
  float reach;          // largest offset of a point, in circumradii
};

// Per wavenumber of a pass: k, x = k / K and the coefficients C_n(x) of the two ranges.
struct PassTable {
  double k[kPass];
  float x[kPass];
  float c[2][kPass][kMoments];      // rows of 48 bytes
  float K, inv;                     // what t carries (1e-20 when every k is 0), its inverse
  float least, most;                // the smallest and the largest |x|
};

// cos: even n; sin: odd n (fit_phase_polys.py 0.8 4 3, errors 6.5e-11 and 2.1e-9; 2.0 5 5, errors
// 4.29e-09 and 3.93e-10)
__constant__ float kPoly[2][kMoments] = {
    {1.0f, 1.0f, -4.999999968e-1f, -1.666664881e-1f, 4.166661828e-2f, 8.331875683e-3f,
     -1.388660219e-3f, -1.948277516e-4f, 2.437514408e-5f, 0.0f, 0.0f, 0.0f},
    {1.0f, 1.0f, -4.999999509e-01f, -1.666666601e-01f, 4.166649215e-02f, 8.333314191e-03f,
     -1.388687057e-03f, -1.983932827e-04f, 2.469945356e-05f, 2.746786451e-06f, -2.519531204e-07f, -2.312569666e-08f}};

__device__ inline void fill_table(PassTable& p, const double* __restrict__ ks, int n) {
  const int t = threadIdx.x;
  if (t >= kPass) return;
  double K = 0.0;
  for (int i = 0; i < n; ++i) {
    const double m = fabs(__ldg(ks + i));
    if (m <= 1e30) K = fmax(K, m);  // one beyond FP32's range has no part in the scale
  }
  if (K < 1e-20) K = 0.0;
  const float Kf = K > 0.0 ? static_cast<float>(K) : 1e-20f;
  auto ratio = [&](int i) { return K > 0.0 ? __ldg(ks + i) / static_cast<double>(Kf) : 0.0; };
  if (t == 0) {
    p.K = Kf;
    p.inv = 1.f / Kf;
    p.least = 1e30f;
    p.most = 0.f;
    for (int i = 0; i < n; ++i) {
      const float v = fabsf(static_cast<float>(ratio(i)));
      p.least = fminf(p.least, v);
      p.most = fmaxf(p.most, v);
    }
  }
  if (t >= n) return;
  const double x = ratio(t);
  p.k[t] = __ldg(ks + t);
  p.x[t] = static_cast<float>(x);
  for (int r = 0; r < 2; ++r) {
    double pw = 1.0;
    for (int m = 0; m < kMoments; ++m) {
      p.c[r][t][m] = static_cast<float>(kPoly[r][m] * pw);
      pw *= x;
    }
  }
}

// The 36 point pairs of a far pair, three packed pairs (trial orbits 0 and 1 of the three
// vertices) at a time: visit(test orbit, 1 / r, t).
template <class F>
__device__ __forceinline__ void far_points(const Tile& T, int it, const Tile& S, int js,
                                           const OrbitSweepRule& rule, float fdx, float fdy,
                                           float fdz, float r0sq, float r0, float K, float inv,
                                           F&& visit) {
  float P[3][3], R[3][3], ex[3], ey[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float4 x = T.R4(a, it), y = S.R4(a, js);
    P[a][0] = x.x;
    P[a][1] = x.y;
    P[a][2] = x.z;
    ex[a] = K * x.w;
    R[a][0] = K * y.x;
    R[a][1] = K * y.y;
    R[a][2] = K * y.z;
    ey[a] = K * y.w;
  }
  float M[3][3], dx[3];
  float2 Y[3];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
      M[a][b] = fmaf(P[a][2], R[b][2], fmaf(P[a][1], R[b][1], P[a][0] * R[b][0]));
    dx[b] = K * fmaf(fdz, P[b][2], fmaf(fdy, P[b][1], fdx * P[b][0]));
    const float dy = fmaf(fdz, R[b][2], fmaf(fdy, R[b][1], fdx * R[b][0]));
    Y[b] = make_float2(fmaf(-2.f, dy, ey[b]), fmaf(rule.kappa2, ey[b], -2.f * rule.kappa * dy));
  }
  const float2 r0sq2 = f2(r0sq), r02 = f2(r0), inv2 = f2(inv);
#pragma unroll
  for (int op = 0; op < 2; ++op) {
    const float2 m2 = make_float2(rule.m[op][0], rule.m[op][1]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float X = op == 0 ? fmaf(2.f, dx[a], ex[a]) : fmaf(rule.kappa2, ex[a], 2.f * rule.kappa * dx[a]);
      float2 rinv[3], t[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const float2 s = ffma2(m2, f2(M[a][b]), fadd2(f2(X), Y[b]));  // K (r^2 - r0^2)
        const float2 r2 = ffma2(s, inv2, r0sq2);
        rinv[b] = rsqrt_approx2(r2);
        t[b] = fmul2(s, rcp_approx2(ffma2(r2, rinv[b], r02)));
      }
      visit(op, rinv, t);
    }
  }
}

// TS: tile shape of a work item, TS x TS tiles of 32 cells on each side (a super-tile
// pair: 1 x 1 or 2 x 2 tile pairs staged together).  Far pairs only: the pairs marked in the
// mesh's near-field masks (near or vertex-sharing) are written by the FP64 launches.
template <int TS>
__global__ void __launch_bounds__(kThreads, 4)
    sweep_sl_dp0(const __grid_constant__ SweepArgs a, const __grid_constant__ OrbitSweepRule rule) {
  constexpr int Q = 6;
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);  // completion of the tile copies
  unsigned char* cursor = smem + 16;
  Tile Tt[TS], St[TS];
#pragma unroll
  for (int i = 0; i < TS; ++i) Tt[i] = carve_tile(cursor, Q, true, 1, false);
#pragma unroll
  for (int i = 0; i < TS; ++i) St[i] = carve_tile(cursor, Q, true, 1, false);
  long long* s_item = reinterpret_cast<long long*>(cursor);
  PassTable& table = *reinterpret_cast<PassTable*>(s_item + 2);
  const int it = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* skip = reinterpret_cast<unsigned*>(s_item + 2 + (sizeof(PassTable) + 15) / 16 * 2);  // [it]: bit js
  float2* mir = reinterpret_cast<float2*>(skip + kTile) +
                warp * (kPass * kMirrorGroup * kMirrorRow);  // [(wavenumber, js)][it], per warp
  if (threadIdx.x == 0) mbar_init(mbar, 1);
  unsigned phase = 0;  // parity of the mbarrier phase of the current item's copies
  for (;;) {
    if (threadIdx.x == 0) *s_item = static_cast<long long>(atomicAdd(a.counter, 1ull));
    __syncthreads();
    const long long item = *s_item;
    if (item >= a.nitems) break;
    int m = 0;
    while (m + 1 < a.nmesh && item >= a.mesh[m + 1].item_begin) ++m;
    const SweepMesh& M = a.mesh[m];
    const long long local = item - M.item_begin;
    // wavenumber chunk outermost: the items resident at one time write one output
    // matrix (one chunk of them), in the banded order of the super-tile pairs
    const int nsup = (M.ntiles + TS - 1) / TS;
    const long long npairs = lower_tile_pair_count(nsup, 0, nsup);
    const int kc = static_cast<int>(local / npairs);
    int TT, ST;
    lower_tile_pair(local % npairs, nsup, 0, nsup, TT, ST);
    const int nc = M.cells.ncells;
    // every tile of the two super-tiles by bulk (TMA) copies on the mbarrier (no FP64
    // points: the far pairs use the FP32 offsets); the previous item's reads of the tiles
    // ended at the barriers that closed it
    if (threadIdx.x == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      unsigned bytes = 0;
      for (int i = 0; i < TS; ++i) {
        if (TS * TT + i < M.ntiles) bytes += bulk_tile_bytes(Q, true, false);
        if (TS * ST + i < M.ntiles) bytes += bulk_tile_bytes(Q, true, false);
      }
      mbar_expect_tx(mbar, bytes);
      for (int i = 0; i < TS; ++i) {
        if (TS * TT + i < M.ntiles)
          stage_tile_bulk(Tt[i], M.cells, (TS * TT + i) * kTile, Q, true, mbar, false);
        if (TS * ST + i < M.ntiles)
          stage_tile_bulk(St[i], M.cells, (TS * ST + i) * kTile, Q, true, mbar, false);
      }
    }
    const bool staged = mbar_wait_bounded(mbar, phase);
    phase ^= 1u;
    if (__syncthreads_or(!staged)) {
      // the copies did not complete in time (never expected): record it, give them a last
      // bounded wait and stop this CTA (the item's entries stay unwritten; the host's
      // completion check reports it)
      if (threadIdx.x == 0) atomicAdd(a.stage_timeouts, 1u);
      mbar_wait_bounded(mbar, phase ^ 1u);
      return;
    }
    const int k1 = min(a.nk, (kc + 1) * a.kchunk);
    for (int k0 = kc * a.kchunk; k0 < k1; k0 += kPass) {
      const int nk = min(kPass, k1 - k0);
      fill_table(table, a.ks + k0, nk);  // published by the barrier after the skip words
#pragma unroll 1
      for (int sub = 0; sub < TS * TS; ++sub) {
        const int tt = TS * TT + sub / TS, st = TS * ST + sub % TS;
        if (tt >= M.ntiles || st >= M.ntiles || tt < st) continue;  // block-uniform
        const Tile& T = Tt[sub / TS];
        const Tile& S = St[sub % TS];
        const bool mirror = tt > st;
        const int ti0 = tt * kTile, sj0 = st * kTile;
        const int nti = min(kTile, nc - ti0), nsj = min(kTile, nc - sj0);
        // the near and vertex-sharing pairs of this tile pair (the relation is symmetric, so
        // the same bits mark the transposed block)
        const int moff = __ldg(M.tile_mask + static_cast<int64_t>(tt) * M.ntiles + st);
        if (threadIdx.x < kTile)
          skip[threadIdx.x] = moff >= 0 ? __ldg(M.masks + static_cast<int64_t>(moff) * kTile + threadIdx.x) : 0u;
        __syncthreads();
        const unsigned skip_it = it < nti ? skip[it] : ~0u;
        const float K = table.K, inv = table.inv;
        const int64_t plane = static_cast<int64_t>(nc) * nc;
        float2* out = M.out + k0 * plane;
        for (int j0 = warp * kMirrorGroup; j0 < nsj; j0 += kWarps * kMirrorGroup) {
#pragma unroll 1
          for (int jj = 0; jj < kMirrorGroup; ++jj) {
            const int js = j0 + jj;
            const bool active = js < nsj && !((skip_it >> js) & 1u);
            if (!__any_sync(0xffffffffu, active)) continue;
            const double dcx = T.G(fCx, it) - S.G(fCx, js), dcy = T.G(fCy, it) - S.G(fCy, js),
                         dcz = T.G(fCz, it) - S.G(fCz, js);
            const double r0sq = dcx * dcx + dcy * dcy + dcz * dcz;
            const double r0 = r0sq * rsqrt_refined(r0sq);
            const double sc = T.G(fJdet, it) * S.G(fJdet, js) * kInv4Pi;
            const float fdx = static_cast<float>(dcx), fdy = static_cast<float>(dcy),
                        fdz = static_cast<float>(dcz);
            const float r0sqf = static_cast<float>(r0sq), r0f = static_cast<float>(r0);
            // largest |t| of the warp's pairs
            const float reach = __uint_as_float(__reduce_max_sync(
                0xffffffffu,
                active ? __float_as_uint(K * rule.reach * static_cast<float>(T.G(fRad, it) + S.G(fRad, js)))
                       : 0u));
            auto store = [&](int kk, float re, float im) {
              // e^{ik r0} from the FP64 phase
              double c, s;
              sincos_any(table.k[kk] * r0, s, c);
              const double dr = re, di = im;
              const float2 v = make_float2(static_cast<float>((dr * c - di * s) * sc),
                                           static_cast<float>((dr * s + di * c) * sc));
              if (active) out[kk * plane + static_cast<int64_t>(sj0 + js) * nc + ti0 + it] = v;
              if (mirror) mir[(kk * kMirrorGroup + jj) * kMirrorRow + it] = v;
            };
            auto by_moments = [&](auto count) {
              constexpr int N = decltype(count)::value;
              float mom[N], comp = 0.f;
              float2 acc[N];
#pragma unroll
              for (int n = 0; n < N; ++n) {
                mom[n] = 0.f;
                acc[n] = f2(0.f);
              }
              int seen = 0;
              far_points(T, it, S, js, rule, fdx, fdy, fdz, r0sqf, r0f, K, inv,
                         [&](int op, const float2 rinv[3], const float2 t[3]) {
                           float2 v[3] = {rinv[0], rinv[1], rinv[2]};
                           const float2 s0 = fadd2(fadd2(v[0], v[1]), v[2]);
                           kahan_add(mom[0], comp, rule.w[op] * fmaf(rule.w[1], s0.y, rule.w[0] * s0.x));
#pragma unroll
                           for (int n = 1; n < N; ++n) {
#pragma unroll
                             for (int b = 0; b < 3; ++b) v[b] = fmul2(v[b], t[b]);
                             acc[n] = fadd2(acc[n], fadd2(fadd2(v[0], v[1]), v[2]));
                           }
                           if (++seen % 3 == 0) {  // the orbit is done
#pragma unroll
                             for (int n = 1; n < N; ++n) {
                               mom[n] = fmaf(rule.w[op], fmaf(rule.w[1], acc[n].y, rule.w[0] * acc[n].x), mom[n]);
                               acc[n] = f2(0.f);
                             }
                           }
                         });
#pragma unroll 2
              for (int kk = 0; kk < nk; ++kk) {
                if (N == kMoments && reach * fabsf(table.x[kk]) > kWide) continue;  // warp-uniform
                const float* c = table.c[N == kMoments][kk];
                constexpr int kEven = (N - 1) & ~1, kOdd = N - 1 - (N & 1);
                float re = c[kEven] * mom[kEven], im = c[kOdd] * mom[kOdd];
#pragma unroll
                for (int n = kEven - 2; n >= 0; n -= 2) re = fmaf(c[n], mom[n], re);
#pragma unroll
                for (int n = kOdd - 2; n > 0; n -= 2) im = fmaf(c[n], mom[n], im);
                store(kk, re, im);
              }
            };
            const float top = reach * table.most;
            if (top <= 0.8f) {
              by_moments(std::integral_constant<int, 9>{});
              continue;
            }
            // every wavenumber is taken by one of the two (a NaN by both)
            const bool moments = top <= kMomentRange;
            if (moments && reach * table.least <= kWide) by_moments(std::integral_constant<int, kMoments>{});
            if (!(top <= kWide)) {
              float2 f[18], t[18];
              int at = 0;
              far_points(T, it, S, js, rule, fdx, fdy, fdz, r0sqf, r0f, K, inv,
                         [&](int op, const float2 rinv[3], const float2 tb[3]) {
                           const float2 w = make_float2(rule.w[op] * rule.w[0], rule.w[op] * rule.w[1]);
#pragma unroll
                           for (int b = 0; b < 3; ++b) {
                             f[at + b] = fmul2(w, rinv[b]);
                             t[at + b] = tb[b];
                           }
                           at += 3;
                         });
#pragma unroll 1
              for (int kk = 0; kk < nk; ++kk) {
                const float2 x = f2(table.x[kk]);
                if (moments && reach * fabsf(x.x) <= kWide) continue;  // warp-uniform: done above
                float re = 0.f, im = 0.f, cre = 0.f, cim = 0.f;
#pragma unroll
                for (int g = 0; g < 18; g += 3) {
                  float2 sr = f2(0.f), si = f2(0.f);
#pragma unroll
                  for (int b = g; b < g + 3; ++b) {
                    float2 cs, sn;
                    reduced_cos_sin2(fmul2(t[b], x), cs, sn);
                    sr = ffma2(f[b], cs, sr);
                    si = ffma2(f[b], sn, si);
                  }
                  kahan_add(re, cre, sr.x + sr.y);
                  kahan_add(im, cim, si.x + si.y);
                }
                store(kk, re, im);
              }
            }
          }
          if (mirror) {
            // the transposed entries (row sj0 + j, column ti0 + i) of four trial cells:
            // 32 contiguous bytes per column
            __syncwarp();
            const int jj = it & (kMirrorGroup - 1), js = j0 + jj;
            for (int kk = 0; kk < nk; ++kk) {
#pragma unroll
              for (int i = it / kMirrorGroup; i < kTile; i += 32 / kMirrorGroup)
                if (i < nti && js < nsj && !((skip[i] >> js) & 1u))
                  out[kk * plane + static_cast<int64_t>(ti0 + i) * nc + sj0 + js] =
                      mir[(kk * kMirrorGroup + jj) * kMirrorRow + i];
            }
            __syncwarp();  // the buffer is reused by the next group
          }
        }
        __syncthreads();  // the skip words and the table are reused
      }
    }
  }
}

// Single-layer DP0 entry of one cell pair (test i, trial j) by the 6-point rule in FP64,
// points and geometry from the grid arrays: phase referenced to the pair when
// |k| (rad_i + rad_j) <= 0.8, else sincos_cw.
__device__ double2 sl_dp0_pair_fp64(const CellSet& cs, int i, int j, const RegularRule& rule,
                                    double k) {
  const int64_t S = cs.stride;
  const double dcx = g(cs.geom, kCx, cs.stride, i) - g(cs.geom, kCx, cs.stride, j);
  const double dcy = g(cs.geom, kCy, cs.stride, i) - g(cs.geom, kCy, cs.stride, j);
  const double dcz = g(cs.geom, kCz, cs.stride, i) - g(cs.geom, kCz, cs.stride, j);
  const bool ref = fabs(k) * (g(cs.geom, kRad, cs.stride, i) + g(cs.geom, kRad, cs.stride, j)) <= 0.8;
  double kr0 = 0.0, pc = 1.0, ps = 0.0;
  if (ref) {
    const double r0sq = dcx * dcx + dcy * dcy + dcz * dcz;
    kr0 = k * (r0sq * rsqrt_refined(r0sq));
    sincos_cw(kr0, ps, pc);
  }
  double yq[6][3];
#pragma unroll
  for (int q = 0; q < 6; ++q)
#pragma unroll
    for (int d = 0; d < 3; ++d) yq[q][d] = __ldg(cs.qpts + (q * 3 + d) * S + j);
  double re = 0.0, im = 0.0;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const double x0 = __ldg(cs.qpts + (p * 3) * S + i), x1 = __ldg(cs.qpts + (p * 3 + 1) * S + i),
                 x2 = __ldg(cs.qpts + (p * 3 + 2) * S + i);
    double ur = 0.0, ui = 0.0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const double dx = x0 - yq[q][0], dy = x1 - yq[q][1], dz = x2 - yq[q][2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      const double rinv = rsqrt_refined(r2);
      const double r = r2 * rinv;
      double sn, cs_;
      if (ref)
        sincos_small(fma(k, r, -kr0), sn, cs_);
      else
        sincos_cw(k * r, sn, cs_);
      const double f = rule.w[q] * rinv;
      ur = fma(f, cs_, ur);
      ui = fma(f, sn, ui);
    }
    re = fma(rule.w[p], ur, re);
    im = fma(rule.w[p], ui, im);
  }
  const double sc = g(cs.geom, kJdet, cs.stride, i) * g(cs.geom, kJdet, cs.stride, j) * kInv4Pi;
  return make_double2((re * pc - im * ps) * sc, (re * ps + im * pc) * sc);
}

// The near pairs (no shared vertex) of every mesh and wavenumber: one thread per (pair,
// wavenumber), wavenumber fastest.
__global__ void __launch_bounds__(kThreads)
    sweep_near_fp64(const __grid_constant__ SweepArgs a, const __grid_constant__ RegularRule rule) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= a.near_begin[a.nmesh]) return;
  int m = 0;
  while (m + 1 < a.nmesh && t >= a.near_begin[m + 1]) ++m;
  const SweepMesh& M = a.mesh[m];
  const long long local = t - a.near_begin[m];
  const int e = static_cast<int>(local / a.nk), kk = static_cast<int>(local % a.nk);
  const int2 pr = __ldg(M.near_pairs + e);
  const double2 v = sl_dp0_pair_fp64(M.cells, pr.x, pr.y, rule, a.ks[kk]);
  const int nc = M.cells.ncells;
  M.out[static_cast<long long>(kk) * nc * nc + static_cast<long long>(pr.y) * nc + pr.x] =
      make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
}

// Offset of a direction of a pair (singular.cu), squared: tangents t0, t1 of both cells.
__device__ __forceinline__ double direction_square(const double2* __restrict__ coef, int i,
                                                   const double tx[2][3], const double ty[2][3]) {
  const double2 cx = __ldg(coef + 2 * i), cy = __ldg(coef + 2 * i + 1);
  double d[3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
    d[c] = fma(cx.x, tx[0][c], fma(cx.y, tx[1][c], fma(-cy.x, ty[0][c], -cy.y * ty[1][c])));
  return fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
}

// The vertex-sharing pairs of every mesh and wavenumber: a pair's Duffy rule as directions and
// radii (singular.cu) for up to kSingularGroup wavenumbers at once: distance and share of a
// direction, then per wavenumber the series of the inner sum (as many terms as the first one
// left out is below 2e-17).  2^lanes threads per pair and group share the directions.  Phases
// beyond the series' range, |theta| > 3.4, are taken at every radius.
__global__ void __launch_bounds__(kThreads, 3)
    sweep_singular_fp64(const __grid_constant__ SweepArgs a, const __grid_constant__ SingularRules rules,
                        int lanes, const __grid_constant__ SeriesRules series) {
  const int ngroups = (a.nk + kSingularGroup - 1) / kSingularGroup;
  const long long total = a.sing_begin[a.nmesh] * ngroups;
  const long long index = (static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x) >> lanes;
  const int sub = threadIdx.x & ((1 << lanes) - 1), step = 1 << lanes;
  const bool valid = index < total;
  const long long flat = valid ? index / ngroups : 0;  // wavenumber groups fastest
  const int k0 = valid ? static_cast<int>(index % ngroups) * kSingularGroup : 0;
  int m = 0;
  while (m + 1 < a.nmesh && flat >= a.sing_begin[m + 1]) ++m;
  const SweepMesh& M = a.mesh[m];
  const int e = static_cast<int>(flat - a.sing_begin[m]);
  const CellSet& cs = M.cells;
  const int tc = __ldg(M.sing.test_cell + e), sc = __ldg(M.sing.trial_cell + e);
  const int cfg = __ldg(M.sing.config + e);
  double tx[2][3], ty[2][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    tx[0][d] = g(cs.geom, kT0x + d, cs.stride, tc);
    tx[1][d] = g(cs.geom, kT1x + d, cs.stride, tc);
    ty[0][d] = g(cs.geom, kT0x + d, cs.stride, sc);
    ty[1][d] = g(cs.geom, kT1x + d, cs.stride, sc);
  }
  const int first = __ldg(rules.dir_offset + cfg);
  const int ndir = valid ? __ldg(rules.dir_offset + cfg + 1) - first : 0;
  const int kind = cfg < 9 ? 0 : cfg < 27 ? 1 : 2;  // common vertex, edge, one cell
  const double2* coef = reinterpret_cast<const double2*>(rules.coef) + 2 * first;
  double k[kSingularGroup], re[kSingularGroup], im[kSingularGroup], kmax = 0.0;
#pragma unroll
  for (int n = 0; n < kSingularGroup; ++n) {
    k[n] = __ldg(a.ks + min(k0 + n, a.nk - 1));
    kmax = fmax(kmax, fabs(k[n]));
    re[n] = im[n] = 0.0;
  }
  const double bound = kmax * (g(cs.geom, kDiam, cs.stride, tc) + g(cs.geom, kDiam, cs.stride, sc));
  // a copy of the loop per kind, so that the coefficients are constant operands
  auto series_of = [&](auto row, auto count) {
    constexpr int N = decltype(count)::value;
    const double* c = series.c[decltype(row)::value];
    for (int i = sub; i < ndir; i += step) {
      const double r2 = direction_square(coef, i, tx, ty), rinv = rsqrt_refined(r2), r = r2 * rinv;
      const double f = __ldg(rules.share + first + i) * rinv;
      double th[kSingularGroup], z[kSingularGroup], pr[kSingularGroup], pi[kSingularGroup];
#pragma unroll
      for (int n = 0; n < kSingularGroup; ++n) {
        th[n] = k[n] * r;
        z[n] = th[n] * th[n];
        pr[n] = c[2 * N - 2];
        pi[n] = c[2 * N - 1];
      }
#pragma unroll
      for (int q = N - 2; q >= 0; --q)
#pragma unroll
        for (int n = 0; n < kSingularGroup; ++n) {
          pr[n] = fma(pr[n], z[n], c[2 * q]);
          pi[n] = fma(pi[n], z[n], c[2 * q + 1]);
        }
#pragma unroll
      for (int n = 0; n < kSingularGroup; ++n) {
        re[n] = fma(f, pr[n], re[n]);
        im[n] = fma(f * th[n], pi[n], im[n]);
      }
    }
  };
  auto by_series = [&](auto count) {
    if (kind == 0)
      series_of(std::integral_constant<int, 0>{}, count);
    else if (kind == 1)
      series_of(std::integral_constant<int, 3>{}, count);
    else
      series_of(std::integral_constant<int, 9>{}, count);
  };
  if (bound <= 0.5171) {
    by_series(std::integral_constant<int, 8>{});
  } else if (bound <= 1.3702) {
    by_series(std::integral_constant<int, 11>{});
  } else if (bound <= 3.4) {
    by_series(std::integral_constant<int, kSeriesTerms>{});
  } else {
    const int n = rules.order, n2 = n * n, n3 = n2 * n;
    const int per = kind == 0 ? n3 : kind == 1 ? n2 : n;    // directions per region
    const int inner = kind == 0 ? n : kind == 1 ? n2 : n3;  // values of rho
    const double2* rho = reinterpret_cast<const double2*>(rules.rho) + (kind == 0 ? 0 : kind == 1 ? n : n + n2);
    const int off = __ldg(rules.offset + cfg);
    for (int i = sub; i < ndir; i += step) {
      const double r2 = direction_square(coef, i, tx, ty), rinv = rsqrt_refined(r2), r = r2 * rinv;
      const double* w = rules.w + off + (i / per) * n2 * n2 + i % per;
      double ar[kSingularGroup], ai[kSingularGroup];
#pragma unroll
      for (int q = 0; q < kSingularGroup; ++q) ar[q] = ai[q] = 0.0;
      for (int j = 0; j < inner; ++j) {
        const double2 rh = __ldg(rho + j);  // rho, 1 / rho
        const double f = __ldg(w + j * per) * rh.y;
        double t[kSingularGroup], sn[kSingularGroup], cn[kSingularGroup];
#pragma unroll
        for (int q = 0; q < kSingularGroup; ++q) t[q] = k[q] * r * rh.x;
        sincos_any_n<kSingularGroup>(t, sn, cn);
#pragma unroll
        for (int q = 0; q < kSingularGroup; ++q) {
          ar[q] = fma(f, cn[q], ar[q]);
          ai[q] = fma(f, sn[q], ai[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < kSingularGroup; ++q) {
        re[q] = fma(rinv, ar[q], re[q]);
        im[q] = fma(rinv, ai[q], im[q]);
      }
    }
  }
  // sums over the pair's threads (every thread of the warp takes part)
  for (int s = step >> 1; s > 0; s >>= 1)
#pragma unroll
    for (int n = 0; n < kSingularGroup; ++n) {
      re[n] += __shfl_xor_sync(0xffffffffu, re[n], s);
      im[n] += __shfl_xor_sync(0xffffffffu, im[n], s);
    }
  if (sub != 0 || !valid) return;
  const double scl = g(cs.geom, kJdet, cs.stride, tc) * g(cs.geom, kJdet, cs.stride, sc) * kInv4Pi;
  const int64_t nc = cs.ncells;
#pragma unroll
  for (int n = 0; n < kSingularGroup; ++n)
    if (k0 + n < a.nk)
      M.out[(k0 + n) * nc * nc + sc * nc + tc] =
          make_float2(static_cast<float>(re[n] * scl), static_cast<float>(im[n] * scl));
}

template <int TS>
cudaError_t launch_sweep_shape(const SweepArgs& args, const OrbitSweepRule& rule, int blocks,
                               cudaStream_t stream) {
  const size_t smem = sweep_smem_bytes(TS);
  auto fn = sweep_sl_dp0<TS>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) {
    cudaGetLastError();  // not sticky: clear it, so that it is not reported by a later launch
    return e;
  }
  fn<<<blocks, kThreads, smem, stream>>>(args, rule);
  return cudaGetLastError();
}

}  // namespace

size_t sweep_smem_bytes(int ts) {
  size_t b = 16;  // the mbarrier
  for (int t = 0; t < 2 * ts; ++t) {  // tiles without FP64 points
    b += sizeof(double) * tile_doubles(6, false) + sizeof(float) * tile_floats(6, true) +
         sizeof(int) * tile_ints(1);
    b = (b + 15) & ~size_t(15);
  }
  return b + 2 * sizeof(long long) + (sizeof(PassTable) + 15) / 16 * 16 + sizeof(unsigned) * kTile +
         sizeof(float2) * kWarps * kPass * kMirrorGroup * kMirrorRow + 16;
}

cudaError_t launch_sweep_sl(const SweepArgs& args, const RegularRule& rule, int blocks_per_sm, int sms,
                            cudaStream_t stream) {
  if (!fp64::has_orbit_form(rule)) return cudaErrorInvalidValue;
  OrbitSweepRule r{};
  double gamma[2];
  for (int o = 0; o < 2; ++o) gamma[o] = (rule.phi[0][3 * o] - 1.0 / 3.0) * 1.5;
  const double kappa[2] = {1.0, gamma[1] / gamma[0]};
  r.kappa = static_cast<float>(kappa[1]);
  r.kappa2 = static_cast<float>(kappa[1] * kappa[1]);
  for (int i = 0; i < 2; ++i) {
    r.w[i] = static_cast<float>(rule.w[3 * i]);
    for (int j = 0; j < 2; ++j) r.m[i][j] = static_cast<float>(-2.0 * kappa[i] * kappa[j]);
  }
  r.reach = static_cast<float>(std::max(std::fabs(gamma[0]), std::fabs(gamma[1])) * (1.0 + 1e-6));
  if (args.tile_shape != 1 && args.tile_shape != 2) return cudaErrorInvalidValue;
  const int blocks = blocks_per_sm * sms;
  return args.tile_shape == 1 ? launch_sweep_shape<1>(args, r, blocks, stream)
                              : launch_sweep_shape<2>(args, r, blocks, stream);
}

cudaError_t launch_sweep_near_singular(const SweepArgs& args, const RegularRule& rule,
                                       const SingularRules& rules, cudaStream_t stream) {
  if (rule.npts != 6 || !rules.host_series) return cudaErrorInvalidValue;
  const long long nn = args.near_begin[args.nmesh];
  const long long ns = args.sing_begin[args.nmesh] * ((args.nk + kSingularGroup - 1) / kSingularGroup);
  if (ns > 0) {
    // threads per pair and group, at most a warp: six times what is resident, since the pairs'
    // kinds differ in their directions (128, 80 and 24 of order 4) and the last ones leave
    // the chip half empty (two threads per pair: 1.1 ms for the case above)
    int lanes = 0;
    while (lanes < 5 && (ns << lanes) < 148LL * 3 * kThreads * 6) ++lanes;
    const long long blocks = ((ns << lanes) + kThreads - 1) / kThreads;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    sweep_singular_fp64<<<static_cast<unsigned>(blocks), kThreads, 0, stream>>>(args, rules, lanes,
                                                                               rules.host_series[0]);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (nn > 0) {
    const long long blocks = (nn + kThreads - 1) / kThreads;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    sweep_near_fp64<<<static_cast<unsigned>(blocks), kThreads, 0, stream>>>(args, rule);
    return cudaGetLastError();
  }
  return cudaSuccess;
}

}  // namespace bempp_b200
