// FP64 mode: the plain double-precision GPU form of the estimator.
//
// The paths of a knot are split into blocks of block_paths; a block is eight
// slots of 32 lanes, slot w starting with the block's paths [32 w, 32 w + 32)
// and every lane taking one of the block's further paths when its own ends,
// by a rule on step counts alone.  Every path
// quantity is FP64 and each stencil exit adds its exact RBF vector
// Y * r_j(X), r_j = exp(-|p_j - X|^2 / c^2), into the FP64 sums S_j of its
// slot.  Afterwards (k_rows_fp64) G_i = -(1/N) sum_j ipsi(j,i) S_j per block.
// Exits are queued per warp (side, coordinate, weight) and the warp adds
// their RBF vectors one exit at a time with the side knots spread over the
// lanes (no atomics), so the n_s exponentials of an exit run at full width.
// By linearity this equals the reference's per-exit
// H_i = sum_j ipsi(j,i) RBF(p_j, X) accumulation (Meshes/stencil.cpp:244-307)
// with n_s instead of n_s^2 exponentials per exit.  It is the all-FP64 GPU
// oracle that MIXED results are compared with.
//
// What bounds it: the FP64 pipe (one warp instruction per 64 cycles and
// scheduler).  A CTA takes all eight slots of a block where there are enough
// blocks to fill the GPU, and fewer of them where there are not (one knot of
// 5,000 paths: 19 blocks, 152 CTAs of one warp); coefficients that reach only
// the sums of B come from tables (fast64.cuh); the exit test of
// constant-sigma kinds compares |x - c| with an edge formed once, as
// integers; the normals of odd and even steps come from one place, so lanes
// of both kinds do not run it twice.  Positions, exponentials and the order
// in which a slot's exits are added have to stay: Psi^-1 has entries of 1e9
// and more, so G carries the rounding of the sums S.  A path that enters
// another slot's sum moves G by 1e-8 to 1e-5 of its size (one knot of 5,000
// paths: 1.3e-6 in the median over 40
// seeds), which is why the hand-out may not depend on which warp comes first.
// With an atomic counter in its place, two runs on the same inputs put 35 %
// of the further paths into different slots; the exchange that replaces it
// costs up to 5 % (one knot 742 against 747 us for the whole call, 4x4/n11
// 24.84 and 24.80 ms, 12x12/n43 in pairs 3.44 to 3.59 and 3.38 to 3.41 s).
// 4x4/n11, N = 1e4, h = 1e-3: 49.7 -> 24.8 ms; one knot of 5,000 paths
// 1.02 -> 0.49 ms; 12x12/n43, 2e4 pairs: 4.64 -> 3.5 s.
#include <cooperative_groups.h>

#include "dev_common.cuh"
#include "fast64.cuh"
#include "kernels.h"

namespace pdds {

namespace {

struct ItemSide64 {
  int n;
  int orient;
  int glob;
  int s_off;         // offset into the shared S arrays
  double origin;
  double inv_c2;
  int64_t t_off;     // shape's local knot coordinates
  double R;          // arc radius (polar stencils): RBF distance = chord 2 R sin(dt / 2)
};

constexpr unsigned FULL = 0xffffffffu;

struct Lvl64 {
  double x, y, Y, Z, xi;
  double phi;  // Z + Y g(X_tau) at the exit (diagnostics)
  Coef<double> k;  // kinds whose sigma varies: the coefficients at (x, y)
  unsigned steps;
};

// Box-Muller in FP64: z0 = rho cos(2 pi u1), z1 = rho sin(2 pi u1).
__device__ __forceinline__ void normals_f64(uint32_t ua, uint32_t ub, double& z0, double& z1) {
  const double u0 = u01_fp64(ua), u1 = u01_fp64(ub);
  const double rho = ::sqrt(-2.0 * ::log(u0));
  double sn, cs;
  sincospi(2.0 * u1, &sn, &cs);
  z0 = rho * cs;
  z1 = rho * sn;
}

// Kinds with sigma = S I and no drift.
template <int KIND>
constexpr bool iso64 = KIND != PK_VARCOEF && !is_lut_kind(KIND);
template <int KIND>
constexpr double sigma64 = KIND == PK_MONEGROS ? 1.41421356237 : 1.4142135623730951;
// Kinds with a reaction term.
template <int KIND>
constexpr bool react64 = KIND == PK_HELMHOLTZ || KIND == PK_VARCOEF || is_lut_kind(KIND);

// coef_f64 with the table functions in the terms that reach only the sums
// of B (f and grad u); sigma, b and c keep coef_f64's rounding.
template <int KIND>
__device__ __forceinline__ void coef_t64(const ProblemDev& P, const Fast64& T, double x, double y, Coef<double>& k) {
  const double PI = 3.141592653589793;
  if constexpr (KIND == PK_POISSON_SINCOS) {
    double sx, cx, sy, cy;
    f64::sincospi(T, x, sx, cx);
    f64::sincospi(T, y, sy, cy);
    k.f = 19.739208802178716 * (sx * cy);
    k.g0 = fma(PI, cx * cy, y);
    k.g1 = fma(-PI, sx * sy, x);
    k.c = 0.0;
  } else if constexpr (KIND == PK_HELMHOLTZ) {
    const double a = P.p[0], b = P.p[1], c = P.p[2];
    double sa, ca, sb, cb;
    f64::sincos(T, a * x, sa, ca);
    f64::sincos(T, b * y, sb, cb);
    k.f = ((a * a + b * b) - c) * (sa * cb);
    k.g0 = a * (ca * cb);
    k.g1 = -(b * (sa * sb));
    k.c = c;
  } else if constexpr (KIND == PK_VARCOEF) {
    const double s1 = 1.0 + 0.5 * (x * x), s2 = 1.0 + 0.5 * (y * y);
    double sn, cs;
    f64::sincos(T, 2.0 * y, sn, cs);
    const double ex = f64::exp(T, x);
    const double ux = ex * cs, uy = -2.0 * (ex * sn), uxx = ux, uyy = -4.0 * ux;
    const double c = -(1.0 + x * x + y * y);
    k.s00 = s1; k.s01 = 0.0; k.s10 = 0.0; k.s11 = s2;
    k.b0 = y; k.b1 = -x; k.c = c;
    k.f = -(0.5 * (s1 * s1 * uxx + s2 * s2 * uyy) + (y * ux - x * uy) + c * (ux + 1.0));
    k.g0 = ux;
    k.g1 = uy;
  } else {
    coef_f64<KIND>(P, x, y, k);
  }
  if (!P.use_cv) { k.g0 = 0.0; k.g1 = 0.0; }
}
// u_f64 likewise (the values of exits on the global boundary)
template <int KIND>
__device__ __forceinline__ double u_t64(const ProblemDev& P, const Fast64& T, double x, double y) {
  if constexpr (KIND == PK_POISSON_SINCOS) {
    double sx, cx, sy, cy;
    f64::sincospi(T, x, sx, cx);
    f64::sincospi(T, y, sy, cy);
    return sx * cy + x * y;
  } else if constexpr (KIND == PK_HELMHOLTZ) {
    double sa, ca, sb, cb;
    f64::sincos(T, P.p[0] * x, sa, ca);
    f64::sincos(T, P.p[1] * y, sb, cb);
    return sa * cb;
  } else if constexpr (KIND == PK_VARCOEF) {
    double sn, cs;
    f64::sincos(T, 2.0 * y, sn, cs);
    return f64::exp(T, x) * cs + 1.0;
  } else {
    return u_f64<KIND>(P, x, y);
  }
}

// |d| < edge for edge >= 0, as integers (no FP64 comparison); false for NaN
__device__ __forceinline__ bool abs_below(double d, double edge) {
  return (unsigned long long)(__double_as_longlong(d) & 0x7fffffffffffffffLL) <
         (unsigned long long)__double_as_longlong(edge);
}

template <int KIND, bool RICH, int GEOM>
__global__ void __launch_bounds__(FP64_THREADS, is_lut_kind(KIND) ? 1 : 2)
k_paths_fp64(const Fp64Args a) {
  extern __shared__ double Ssum[];  // [warps][sum n] the slots' RBF sums, then [sum n] local t
  __shared__ double s_qs[FP64_THREADS / 32][FP64_QCAP], s_qy[FP64_THREADS / 32][FP64_QCAP];
  __shared__ int s_qd[FP64_THREADS / 32][FP64_QCAP];
  __shared__ int s_qn[FP64_THREADS / 32];
  __shared__ ItemSide64 s_side[4];
  __shared__ double s_rect[4];
  __shared__ int s_item, s_knot, s_nall;
  // slots: ends in this iteration (6 bits), queued exits (8), iterations with ends before
  __shared__ unsigned s_ends[2][FP64_SLOTS];
  __shared__ double s_h;
  __shared__ double s_red[FP64_THREADS / 32][2];
  __shared__ double s_diag[PDDS_DIAG_N];
  __shared__ unsigned long long s_redi[FP64_THREADS / 32][3];
  const DevLayout& L = a.L;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthr = blockDim.x, NW = nthr >> 5;  // NW slots of a block
  const unsigned lt = (1u << lane) - 1u;

  for (;;) {
    // blocks spread over CTAs: one item per CTA, a block's CTAs next to each other
    if (tid == 0) s_item = a.spread ? (int)blockIdx.x : atomicAdd(a.item_counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= a.n_items) break;
    // item = (block, group of NW slots); block = (knot, chunk of paths)
    const int groups = (a.slots + NW - 1) / NW;
    const int block = item / groups, slot = (item - block * groups) * NW + warp;
    const int kn = block / a.blocks, p0 = (block - kn * a.blocks) * a.block_paths;
    const unsigned path_end = (unsigned)min((int64_t)a.N, (int64_t)p0 + a.block_paths);
    if (tid == 0) {
      const int k = a.mc_knots[kn];
      s_knot = k;
      for (int q = 0; q < PDDS_DIAG_N; q++) s_diag[q] = 0.0;
      const int st = L.knot_stencil[k];
      for (int q = 0; q < 4; q++) s_rect[q] = L.st_rect[4 * st + q];
      s_h = a.h;
      if (a.adaptive_h) {
        Coef<double> kd;
        coef_f64<KIND>(a.P, L.kx[k], L.ky[k], kd);
        s_h = GEOM == 1 ? adaptive_step_polar(L.st_rect + 4 * st, L.kx[k], L.ky[k], a.h, kd)
                        : adaptive_step<double>(L.st_rect + 4 * st, L.kx[k], L.ky[k], a.h, kd);
      }
      int off = 0;
      for (int d = 0; d < 4; d++) {
        const int sd = L.st_side[4 * st + d];
        ItemSide64 is;
        is.glob = L.st_glob[4 * st + d];
        if (sd < 0) {
          is.n = 0; is.orient = 0; is.s_off = off; is.origin = 0.0; is.inv_c2 = 0.0;
          is.t_off = 0; is.R = 0.0;
        } else {
          const int sh = L.sd_shape[sd];
          is.n = L.sd_n[sd];
          is.orient = L.sd_orient[sd];
          is.s_off = off;
          is.origin = L.sd_origin[sd];
          is.R = L.sh_R ? L.sh_R[sh] : 0.0;
          if (GEOM == 1 && is.orient == 0) {  // arc: the side's angles in this stencil's turn
            const double tw = 6.283185307179586;
            is.origin += tw * nearbyint((L.st_rect[4 * st + 1] - is.origin) / tw);
          }
          const double c = L.sh_c[sh];
          is.inv_c2 = 1.0 / (c * c);
          is.t_off = L.sh_t_off[sh];
          off += is.n;
        }
        s_side[d] = is;
      }
      s_nall = off;
    }
    __syncthreads();
    const int knot = s_knot, nall = s_nall;
    const double h = s_h, sqrth = ::sqrt(s_h);
    double* tloc = Ssum + NW * nall;
    double* Sw = Ssum + warp * nall;  // this warp's sums
    for (int i = tid; i < NW * nall; i += nthr) Ssum[i] = 0.0;
    if (lane == 0) s_qn[warp] = 0;
    for (int d = 0; d < 4; d++)
      for (int i = tid; i < s_side[d].n; i += nthr)
        tloc[s_side[d].s_off + i] = L.sh_t[s_side[d].t_off + i];
    __syncthreads();

    const double x0 = L.kx[knot], y0 = L.ky[knot];
    const double rect[4] = {s_rect[0], s_rect[1], s_rect[2], s_rect[3]};
    const double pa0 = GEOM == 1 ? ::cos(rect[1]) : 0.0, pa1 = GEOM == 1 ? ::sin(rect[1]) : 0.0;
    const double pb0 = GEOM == 1 ? ::cos(rect[3]) : 0.0, pb1 = GEOM == 1 ? ::sin(rect[3]) : 0.0;
    // PK_ROBIN: the reflecting stencil side (a global side in the Robin set
    // P.p[0], bits N 1, S 2, E 4, W 8), its line n . (x, y) = rc
    const int globmask = (s_side[0].glob ? 1 : 0) | (s_side[1].glob ? 2 : 0) | (s_side[2].glob ? 4 : 0) |
                         (s_side[3].glob ? 8 : 0);
    const int rmask = KIND == PK_ROBIN ? (globmask & (int)a.P.p[0]) : 0;
    double rn0 = 0.0, rn1 = 0.0, rc = 0.0;
    if (rmask & 1) { rn1 = 1.0; rc = rect[3]; }
    else if (rmask & 2) { rn1 = -1.0; rc = -rect[1]; }
    else if (rmask & 4) { rn0 = 1.0; rc = rect[2]; }
    else if (rmask & 8) { rn0 = -1.0; rc = -rect[0]; }
    const Fast64& T = a.T;
    constexpr double S = iso64<KIND> ? sigma64<KIND> : 1.0;
    const double hf = 0.5 * h, sqf = ::sqrt(hf);
    const double cx = 0.5 * (rect[0] + rect[2]), cy = 0.5 * (rect[1] + rect[3]);
    // constant sigma: a path is inside while |x - cx| < ex and |y - cy| < ey
    const double thr_c = -0.5826 * S * sqrth, thr_f = -0.5826 * S * sqf;
    const double exc = ::fmax((rect[2] - cx) + thr_c, 0.0), eyc = ::fmax((rect[3] - cy) + thr_c, 0.0);
    const double exf = ::fmax((rect[2] - cx) + thr_f, 0.0), eyf = ::fmax((rect[3] - cy) + thr_f, 0.0);
    Coef<double> k0;
    if constexpr (!iso64<KIND>) coef_t64<KIND>(a.P, T, x0, y0, k0);
    unsigned path = (unsigned)(p0 + 32 * slot + lane);
    bool active = path < path_end;
    // Hand-out of the block's paths beyond the slots' first ones: by the
    // iteration in which a lane's path ends, then the slot with fewer such
    // iterations so far, the higher slot, the lower lane.  A path's slot
    // decides which of the sums S its exits enter, so no timing may enter
    // here; while paths are left (every lane of the block then has one) the
    // block's warps exchange their ends after every iteration.  The rule is
    // the order in which the warps of one CTA come to an atomic counter,
    // nearly: of 22,261 hand-outs to two slots in one iteration 1,178 came
    // first to the one with fewer ends and 52 to the other.
    unsigned next = (unsigned)p0 + 32u * FP64_SLOTS;  // next path to hand out, the same in every warp
    unsigned ends = 0;                                // iterations of this slot with ends
    unsigned phase = 0;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (a.spread && next < path_end) cluster.sync();  // every CTA of the block has started
    double b = 0.0, bb = 0.0;
    unsigned long long nsteps = 0, nglob = 0, nsten = 0;
    // exit on side d at side coordinate `along` (x or y on rectangles, angle
    // or radius on polar stencils), projection (Ex, Ey)
    auto exit_level = [&](Lvl64& s, double wgt, double Ex, double Ey, int d, bool glob,
                          double along) -> double {
      if (isnan(s.x) || isnan(s.y)) {
        // a position that is not a number lies on no side: reported, scores nothing
        atomicOr(a.err_flags, ERR_FLAG_EXIT_SIDE);
        return 0.0;
      }
      if (glob) {
        ++nglob;
        s.phi = s.Z + s.Y * u_t64<KIND>(a.P, T, Ex, Ey);
        return s.phi + s.xi;
      }
      if (a.diag) s.phi = s.Z + s.Y * u_t64<KIND>(a.P, T, Ex, Ey);
      ++nsten;
      if (d < 0) {
        atomicOr(a.err_flags, ERR_FLAG_EXIT_SIDE);
      } else {
        // queue the exit: FP64_QCAP - 64 left over + at most 2 exits per lane
        // and iteration fit in FP64_QCAP
        const int e = atomicAdd(&s_qn[warp], 1);
        if (idx_ok(e, FP64_QCAP, a.err_flags)) {
          s_qd[warp][e] = d;
          s_qs[warp][e] = along - s_side[d].origin;
          s_qy[warp][e] = wgt * s.Y;
        }
      }
      return s.Z + s.xi;
    };
    // Add the queued exits' RBF vectors to this warp's sums (warp-uniform
    // call; only when at least minq exits are queued).
    auto flush = [&](int minq) {
      __syncwarp();
      const int n = s_qn[warp];
      if (n < minq) return;
      for (int e = 0; e < min(n, FP64_QCAP); e++) {
        const ItemSide64& is = s_side[s_qd[warp][e]];
        const double sc = s_qs[warp][e], yw = s_qy[warp][e];
        for (int j = lane; j < is.n; j += 32) {
          const double dt0 = tloc[is.s_off + j] - sc;
          const double dt = GEOM == 1 && is.R > 0.0 ? 2.0 * is.R * ::sin(0.5 * dt0) : dt0;
          Sw[is.s_off + j] += yw * ::exp(-(dt * dt) * is.inv_c2);
        }
      }
      __syncwarp();
      if (lane == 0) s_qn[warp] = 0;
      __syncwarp();
    };
    // One step of a level with the increments i0, i1 = sqrt(h) z and its
    // exit; ex, ey: the level's exit edges.
    // exs: Exp(1) sample of the reflected step (PK_ROBIN), see k_mixed.cu
    auto step_level = [&](Lvl64& s, double i0, double i1, double hh, double sq, double ex, double ey, double wgt,
                          double& val, double exs) -> bool {
      if constexpr (iso64<KIND>) {
        Coef<double> k;
        coef_t64<KIND>(a.P, T, s.x, s.y, k);
        // Robin: the increment's product may be fused with the push along the
        // normal below, which is the rounding that this step has always had
        const double d0 = KIND == PK_ROBIN ? S * i0 : __dmul_rn(S, i0);
        const double d1 = KIND == PK_ROBIN ? S * i1 : __dmul_rn(S, i1);
        const double gd = fma(k.g0, d0, k.g1 * d1);
        if constexpr (react64<KIND> || KIND == PK_ROBIN) {
          s.xi = fma(-s.Y, gd, s.xi);
          s.Z = fma(k.f * s.Y, hh, s.Z);
          if constexpr (react64<KIND>) s.Y = fma(k.c * s.Y, hh, s.Y);
        } else {  // Y stays 1
          s.xi -= gd;
          s.Z = fma(k.f, hh, s.Z);
        }
        if constexpr (KIND == PK_ROBIN) {
          double dL = 0.0;
          if (rmask) {
            const double dR = rn0 * s.x + rn1 * s.y - rc;
            const double U = rn0 * d0 + rn1 * d1;
            const double M = 0.5 * (U + ::sqrt(U * U + 4.0 * hh * exs));  // |sigma^T n|^2 = 2
            dL = ::fmax(0.0, M + dR);
            if (dL > 0.0) {  // exact in dL, as in k_mixed.cu
              double vphi, psi;
              robin_data<double>(s.x - dR * rn0, s.y - dR * rn1, rn0, rn1, vphi, psi);
              const double t = vphi * dL;
              const double em1 = ::expm1(t);
              s.Z += psi * s.Y * (t != 0.0 ? em1 / vphi : dL);
              s.Y += s.Y * em1;
            }
          }
          s.x += d0 - dL * rn0;
          s.y += d1 - dL * rn1;
        } else {
          s.x = __dadd_rn(s.x, d0);
          s.y = __dadd_rn(s.y, d1);
        }
      } else {
        const double d0 = __dmul_rn(s.k.s00, i0), d1 = __dmul_rn(s.k.s11, i1);
        s.xi = fma(-s.Y, fma(s.k.g0, d0, s.k.g1 * d1), s.xi);
        s.Z = fma(s.k.f * s.Y, hh, s.Z);
        s.Y = fma(s.k.c * s.Y, hh, s.Y);
        s.x += fma(s.k.b0, hh, d0);
        s.y += fma(s.k.b1, hh, d1);
        coef_t64<KIND>(a.P, T, s.x, s.y, s.k);
      }
      ++s.steps;
      if constexpr (GEOM == 1) {
        // polar stencil, isotropic sigma: outside distances beyond the inner
        // arc (none at the centre), the outer arc and the two rays
        const double rho = ::sqrt(s.x * s.x + s.y * s.y);
        const double d_in = rect[0] > 0.0 ? rect[0] - rho : -1e300;
        const double d_out = rho - rect[2];
        const bool has_rays = rect[3] - rect[1] < 6.2;  // a full disk has one side, its arc
        const double d_a = has_rays ? pa1 * s.x - pa0 * s.y : -1e300;
        const double d_b = has_rays ? pb0 * s.y - pb1 * s.x : -1e300;
        int d = 1;
        double mx = d_in;
        if (d_out > mx) { mx = d_out; d = 0; }
        if (d_a > mx) { mx = d_a; d = 3; }
        if (d_b > mx) { mx = d_b; d = 2; }
        if (mx < -0.5826 * S * sq) {
          if (s.steps < (unsigned)a.max_steps) return false;
          atomicOr(a.err_flags, ERR_FLAG_STEP_LIMIT);
          val = 0.0;
          return true;
        }
        double along, Ex = 0.0, Ey = 0.0;
        if (d <= 1) {
          // (the roundings of both forms stated: left to the compiler, they depend on the code around)
          const double sn = RICH ? __dsub_rn(__dmul_rn(pa0, s.y), __dmul_rn(pa1, s.x))
                                 : fma(pa0, s.y, -__dmul_rn(pa1, s.x));
          const double rel = ::atan2(sn, fma(pa0, s.x, __dmul_rn(pa1, s.y)));
          along = rect[1] + (has_rays ? ::fmin(::fmax(rel, 0.0), rect[3] - rect[1])
                                      : (rel < 0.0 ? rel + 6.283185307179586 : rel));
          ::sincos(along, &Ey, &Ex);
          Ex *= rect[d == 0 ? 2 : 0];
          Ey *= rect[d == 0 ? 2 : 0];
        } else {
          const double t = d == 3 ? pa0 * s.x + pa1 * s.y : pb0 * s.x + pb1 * s.y;
          along = ::fmin(::fmax(t, rect[0]), rect[2]);
        }
        val = exit_level(s, wgt, Ex, Ey, d, d == 0 && s_side[0].glob, along);
        return true;
      } else if constexpr (KIND == PK_ROBIN) {
        // absorbing sides only; the exit side is the one with the largest
        // outside distance (ties S, N, W, E), the other coordinate clamped
        const double o0 = (rmask & 1) ? -1e300 : s.y - rect[3], o1 = (rmask & 2) ? -1e300 : rect[1] - s.y;
        const double o2 = (rmask & 4) ? -1e300 : s.x - rect[2], o3 = (rmask & 8) ? -1e300 : rect[0] - s.x;
        int d = 1;
        double mx = o1;
        if (o0 > mx) { mx = o0; d = 0; }
        if (o3 > mx) { mx = o3; d = 3; }
        if (o2 > mx) { mx = o2; d = 2; }
        if (mx < -0.5826 * 1.4142135623730951 * sq) {
          if (s.steps < (unsigned)a.max_steps) return false;
          atomicOr(a.err_flags, ERR_FLAG_STEP_LIMIT);
          val = 0.0;
          return true;
        }
        const double Ex = d == 3 ? rect[0] : (d == 2 ? rect[2] : ::fmin(::fmax(s.x, rect[0]), rect[2]));
        const double Ey = d == 1 ? rect[1] : (d == 0 ? rect[3] : ::fmin(::fmax(s.y, rect[1]), rect[3]));
        val = exit_level(s, wgt, Ex, Ey, d, s_side[d].glob != 0, s_side[d].orient == 0 ? Ex : Ey);
        return true;
      } else {
        // inside: the larger of |x - cx| - hx and |y - cy| - hy is below the
        // threshold -0.5826 |N^T sigma| sqrt(h), N the normal of that side
        // (beyond a corner the distance is positive and the threshold is not)
        bool inside;
        if constexpr (iso64<KIND>) {
          inside = abs_below(s.x - cx, ex) && abs_below(s.y - cy, ey);
        } else {
          const double dx = ::fabs(s.x - cx) - (rect[2] - cx), dy = ::fabs(s.y - cy) - (rect[3] - cy);
          const bool xs = dx > dy;
          inside = (xs ? dx : dy) < -0.5826 * ::fabs(xs ? s.k.s00 : s.k.s11) * sq;
        }
        if (inside) {
          if (s.steps < (unsigned)a.max_steps) return false;
          atomicOr(a.err_flags, ERR_FLAG_STEP_LIMIT);
          val = 0.0;
          return true;
        }
        double Ex, Ey, Nx, Ny;
        int onmask;
        rect2d<double>(rect, s.x, s.y, Ex, Ey, Nx, Ny, onmask);
        const int d = exit_side(onmask);
        const bool glob = ((onmask & 1) && s_side[0].glob) || ((onmask & 2) && s_side[1].glob) ||
                          ((onmask & 4) && s_side[2].glob) || ((onmask & 8) && s_side[3].glob);
        val = exit_level(s, wgt, Ex, Ey, d, glob, d >= 0 && s_side[d].orient == 0 ? Ex : Ey);
        return true;
      }
    };
    Lvl64 fine, coarse;
    auto reset = [&]() {
      fine.x = x0; fine.y = y0; fine.Y = 1.0; fine.Z = 0.0; fine.xi = 0.0; fine.phi = 0.0;
      if constexpr (!iso64<KIND>) fine.k = k0;
      fine.steps = 0;
      coarse = fine;
    };
    reset();
    bool fine_alive = active, coarse_alive = RICH && active;
    double val_f = 0.0, val_c = 0.0;
    unsigned m = 0;
    u32x4 blk;
    blk.v[0] = blk.v[1] = blk.v[2] = blk.v[3] = 0;
    while (__any_sync(FULL, active)) {
      bool fin = false;  // the lane's path (pair) finished in this iteration
      if (active) {
        if (RICH) {
          const unsigned mi = m++;
          blk = path_block(a.seed, a.instance, knot_word(a.L, knot), path, mi);
          double za0, za1, zb0, zb1;
          normals_f64(blk.v[0], blk.v[1], za0, za1);
          normals_f64(blk.v[2], blk.v[3], zb0, zb1);
          double x0e = 0.0, x1e = 0.0, x2e = 0.0;  // Exp(1) samples of reflected steps
          if (KIND == PK_ROBIN && rmask) {
            const u32x4 bx = path_block(a.seed, a.instance, knot_word(a.L, knot) | 0x80000000u, path, mi);
            x0e = -::log(u01_fp64(bx.v[0]));
            x1e = -::log(u01_fp64(bx.v[1]));
            x2e = -::log(u01_fp64(bx.v[2]));
          }
          if (fine_alive) fine_alive = !step_level(fine, sqf * za0, sqf * za1, hf, sqf, exf, eyf, 2.0, val_f, x0e);
          if (fine_alive) fine_alive = !step_level(fine, sqf * zb0, sqf * zb1, hf, sqf, exf, eyf, 2.0, val_f, x1e);
          if (coarse_alive)
            coarse_alive = !step_level(coarse, sqf * (za0 + zb0), sqf * (za1 + zb1), h, sqrth, exc, eyc, -1.0, val_c,
                                       x2e);
          if (!fine_alive && !coarse_alive) {
            const double v = 2.0 * val_f - val_c;
            b += v;
            bb += v * v;
            nsteps += fine.steps + coarse.steps;
            fin = true;
            if (a.diag)
              diag_add(s_diag, 2.0 * fine.phi - coarse.phi, 2.0 * fine.xi - coarse.xi, fine.steps * hf,
                       2.0 * fine.steps);
          }
        } else {
          if ((m & 1u) == 0) blk = path_block(a.seed, a.instance, knot_word(a.L, knot), path, m >> 1);
          double z0, z1;
          normals_f64(m & 1u ? blk.v[2] : blk.v[0], m & 1u ? blk.v[3] : blk.v[1], z0, z1);
          double xe = 0.0;
          if (KIND == PK_ROBIN && rmask) {
            const u32x4 bx = path_block(a.seed, a.instance, knot_word(a.L, knot) | 0x80000000u, path, m >> 1);
            xe = -::log(u01_fp64(bx.v[m & 1u]));
          }
          ++m;
          if (step_level(fine, sqrth * z0, sqrth * z1, h, sqrth, exc, eyc, 1.0, val_f, xe)) {
            b += val_f;
            bb += val_f * val_f;
            nsteps += fine.steps;
            fin = true;
            if (a.diag) diag_add(s_diag, fine.phi, fine.xi, fine.steps * h, 2.0 * fine.steps);
          }
        }
      }
      const unsigned fm = __ballot_sync(FULL, fin);
      unsigned take = path_end;
      int minq = 32;
      if (next < path_end) {
        __syncwarp();  // every lane's exits are queued
        const unsigned mine = (unsigned)__popc(fm) | (unsigned)s_qn[warp] << 6 | ends << 14;
        unsigned* slots = s_ends[phase];
        if (a.spread) {
          if (lane < groups) *cluster.map_shared_rank(slots + slot, lane) = mine;
          cluster.sync();
        } else {
          if (lane == 0) slots[slot] = mine;
          __syncthreads();
        }
        const unsigned other = lane < FP64_SLOTS ? slots[lane] : 0u, n = other & 0x3fu, before = other >> 14;
        const bool first = before < ends || (before == ends && lane > slot);
        take = next + __reduce_add_sync(FULL, first ? n : 0u) + (unsigned)__popc(fm & lt);
        next += __reduce_add_sync(FULL, n);
        ends = min(ends + (fm != 0u ? 1u : 0u), 0x3ffffu);
        phase ^= 1u;
        // warps in step add their exits together: one that did it alone would
        // hold up the others (for as long as seven iterations with 127 side
        // knots: 12x12/n43 5.5 s, together 3.4)
        minq = __reduce_max_sync(FULL, other >> 6 & 0xffu) > FP64_QCAP - 64 ? 1 : FP64_QCAP + 1;
      }
      if (fin) {
        path = take;
        if (path >= path_end) {
          active = false;
        } else {
          reset();
          fine_alive = true;
          coarse_alive = RICH;
          m = 0;
        }
      }
      flush(minq);
    }
    flush(1);
    __syncthreads();
    // the slot's sums
    {
      double* out = a.S + ((int64_t)block * FP64_SLOTS + slot) * a.sum_stride;
      for (int i = lane; i < nall; i += 32) out[i] = Sw[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      b += __shfl_xor_sync(FULL, b, o);
      bb += __shfl_xor_sync(FULL, bb, o);
      nsteps += __shfl_xor_sync(FULL, nsteps, o);
      nglob += __shfl_xor_sync(FULL, nglob, o);
      nsten += __shfl_xor_sync(FULL, nsten, o);
    }
    if (lane == 0) {
      s_red[warp][0] = b;
      s_red[warp][1] = bb;
      s_redi[warp][0] = nsteps;
      s_redi[warp][1] = nglob;
      s_redi[warp][2] = nsten;
    }
    __syncthreads();
    if (tid == 0) {
      double tb = 0.0, tbb = 0.0;
      unsigned long long ts = 0, tg = 0, tt = 0;
      for (int w = 0; w < NW; w++) {
        tb += s_red[w][0]; tbb += s_red[w][1];
        ts += s_redi[w][0]; tg += s_redi[w][1]; tt += s_redi[w][2];
      }
      atomicAdd(a.Bsum + knot, tb);
      atomicAdd(a.BBsum + knot, tbb);
      atomicAdd(a.stats + 0, ts);
      atomicAdd(a.stats + 2, tg);
      atomicAdd(a.stats + 3, tt);
    }
    if (a.diag) diag_flush(s_diag, a.diag + (int64_t)knot * PDDS_DIAG_N, tid);
    if (a.spread) break;
    __syncthreads();
  }
}

// G_i = -(1/N) sum_j ipsi(j,i) S_j of one block of paths, S_j the slots'
// sums added in order.
constexpr int ROWS64_THREADS = 128;
__global__ void __launch_bounds__(ROWS64_THREADS) k_rows_fp64(const Fp64Args a) {
  extern __shared__ double S[];
  __shared__ int s_n[4], s_soff[4];
  __shared__ int64_t s_ip[4], s_map[4];
  const DevLayout& L = a.L;
  const int block = blockIdx.x, tid = threadIdx.x;
  const int knot = a.mc_knots[block / a.blocks];
  const int st = L.knot_stencil[knot];
  if (tid == 0) {
    int off = 0;
    int64_t moff = L.st_map_off[st];
    for (int d = 0; d < 4; d++) {
      const int sd = L.st_side[4 * st + d];
      s_n[d] = sd < 0 ? 0 : L.sd_n[sd];
      s_soff[d] = off;
      s_map[d] = moff;
      s_ip[d] = sd < 0 ? 0 : L.sh_ipsi_off[L.sd_shape[sd]];
      off += s_n[d];
      moff += s_n[d];
    }
  }
  __syncthreads();
  const int nall = s_soff[3] + s_n[3];
  const double* src = a.S + (int64_t)block * FP64_SLOTS * a.sum_stride;
  for (int i = tid; i < nall; i += ROWS64_THREADS) {
    double t = src[i];
#pragma unroll
    for (int w = 1; w < FP64_SLOTS; w++)
      if (w < a.slots) t += src[w * a.sum_stride + i];
    S[i] = t;
  }
  __syncthreads();
  const int64_t row0 = L.row_ptr[knot];
  for (int pr = tid; pr < nall; pr += ROWS64_THREADS) {
    int d = 0, i = pr;
    while (i >= s_n[d]) { i -= s_n[d]; ++d; }
    const int n = s_n[d];
    const int64_t mp = s_map[d] + i;
    if (!a.dup_sum && !L.map_owner[mp]) continue;
    const double* ip = L.ipsi + s_ip[d] + i;
    const double* Sd = S + s_soff[d];
    double acc = 0.0;
#pragma unroll 8
    for (int j = 0; j < n; j++) acc = fma(__ldg(ip + (int64_t)j * n), Sd[j], acc);
    if (idx_ok(L.map_pos[mp], L.row_ptr[knot + 1] - row0, a.err_flags))
      atomicAdd(a.G + row0 + L.map_pos[mp], -acc * a.inv_N);
  }
}

}  // namespace

// Dynamic shared memory of the largest launch (eight slots' sums and the side
// knots' coordinates, four sides of 160 knots).  The kernels' limit is always
// set to this: with the launch's own size, a launch of another context in
// another thread could lower it in between.
constexpr int FP64_SMEM_MAX = (FP64_SLOTS + 1) * 4 * 160 * (int)sizeof(double);

template <bool RICH>
static cudaError_t launch_fp64_t(const Fp64Args& a, int kind, int grid, int threads, size_t smem, cudaStream_t s) {
#define PDDS_FP64_CASE(KK, GG)                                                                           \
  case KK:                                                                                               \
    cudaFuncSetAttribute(k_paths_fp64<KK, RICH, GG>, cudaFuncAttributeMaxDynamicSharedMemorySize, FP64_SMEM_MAX); \
    return cudaLaunchKernelEx(&cfg, k_paths_fp64<KK, RICH, GG>, a);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  // the CTAs of a spread block with paths to hand out (all of its slots are
  // filled) exchange their ends through distributed shared memory
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = (unsigned)(a.slots * 32 / threads);
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cfg.attrs = &cluster;
  cfg.numAttrs = a.spread && a.block_paths > 32 * FP64_SLOTS ? 1 : 0;
  if (a.L.geom == 1) {
    switch (kind) {
      PDDS_FP64_CASE(0, 1)
      PDDS_FP64_CASE(5, 1)
      default: return cudaErrorInvalidValue;
    }
  } else {
    switch (kind) {
      PDDS_FP64_CASE(0, 0)
      PDDS_FP64_CASE(1, 0)
      PDDS_FP64_CASE(2, 0)
      PDDS_FP64_CASE(3, 0)
      PDDS_FP64_CASE(4, 0)
      PDDS_FP64_CASE(5, 0)
      PDDS_FP64_CASE(6, 0)
      default: return cudaErrorInvalidValue;
    }
  }
#undef PDDS_FP64_CASE
}

cudaError_t launch_paths_fp64(const Fp64Args& a, int kind, int grid, int threads, size_t smem, cudaStream_t s) {
  return a.richardson ? launch_fp64_t<true>(a, kind, grid, threads, smem, s)
                      : launch_fp64_t<false>(a, kind, grid, threads, smem, s);
}

cudaError_t launch_rows_fp64(const Fp64Args& a, int n_blocks, cudaStream_t s) {
  k_rows_fp64<<<n_blocks, ROWS64_THREADS, a.sum_stride * sizeof(double), s>>>(a);
  return cudaGetLastError();
}

template <bool RICH>
static int blocks64_t(int kind, size_t smem, int threads) {
  int nb = 0;
  switch (kind) {
    case 0: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<0, RICH, 0>, threads, smem); break;
    case 1: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<1, RICH, 0>, threads, smem); break;
    case 2: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<2, RICH, 0>, threads, smem); break;
    case 4: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<4, RICH, 0>, threads, smem); break;
    case 5: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<5, RICH, 0>, threads, smem); break;
    default: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_paths_fp64<3, RICH, 0>, threads, smem); break;
  }
  return nb;
}

int fp64_blocks_per_sm(int kind, size_t smem, int richardson, int threads) {
  return richardson ? blocks64_t<true>(kind, smem, threads) : blocks64_t<false>(kind, smem, threads);
}

}  // namespace pdds
