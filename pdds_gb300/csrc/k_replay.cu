// REPLAY_FP64 mode: bit-exact replay of the CPU restatement of the reference.
//
// Compiled with -fmad=false so no multiply-add is contracted, and every
// elementary function comes from pdds_portable.h, so each operation below
// rounds exactly as the host restatement does.  The path phase follows
//   Step (control variate)   Integrators/FKACIntegrator.hpp:46-57
//   Inside (Gobet shift)     Integrators/FKACIntegrator.hpp:168-222
//   Simulate_OMP             Solvers/EMFKACSolver.hpp:138-213 (linear + sublinear legs)
// one lane per path, lanes taking the next path when theirs ends.  The
// reduction keeps the reference's serial order:
//   Reduce_Analytic          Solvers/EMFKACSolver.hpp:514-575 (paths in order)
//   G_update                 Meshes/stencil.cpp:244-307 (H_i over j in order)
//   G_return_withrep         Meshes/stencil.cpp:343-406 (sides N,S,E,W)
// but only the additions into the sums are serial: the terms (the score of a
// path, H_i Y of an exit) are formed by whole CTAs first.
//
// What bounds it: the FP64 pipe (one warp instruction per 64 cycles and
// scheduler).  So operations whose outcome is known are left out where no
// bit can change: products with the zeros of a diagonal sigma, products with
// a Y that stays 1, the normal's length (sqrt(s s) = |s| exactly), and the
// distance once a path is outside the stencil, where it is positive and the
// threshold is not.
//
// 4x4/n11, N = 1e4, h = 1e-3 (one thread per path, and one per side knot that
// walked every path, -> now): paths 216 -> 38 ms, G 626 -> 12 ms, B 43 -> 1.0 ms.
#include <algorithm>

#include "dev_common.cuh"
#include "kernels.h"

namespace pdds {

namespace {

constexpr int DIR_N_ = 0, DIR_S_ = 1, DIR_E_ = 2, DIR_W_ = 3;

template <int KIND>
__device__ void coef_port(const ProblemDev& P, double x, double y, Coef<double>& k) {
  const double PI = pm::PI;
  if (KIND == PK_LUT) {
    double v[8];
    lut_sample<double, 8>(P.lut, x, y, v);
    k.s00 = v[0]; k.s01 = 0.0; k.s10 = 0.0; k.s11 = v[1];
    k.b0 = v[2]; k.b1 = v[3]; k.c = v[4]; k.f = v[5]; k.g0 = v[6]; k.g1 = v[7];
  } else if (KIND == PK_POISSON_SINCOS) {
    double sx, cx, sy, cy;
    pm::sincos(PI * x, &sx, &cx);
    pm::sincos(PI * y, &sy, &cy);
    k.s00 = 1.4142135623730951; k.s01 = 0.0; k.s10 = 0.0; k.s11 = 1.4142135623730951;
    k.b0 = 0.0; k.b1 = 0.0; k.c = 0.0;
    k.f = 19.739208802178716 * (sx * cy);
    k.g0 = PI * (cx * cy) + y;
    k.g1 = x - PI * (sx * sy);
  } else if (KIND == PK_HELMHOLTZ) {
    const double a = P.p[0], b = P.p[1], c = P.p[2];
    double sa, ca, sb, cb;
    pm::sincos(a * x, &sa, &ca);
    pm::sincos(b * y, &sb, &cb);
    k.s00 = 1.4142135623730951; k.s01 = 0.0; k.s10 = 0.0; k.s11 = 1.4142135623730951;
    k.b0 = 0.0; k.b1 = 0.0; k.c = c;
    k.f = ((a * a + b * b) - c) * (sa * cb);
    k.g0 = a * (ca * cb);
    k.g1 = -(b * (sa * sb));
  } else {  // PK_VARCOEF (the Monegros problem has no portable form)
    const double s1 = 1.0 + 0.5 * (x * x), s2 = 1.0 + 0.5 * (y * y);
    double sn, cs;
    pm::sincos(2.0 * y, &sn, &cs);
    const double ex = pm::exp(x);
    const double ux = ex * cs, uy = -2.0 * (ex * sn), uxx = ux, uyy = -4.0 * ux;
    const double c = -(1.0 + x * x + y * y);
    const double u = ux + 1.0;
    k.s00 = s1; k.s01 = 0.0; k.s10 = 0.0; k.s11 = s2;
    k.b0 = y; k.b1 = -x; k.c = c;
    k.f = -(0.5 * (s1 * s1 * uxx + s2 * s2 * uyy) + (y * ux - x * uy) + c * u);
    k.g0 = ux;
    k.g1 = uy;
  }
  if (!P.use_cv) { k.g0 = 0.0; k.g1 = 0.0; }
}

template <int KIND>
__device__ double u_port(const ProblemDev& P, double x, double y) {
  if (KIND == PK_LUT) {
    return lut_sample_g<double>(P.lut, x, y);
  } else if (KIND == PK_POISSON_SINCOS) {
    double sx, cx, sy, cy;
    pm::sincos(pm::PI * x, &sx, &cx);
    pm::sincos(pm::PI * y, &sy, &cy);
    return sx * cy + x * y;
  } else if (KIND == PK_HELMHOLTZ) {
    double sa, ca, sb, cb;
    pm::sincos(P.p[0] * x, &sa, &ca);
    pm::sincos(P.p[1] * y, &sb, &cb);
    return sa * cb;
  } else {
    double s2, c2;
    pm::sincos(2.0 * y, &s2, &c2);
    return pm::exp(x) * c2 + 1.0;
  }
}

// Kinds with sigma = sqrt2 I and no drift; of those, kinds without a
// reaction term keep Y = 1.
template <int KIND>
constexpr bool iso64 = KIND == PK_POISSON_SINCOS || KIND == PK_HELMHOLTZ;
template <int KIND>
constexpr bool unit_y64 = KIND == PK_POISSON_SINCOS;

// (2 a + 1) 2^-33, the uniform u01_fp64(a), as exponent and mantissa bits:
// the same double without a conversion and two FP64 operations.
__device__ __forceinline__ uint64_t u01_bits(uint32_t a) {
  const uint64_t n = 2 * (uint64_t)a + 1;  // 1 .. 2^33 - 1
  const int lz = __clzll((long long)n);    // 31 .. 63
  const uint64_t frac = (n << lz) << 1;    // the leading one shifted out
  return ((uint64_t)(1023 + 30 - lz) << 52) | (frac >> 12);
}

// Products e ln2 of pm::log for the exponents of uniforms, e = -33 .. 0.
struct LogTab {
  double hi[34], lo[34];
};

// pm::log of a normal number in (0, 1) given by its bits: the same
// operations; the exponent's products with ln2 come from the table.
__device__ __forceinline__ double log_u01(uint64_t b, const LogTab& t) {
  int e = (int)(b >> 52) - 1023;
  uint64_t mb = (b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL;
  if (mb > 0x3ff6a09e667f3bcdULL) {  // m > sqrt2 (the double 1.4142135623730951): m / 2
    mb -= 0x0010000000000000ULL;
    e += 1;
  }
  const double m = pm::bits_to_double(mb);
  const double f = (m - 1.0) / (m + 1.0);
  const double s = f * f;
  double p = 0.04;
  p = p * s + 0.043478260869565216;
  p = p * s + 0.047619047619047616;
  p = p * s + 0.05263157894736842;
  p = p * s + 0.058823529411764705;
  p = p * s + 0.06666666666666667;
  p = p * s + 0.07692307692307693;
  p = p * s + 0.09090909090909091;
  p = p * s + 0.1111111111111111;
  p = p * s + 0.14285714285714285;
  p = p * s + 0.2;
  p = p * s + 0.3333333333333333;
  const double f2 = 2.0 * f;
  const double lm = f2 + f2 * (s * p);
  return t.hi[-e] + (lm + t.lo[-e]);
}

// box_muller_portable
__device__ __forceinline__ void box_muller_bits(uint32_t a, uint32_t b, const LogTab& t, double* z0, double* z1) {
  const double rho = ::sqrt(-2.0 * log_u01(u01_bits(a), t));
  double s, c;
  pm::sincos(pm::TWO_PI * pm::bits_to_double(u01_bits(b)), &s, &c);
  *z0 = rho * c;
  *z1 = rho * s;
}

// h and sqrt(h) of the range's knots.
template <int KIND>
__global__ void k_replay_h(const ReplayArgs a) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.n_mc) return;
  double h = a.h, sq = a.sqrth;
  if (a.adaptive_h) {
    const int knot = a.mc_knots[m];
    Coef<double> k0;
    coef_port<KIND>(a.P, a.L.kx[knot], a.L.ky[knot], k0);
    h = adaptive_step<double>(a.L.st_rect + 4 * a.L.knot_stencil[knot], a.L.kx[knot], a.L.ky[knot], a.h, k0);
    sq = ::sqrt(h);
  }
  a.knot_h[2 * m] = h;
  a.knot_h[2 * m + 1] = sq;
}

constexpr int RP_THREADS = 128;

template <int KIND>
__global__ void __launch_bounds__(RP_THREADS) k_replay_paths(const ReplayArgs a) {
  __shared__ LogTab tab;
  for (int i = threadIdx.x; i < 34; i += RP_THREADS) {
    const double ed = (double)(-i);
    tab.hi[i] = ed * pm::LN2_HI;
    tab.lo[i] = ed * pm::LN2_LO;
  }
  __syncthreads();
  const DevLayout& L = a.L;
  const int lane = threadIdx.x & 31;
  const unsigned long long total = (unsigned long long)a.n_mc * a.N;
  // the lane's path
  unsigned long long gid = 0;
  int m = 0;
  uint32_t word = 0, path = 0, step = 0;
  u32x4 blk;
  blk.v[0] = blk.v[1] = blk.v[2] = blk.v[3] = 0;
  double X0 = 0.0, X1 = 0.0, Y = 1.0, Z = 0.0, xi = 0.0, E0 = 0.0, E1 = 0.0, h = 0.0, sqrth = 0.0, thr = 0.0;
  double c0 = 0.0, c1 = 0.0, h0 = 0.0, h1 = 0.0;  // centre and half widths of the stencil
  Coef<double> k;
  bool have = false;  // k holds the coefficients at (X0, X1)
  long long nl = 0, ns = 0;
  int side = -2;
  bool sub = false;   // in the sublinear leg
  bool capped = false, active = true, want = true;
  const double S2 = 1.4142135623730951;
  for (;;) {
    // lanes without a path take the next ones
    const unsigned wm = __ballot_sync(0xffffffffu, want);
    if (wm) {
      const int leader = __ffs(wm) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(a.path_counter, (unsigned long long)__popc(wm));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (want) {
        want = false;
        gid = base + __popc(wm & ((1u << lane) - 1u));
        active = gid < total;
        if (active) {
          m = (int)(gid / (unsigned)a.N);
          path = (uint32_t)(gid - (unsigned long long)m * a.N);
          const int knot = a.mc_knots[m];
          const double* sp = L.st_rect + 4 * L.knot_stencil[knot];
          c0 = 0.5 * (sp[0] + sp[2]);
          c1 = 0.5 * (sp[1] + sp[3]);
          h0 = sp[2] - c0;
          h1 = sp[3] - c1;
          X0 = L.kx[knot];
          X1 = L.ky[knot];
          E0 = X0;
          E1 = X1;
          Y = 1.0; Z = 0.0; xi = 0.0;
          h = a.knot_h[2 * m];
          sqrth = a.knot_h[2 * m + 1];
          thr = iso64<KIND> ? -0.5826 * S2 * sqrth : 0.0;
          word = knot_word(L, knot);
          step = 0;
          nl = ns = 0;
          sub = capped = have = false;
        }
      }
    }
    if (!__any_sync(0xffffffffu, active)) break;
    bool done = false;
    if (active) {
      // one step (Step with the control variate)
      if (!have) coef_port<KIND>(a.P, X0, X1, k);
      if ((step & 1u) == 0) blk = path_block(a.seed, a.instance, word, path, step >> 1);
      double z0, z1;
      box_muller_bits(step & 1u ? blk.v[2] : blk.v[0], step & 1u ? blk.v[3] : blk.v[1], tab, &z0, &z1);
      step++;
      const double i0 = sqrth * z0, i1 = sqrth * z1;
      const double v0 = (-k.s00) * k.g0, v1 = (-k.s11) * k.g1;
      if constexpr (unit_y64<KIND>) {
        xi += v0 * i0 + v1 * i1;
        Z += k.f * h;
        X0 += k.s00 * i0;
        X1 += k.s11 * i1;
      } else {
        xi += Y * (v0 * i0 + v1 * i1);
        Z += k.f * Y * h;
        Y += k.c * Y * h;
        if constexpr (iso64<KIND>) {
          X0 += k.s00 * i0;
          X1 += k.s11 * i1;
        } else {
          X0 += k.b0 * h + k.s00 * i0;
          X1 += k.b1 * h + k.s11 * i1;
        }
      }
      // the exit test (Inside) with Rectangle2D's branches: outside the
      // rectangle the distance is positive and the threshold is not
      if ((sub ? ++ns : ++nl) > a.max_steps) {
        capped = true;
        done = true;
        if (!sub) {
          const int64_t o = (int64_t)gid;
          a.ex[o] = E0; a.ey[o] = E1; a.eY[o] = Y; a.eZ[o] = Z; a.exi[o] = xi;
        }
      } else {
        const double d0 = fabs(X0 - c0), d1 = fabs(X1 - c1);
        const bool ox = d0 > h0, oy = d1 > h1;
        const double dx = d0 - h0, dy = d1 - h1;
        const bool xs = dx > dy;
        bool out = ox || oy;
        have = false;
        if (!out) {
          double t = thr;
          if constexpr (!iso64<KIND>) {
            if constexpr (KIND == PK_LUT) {
              coef_port<KIND>(a.P, X0, X1, k);
              have = true;
              t = (sub ? 0.0 : -0.5826) * fabs(xs ? k.s00 : k.s11) * sqrth;
            } else {
              Coef<double> ks;
              coef_port<KIND>(a.P, X0, X1, ks);
              t = (sub ? 0.0 : -0.5826) * fabs(xs ? ks.s00 : ks.s11) * sqrth;
            }
          }
          out = !((xs ? dx : dy) < t);
        }
        if (out) {
          const bool px = ox || oy ? ox : xs;       // the projection moves x
          const bool py = ox || oy ? oy || !ox : !xs;  // and y
          E0 = px ? (X0 > c0 ? h0 + c0 : -h0 + c0) : X0;
          E1 = py ? (X1 > c1 ? h1 + c1 : -h1 + c1) : X1;
          if (!sub) {
            // exit classification of Reduce_Analytic (:559) and G_update (stencil.cpp:246-301)
            const int64_t o = (int64_t)gid;
            a.ex[o] = E0; a.ey[o] = E1; a.eY[o] = Y; a.eZ[o] = Z; a.exi[o] = xi;
            const double* sp = L.st_rect + 4 * L.knot_stencil[a.mc_knots[m]];
            double g0, g1, Nx, Ny;
            int onm;
            const double gd = rect2d<double>(L.dom, E0, E1, g0, g1, Nx, Ny, onm);
            if (gd >= -1e-08) side = -1;
            else if (fabs(E1 - sp[1]) < 1e-8) side = DIR_S_;
            else if (fabs(E1 - sp[3]) < 1e-8) side = DIR_N_;
            else if (fabs(E0 - sp[0]) < 1e-8) side = DIR_W_;
            else if (fabs(E0 - sp[2]) < 1e-8) side = DIR_E_;
            else side = -2;
            sub = true;
            thr = 0.0;
            done = !a.sublinear;
          } else {
            done = true;
          }
        }
      }
    }
    if (done) {
      const int64_t o = (int64_t)gid;
      if (isnan(X0) || isnan(X1)) side = -2;  // a position that is not a number lies on no side
      if (a.diag) {  // the sublinear leg's end (the linear one's when it did not run)
        a.sx[o] = E0; a.sy[o] = E1; a.sY[o] = Y; a.sZ[o] = Z; a.sxi[o] = xi;
      }
      a.esteps_l[o] = (int)nl;
      a.esteps_s[o] = (int)ns;
      a.eside[o] = capped ? -4 : side;
      if (capped) atomicOr(a.err_flags, ERR_FLAG_STEP_LIMIT);
      if (!capped && side == -2) atomicOr(a.err_flags, ERR_FLAG_EXIT_SIDE);
      want = true;
    }
  }
}

// B and BB of one knot: Reduce_Analytic's serial loop over the paths.  The
// CTA forms RB_CHUNK paths' terms, then one lane per sum adds them in order.
constexpr int RB_CHUNK = 256;
constexpr int RB_STRIDE = RB_CHUNK + 1;  // the summing lanes read different banks
constexpr int RB_TERMS = 2 + PDDS_DIAG_N;

template <int KIND>
__global__ void __launch_bounds__(RB_CHUNK) k_replay_b(const ReplayArgs a) {
  extern __shared__ double term[];  // [terms][RB_STRIDE]
  __shared__ unsigned char counts[RB_CHUNK];
  const int m = blockIdx.x, tid = threadIdx.x;
  const int knot = a.mc_knots[m];
  const int nt = a.diag ? RB_TERMS : 2;
  // lane t of warp 0: sum t (b, bb, then the diagnostic sums)
  double acc = 0.0;
  unsigned long long steps = 0;
  unsigned ng = 0, nst = 0;
  const double hk = a.knot_h[2 * m];
  for (int n0 = 0; n0 < a.N; n0 += RB_CHUNK) {
    const int n = n0 + tid;
    if (n < a.N) {
      const int64_t o = (int64_t)m * a.N + n;
      const int side = a.eside[o];
      const double Z = a.eZ[o], Y = a.eY[o], xi = a.exi[o];
      double v = Z + xi;
      if (side == -1) {
        const double score = Z + Y * u_port<KIND>(a.P, a.ex[o], a.ey[o]);
        v = score + xi;
      }
      counts[tid] = side >= -1;
      term[tid] = v;
      term[RB_STRIDE + tid] = v * v;
      steps += (unsigned)a.esteps_l[o];
      ng += side == -1;
      nst += side >= 0;
      if (a.diag) {
        // the diagnostic sums of Reduce_Analytic (Solvers/EMFKACSolver.hpp:542-558),
        // paths in order; tau = steps x h (elapsed time)
        double* d = term + 2 * RB_STRIDE + tid;
        const double phl = Z + Y * u_port<KIND>(a.P, a.ex[o], a.ey[o]);
        const double phs = a.sZ[o] + a.sY[o] * u_port<KIND>(a.P, a.sx[o], a.sy[o]);
        const double xl = xi, xs = a.sxi[o];
        const double sl = (double)a.esteps_l[o], ss = sl + (double)a.esteps_s[o];
        for (int q = 0; q < PDDS_DIAG_N; q++) d[q * RB_STRIDE] = 0.0;
        d[PDDS_DIAG_SCORE * RB_STRIDE] = phl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_SCORE) * RB_STRIDE] = phs;
        d[PDDS_DIAG_SCORE2 * RB_STRIDE] = phl * phl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_SCORE2) * RB_STRIDE] = phs * phs;
        d[PDDS_DIAG_XI * RB_STRIDE] = xl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_XI) * RB_STRIDE] = xs;
        d[PDDS_DIAG_XI2 * RB_STRIDE] = xl * xl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_XI2) * RB_STRIDE] = xs * xs;
        d[PDDS_DIAG_SCORE_VR * RB_STRIDE] = phl + xl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_SCORE_VR) * RB_STRIDE] = phs + xs;
        d[PDDS_DIAG_SCORE_VR2 * RB_STRIDE] = (phl + xl) * (phl + xl);
        d[(PDDS_DIAG_SUB + PDDS_DIAG_SCORE_VR2) * RB_STRIDE] = (phs + xs) * (phs + xs);
        d[PDDS_DIAG_XI_SCORE * RB_STRIDE] = xl * phl;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_XI_SCORE) * RB_STRIDE] = xs * phs;
        d[PDDS_DIAG_RNG * RB_STRIDE] = 2.0 * ss;
        d[PDDS_DIAG_TAU * RB_STRIDE] = sl * hk;
        d[(PDDS_DIAG_SUB + PDDS_DIAG_TAU) * RB_STRIDE] = ss * hk;
        d[PDDS_DIAG_PATHS * RB_STRIDE] = 1.0;
      }
    }
    __syncthreads();
    if (tid < nt) {
      const int n1 = min(RB_CHUNK, a.N - n0);
      const double* t = term + tid * RB_STRIDE;
      for (int q = 0; q < n1; q++)
        if (tid >= 2 || counts[q]) acc += t[q];
    }
    __syncthreads();
  }
  if (tid == 0) a.B[knot] = acc / a.N;
  if (tid == 1) a.BB[knot] = acc / a.N;
  if (tid >= 2 && tid < nt) a.diag[(int64_t)knot * PDDS_DIAG_N + tid - 2] = acc;
  for (int o = 16; o > 0; o >>= 1) {
    steps += __shfl_xor_sync(0xffffffffu, steps, o);
    ng += __shfl_xor_sync(0xffffffffu, ng, o);
    nst += __shfl_xor_sync(0xffffffffu, nst, o);
  }
  if ((tid & 31) == 0) {
    atomicAdd(a.stats + 0, steps);
    atomicAdd(a.stats + 2, (unsigned long long)ng);
    atomicAdd(a.stats + 3, (unsigned long long)nst);
  }
}

// G_update accumulation in two launches, for paths [p0, p1) of every knot.
//
// First the exits' terms H_i Y, in any order: a CTA collects the exits of one
// (knot, side, RG_PATHS paths), RG_EXITS at a time, forms their RBF values r_j
// (each used by every side knot; the per-knot loop this replaces took the n
// exponentials anew for each of the n knots), then
// H_i Y = (sum_j ipsi(j, i) r_j) Y with j in order, into hy[path][i].  FP64
// instructions bound it, so it has to fill every SM: with a CTA per (knot,
// side) and all of its paths, which also added the terms, the side nearest to
// its knot (nine tenths of the exits) set the end: 26.3 ms at 225 knots x 10^4
// paths; the two launches take 10.5 and 1.6 ms.
constexpr int RG_THREADS = 256;
constexpr int RG_EXITS = 32;
constexpr int RG_PATHS = 512;

__global__ void __launch_bounds__(RG_THREADS) k_replay_terms(const ReplayArgs a, int p0, int p1, double* hy, int ld) {
  extern __shared__ double r[];  // [RG_EXITS][n]
  __shared__ int queue[RG_PATHS];
  __shared__ int s_cnt[RG_THREADS / 32];
  __shared__ double s_x[RG_EXITS], s_y[RG_EXITS], s_Y[RG_EXITS];
  const int m = blockIdx.x, d = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const DevLayout& L = a.L;
  const int sd = L.st_side[4 * L.knot_stencil[a.mc_knots[m]] + d];
  if (sd < 0) return;
  const int n = L.sd_n[sd];
  const double c = L.sd_c[sd];
  const double c2 = c * c;
  const double* px = L.side_px + L.sd_knot_off[sd];
  const double* py = L.side_py + L.sd_knot_off[sd];
  const double* ip = a.knot_ipsi_off ? a.ipsi_knot + a.knot_ipsi_off[4 * m + d]
                                     : L.ipsi + L.sh_ipsi_off[L.sd_shape[sd]];
  const int b0 = p0 + blockIdx.z * RG_PATHS, b1 = min(p1, b0 + RG_PATHS);
  int all = 0;
  for (int q0 = b0; q0 < b1; q0 += RG_THREADS) {
    const int p = q0 + tid;
    const bool hit = p < b1 && a.eside[(int64_t)m * a.N + p] == d;
    const unsigned mk = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) s_cnt[warp] = __popc(mk);
    __syncthreads();
    int at = all + __popc(mk & ((1u << lane) - 1u));
    for (int w = 0; w < RG_THREADS / 32; w++) {
      if (w < warp) at += s_cnt[w];
      all += s_cnt[w];
    }
    if (hit) queue[at] = p;
    __syncthreads();
  }
  for (int q0 = 0; q0 < all; q0 += RG_EXITS) {
    const int ne = min(RG_EXITS, all - q0);
    if (tid < ne) {
      const int64_t o = (int64_t)m * a.N + queue[q0 + tid];
      s_x[tid] = a.ex[o];
      s_y[tid] = a.ey[o];
      s_Y[tid] = a.eY[o];
    }
    __syncthreads();
    for (int e = tid; e < ne * n; e += RG_THREADS) {
      const int x = e / n, j = e - x * n;
      // the RBF of the reference (BVPs/BVP.hpp:84-87), c^2 formed once
      const double d0 = px[j] - s_x[x], d1 = py[j] - s_y[x];
      const double nrm = ::sqrt(d0 * d0 + d1 * d1);
      r[e] = pm::exp(-(nrm * nrm) / c2);
    }
    __syncthreads();
    for (int e = tid; e < ne * n; e += RG_THREADS) {
      const int x = e / n, i = e - x * n;
      const double* rx = r + x * n;
      double H = 0.0;
#pragma unroll 4
      for (int j = 0; j < n; j++) H += __ldg(ip + (int64_t)j * n + i) * rx[j];
      hy[((int64_t)m * (p1 - p0) + queue[q0 + x] - p0) * ld + i] = H * s_Y[x];
    }
    __syncthreads();
  }
}

// Then their sums in path order, a thread per (knot, side, side knot): a
// chain of additions, fed by loads RS_AHEAD exits ahead.
constexpr int RS_THREADS = 160;  // side knots of a stencil side, at most
constexpr int RS_PATHS = 640;
constexpr int RS_AHEAD = 16;

__global__ void __launch_bounds__(RS_THREADS) k_replay_sum(const ReplayArgs a, int p0, int p1, const double* hy, int ld,
                                                          const int64_t* knot_task_off, double* Gside,
                                                          double* GGside) {
  __shared__ int queue[RS_PATHS];
  __shared__ int s_cnt[RS_THREADS / 32];
  const int m = blockIdx.x, d = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const DevLayout& L = a.L;
  const int st = L.knot_stencil[a.mc_knots[m]];
  const int sd = L.st_side[4 * st + d];
  if (sd < 0) return;
  int64_t out = knot_task_off[m];
  for (int q = 0; q < d; q++) {
    const int s2 = L.st_side[4 * st + q];
    if (s2 >= 0) out += L.sd_n[s2];
  }
  const int n = L.sd_n[sd];
  const bool mine = tid < n;
  double G = 0.0, GG = 0.0;  // of side knot tid
  if (mine && p0 > 0) {
    G = Gside[out + tid];
    GG = GGside[out + tid];
  }
  const double* h0 = hy + (int64_t)m * (p1 - p0) * ld + tid;
  for (int b0 = p0; b0 < p1; b0 += RS_PATHS) {
    int all = 0;
    for (int q0 = b0; q0 < min(p1, b0 + RS_PATHS); q0 += RS_THREADS) {
      const int p = q0 + tid;
      const bool hit = p < p1 && a.eside[(int64_t)m * a.N + p] == d;
      const unsigned mk = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) s_cnt[warp] = __popc(mk);
      __syncthreads();
      int at = all + __popc(mk & ((1u << lane) - 1u));
      for (int w = 0; w < RS_THREADS / 32; w++) {
        if (w < warp) at += s_cnt[w];
        all += s_cnt[w];
      }
      if (hit) queue[at] = p - p0;
      __syncthreads();
    }
    if (mine) {
      double t[RS_AHEAD];
      int q = 0;
      for (; q + RS_AHEAD <= all; q += RS_AHEAD) {
#pragma unroll
        for (int u = 0; u < RS_AHEAD; u++) t[u] = __ldcs(h0 + (int64_t)queue[q + u] * ld);
#pragma unroll
        for (int u = 0; u < RS_AHEAD; u++) {
          G -= t[u];
          GG += t[u] * t[u];
        }
      }
      for (; q < all; q++) {
        const double v = __ldcs(h0 + (int64_t)queue[q] * ld);
        G -= v;
        GG += v * v;
      }
    }
    __syncthreads();
  }
  if (mine) {
    Gside[out + tid] = G;
    GGside[out + tid] = GG;
  }
}

// G_return_withrep for one knot: sides N, S, E, W in order, G = G_side * (1/N).
__global__ void k_replay_row(const ReplayArgs a, const int64_t* knot_task_off, const double* Gside,
                             const double* GGside) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= a.n_mc) return;
  const DevLayout& L = a.L;
  const int knot = a.mc_knots[m];
  const int st = L.knot_stencil[knot];
  const int64_t r0 = L.row_ptr[knot], r1 = L.row_ptr[knot + 1];
  for (int64_t e = r0; e < r1; e++) { a.G[e] = 0.0; a.GG[e] = 0.0; }
  const double norm = 1.0 / (a.N * 1.0);
  int64_t mo = L.st_map_off[st];
  int64_t to = knot_task_off[m];
  for (int d = 0; d < 4; d++) {
    const int sd = L.st_side[4 * st + d];
    if (sd < 0) continue;
    const int n = L.sd_n[sd];
    for (int i = 0; i < n; i++, mo++, to++) {
      const int64_t e = r0 + L.map_pos[mo];
      if (!idx_ok(e - r0, r1 - r0, a.err_flags)) continue;
      if (a.dup_sum) {
        a.G[e] += Gside[to] * norm;
        a.GG[e] += GGside[to] * norm;
      } else {
        a.G[e] = Gside[to] * norm;
        a.GG[e] = GGside[to] * norm;
      }
    }
  }
  for (int64_t e = r0; e < r1; e++) a.GG[e] = a.GG[e] - a.G[e] * a.G[e];
}

}  // namespace

template <int KIND>
static cudaError_t launch_paths_t(const ReplayArgs& a, int num_sms, cudaStream_t s) {
  int bps = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_replay_paths<KIND>, RP_THREADS, 0);
  const int64_t want = ((int64_t)a.n_mc * a.N + RP_THREADS - 1) / RP_THREADS;
  const int grid = (int)std::min<int64_t>(want, (int64_t)std::max(bps, 1) * std::max(num_sms, 1));
  k_replay_h<KIND><<<(a.n_mc + 127) / 128, 128, 0, s>>>(a);
  k_replay_paths<KIND><<<grid, RP_THREADS, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_replay_paths(const ReplayArgs& a, int kind, int num_sms, cudaStream_t s) {
  if ((int64_t)a.n_mc * a.N == 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(a.path_counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  switch (kind) {
    case PK_POISSON_SINCOS: return launch_paths_t<PK_POISSON_SINCOS>(a, num_sms, s);
    case PK_HELMHOLTZ: return launch_paths_t<PK_HELMHOLTZ>(a, num_sms, s);
    case PK_VARCOEF: return launch_paths_t<PK_VARCOEF>(a, num_sms, s);
    case PK_LUT: return launch_paths_t<PK_LUT>(a, num_sms, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND>
static void launch_b_t(const ReplayArgs& a, cudaStream_t s) {
  const size_t smem = (size_t)(a.diag ? RB_TERMS : 2) * RB_STRIDE * sizeof(double);
  k_replay_b<KIND><<<a.n_mc, RB_CHUNK, smem, s>>>(a);
}

int replay_terms_paths(int n_mc, int N, int max_n) {
  // 512 MB of terms, but at least 128 paths, and at most 65,535 blocks of
  // paths (the grid's z)
  const int64_t per_path = std::max<int64_t>(1, (int64_t)n_mc * max_n * (int64_t)sizeof(double));
  const int64_t fit = std::max<int64_t>(128, ((int64_t)512 << 20) / per_path);
  return (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(N, (int64_t)65535 * RG_PATHS), fit));
}

cudaError_t launch_replay_reduce(const ReplayArgs& a, int kind, int max_n, const int64_t* knot_task_off,
                                 double* Gside, double* GGside, double* hy, int* launches, cudaStream_t s) {
  if (a.n_mc == 0) return cudaSuccess;
  switch (kind) {
    case PK_POISSON_SINCOS: launch_b_t<PK_POISSON_SINCOS>(a, s); break;
    case PK_HELMHOLTZ: launch_b_t<PK_HELMHOLTZ>(a, s); break;
    case PK_VARCOEF: launch_b_t<PK_VARCOEF>(a, s); break;
    case PK_LUT: launch_b_t<PK_LUT>(a, s); break;
    default: return cudaErrorInvalidValue;
  }
  if (max_n > RS_THREADS) return cudaErrorInvalidValue;
  if (max_n > 0) {
    const size_t smem = (size_t)RG_EXITS * max_n * sizeof(double);  // at most 40 KB
    const int part = replay_terms_paths(a.n_mc, a.N, max_n);
    for (int p0 = 0; p0 < a.N; p0 += part) {
      const int p1 = std::min(a.N, p0 + part);
      const int blocks = (p1 - p0 + RG_PATHS - 1) / RG_PATHS;
      k_replay_terms<<<dim3(a.n_mc, 4, blocks), RG_THREADS, smem, s>>>(a, p0, p1, hy, max_n);
      k_replay_sum<<<dim3(a.n_mc, 4), RS_THREADS, 0, s>>>(a, p0, p1, hy, max_n, knot_task_off, Gside, GGside);
      *launches += 2;
    }
  }
  k_replay_row<<<(a.n_mc + 127) / 128, 128, 0, s>>>(a, knot_task_off, Gside, GGside);
  return cudaGetLastError();
}

}  // namespace pdds
