// Launch arguments and entry points of the device kernels (host-visible).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pdds.h"
#include "dev_common.cuh"
#include "fast64.cuh"

namespace pdds {

constexpr int MIXED_MAX_THREADS = 256;
// Block size of the MIXED path kernel: 128-thread CTAs (8 per SM) for large
// layouts, 256 (4 per SM) below 8192 Monte Carlo knots, except for short work
// items and long continuations (short_items and adaptive_continue in capi.cu).
// 128 against 256, 20,000 paths: 10,989 knots in pairs 22.5 and 22.8 ms, with
// variances (whose histograms leave 128-thread CTAs fewer lanes per SM) 9.1 and
// 7.4; 3,325 knots in pairs 6.9 and 6.6, with variances 2.5 and 2.2.
inline int mixed_threads(int n_mc) { return n_mc >= 8192 ? 128 : 256; }
constexpr int FP64_SLOTS = 8;      // warps that share a block of paths in the FP64 kernel
constexpr int FP64_THREADS = 32 * FP64_SLOTS;  // at most (a CTA may take fewer slots)
constexpr int FP64_QCAP = 160;  // exits queued per warp in the FP64 kernel
constexpr unsigned ERR_FLAG_STEP_LIMIT = 1u;
constexpr unsigned ERR_FLAG_EXIT_SIDE = 2u;
constexpr unsigned ERR_FLAG_SINGULAR = 4u;
constexpr unsigned ERR_FLAG_TIMEOUT = 8u;  // a bounded device wait ran out
constexpr unsigned ERR_FLAG_SUB_NOCONV = 16u;  // a subdomain solve missed its tolerance
constexpr unsigned ERR_FLAG_BOUNDS = 32u;      // an index check of the checked build failed

// Index check of the checked build (compiled with -DPDDS_CHECKED,
// pdds_gb300.build.build(checked=True)): i must lie in [0, n); a failed
// check sets ERR_FLAG_BOUNDS and the caller skips the access.  The default
// build compiles every check to true.
__device__ __forceinline__ bool idx_ok(long long i, long long n, unsigned* flags) {
#ifdef PDDS_CHECKED
  if (i >= 0 && i < n) return true;
  if (flags) atomicOr(flags, ERR_FLAG_BOUNDS);
  return false;
#else
  (void)i;
  (void)n;
  (void)flags;
  return true;
#endif
}

// Diagnostic sums of one finished path (or Richardson pair) into a CTA's
// shared sums: phi, phi^2, xi, xi^2, phi + xi, (phi + xi)^2, xi phi, tau, normals.
__device__ __forceinline__ void diag_add(double* sd, double phi, double xi, double tau, double rng) {
  atomicAdd(sd + PDDS_DIAG_SCORE, phi);
  atomicAdd(sd + PDDS_DIAG_SCORE2, phi * phi);
  atomicAdd(sd + PDDS_DIAG_XI, xi);
  atomicAdd(sd + PDDS_DIAG_XI2, xi * xi);
  atomicAdd(sd + PDDS_DIAG_SCORE_VR, phi + xi);
  atomicAdd(sd + PDDS_DIAG_SCORE_VR2, (phi + xi) * (phi + xi));
  atomicAdd(sd + PDDS_DIAG_XI_SCORE, xi * phi);
  atomicAdd(sd + PDDS_DIAG_TAU, tau);
  atomicAdd(sd + PDDS_DIAG_RNG, rng);
  atomicAdd(sd + PDDS_DIAG_PATHS, 1.0);
}
// A CTA's sums into the knot's (the linear sums also fill the sublinear
// slots: the FP64 and MIXED forms run no sublinear leg).
__device__ __forceinline__ void diag_flush(const double* sd, double* out, int tid) {
  if (tid < PDDS_DIAG_SUB) {
    atomicAdd(out + tid, sd[tid]);
    atomicAdd(out + PDDS_DIAG_SUB + tid, sd[tid]);
  } else if (tid == PDDS_DIAG_SUB || tid == PDDS_DIAG_SUB + 1) {
    const int q = tid == PDDS_DIAG_SUB ? PDDS_DIAG_RNG : PDDS_DIAG_PATHS;
    atomicAdd(out + q, sd[q]);
  }
}

struct MixedArgs {
  DevLayout L;
  ProblemDev P;
  int N;                 // paths per knot
  float h, sqrth;
  // Philox-4x32-10 round keys of the seed (k0 + r W0, k1 + r W1 for rounds
  // r = 0..9, set by mixed_set_rng): kernel parameters, so every round's key
  // is an operand of its XOR instead of a key-schedule addition per call
  uint32_t rk[20];
  uint32_t instance;
  int chunks, paths_per_chunk, n_items;
  int want_var;
  int adaptive_h;
  int richardson;        // 1: common-random-number Richardson pair (h/2, h)
  double h64;            // h in FP64 (for the adaptive step)
  long long max_steps;
  const int* mc_knots;   // knots that need paths, in hand-out order
  int hist_cap;          // words reserved for one exit histogram
  // the items' histograms: item i of a list at slot i, chunk c of a knot at
  // slot (mc_pos[knot] - mc0) chunks + c, hist_stride words each, the Y^2
  // histogram var_off words after the first
  float* hist_out;
  int64_t hist_stride;
  int var_off;
  const int* mc_pos;     // position of each knot in the hand-out order
  int mc0;
  int lut_nodes;         // table nodes that can be staged in shared memory (PK_LUT)
  int* item_counter;
  double* Bsum;          // [K]
  double* BBsum;         // [K]
  unsigned long long* stats;  // [0] steps [1] unused [2] global exits [3] stencil exits
  unsigned* err_flags;
  // optional explicit items (knot, paths [p0, p1)) instead of n_mc x chunks
  const int* item_knot;
  const int* item_p0;
  const int* item_p1;
  unsigned long long* knot_steps;  // optional: path steps per knot (both levels)
  // optional [32]: paths (each level of a Richardson pair counts) by their
  // steps, bin b = steps in [2^b, 2^(b+1))
  unsigned long long* step_hist;
  // optional [K][PDDS_DIAG_N]: the reduction's diagnostic sums per knot
  double* diag;
};

// G from the path kernel's histograms (k_contract.cu), one row per work item.
struct ContractArgs {
  DevLayout L;
  const float* hist;     // slots of `stride` words
  int64_t stride;
  int var_off;           // words from a slot's histogram to its Y^2 histogram
  int n_rows;            // work items
  const int* rows;       // knots, in hand-out order: item r is of knot rows[r / chunks]
  int chunks;
  const int* row_slot;   // optional: each item's slot (else r)
  double inv_N;
  const double* knot_invN;  // optional: 1/N_k instead of inv_N (variance-adaptive paths)
  int dup_sum;
  double* G;             // [nnz] accumulates -sum Y H / N
  double* GG;            // [nnz] accumulates sum (Y H)^2 / N; null without variances
  unsigned* err_flags;
};

struct Fp64Args {
  DevLayout L;
  ProblemDev P;
  Fast64 T;
  int N;
  double h, sqrth, inv_N;
  uint64_t seed;
  uint32_t instance;
  int blocks, block_paths;  // blocks of paths per knot, paths per block
  int slots;                // slots of a block that have paths
  int n_items;              // knots x blocks x (slots / slots per CTA)
  int dup_sum;
  int adaptive_h;
  int richardson;
  long long max_steps;
  const int* mc_knots;
  int* item_counter;
  int spread;               // 1: a block takes several CTAs, one item per CTA
  double* S;                // [knots x blocks][FP64_SLOTS][sum_stride]: the slots' RBF sums
  int sum_stride;
  double* G;
  double* Bsum;
  double* BBsum;
  unsigned long long* stats;
  unsigned* err_flags;
  double* diag;          // optional [K][PDDS_DIAG_N]: diagnostic sums per knot
};

struct ReplayArgs {
  DevLayout L;
  ProblemDev P;
  int N;
  double h, sqrth;
  uint64_t seed;
  uint32_t instance;
  int sublinear;
  int adaptive_h;
  long long max_steps;
  const int* mc_knots;   // knots with paths
  int n_mc;
  // per-knot side data for the reduction (actual positions, ipsi per knot)
  const int64_t* knot_ipsi_off;  // [n_mc][4] offset into ipsi_knot, -1 if none
  const double* ipsi_knot;
  // exit records [n_mc * N]
  double* ex;
  double* ey;
  double* eY;
  double* eZ;
  double* exi;
  int* eside;            // -1 global, 0..3 stencil side, -2 no side
  int* esteps_l;
  int* esteps_s;
  // diagnostics (all null when off): sums [K][PDDS_DIAG_N], the sublinear
  // leg's end states [n_mc * N]
  double* diag;
  double* sx;
  double* sy;
  double* sY;
  double* sZ;
  double* sxi;
  double* knot_h;        // [n_mc][2]: each knot's step and its square root
  unsigned long long* path_counter;  // next path to hand out
  unsigned long long* stats;         // as in MixedArgs
  // outputs
  double* G;             // [nnz] final values
  double* GG;            // [nnz] final GG/N values (before - G^2)
  double* B;             // [K]
  double* BB;            // [K]
  int dup_sum;
  unsigned* err_flags;
};

// The FP32 path-kernel instantiation of a problem: table-served problems
// with textures run PK_LUT_TEX, every other problem its own kind.
inline int mixed_kind(const ProblemDev& P) { return P.kind == PK_LUT && P.lut.tex_mode ? PK_LUT_TEX : P.kind; }

// smem: mixed_queue_smem(threads, richardson) + the exit histograms
cudaError_t launch_paths_mixed(const MixedArgs& a, int kind, int grid, int threads, size_t smem, cudaStream_t s);
size_t mixed_queue_smem(int threads, int richardson);
// max_n, max_nbins: of the layout's shapes
cudaError_t launch_contract(const ContractArgs& a, int max_n, int max_nbins, int num_sms, int* launches,
                            cudaStream_t s);
// Buffers to be zeroed in one launch (4-byte words each, 4-byte aligned).
struct ZeroList {
  static constexpr int MAX = 8;
  int n = 0;
  unsigned* p[MAX];
  size_t words[MAX];
  template <typename T>
  void add(T* q, size_t count) {
    static_assert(sizeof(T) % 4 == 0, "words");
    p[n] = reinterpret_cast<unsigned*>(q);
    words[n++] = count * (sizeof(T) / 4);
  }
};
cudaError_t launch_zero(const ZeroList& z, int num_sms, cudaStream_t s);
// knots mc[n] reordered heaviest first by steps[knot] (quarter-octave groups)
cudaError_t launch_lpt_order(const int* mc, int n, const unsigned long long* steps, int* out, cudaStream_t s);
// Sets the Philox key schedule (rk) of `seed` and the instance word.
void mixed_set_rng(MixedArgs& a, uint64_t seed, uint32_t instance);
// out[4i..4i+3] = the MIXED kernel's Philox block for counter ctr[4i..4i+3]
// and the 64-bit key (low word first), device arrays.
cudaError_t launch_philox_rk_check(uint64_t key, const uint32_t* ctr, int n, uint32_t* out, cudaStream_t s);
// The portable Philox (form 0) and FP64 functions (selfcheck.cu).
cudaError_t launch_philox_check(const uint32_t* ctr, const uint32_t* key, int n, uint32_t* out, cudaStream_t s);
cudaError_t launch_portable_math_check(int fn, const double* x, int n, double* out, cudaStream_t s);
void philox_check_host(const uint32_t* ctr, const uint32_t* key, int n, uint32_t* out);
void portable_math_check_host(int fn, const double* x, int n, double* out);
// True when `func` is one of the MIXED path kernels (a captured graph's
// nodes are re-keyed with a new seed through their parameters).
bool is_mixed_path_kernel(const void* func);
int mixed_blocks_per_sm(int kind, size_t smem, int richardson, int threads, bool diag = false);
cudaError_t launch_paths_fp64(const Fp64Args& a, int kind, int grid, int threads, size_t smem, cudaStream_t s);
int fp64_blocks_per_sm(int kind, size_t smem, int richardson, int threads);
cudaError_t launch_rows_fp64(const Fp64Args& a, int n_blocks, cudaStream_t s);
cudaError_t launch_replay_paths(const ReplayArgs& a, int kind, int num_sms, cudaStream_t s);
// max_n: side knots of the largest side; knot_task_off: first side entry of
// each knot in Gside and GGside (sides N, S, E, W one after the other)
cudaError_t launch_replay_reduce(const ReplayArgs& a, int kind, int max_n, const int64_t* knot_task_off,
                                 double* Gside, double* GGside, double* hy, int* launches, cudaStream_t s);
// paths whose RBF terms are held at once: hy has n_mc x that x max_n words
int replay_terms_paths(int n_mc, int N, int max_n);
// FP64 factorisation of every shape's Psi and the cardinal-function tables.
// lu: scratch of the ipsi layout; piv, uinv: scratch of the sh_t layout
cudaError_t launch_rbf_setup(const DevLayout& L, int max_n, int max_nbins, double* ipsi, float* tab,
                             double* lu, int* piv, double* uinv,
                             unsigned* err_flags, cudaStream_t s);
// CSR column indices of G from the stencils' column lists
cudaError_t launch_expand_cols(int K, const int64_t* row_ptr, const int* knot_stencil, const int64_t* st_off,
                               const int* st_cols, int* col, cudaStream_t s);
// B = g(x0) for boundary knots; finalisation of B, BB, G_var.
cudaError_t launch_boundary_b(const DevLayout& L, const ProblemDev& P, int mode, const int* knots,
                              int n, double* B, double* BB, cudaStream_t s);
// Variance-adaptive paths: rescale the pilot's G/GG rows, finalise with per-knot N.
cudaError_t launch_scale_rows(const int* mc, int n, const int64_t* row_ptr, const double* scale, double* G,
                              double* GG, cudaStream_t s);
cudaError_t launch_finalize_n(const int* mc_knots, int n_mc, const int* knot_N, const double* Bsum,
                              const double* BBsum, double* B, double* BB, int64_t nnz, const double* G,
                              double* GG_to_var, int want_var, cudaStream_t s);
// Subdomain interior solves (k_subdomain.cu).
size_t subdomain_smem(int m);
// grid: optional nsub (m + 1) + 1 nodes per side, the solution with its edges
cudaError_t launch_subdomain(const DevLayout& L, const ProblemDev& P, int nsub, int m, int n, const int* edge_knots,
                             const double* u, double* out, double* grid, cudaStream_t s);
// table-served problems (PK_LUT): BiCGSTAB with a sine-transform preconditioner;
// work = 13 m^2 doubles per subdomain
cudaError_t launch_subdomain_lut(const DevLayout& L, const ProblemDev& P, int nsub, int m, int n, const int* edge_knots,
                                 const double* u, double* out, double* work, double* grid, int max_iter, double tol,
                                 int* iters, unsigned* err, cudaStream_t s);
// tables of one outer-loop step around the grid (or the constant u0)
enum { OUTER_NEWTON_U3 = 0, OUTER_LINEAR_SHIFT = 1 };
struct OuterStep {
  int equation;                  // OUTER_*
  double u0;                     // constant iterate when there is no grid
  double a;                      // NEWTON_U3: u = a + sin(pi x) sin(pi y)
  double c2, alpha, k;           // LINEAR_SHIFT: Lap u + c2 u + F = 0, shift alpha, rescale k
};
cudaError_t launch_newton_tables(const double* grid, int G, double x0, double y0, double hx, double hy,
                                 const OuterStep& eq, float* coef, float* gtab, cudaStream_t s);
cudaError_t launch_finalize(const int* mc_knots, int n_mc, int N, const double* Bsum,
                            const double* BBsum, double* B, double* BB, const int64_t* row_ptr,
                            int64_t nnz, const double* G, double* GG_to_var, int want_var,
                            cudaStream_t s);

}  // namespace pdds
