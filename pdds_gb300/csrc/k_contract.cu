// Rows of G from the MIXED path kernel's exit histograms: for every work item
// and stencil side, G[knot, i] -= sum_b hist[b] H[b][i] / N over the side's
// bins b (and the same with squares for G's variances), H the shape's RBF
// weights.
//
// Counterpart of the reference's per-exit loop over the side's RBF centres
// (G_update, Meshes/stencil.cpp:244-307); the path kernel used to do this
// at the end of each work item, with its own 128 or 256 threads.
//
// What bounds it: instruction issue (60 % at 12x12/n43), of FMAs to a third.
// In the path kernel a thread had one column and read a weight from L2 for
// every product, with the CTA's paths waiting: 2.9 ms of 25.0 at 12x12/n43
// (10,945 knots, 4 sides of up to 127 columns x 1,348 bins).  Here 32 items
// of knots that are neighbours in hand-out order, so mostly of one shape,
// share the weights, and a thread has 8 items x up to 4 columns: a weight
// serves 8 products and a 16-byte read of the histograms 16, and an
// instruction forms the products of two items.  The stages come by
// asynchronous copies, two ahead (a shape's CT_BINS x n weights are
// contiguous).  Loads into registers, one ahead, took 0.63 ms at 12x12/n43,
// the copies 0.52, two products per instruction 0.46, the third float of the
// sums 0.51.  Path kernel and contraction: 24.9 -> 22.6 ms there; 237 knots
// 0.433 -> 0.404 ms; 741 knots with variances 3.50 -> 3.43.
//
// Rounding is that of the loop it replaces: FP32 sums of 64 products in the
// same order for each item, added to more than FP64 accuracy in three floats
// (pair_sum.cuh) and over the items in FP64.  Adding a knot's items
// before the products would save 0.04 of 3.42 ms at 741 knots, but the
// products' rounding would not average over the items.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "kernels.h"
#include "pair_sum.cuh"

namespace pdds {

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int CT_ROWS = 32;  // work items of a CTA
constexpr int CT_BINS = 32;  // bins of a stage
constexpr int CT_SUM = 2;   // stages of one FP32 sum
constexpr int CT_RING = 3;   // stages in shared memory
constexpr int CT_LD = CT_ROWS + 4;  // stride of a bin's values: 16-byte aligned

// Asynchronous copies into shared memory, 16 bytes, and 4 bytes or zero.
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}

struct RowInfo {
  int64_t hist;  // word of the row's histogram of this side
  int64_t tab;   // the shape's weights, -1 without a side
  int64_t map;   // side-knot -> row position map
  int64_t e0;    // first entry of the row
  int n, nbins, knot;
};

// VAR: the squares too (4 items and up to 2 columns per thread instead of 8
// and 4, twice the warps).
template <bool VAR>
struct Tile {
  static constexpr int RT = VAR ? 4 : 8;
  static constexpr int NJ = VAR ? 2 : 4;
  static constexpr int WARPS = CT_ROWS / RT;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int A_WORDS = (VAR ? 2 : 1) * CT_BINS * CT_LD;  // histograms of a stage
};

// Columns c0 .. c0 + 32 NJ - 1 of the rows in `rows` (one shape), stages
// [st0, st1).  ring: CT_RING stages of the histograms, transposed, and of the
// weights (CT_BINS bins of all columns, contiguous in the table).
template <int NJ, bool VAR>
__device__ __forceinline__ void contract_columns(const ContractArgs& a, const RowInfo* s_row, float* ring,
                                                 int stage_words, unsigned rows, int first, int c0, int st0, int st1) {
  using T = Tile<VAR>;
  constexpr int RT = T::RT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = s_row[first].n, nb = s_row[first].nbins;
  const float* tab = a.L.tab + s_row[first].tab;
  const bool busy = (rows >> (warp * RT)) & ((1u << RT) - 1u);
  // rows in pairs: one instruction for two products
  constexpr int RP = RT / 2;
  const float2 zero = make_float2(0.f, 0.f);
  PairSum sum[RP][NJ], sum2[VAR ? RP : 1][NJ];
  float2 p[RP][NJ], p2[VAR ? RP : 1][NJ];
#pragma unroll
  for (int r = 0; r < RP; r++)
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      p[r][j] = zero;
      sum[r][j] = {zero, zero, zero};
      if (VAR) {
        p2[r][j] = zero;
        sum2[r][j] = {zero, zero, zero};
      }
    }
  auto issue = [&](int st) {
    if (st < st1) {
      float* A = ring + (st % CT_RING) * stage_words;
      float* W = A + T::A_WORDS;
      const int q0 = st * CT_BINS, qn = min(CT_BINS, nb - q0);
      // the table's shapes start at multiples of 4 words (16 bytes), so the
      // last words copied are at most the padding after this one
      const float* src = tab + (int64_t)q0 * n;
      for (int i = 4 * tid; i < qn * n; i += 4 * T::THREADS) copy16(W + i, src + i);
      for (int r = warp; r < CT_ROWS; r += T::WARPS) {
        const bool in = ((rows >> r) & 1u) && lane < qn;
        const float* h = a.hist + (in ? s_row[r].hist + q0 + lane : 0);
        copy4(A + lane * CT_LD + r, h, in);
        if (VAR) copy4(A + (CT_BINS + lane) * CT_LD + r, h + (in ? a.var_off : 0), in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int k = 0; k < CT_RING - 1; k++) issue(st0 + k);
  for (int st = st0; st < st1; st++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(CT_RING - 2) : "memory");
    __syncthreads();  // stage st is there, and the stage before it is read
    issue(st + CT_RING - 1);
    if (!busy) continue;
    const int qn = min(CT_BINS, nb - st * CT_BINS);
    const float* A = ring + (st % CT_RING) * stage_words + warp * RT;
    const float* A2 = A + CT_BINS * CT_LD;
    // columns past n read the next bin's weights (or padding): not written
    const float* W = ring + (st % CT_RING) * stage_words + T::A_WORDS + c0 + lane;
    auto bin = [&](int q) {
      float2 x[RP], x2[VAR ? RP : 1];
#pragma unroll
      for (int r = 0; r < RP; r += 2) {
        const float4 v = *reinterpret_cast<const float4*>(A + q * CT_LD + 2 * r);
        x[r] = make_float2(v.x, v.y);
        x[r + 1] = make_float2(v.z, v.w);
        if (VAR) {
          const float4 v2 = *reinterpret_cast<const float4*>(A2 + q * CT_LD + 2 * r);
          x2[r] = make_float2(v2.x, v2.y);
          x2[r + 1] = make_float2(v2.z, v2.w);
        }
      }
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const float h = W[32 * j];
        const float2 hv = make_float2(h, h);
#pragma unroll
        for (int r = 0; r < RP; r++) p[r][j] = __ffma2_rn(x[r], hv, p[r][j]);
        if (VAR) {
          const float2 h2 = __fmul2_rn(hv, hv);
#pragma unroll
          for (int r = 0; r < RP; r++) p2[r][j] = __ffma2_rn(x2[r], h2, p2[r][j]);
        }
      }
      W += n;
    };
    if (qn == CT_BINS) {
#pragma unroll 8
      for (int q = 0; q < CT_BINS; q++) bin(q);
    } else {
      for (int q = 0; q < qn; q++) bin(q);
    }
    if ((st + 1) % CT_SUM == 0 || st == st1 - 1) {
#pragma unroll
      for (int r = 0; r < RP; r++)
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          pair_add(sum[r][j], p[r][j]);
          p[r][j] = zero;
          if (VAR) {
            pair_add(sum2[r][j], p2[r][j]);
            p2[r][j] = zero;
          }
        }
    }
  }
  __syncthreads();  // the ring is free
  if (!busy) return;
#pragma unroll
  for (int r = 0; r < RT; r++) {
    const int row = warp * RT + r;
    if (!((rows >> row) & 1u)) continue;
    const RowInfo& ri = s_row[row];
    const double invN = a.knot_invN ? a.knot_invN[ri.knot] : a.inv_N;
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      const int c = c0 + lane + 32 * j;
      if (c >= n) continue;
      const int64_t m = ri.map + c;
      if (!a.dup_sum && !a.L.map_owner[m]) continue;
      const int64_t e = a.L.map_pos[m];
      if (!idx_ok(e, a.L.row_ptr[ri.knot + 1] - ri.e0, a.err_flags)) continue;
      atomicAdd(a.G + ri.e0 + e, -pair_total(sum[r / 2][j], r & 1) * invN);
      if (VAR) atomicAdd(a.GG + ri.e0 + e, pair_total(sum2[r / 2][j], r & 1) * invN);
    }
  }
}

template <bool VAR>
__global__ void __launch_bounds__(Tile<VAR>::THREADS, VAR ? 2 : 3) k_contract(const ContractArgs a, int stage_words) {
  extern __shared__ __align__(16) float ring[];
  __shared__ RowInfo s_row[CT_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, d = blockIdx.y;
  if (tid < CT_ROWS) {
    const int64_t r = (int64_t)blockIdx.x * CT_ROWS + tid;
    RowInfo ri;
    ri.tab = -1;
    ri.n = ri.nbins = ri.knot = 0;
    ri.hist = ri.map = ri.e0 = 0;
    if (r < a.n_rows) {
      const DevLayout& L = a.L;
      const int k = a.rows[r / a.chunks], st = L.knot_stencil[k], sd = L.st_side[4 * st + d];
      if (sd >= 0) {
        int off = 0;
        int64_t map = L.st_map_off[st];
        for (int q = 0; q < d; q++) {
          const int sq = L.st_side[4 * st + q];
          if (sq < 0) continue;
          off += L.sh_nbins[L.sd_shape[sq]];
          map += L.sd_n[sq];
        }
        const int sh = L.sd_shape[sd];
        ri.knot = k;
        ri.n = L.sd_n[sd];
        ri.nbins = L.sh_nbins[sh];
        ri.tab = L.sh_tab_off[sh];
        ri.map = map;
        ri.e0 = L.row_ptr[k];
        ri.hist = (a.row_slot ? a.row_slot[r] : r) * a.stride + off;
        if (ri.n < 1 || ri.nbins < 1) ri.tab = -1;
      }
    }
    s_row[tid] = ri;
  }
  __syncthreads();
  const int64_t mine = s_row[lane].tab;
  unsigned todo = __ballot_sync(FULLM, mine >= 0);
  while (todo) {  // one pass per distinct shape
    const int first = __ffs(todo) - 1;
    const unsigned rows = __ballot_sync(FULLM, mine == s_row[first].tab) & todo;
    const int n = s_row[first].n, stages = (s_row[first].nbins + CT_BINS - 1) / CT_BINS;
    const int sums = (stages + CT_SUM - 1) / CT_SUM;
    const int st0 = CT_SUM * (int)((int64_t)sums * blockIdx.z / gridDim.z);
    const int st1 = min(stages, CT_SUM * (int)((int64_t)sums * (blockIdx.z + 1) / gridDim.z));
    if (st0 < st1)
      for (int c0 = 0; c0 < n; c0 += 32 * Tile<VAR>::NJ) {
        const int left = n - c0;
        if constexpr (!VAR) {
          if (left > 96) {
            contract_columns<4, VAR>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
            continue;
          }
          if (left > 64) {
            contract_columns<3, VAR>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
            continue;
          }
        }
        if (left > 32) contract_columns<2, VAR>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
        else contract_columns<1, VAR>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
      }
    todo &= ~rows;
  }
}

}  // namespace

// three stages of 32 bins x 160 columns and both histograms, with room
constexpr int CT_SMEM_MAX = 96 * 1024;

cudaError_t launch_contract(const ContractArgs& a, int max_n, int max_nbins, int num_sms, int* launches,
                            cudaStream_t s) {
  if (a.n_rows < 1 || max_n < 1) return cudaSuccess;
  // bins split over CTAs until there are about eight tiles per SM
  const int tiles = (a.n_rows + CT_ROWS - 1) / CT_ROWS;
  const int sums = (max_nbins + CT_SUM * CT_BINS - 1) / (CT_SUM * CT_BINS);
  const int split = std::max(1, std::min(sums, (8 * num_sms + 4 * tiles - 1) / (4 * tiles)));
  const dim3 grid(tiles, 4, split);
  auto run = [&](auto kernel, int threads, int a_words) -> cudaError_t {
    const int stage_words = a_words + ((CT_BINS * max_n + 3) & ~3);
    const size_t smem = ((size_t)CT_RING * stage_words + 128) * sizeof(float);
    if (smem > CT_SMEM_MAX) return cudaErrorInvalidValue;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_SMEM_MAX);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, s>>>(a, stage_words);
    ++*launches;
    return cudaGetLastError();
  };
  return a.GG ? run(k_contract<true>, Tile<true>::THREADS, Tile<true>::A_WORDS)
              : run(k_contract<false>, Tile<false>::THREADS, Tile<false>::A_WORDS);
}

}  // namespace pdds
