// Rows of G from the MIXED path kernel's exit histograms: for every knot and
// stencil side, G[knot, i] -= sum_b hist[b] H[b][i] / N over the side's bins b
// (and the same with squares for G's variances), H the shape's RBF weights.
//
// Counterpart of the reference's per-exit loop over the side's RBF centres
// (PDDAlgorithms/PDDSparseGM.cpp, Update_G); the path kernel used to do this
// for each of its work items, with its own 128 or 256 threads.
//
// What bounds it: shared-memory reads and the FP32 pipe.  In the path kernel
// a thread had one column and read a weight from L2 for every product, with
// the CTA's other work waiting: 2.9 ms of 25.0 at 12x12/n43 (10,945 knots, 4
// sides of up to 127 columns x 1,348 bins).  Here 32 knots, neighbours in
// hand-out order and so mostly of one shape, share the weights, and a thread
// has 8 knots x up to 4 columns: a weight serves 8 products and a 16-byte
// read of the histograms 16.  The stages come by asynchronous copies, two
// ahead (a shape's CT_BINS x n weights are contiguous); with loads into
// registers, one ahead, it took 0.63 ms there, now 0.52 (path kernel and
// contraction: 24.9 -> 22.7 ms; 741 knots with variances 3.50 -> 3.35; 237
// knots 0.433 -> 0.404).
//
// Rounding: before, each work item had FP32 sums of 64 products, added up in
// FP64.  With one item per knot it is the same here, the 64-product sums added
// in two floats (TwoSum, 48 bits; FP64 issues at 1/64 of the rate).  Several
// items of a knot are added first, in two floats rounded once, so the
// products' rounding no longer averages over the items: the FP32 sums are
// then 8 products long, 4 from 5 items on.  Against exact sums of the same
// histograms, G is off by (rms, before and now) 4.0e-8 and 2.0e-8 with 11
// items per knot, 6.5e-8 and 3.4e-8 with 4 (with sums of 16 products 5.6e-8
// and 5.8e-8); the time is the same.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "kernels.h"

namespace pdds {

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int CT_ROWS = 32;  // knots of a CTA
constexpr int CT_BINS = 32;  // bins of a stage
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

// s + e exactly (e the running error): TwoSum
__device__ __forceinline__ void add2(float& s, float& e, float v) {
  const float t = s + v, b = t - s;
  e += (s - (t - b)) + (v - b);
  s = t;
}
// an infinite sum has no error term
__device__ __forceinline__ float fin(float s, float e) { return isfinite(s) ? e : 0.f; }

// a slot per work item -> the first slot of its row: the sum of the row's
// slots, in two floats and rounded once
__global__ void k_hist_sum(float* hist, int64_t stride, int words, const int* row_slot, const int* row_cnt,
                           int chunks) {
  const int r = blockIdx.y;
  const int cnt = row_cnt ? row_cnt[r] : chunks;
  if (cnt < 2) return;
  float* h0 = hist + (row_slot ? (int64_t)row_slot[r] : (int64_t)r * chunks) * stride;
  const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= words) return;
  float4 hi = *reinterpret_cast<const float4*>(h0 + i);
  float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int c = 1; c < cnt; c++) {
    const float4 v = *reinterpret_cast<const float4*>(h0 + c * stride + i);
    add2(hi.x, lo.x, v.x);
    add2(hi.y, lo.y, v.y);
    add2(hi.z, lo.z, v.z);
    add2(hi.w, lo.w, v.w);
  }
  *reinterpret_cast<float4*>(h0 + i) =
      make_float4(hi.x + fin(hi.x, lo.x), hi.y + fin(hi.y, lo.y), hi.z + fin(hi.z, lo.z), hi.w + fin(hi.w, lo.w));
}

struct RowInfo {
  int64_t hist;  // word of the row's histogram of this side
  int64_t tab;   // the shape's weights, -1 without a side
  int64_t map;   // side-knot -> row position map
  int64_t e0;    // first entry of the row
  int n, nbins, knot;
};

// VAR: the squares too (4 knots and up to 2 columns per thread instead of 8
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
template <int NJ, bool VAR, int SUM>
__device__ __forceinline__ void contract_columns(const ContractArgs& a, const RowInfo* s_row, float* ring,
                                                 int stage_words, unsigned rows, int first, int c0, int st0, int st1) {
  using T = Tile<VAR>;
  constexpr int RT = T::RT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = s_row[first].n, nb = s_row[first].nbins;
  const float* tab = a.L.tab + s_row[first].tab;
  const bool busy = (rows >> (warp * RT)) & ((1u << RT) - 1u);
  int col[NJ];
#pragma unroll
  for (int j = 0; j < NJ; j++) col[j] = min(c0 + lane + 32 * j, n - 1);
  float hi[RT][NJ], lo[RT][NJ], p[RT][NJ];
  float hi2[VAR ? RT : 1][NJ], lo2[VAR ? RT : 1][NJ], p2[VAR ? RT : 1][NJ];
#pragma unroll
  for (int r = 0; r < RT; r++)
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      hi[r][j] = lo[r][j] = p[r][j] = 0.f;
      if (VAR) hi2[r][j] = lo2[r][j] = p2[r][j] = 0.f;
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
    const float* W = ring + (st % CT_RING) * stage_words + T::A_WORDS;
    auto bin = [&](int q) {
      float hv[NJ], x[RT], x2[VAR ? RT : 1];
#pragma unroll
      for (int j = 0; j < NJ; j++) hv[j] = W[q * n + col[j]];
#pragma unroll
      for (int r = 0; r < RT; r += 4) {
        *reinterpret_cast<float4*>(x + r) = *reinterpret_cast<const float4*>(A + q * CT_LD + r);
        if (VAR) *reinterpret_cast<float4*>(x2 + r) = *reinterpret_cast<const float4*>(A2 + q * CT_LD + r);
      }
#pragma unroll
      for (int j = 0; j < NJ; j++) {
#pragma unroll
        for (int r = 0; r < RT; r++) p[r][j] = fmaf(x[r], hv[j], p[r][j]);
        if (VAR) {
          const float h2 = hv[j] * hv[j];
#pragma unroll
          for (int r = 0; r < RT; r++) p2[r][j] = fmaf(x2[r], h2, p2[r][j]);
        }
      }
    };
    auto flush = [&]() {
#pragma unroll
      for (int r = 0; r < RT; r++)
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          add2(hi[r][j], lo[r][j], p[r][j]);
          p[r][j] = 0.f;
          if (VAR) {
            add2(hi2[r][j], lo2[r][j], p2[r][j]);
            p2[r][j] = 0.f;
          }
        }
    };
    if constexpr (SUM > CT_BINS) {
      if (qn == CT_BINS) {
#pragma unroll 8
        for (int q = 0; q < CT_BINS; q++) bin(q);
      } else {
        for (int q = 0; q < qn; q++) bin(q);
      }
      if ((st + 1) % (SUM / CT_BINS) == 0 || st == st1 - 1) flush();
    } else {
      int q = 0;
#pragma unroll 1
      for (; q + SUM <= qn; q += SUM) {
#pragma unroll
        for (int k = 0; k < SUM; k++) bin(q + k);
        flush();
      }
      if (q < qn) {
        for (; q < qn; q++) bin(q);
        flush();
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
      atomicAdd(a.G + ri.e0 + e, -((double)hi[r][j] + (double)fin(hi[r][j], lo[r][j])) * invN);
      if (VAR) atomicAdd(a.GG + ri.e0 + e, ((double)hi2[r][j] + (double)fin(hi2[r][j], lo2[r][j])) * invN);
    }
  }
}

template <bool VAR, int SUM>
__global__ void __launch_bounds__(Tile<VAR>::THREADS, VAR ? 2 : 3) k_contract(const ContractArgs a, int stage_words) {
  extern __shared__ __align__(16) float ring[];
  __shared__ RowInfo s_row[CT_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, d = blockIdx.y;
  if (tid < CT_ROWS) {
    const int r = blockIdx.x * CT_ROWS + tid;
    RowInfo ri;
    ri.tab = -1;
    ri.n = ri.nbins = ri.knot = 0;
    ri.hist = ri.map = ri.e0 = 0;
    if (r < a.n_rows) {
      const DevLayout& L = a.L;
      const int k = a.rows[r], st = L.knot_stencil[k], sd = L.st_side[4 * st + d];
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
        ri.hist = (a.row_slot ? (int64_t)a.row_slot[r] : (int64_t)r * a.chunks) * a.stride + off;
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
    const int pair = (stages + 1) / 2;  // the split leaves every 64 bins together
    const int st0 = 2 * (int)((int64_t)pair * blockIdx.z / gridDim.z);
    const int st1 = min(stages, 2 * (int)((int64_t)pair * (blockIdx.z + 1) / gridDim.z));
    if (st0 < st1)
      for (int c0 = 0; c0 < n; c0 += 32 * Tile<VAR>::NJ) {
        const int left = n - c0;
        if constexpr (!VAR) {
          if (left > 96) {
            contract_columns<4, VAR, SUM>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
            continue;
          }
          if (left > 64) {
            contract_columns<3, VAR, SUM>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
            continue;
          }
        }
        if (left > 32) contract_columns<2, VAR, SUM>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
        else contract_columns<1, VAR, SUM>(a, s_row, ring, stage_words, rows, first, c0, st0, st1);
      }
    todo &= ~rows;
  }
}

}  // namespace

cudaError_t launch_contract(const ContractArgs& a, int words, int max_n, int max_nbins, int max_cnt, int num_sms,
                            int* launches, cudaStream_t s) {
  if (a.n_rows < 1 || words < 1) return cudaSuccess;
  if (max_cnt > 1) {
    // at most 65,535 rows per launch (the grid's y)
    for (int r0 = 0; r0 < a.n_rows; r0 += 65535) {
      const int nr = std::min(a.n_rows - r0, 65535);
      const dim3 grid((words / 4 + 127) / 128, nr);
      k_hist_sum<<<grid, 128, 0, s>>>(a.row_slot ? a.hist : a.hist + (int64_t)r0 * a.chunks * a.stride, a.stride,
                                      words, a.row_slot ? a.row_slot + r0 : nullptr,
                                      a.row_cnt ? a.row_cnt + r0 : nullptr, a.chunks);
      ++*launches;
    }
  }
  // bins split over CTAs until there are about eight tiles per SM
  const int tiles = (a.n_rows + CT_ROWS - 1) / CT_ROWS;
  const int stages = (max_nbins + CT_BINS - 1) / CT_BINS;
  const int split = std::max(1, std::min((stages + 1) / 2, (8 * num_sms + 4 * tiles - 1) / (4 * tiles)));
  const dim3 grid(tiles, 4, split);
  auto run = [&](auto kernel, int threads, int a_words) -> cudaError_t {
    const int stage_words = a_words + ((CT_BINS * max_n + 3) & ~3);
    const size_t smem = (size_t)CT_RING * stage_words * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, s>>>(a, stage_words);
    ++*launches;
    return cudaGetLastError();
  };
  // FP32 sums as long as the rounding allows (see above)
  if (a.GG)
    return max_cnt > 4   ? run(k_contract<true, 4>, Tile<true>::THREADS, Tile<true>::A_WORDS)
           : max_cnt > 1 ? run(k_contract<true, 8>, Tile<true>::THREADS, Tile<true>::A_WORDS)
                         : run(k_contract<true, 64>, Tile<true>::THREADS, Tile<true>::A_WORDS);
  return max_cnt > 4   ? run(k_contract<false, 4>, Tile<false>::THREADS, Tile<false>::A_WORDS)
         : max_cnt > 1 ? run(k_contract<false, 8>, Tile<false>::THREADS, Tile<false>::A_WORDS)
                       : run(k_contract<false, 64>, Tile<false>::THREADS, Tile<false>::A_WORDS);
}

}  // namespace pdds
