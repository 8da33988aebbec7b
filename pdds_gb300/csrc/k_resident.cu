// Interface solve (I + G) u = B with the system resident on chip: one launch,
// every CTA keeps its rows of G (FP32), its rows of the Krylov basis and the
// list of the columns its rows touch in shared memory, so that a product
// reads no matrix from L2.
//
// The reference solves the system with Eigen's BiCGSTAB
// (PDDAlgorithms/PDDSparseGM.cpp:3168-3246).  Two methods here: pipelined
// GMRES(m) in FP32 inside FP64 refinement (the recurrences are those of
// gmres_body_p1 in k_gmres_cluster.cu), and BiCGSTAB in FP64.
//
// What bounds it: latency, of the exchange between the CTAs and of the serial
// parts of a step.  The kernels this one replaces read 8 bytes per entry
// (value and column) from L2 in every step, staged the whole vector in every
// CTA, and put a counting barrier between publishing and reading.  Here:
//  * a CTA of the 12x12/n43 system (10,989 rows, 4.0 M entries, 152 CTAs)
//    holds its 26.5 k entries, 106 KB of FP32 values.  The columns are stored
//    once per run of rows with the same stencil (such rows share their column
//    list), as 16-bit indices into the CTA's ~1 k distinct columns, whose
//    values are all it gathers; four rows of a run are multiplied at once, so
//    an index and a vector element are read once for four entries.
//  * there is no barrier: every published word carries a sequence number next
//    to 32 bits of data (one 8-byte access), and a reader polls the words it
//    needs until they have the number it waits for.  A buffer is written
//    again only two publications later; by then every CTA has read it,
//    because the publication in between was computed from it.
//  * FP64 issues at 1/64 of the FP32 rate, one warp instruction per 64 cycles
//    and scheduler: FP64 scalars are formed by one warp and passed through
//    shared memory, and sums involve only the warps that hold rows.
//  * of a larger system the entries that do not fit are read from L2 as FP32
//    (up to half of a CTA's): 19,005 rows, 6.9 M entries, GMRES(20) 1,665 ->
//    1,526 us against the kernel that reads values and columns from L2.
// Measured (median of 5, before -> now): GMRES(20) 237 rows 501 -> 165 us,
// 741 rows 847 -> 214, 2,205 rows 1,500 -> 365, 3,325 rows 2,780 -> 508,
// 10,989 rows (120 steps) 1,945 -> 980 us; BiCGSTAB 3,325 rows 2,956 -> 890,
// 10,989 rows (52 iterations) 5,140 -> 2,480 us.  A step of the 10,989-row
// GMRES is about 4.5 k cycles of waiting for the slowest CTA's words, 3.3 k to
// gather and sum them, 1.1 to 2.7 k of products, 2.3 k for v and z, 0.9 k for
// the dots.  A counting barrier in their place measured 1,174 us, polling
// with every warp instead of one 1,579 us, 1,024 threads 1,370 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "solve.h"

namespace pdds {

namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_MAXM = GMRES_CLUSTER_MAX_M;
constexpr int RS_MAXV = RS_MAXM + 2;   // values of one group sum
constexpr int RS_RANKS = RESIDENT_MAX_CTAS;  // 5 per lane
constexpr int QUAD = 4;                // rows multiplied at once
constexpr int MAX_SEG = 4;             // column segments of a quad's product
constexpr unsigned FIRST_POLL_NS = 300;  // before the first poll: polls in vain delay the words on their way
constexpr unsigned RS_SPIN_LIMIT = 1u << 21;  // polls of one wait, about a second

// ------------------------------------------------------------ tagged words
// 32 bits of data and a sequence number in one 8-byte word (one relaxed
// access, so neither is seen without the other).
__device__ __forceinline__ unsigned long long tagged(unsigned data, unsigned seq) {
  return (unsigned long long)data | ((unsigned long long)seq << 32);
}
__device__ __forceinline__ void put1(unsigned long long* p, unsigned data, unsigned seq) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(tagged(data, seq)) : "memory");
}
__device__ __forceinline__ unsigned long long get1(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// two words side by side: both halves of a double, or of a two-float sum
__device__ __forceinline__ void put2(ulonglong2* p, unsigned a, unsigned b, unsigned seq) {
  put1(&p->x, a, seq);
  put1(&p->y, b, seq);
}
__device__ __forceinline__ ulonglong2 get2(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool has(unsigned long long v, unsigned seq) { return (unsigned)(v >> 32) == seq; }
__device__ __forceinline__ bool has(const ulonglong2& v, unsigned seq) { return has(v.x, seq) && has(v.y, seq); }
__device__ __forceinline__ double as_double(const ulonglong2& v) {
  return __hiloint2double((int)(unsigned)v.x, (int)(unsigned)v.y);
}
__device__ __forceinline__ float2 as_float2(const ulonglong2& v) {
  return make_float2(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y));
}
__device__ __forceinline__ void put_double(ulonglong2* p, double d, unsigned seq) {
  put2(p, (unsigned)__double2hiint(d), (unsigned)__double2loint(d), seq);
}
// polls *p until it has seq; false when the limit runs out
__device__ __forceinline__ bool await(const unsigned long long* p, unsigned long long& v, unsigned seq, unsigned limit) {
  for (unsigned n = 0; !has(v, seq); n++) {
    if (n >= limit) return false;
    v = get1(p);
  }
  return true;
}
__device__ __forceinline__ bool await(const ulonglong2* p, ulonglong2& v, unsigned seq, unsigned limit) {
  for (unsigned n = 0; !has(v, seq); n++) {
    if (n >= limit) return false;
    v = get2(p);
  }
  return true;
}

// ------------------------------------------------------------ sums
// Two-float sums (see k_gmres_cluster.cu): TwoSum and the FMA product error.
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
  const float s = a.x + b.x;
  const float bb = s - a.x;
  const float e = (a.x - (s - bb)) + (b.x - bb) + (a.y + b.y);
  const float hi = s + e;
  return make_float2(hi, e - (hi - s));
}
__device__ __forceinline__ float2 df_sq(float a) {
  const float p = a * a;
  return make_float2(p, fmaf(a, a, -p));
}
__device__ __forceinline__ float2 df_from(double v) {
  const float hi = (float)v;
  return make_float2(hi, (float)(v - (double)hi));
}
__device__ __forceinline__ double df_val(float2 v) { return (double)v.x + (double)v.y; }
template <int W>
__device__ __forceinline__ float2 sum_df(float2 v) {  // over groups of W lanes
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1)
    v = df_add(v, make_float2(__shfl_xor_sync(FULLM, v.x, o), __shfl_xor_sync(FULLM, v.y, o)));
  return v;
}
__device__ __forceinline__ double sum_f64(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLM, v, o);
  return v;
}
// Sums over the warp of four values per lane with 6 exchanges instead of 20:
// lane l ends with the sum of value ((l >> 4) & 1) + 2 ((l >> 3) & 1).
template <typename T>
__device__ __forceinline__ T warp_sum4(const T (&a)[QUAD], int lane) {
  const bool h = (lane & 16) != 0, g = (lane & 8) != 0;
  T k0 = h ? a[1] : a[0], k1 = h ? a[3] : a[2];
  k0 += __shfl_xor_sync(FULLM, h ? a[0] : a[1], 16);
  k1 += __shfl_xor_sync(FULLM, h ? a[2] : a[3], 16);
  T k = g ? k1 : k0;
  k += __shfl_xor_sync(FULLM, g ? k0 : k1, 8);
  k += __shfl_xor_sync(FULLM, k, 4);
  k += __shfl_xor_sync(FULLM, k, 2);
  k += __shfl_xor_sync(FULLM, k, 1);
  return k;
}

// ------------------------------------------------------------ the CTA's part
__host__ __device__ constexpr size_t up16(size_t n) { return (n + 15) & ~size_t(15); }

// Dynamic shared memory of a CTA, carved the same way on the host (size) and
// in the kernel.
struct Carve {
  size_t xloc, own64, basis, w, val, gl, voff, loff, runs, quads, list, bits, pre, total;
};
__host__ __device__ inline Carve carve(int method, int K, int m, int per, int cap_nnz, int cap_list, int cap_loc) {
  Carve c;
  size_t o = 0;
  const int nw = (K + 31) / 32;
  const bool bicg = method == RESIDENT_BICGSTAB;
  c.xloc = o;   // gathered vectors: x in FP64 (GMRES, over the FP32 one); p, r/s, v in FP64 (BiCGSTAB)
  o += up16((size_t)cap_loc * 8 * (bicg ? 3 : 1));
  c.own64 = o;  // own rows in FP64: b, r, x (GMRES); x, r, r0, p, v, s, t (BiCGSTAB)
  o += up16((size_t)per * 8 * (bicg ? 7 : 3));
  c.basis = o;  // own rows of V and Z
  if (!bicg) o += up16((size_t)2 * m * per * 4);
  c.w = o;      // products of the own rows, by column segment
  o += up16((size_t)MAX_SEG * per * (bicg ? 8 : 4));
  if (!bicg) o += up16((size_t)MAX_SEG * per * 8);  // and of the FP64 residual
  c.val = o;    // own entries: FP32 (GMRES), FP64 where they fit (BiCGSTAB, cap_nnz 0: read from L2)
  o += up16((size_t)cap_nnz * (bicg ? 8 : 4));
  c.gl = o;     // global column of each distinct one
  o += up16((size_t)cap_loc * 4);
  c.voff = o;
  o += up16((size_t)(per + 1) * 4);
  c.loff = o;
  o += up16((size_t)per * 4);
  c.runs = o;
  o += up16((size_t)per * 4);
  c.quads = o;
  o += up16((size_t)(per + 1) * 4);
  c.list = o;   // column lists, as indices of distinct columns
  o += up16((size_t)cap_list * 2);
  c.bits = o;   // columns present, one bit each, and the ranks of its words
  o += up16((size_t)nw * 4);
  c.pre = o;
  o += up16((size_t)nw * 4);
  c.total = o;
  return c;
}

struct Part {
  int nown, nloc, nquad, nseg;
  int64_t e0;        // first entry
  const int* gl;     // distinct columns
  const int* voff;   // row -> entries (from e0)
  const int* loff;   // row -> column list
  const int* quads;  // first row of each group of up to QUAD rows of one run
  const unsigned short* list;
};

// Row offsets, column lists and distinct columns of the CTA's rows.  Rows
// that follow each other with the same stencil and length share a list.
__device__ Part build_part(const ResidentArgs& a, const Carve& c, unsigned char* dyn, int r0, int nown) {
  __shared__ int s_nrun, s_nloc, s_nquad;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = (a.K + 31) / 32;
  int* voff = reinterpret_cast<int*>(dyn + c.voff);
  int* loff = reinterpret_cast<int*>(dyn + c.loff);
  int* runs = reinterpret_cast<int*>(dyn + c.runs);
  int* quads = reinterpret_cast<int*>(dyn + c.quads);
  int* gl = reinterpret_cast<int*>(dyn + c.gl);
  unsigned short* list = reinterpret_cast<unsigned short*>(dyn + c.list);
  unsigned* bits = reinterpret_cast<unsigned*>(dyn + c.bits);
  int* pre = reinterpret_cast<int*>(dyn + c.pre);
  Part p;
  p.nown = nown;
  p.e0 = nown > 0 ? a.row_ptr[r0] : 0;
  for (int q = tid; q <= nown; q += RS_THREADS) voff[q] = nown > 0 ? (int)(a.row_ptr[r0 + q] - p.e0) : 0;
  for (int w = tid; w < nw; w += RS_THREADS) bits[w] = 0u;
  __syncthreads();
  if (warp == 0) {
    int carry = 0, nrun = 0, nquad = 0, start = 0;
    for (int q0 = 0; q0 < nown; q0 += 32) {
      const int q = q0 + lane;
      const bool in = q < nown;
      const int len = in ? voff[q + 1] - voff[q] : 0;
      bool first = in;
      if (in && q > 0)
        first = a.knot_stencil[r0 + q] != a.knot_stencil[r0 + q - 1] || len != voff[q] - voff[q - 1];
      int incl = first ? len : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULLM, incl, o);
        if (lane >= o) incl += t;
      }
      if (in) loff[q] = carry + incl - len;
      const unsigned lt = (1u << lane) - 1u;
      const unsigned mk = __ballot_sync(FULLM, first);
      if (first) runs[nrun + __popc(mk & lt)] = q;
      const unsigned upto = mk & (lt | (1u << lane));
      const int run0 = upto ? q0 + 31 - __clz(upto) : start;  // first row of q's run
      const bool qfirst = in && ((q - run0) & (QUAD - 1)) == 0;
      const unsigned mq = __ballot_sync(FULLM, qfirst);
      if (qfirst) quads[nquad + __popc(mq & lt)] = q;
      nrun += __popc(mk);
      nquad += __popc(mq);
      if (mk) start = q0 + 31 - __clz(mk);
      carry += __shfl_sync(FULLM, incl, 31);
    }
    if (lane == 0) {
      s_nrun = nrun;
      s_nquad = nquad;
      quads[nquad] = nown;
    }
  }
  __syncthreads();
  const int nrun = s_nrun;
  for (int k = warp; k < nrun; k += RS_WARPS) {
    const int q = runs[k], len = voff[q + 1] - voff[q];
    if (len == 0) continue;
    const int* cols = a.st_cols + a.st_off[a.knot_stencil[r0 + q]];
    for (int i = lane; i < len; i += 32) {
      const int col = __ldg(cols + i) - a.col0;
      if (idx_ok(col, a.K, a.err_flags)) atomicOr(&bits[col >> 5], 1u << (col & 31));
    }
  }
  __syncthreads();
  if (warp == 0) {
    int carry = 0;
    for (int w0 = 0; w0 < nw; w0 += 32) {
      const int w = w0 + lane, n = w < nw ? __popc(bits[w]) : 0;
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULLM, incl, o);
        if (lane >= o) incl += t;
      }
      if (w < nw) pre[w] = carry + incl - n;
      carry += __shfl_sync(FULLM, incl, 31);
    }
    if (lane == 0) s_nloc = carry;
  }
  __syncthreads();
  for (int w = tid; w < nw; w += RS_THREADS) {
    unsigned b = bits[w];
    int at = pre[w];
    while (b) {
      gl[at++] = 32 * w + __ffs(b) - 1;
      b &= b - 1;
    }
  }
  for (int k = warp; k < nrun; k += RS_WARPS) {
    const int q = runs[k], len = voff[q + 1] - voff[q], at = loff[q];
    if (len == 0) continue;
    const int* cols = a.st_cols + a.st_off[a.knot_stencil[r0 + q]];
    for (int i = lane; i < len; i += 32) {
      const int col = __ldg(cols + i) - a.col0;
      if (!idx_ok(col, a.K, a.err_flags)) continue;
      list[at + i] = (unsigned short)(pre[col >> 5] + __popc(bits[col >> 5] & ((1u << (col & 31)) - 1u)));
    }
  }
  p.nloc = s_nloc;
  p.nquad = s_nquad;
  // enough units of work (quad, column segment) for the CTA's warps
  p.nseg = 8 * p.nquad >= 5 * RS_WARPS ? 1 : (16 * p.nquad >= 5 * RS_WARPS ? 2 : MAX_SEG);
  p.gl = gl;
  p.voff = voff;
  p.loff = loff;
  p.quads = quads;
  p.list = list;
  __syncthreads();
  return p;
}

// Products of the CTA's rows with the gathered vector x, by column segment:
// out[s * per + q], to be added over the segments.  The first `warps` warps
// take part, one (quad, segment) each at a time; val(e): the CTA's entries.
template <typename T, typename Load>
__device__ __forceinline__ void products(const Part& p, int per, const T* x, int warp, int warps, int lane, Load val,
                                         T* out) {
  if (warp >= warps) return;
  const int units = p.nquad * p.nseg;
  for (int un = warp; un < units; un += warps) {
    const int k = un / p.nseg, seg = un - k * p.nseg;
    const int q = p.quads[k], nr = p.quads[k + 1] - q;
    const int v0 = p.voff[q], len = p.voff[q + 1] - v0;
    const int chunk = ((len + p.nseg - 1) / p.nseg + 31) & ~31;
    const int e1 = min(len, (seg + 1) * chunk);
    const unsigned short* ls = p.list + p.loff[q];
    T acc[QUAD];
#pragma unroll
    for (int r = 0; r < QUAD; r++) acc[r] = T(0);
    if (nr == QUAD) {
      int e = seg * chunk + lane;
      for (; e + 32 < e1; e += 64) {
        T a[QUAD], b[QUAD];
#pragma unroll
        for (int r = 0; r < QUAD; r++) {
          a[r] = val(v0 + r * len + e);
          b[r] = val(v0 + r * len + e + 32);
        }
        const T xa = x[ls[e]], xb = x[ls[e + 32]];
#pragma unroll
        for (int r = 0; r < QUAD; r++) acc[r] += a[r] * xa;
#pragma unroll
        for (int r = 0; r < QUAD; r++) acc[r] += b[r] * xb;
      }
      if (e < e1) {
        const T xa = x[ls[e]];
#pragma unroll
        for (int r = 0; r < QUAD; r++) acc[r] += val(v0 + r * len + e) * xa;
      }
    } else {
      for (int e = seg * chunk + lane; e < e1; e += 32) {
        const T xa = x[ls[e]];
#pragma unroll
        for (int r = 0; r < QUAD; r++)
          if (r < nr) acc[r] += val(v0 + r * len + e) * xa;
      }
    }
    const T s = warp_sum4(acc, lane);
    const int r = ((lane >> 4) & 1) + 2 * ((lane >> 3) & 1);
    if ((lane & 7) == 0 && r < nr) out[seg * per + q + r] = s;
  }
}
template <typename T>
__device__ __forceinline__ T seg_sum(const Part& p, int per, const T* out, int q) {
  T s = out[q];
  for (int g = 1; g < p.nseg; g++) s += out[g * per + q];
  return s;
}

__device__ __forceinline__ void write_out(const ResidentArgs& a, bool alive, int total, int ref, double relres) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!a.out) {
      *a.out_iters = total;
      *a.out_refines = ref;
      *a.out_relres = alive ? relres : -1.0;
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      *a.out_t_end = t;
      return;
    }
    a.out[0] = alive ? relres : -1.0;
    reinterpret_cast<int*>(a.out + 1)[0] = total;
    reinterpret_cast<int*>(a.out + 1)[1] = ref;
  }
}

// The partials of a group sum: value i of rank k of publication n at
// part[((n & 1) RS_MAXV + i) RS_RANKS + k].
__device__ __forceinline__ ulonglong2* partial(const ResidentArgs& a, unsigned seq, int i) {
  return a.part + ((size_t)(seq & 1u) * RS_MAXV + i) * RS_RANKS;
}

// ------------------------------------------------------------------ GMRES
__global__ void __launch_bounds__(RS_THREADS, 1) k_resident_gmres(const ResidentArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ float2 s_red[RS_MAXV];
  __shared__ float s_H[(RS_MAXM + 1) * RS_MAXM];  // column j at s_H[j * (m + 1)]
  __shared__ float s_cs[RS_MAXM], s_sn[RS_MAXM], s_g[RS_MAXM + 1], s_y[RS_MAXM];
  __shared__ float2 s_bsum[RS_WARPS];
  __shared__ int s_flag;
  __shared__ float s_inv;
  __shared__ double s_beta[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = a.m, per = a.per, size = gridDim.x;
  unsigned limit = a.spin_limit ? a.spin_limit : RS_SPIN_LIMIT;  // 0 once a wait ran out
  const int r0 = a.row0[blockIdx.x], nown = a.row0[blockIdx.x + 1] - r0;
  const Carve c = carve(RESIDENT_GMRES, a.K, m, per, a.cap_nnz, a.cap_list, a.cap_loc);
  const Part p = build_part(a, c, dyn, r0, nown);
  float* xf = reinterpret_cast<float*>(dyn + c.xloc);
  double* xd = reinterpret_cast<double*>(dyn + c.xloc);
  double* ob = reinterpret_cast<double*>(dyn + c.own64);
  double* orr = ob + per;
  double* ox = orr + per;
  float* V = reinterpret_cast<float*>(dyn + c.basis);  // V[i * per + q]
  float* Z = V + (size_t)m * per;
  float* w = reinterpret_cast<float*>(dyn + c.w);
  double* wd = reinterpret_cast<double*>(dyn + c.w + up16((size_t)MAX_SEG * per * 4));
  float* val = reinterpret_cast<float*>(dyn + c.val);
  const double* v64 = a.val64 + p.e0;
  const int own_warps = (nown + 31) / 32;
  {
    const int nn = p.voff[nown];
    constexpr int U = 8;
    for (int e0 = tid; e0 < nn; e0 += RS_THREADS * U) {
      double t[U];
#pragma unroll
      for (int u = 0; u < U; u++) t[u] = e0 + RS_THREADS * u < nn ? __ldg(v64 + e0 + RS_THREADS * u) : 0.0;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (const int e = e0 + RS_THREADS * u; e < nn) {
          if (e < a.cap_nnz) val[e] = (float)t[u];
          else a.rest[p.e0 + e] = (float)t[u];
        }
    }
  }
  const bool all_here = p.voff[nown] <= a.cap_nnz;
  const float* rest = all_here ? nullptr : a.rest + p.e0;
  unsigned seqp = 0, seqt = 0, seqx = 0;  // publications of partials, of Krylov vectors, of x
  bool alive = true;                      // false once a wait ran out: the CTA winds down
  auto all_ok = [&](bool ok) -> bool {    // CTA barrier; later waits do not wait again
    const bool r = __syncthreads_and(ok) && alive;
    if (!r) limit = 0;
    return r;
  };
  // One warp waits until value 0 of partials seqp has arrived from every CTA;
  // the others' reads of tagged words then hardly ever have to poll (polling
  // with every warp slowed the very stores that were waited for).
  auto arrived = [&]() {
    bool ok = true;
    if (warp == 0) {
      __nanosleep(FIRST_POLL_NS);
      const ulonglong2* b = partial(a, seqp, 0);
      for (int rk = lane; rk < size; rk += 32) {
        unsigned long long v = get1(&b[rk].x);
        ok = ok && await(&b[rk].x, v, seqp, limit);
      }
    }
    alive = all_ok(ok);
  };
  // sum over the CTAs of value i of partials seqp, by one warp
  auto rank_sum = [&](int i, ulonglong2 (&t)[RS_RANKS / 32], bool& ok) -> float2 {
    const ulonglong2* b = partial(a, seqp, i);
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < RS_RANKS / 32; u++) {
      const int rk = lane + 32 * u;
      if (rk < size) {
        ok = ok && await(b + rk, t[u], seqp, limit);
        s = df_add(s, as_float2(t[u]));
      }
    }
    return sum_df<32>(s);
  };
  auto rank_load = [&](int i, ulonglong2 (&t)[RS_RANKS / 32]) {
    const ulonglong2* b = partial(a, seqp, i);
#pragma unroll
    for (int u = 0; u < RS_RANKS / 32; u++) {
      const int rk = lane + 32 * u;
      if (rk < size) t[u] = get2(b + rk);
    }
  };
  // group sum of the two-float value that the own rows' threads hold
  auto group_sum = [&](float2 t) -> double {
    t = sum_df<32>(t);
    if (lane == 0) s_bsum[warp] = t;
    __syncthreads();
    ++seqp;
    bool ok = true;
    if (warp == 0) {
      t = sum_df<32>(lane < RS_WARPS ? s_bsum[lane] : make_float2(0.f, 0.f));
      if (lane == 0) put2(partial(a, seqp, 0) + blockIdx.x, __float_as_uint(t.x), __float_as_uint(t.y), seqp);
      ulonglong2 v[RS_RANKS / 32];
      rank_load(0, v);
      t = rank_sum(0, v, ok);
      if (lane == 0) s_beta[2] = df_val(t);
    }
    alive = all_ok(ok);
    return s_beta[2];
  };
  // own squares of an FP64 vector as a two-float value per thread; only the
  // warps that hold rows take part
  auto own_sq = [&](const double* v) -> float2 {
    double s = 0.0;
    if (warp < own_warps)
      for (int q = tid; q < nown; q += RS_THREADS) s += v[q] * v[q];
    return warp < own_warps ? df_from(s) : make_float2(0.f, 0.f);
  };
  // the first residual is b (x = 0)
  for (int q = tid; q < nown; q += RS_THREADS) {
    const double v = a.b[r0 + q];
    ob[q] = v;
    orr[q] = v;
    ox[q] = 0.0;
  }
  const double bnorm2 = group_sum(own_sq(orr));
  int total = 0, ref = 0;
  double rr = bnorm2;
  if (bnorm2 > 0.0 && alive) {
    const double tol2 = a.tol * a.tol * bnorm2;
    for (ref = 0;; ref++) {
      if (ref > 0) {
        // FP64 residual r = b - x - G x of the own rows
        arrived();
        bool ok = true;
        for (int l = tid; l < p.nloc; l += RS_THREADS) {
          const ulonglong2* at = a.pub + p.gl[l];
          ulonglong2 v = get2(at);
          ok = ok && await(at, v, seqx, limit);
          xd[l] = as_double(v);
        }
        alive = all_ok(ok);
        products<double>(p, per, xd, warp, RS_WARPS, lane, [&](int e) { return __ldg(v64 + e); }, wd);
        __syncthreads();
        for (int q = tid; q < nown; q += RS_THREADS) orr[q] = ob[q] - ox[q] - seg_sum(p, per, wd, q);
        rr = group_sum(own_sq(orr));
      }
      if (!(rr > tol2) || ref >= a.max_refine || total >= a.max_iter || !alive) break;
      if (tid == 0) {
        s_beta[0] = sqrt(rr);
        s_beta[1] = 1.0 / s_beta[0];
        for (int i = 0; i <= m; i++) s_g[i] = 0.f;
        s_g[0] = 1.f;
      }
      __syncthreads();
      const double beta = s_beta[0], ibeta = s_beta[1];
      // t_0 = v_0 = r / |r|
      ++seqt;
      for (int q = tid; q < nown; q += RS_THREADS) {
        const float v = (float)(orr[q] * ibeta);
        V[q] = v;
        put1(a.T + (size_t)(seqt & 1u) * a.K + r0 + q, __float_as_uint(v), seqt);
      }
      ++seqp;  // no partials with v_0: value 0 only tells that it is there
      if (tid == 0) put2(partial(a, seqp, 0) + blockIdx.x, 0u, 0u, seqp);
      int jdim = 0;
      // Step j: gather t_j (= v_0, then z_{j-1}) and sum the partials (its
      // dots with v_0 .. v_{j-1} and |t_j|^2); form the products G t_j while
      // the last warp turns the sums into column j - 1 of the Hessenberg
      // matrix; then v_j and z_j of the own rows, published, and z_j's dots.
      for (int j = 0;; j++) {
        arrived();
        bool ok = true;
        {
          const unsigned long long* tj = a.T + (size_t)(seqt & 1u) * a.K;
          const int nv = j > 0 ? j + 1 : 0;
          ulonglong2 t[RS_RANKS / 32];
          // all loads in flight before the first wait
          if (warp < nv) rank_load(warp, t);
          const int l0 = tid, l1 = tid + RS_THREADS;
          unsigned long long g0 = 0, g1 = 0;
          if (l0 < p.nloc) g0 = get1(tj + p.gl[l0]);
          if (l1 < p.nloc) g1 = get1(tj + p.gl[l1]);
          if (l0 < p.nloc) {
            ok = ok && await(tj + p.gl[l0], g0, seqt, limit);
            xf[l0] = __uint_as_float((unsigned)g0);
          }
          if (l1 < p.nloc) {
            ok = ok && await(tj + p.gl[l1], g1, seqt, limit);
            xf[l1] = __uint_as_float((unsigned)g1);
          }
          for (int l = tid + 2 * RS_THREADS; l < p.nloc; l += RS_THREADS) {
            g0 = get1(tj + p.gl[l]);
            ok = ok && await(tj + p.gl[l], g0, seqt, limit);
            xf[l] = __uint_as_float((unsigned)g0);
          }
          for (int i = warp; i < nv; i += RS_WARPS) {
            if (i != warp) rank_load(i, t);
            const float2 s = rank_sum(i, t, ok);
            if (lane == 0) s_red[i] = s;
          }
        }
        alive = all_ok(ok);
        // column j - 1: h_i = s_red[i], beta = |t_j - V h|, Givens update
        if (j > 0 && warp == RS_WARPS - 1) {
          float2 hh = make_float2(0.f, 0.f);
          for (int i = lane; i < j; i += 32) {
            float2 t = df_sq(s_red[i].x);
            t.y = fmaf(2.f * s_red[i].x, s_red[i].y, t.y);
            hh = df_add(hh, t);
          }
          hh = sum_df<32>(hh);
          if (lane == 0) {
            const float2 d = df_add(s_red[j], make_float2(-hh.x, -hh.y));
            const float hn = sqrtf(fmaxf(d.x + d.y, 0.f));
            s_inv = hn > 0.f ? 1.f / hn : 0.f;
            float* col = s_H + (j - 1) * (m + 1);
            float cur = s_red[0].x + (j == 1 ? 1.f : 0.f);  // + 1: the identity of I + G
#pragma unroll 4
            for (int i = 0; i < j - 1; i++) {
              const float cs = s_cs[i], sn = s_sn[i];
              const float nx = s_red[i + 1].x + (i + 1 == j - 1 ? 1.f : 0.f);
              col[i] = cs * cur + sn * nx;
              cur = cs * nx - sn * cur;
            }
            const float rho = sqrtf(cur * cur + hn * hn);
            const float irho = rho > 0.f ? 1.f / rho : 0.f;
            const float cs = rho > 0.f ? cur * irho : 1.f, sn = hn * irho;
            s_cs[j - 1] = cs;
            s_sn[j - 1] = sn;
            col[j - 1] = rho;
            const float g = s_g[j - 1], gj = -sn * g;
            s_g[j] = gj;
            s_g[j - 1] = cs * g;
            s_flag = (fabsf(gj) <= (float)a.inner_tol || !(hn > 0.f)) ? 1 : 0;
          }
        }
        if (j < m) {
          const int warps = j > 0 ? RS_WARPS - 1 : RS_WARPS;
          if (all_here)
            products<float>(p, per, xf, warp, warps, lane, [&](int e) { return val[e]; }, w);
          else
            products<float>(p, per, xf, warp, warps, lane,
                            [&](int e) { return e < a.cap_nnz ? val[e] : rest[e]; }, w);
        }
        __syncthreads();
        if (j > 0) {
          jdim = j;
          if (s_flag || j >= m || total >= a.max_iter || !alive) break;
        }
        if (!alive) break;
        // v_j = (t_j - sum_i h_i v_i) / beta, z_j = (G t_j - sum_i h_i z_i) / beta
        // of the own rows: the j terms of a row split over pp lanes
        ++seqt;
        unsigned long long* zpub = a.T + (size_t)(seqt & 1u) * a.K + r0;
        if (j == 0) {
          for (int q = tid; q < nown; q += RS_THREADS) {
            const float z = seg_sum(p, per, w, q);
            Z[q] = z;
            put1(zpub + q, __float_as_uint(z), seqt);
          }
        } else {
          const float inv = s_inv;
          int pp = 1;
          while (pp < 32 && pp < j && 2 * pp * nown <= RS_THREADS) pp *= 2;
          const int rows_w = 32 / pp, part = lane & (pp - 1);
          for (int base = warp * rows_w; base < nown; base += RS_WARPS * rows_w) {
            const int q = base + lane / pp;
            float v = 0.f, z = 0.f;
            if (q < nown) {
              for (int i = part; i < j; i += pp) {
                const float hi = s_red[i].x;
                v = fmaf(-hi, V[i * per + q], v);
                z = fmaf(-hi, Z[i * per + q], z);
              }
            }
            for (int o = pp >> 1; o > 0; o >>= 1) {
              z += __shfl_xor_sync(FULLM, z, o);
              v += __shfl_xor_sync(FULLM, v, o);
            }
            if (q < nown && part == 0) {
              const float zj = (seg_sum(p, per, w, q) + z) * inv;
              put1(zpub + q, __float_as_uint(zj), seqt);
              V[j * per + q] = (Z[(j - 1) * per + q] + v) * inv;
              Z[j * per + q] = zj;
            }
          }
        }
        __syncthreads();
        // partial dots of z_j with v_0 .. v_j, and |z_j|^2: 8 lanes each
        ++seqp;
        {
          const float* zj = Z + j * per;
          const int i = tid >> 3, l8 = tid & 7;
          if ((tid & ~31) >> 3 <= j + 1) {  // warp-uniform: 4 values per warp
            float2 t = make_float2(0.f, 0.f);
            if (i <= j) {
              const float* vi = V + i * per;
              float acc = 0.f;
              for (int q = l8; q < nown; q += 8) acc = fmaf(vi[q], zj[q], acc);
              t.x = acc;
            } else if (i == j + 1) {
              for (int q = l8; q < nown; q += 8) t = df_add(t, df_sq(zj[q]));
            }
            t = sum_df<8>(t);
            if (l8 == 0 && i <= j + 1)
              put2(partial(a, seqp, i) + blockIdx.x, __float_as_uint(t.x), __float_as_uint(t.y), seqp);
          }
        }
        ++total;
      }
      // y = H^-1 g (upper triangular, FP32), one warp, rows lane and lane + 32
      if (warp == 0) {
        float g0 = lane < jdim ? s_g[lane] : 0.f, g1 = lane + 32 < jdim ? s_g[lane + 32] : 0.f;
        const float d0 = lane < jdim ? s_H[lane * (m + 1) + lane] : 0.f;
        const float d1 = lane + 32 < jdim ? s_H[(lane + 32) * (m + 1) + lane + 32] : 0.f;
        const float i0 = d0 != 0.f ? 1.f / d0 : 0.f, i1 = d1 != 0.f ? 1.f / d1 : 0.f;
        for (int i = jdim - 1; i >= 0; i--) {
          const float y = __shfl_sync(FULLM, i < 32 ? g0 * i0 : g1 * i1, i & 31);
          const float* col = s_H + i * (m + 1);
          if (lane < i) g0 = fmaf(-col[lane], y, g0);
          if (lane + 32 < i) g1 = fmaf(-col[lane + 32], y, g1);
          if (lane == 0) s_y[i] = y;
        }
      }
      __syncthreads();
      // x += beta V y (FP64 iterate), published for the next residual
      ++seqx;
      for (int q = tid; q < nown; q += RS_THREADS) {
        float acc = 0.f;
        for (int i = 0; i < jdim; i++) acc = fmaf(s_y[i], V[i * per + q], acc);
        const double v = ox[q] + beta * (double)acc;
        ox[q] = v;
        put_double(a.pub + r0 + q, v, seqx);
      }
      ++seqp;
      if (tid == 0) put2(partial(a, seqp, 0) + blockIdx.x, 0u, 0u, seqp);
      if (!alive) break;
    }
  }
  for (int q = tid; q < nown; q += RS_THREADS) a.x[r0 + q] = ox[q];
  if (!alive && tid == 0) atomicOr(a.err_flags, ERR_FLAG_TIMEOUT);
  write_out(a, alive, total, ref, bnorm2 > 0.0 ? sqrt(rr / bnorm2) : 0.0);
}

// --------------------------------------------------------------- BiCGSTAB
// van der Vorst's iteration in FP64 from x = 0 (the diagonal of I + G is 1,
// so the reference's Jacobi preconditioner is the identity).  Three group
// sums per iteration; r and v are published, and every CTA forms p and s at
// its own columns from them, so neither has to be published itself.
__global__ void __launch_bounds__(RS_THREADS, 1) k_resident_bicgstab(const ResidentArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double s_red[2], s_part[2][32], s_sc[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = a.per, size = gridDim.x;
  unsigned limit = a.spin_limit ? a.spin_limit : RS_SPIN_LIMIT;  // 0 once a wait ran out
  const int r0 = a.row0[blockIdx.x], nown = a.row0[blockIdx.x + 1] - r0;
  const Carve c = carve(RESIDENT_BICGSTAB, a.K, a.m, per, a.cap_nnz, a.cap_list, a.cap_loc);
  const Part p = build_part(a, c, dyn, r0, nown);
  double* pl = reinterpret_cast<double*>(dyn + c.xloc);  // p, r (then s) and v at the CTA's columns
  double* rl = pl + a.cap_loc;
  double* vl = rl + a.cap_loc;
  double* ox = reinterpret_cast<double*>(dyn + c.own64);
  double *orr = ox + per, *or0 = orr + per, *op = or0 + per, *ov = op + per, *os = ov + per, *ot = os + per;
  double* w = reinterpret_cast<double*>(dyn + c.w);
  double* val = reinterpret_cast<double*>(dyn + c.val);
  ulonglong2* rpub = a.pub;
  ulonglong2* vpub = a.pub + a.K;
  const double* v64 = a.val64 + p.e0;
  const bool res = a.cap_nnz > 0;  // entries in shared memory
  const int own_warps = (nown + 31) / 32;
  if (res)
    for (int e = tid; e < p.voff[nown]; e += RS_THREADS) val[e] = __ldg(v64 + e);
  for (int l = tid; l < p.nloc; l += RS_THREADS) pl[l] = vl[l] = 0.0;
  if (tid < 32) s_part[0][tid] = s_part[1][tid] = 0.0;
  unsigned seqp = 0, seqr = 0, seqv = 0;
  bool alive = true;
  auto all_ok = [&](bool ok) -> bool {
    const bool r = __syncthreads_and(ok) && alive;
    if (!r) limit = 0;
    return r;
  };
  // group sums of nv values that the own rows' threads hold, into s_red; the
  // sum over a warp only where it holds rows (FP64 adds are what this costs)
  auto group_sum = [&](double u, double v, int nv) {
    if (warp < own_warps) {
      u = sum_f64(u);
      if (nv > 1) v = sum_f64(v);
      if (lane == 0) { s_part[0][warp] = u; s_part[1][warp] = v; }
    }
    __syncthreads();
    ++seqp;
    bool ok = true;
    if (warp < nv) {
      double t = s_part[warp][lane];
      for (int o = 16; o > 0; o >>= 1) {
        const double n = __shfl_xor_sync(FULLM, t, o);
        if (o < own_warps) t += n;  // lanes from own_warps on hold zeros
      }
      if (lane == 0) put_double(partial(a, seqp, warp) + blockIdx.x, t, seqp);
      const ulonglong2* b = partial(a, seqp, warp);
      ulonglong2 g[RS_RANKS / 32];
#pragma unroll
      for (int k = 0; k < RS_RANKS / 32; k++)
        if (lane + 32 * k < size) g[k] = get2(b + lane + 32 * k);
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < RS_RANKS / 32; k++)
        if (32 * k < size) {
          const bool in = lane + 32 * k < size;
          if (in) ok = ok && await(b + lane + 32 * k, g[k], seqp, limit);
          s += in ? as_double(g[k]) : 0.0;
        }
      s = sum_f64(s);
      if (lane == 0) s_red[warp] = s;
    }
    alive = all_ok(ok);
  };
  auto product = [&](const double* x) {
    if (res) products<double>(p, per, x, warp, RS_WARPS, lane, [&](int e) { return val[e]; }, w);
    else products<double>(p, per, x, warp, RS_WARPS, lane, [&](int e) { return __ldg(v64 + e); }, w);
    __syncthreads();
  };
  double bb = 0.0;
  ++seqr;
  for (int q = tid; q < nown; q += RS_THREADS) {
    const double v = a.b[r0 + q];
    orr[q] = or0[q] = v;
    ox[q] = op[q] = ov[q] = 0.0;
    put_double(rpub + r0 + q, v, seqr);
    bb += v * v;
  }
  group_sum(bb, bb, 2);  // |r|^2 and r0 . r
  const double rhs = s_red[0], tol2 = a.tol * a.tol * rhs;
  double rr = rhs, rho_new = s_red[1], rho = 1.0, alpha = 1.0, om = 1.0;
  int it = 0;
  while (rhs != 0.0 && it < a.max_iter && rr > tol2 && alive) {
    // beta = (rho_new / rho) (alpha / om), its two quotients in two lanes of one warp
    if (warp == RS_WARPS - 1) {
      const double qt = (lane & 1 ? alpha : rho_new) / (lane & 1 ? om : rho);
      const double b = qt * __shfl_xor_sync(FULLM, qt, 1);
      if (lane == 0) s_sc[0] = b;
    }
    rho = rho_new;
    bool ok = true;
    for (int l = tid; l < p.nloc; l += RS_THREADS) {
      const ulonglong2* at = rpub + p.gl[l];
      ulonglong2 v = get2(at);
      ok = ok && await(at, v, seqr, limit);
      rl[l] = as_double(v);
    }
    alive = all_ok(ok);
    const double beta = s_sc[0];
    for (int l = tid; l < p.nloc; l += RS_THREADS) pl[l] = rl[l] + beta * (pl[l] - om * vl[l]);
    for (int q = tid; q < nown; q += RS_THREADS) op[q] = orr[q] + beta * (op[q] - om * ov[q]);
    __syncthreads();
    product(pl);  // v = A p
    double d = 0.0, d2 = 0.0;
    ++seqv;
    for (int q = tid; q < nown; q += RS_THREADS) {
      const double v = op[q] + seg_sum(p, per, w, q);
      ov[q] = v;
      put_double(vpub + r0 + q, v, seqv);
      d += or0[q] * v;
    }
    group_sum(d, 0.0, 1);
    if (warp == RS_WARPS - 1) {
      const double al = rho / s_red[0];
      if (lane == 0) s_sc[1] = al;
    }
    ok = true;
    for (int l = tid; l < p.nloc; l += RS_THREADS) {
      const ulonglong2* at = vpub + p.gl[l];
      ulonglong2 v = get2(at);
      ok = ok && await(at, v, seqv, limit);
      vl[l] = as_double(v);
    }
    alive = all_ok(ok);
    alpha = s_sc[1];
    for (int l = tid; l < p.nloc; l += RS_THREADS) rl[l] -= alpha * vl[l];
    for (int q = tid; q < nown; q += RS_THREADS) os[q] = orr[q] - alpha * ov[q];
    __syncthreads();
    product(rl);  // t = A s
    d = d2 = 0.0;
    for (int q = tid; q < nown; q += RS_THREADS) {
      const double t = os[q] + seg_sum(p, per, w, q);
      ot[q] = t;
      d += t * os[q];
      d2 += t * t;
    }
    group_sum(d, d2, 2);
    if (warp == RS_WARPS - 1) {
      const double wv = s_red[1] > 0.0 ? s_red[0] / s_red[1] : 0.0;
      if (lane == 0) s_sc[0] = wv;
    }
    __syncthreads();
    om = s_sc[0];
    d = d2 = 0.0;
    ++seqr;
    for (int q = tid; q < nown; q += RS_THREADS) {
      ox[q] += alpha * op[q] + om * os[q];
      const double r = os[q] - om * ot[q];
      orr[q] = r;
      put_double(rpub + r0 + q, r, seqr);
      d += r * r;
      d2 += or0[q] * r;
    }
    group_sum(d, d2, 2);
    rr = s_red[0];
    rho_new = s_red[1];
    ++it;
  }
  for (int q = tid; q < nown; q += RS_THREADS) a.x[r0 + q] = ox[q];
  if (!alive && tid == 0) atomicOr(a.err_flags, ERR_FLAG_TIMEOUT);
  write_out(a, alive, it, 0, rhs != 0.0 ? sqrt(rr / rhs) : 0.0);
}

const void* resident_kernel(int method) {
  return method == RESIDENT_GMRES ? (const void*)k_resident_gmres : (const void*)k_resident_bicgstab;
}

constexpr int RES_ROWS = 32;
constexpr size_t RES_SMEM_CAP = 216 * 1024;  // dynamic; the kernels' static shared memory is under 10 KB

// Consecutive rows for each of `ctas` CTAs, about equal in entries (a row
// counts as ROW_COST more), and what the largest CTA needs.
constexpr int ROW_COST = 32;
void plan_rows(const ResidentRows& rows, int ctas, ResidentPlan& p) {
  const int64_t e0 = rows.row_ptr[0], all = rows.row_ptr[rows.K] - e0 + (int64_t)ROW_COST * rows.K;
  p.ctas = ctas;
  p.per = p.cap_nnz = p.cap_list = p.cap_loc = 0;
  int r = 0;
  for (int c = 0; c < ctas; c++) {
    p.row0[c] = r;
    const int64_t upto = all * (c + 1) / ctas;
    int64_t list = 0, nnz = 0;
    const int first = r;
    while (r < rows.K && (c == ctas - 1 || rows.row_ptr[r + 1] - e0 + (int64_t)ROW_COST * (r + 1) <= upto)) {
      const int64_t len = rows.row_ptr[r + 1] - rows.row_ptr[r];
      if (r == first || rows.knot_stencil[r] != rows.knot_stencil[r - 1] ||
          len != rows.row_ptr[r] - rows.row_ptr[r - 1])
        list += len;
      nnz += len;
      r++;
    }
    p.per = std::max(p.per, r - first);
    p.cap_nnz = std::max(p.cap_nnz, (int)std::min<int64_t>(nnz, 1 << 28));
    p.cap_list = std::max(p.cap_list, (int)std::min<int64_t>(list, 1 << 28));
    p.cap_loc = std::max(p.cap_loc, (int)std::min<int64_t>(rows.K, list));
  }
  p.row0[ctas] = r;
  p.per = std::max(p.per, 1);
}

bool plan_fits(const ResidentRows& rows, int method, int m, ResidentPlan& p) {
  if (p.cap_loc > 65535) return false;  // 16-bit indices
  p.smem = carve(method, rows.K, m, p.per, p.cap_nnz, p.cap_list, p.cap_loc).total;
  if (p.smem > RES_SMEM_CAP && method == RESIDENT_BICGSTAB) {
    // the FP64 entries stay in L2 (the FP64 pipe sets the pace: keeping 80 % of
    // the 12x12/n43 entries on chip measured no faster)
    p.cap_nnz = 0;
    p.smem = carve(method, rows.K, m, p.per, 0, p.cap_list, p.cap_loc).total;
  } else if (p.smem > RES_SMEM_CAP) {
    // what does not fit is read from L2, as long as it is the smaller part
    const size_t over = p.smem - RES_SMEM_CAP;
    const int keep = p.cap_nnz - (int)((over + 15) / 16 * 4) - 4;
    if (2 * (int64_t)keep < p.cap_nnz) return false;
    p.cap_nnz = keep & ~3;
    p.rest = true;
    p.smem = carve(method, rows.K, m, p.per, p.cap_nnz, p.cap_list, p.cap_loc).total;
  }
  return p.smem <= RES_SMEM_CAP;
}

}  // namespace


ResidentPlan resident_plan(const ResidentRows& rows, int method, int m, int grid_ctas) {
  ResidentPlan p;
  if (rows.K < 1) return p;
  int dev = 0, sms = 0, coop = 0, per_sm = 0;
  const void* f = resident_kernel(method);
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (!coop || sms < 1) return p;
  // one CTA per SM, but at least RES_ROWS rows each: a step's exchange takes
  // longer over more CTAs (1.0 k cycles to arrive for 6, 1.7 k for 30, 4 to
  // 5 k from 47 on) than small products gain from them.  16, 32 and 64 rows:
  // 2,205 rows 484, 411 and 390 us by GMRES, 1,014, 832 and 866 by BiCGSTAB;
  // 3,325 rows 668, 649 and 573 us, 1,037, 931 and 1,162
  const int most = std::min(RS_RANKS, grid_ctas > 0 ? std::min(grid_ctas, sms) : sms);
  plan_rows(rows, std::max(1, std::min(most, (rows.K + RES_ROWS - 1) / RES_ROWS)), p);
  if (!plan_fits(rows, method, m, p) ||
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RES_SMEM_CAP) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, RS_THREADS, p.smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    p.ctas = 0;
  }
  return p;
}

size_t resident_exchange_bytes(int K) {
  return (size_t)2 * RS_MAXV * RS_RANKS * sizeof(ulonglong2) + (size_t)2 * K * sizeof(unsigned long long) +
         (size_t)2 * K * sizeof(ulonglong2);
}

cudaError_t launch_resident(const ResidentArgs& a0, const ResidentPlan& p, int method, void* exchange,
                            cudaStream_t s) {
  if (p.ctas < 1 || a0.m < 2 || a0.m > RS_MAXM) return cudaErrorInvalidValue;
  ResidentArgs a = a0;
  for (int c = 0; c <= p.ctas; c++) a.row0[c] = p.row0[c];
  a.per = p.per;
  a.cap_nnz = p.cap_nnz;
  a.cap_list = p.cap_list;
  a.cap_loc = p.cap_loc;
  a.part = static_cast<ulonglong2*>(exchange);
  a.pub = a.part + (size_t)2 * RS_MAXV * RS_RANKS;
  a.T = reinterpret_cast<unsigned long long*>(a.pub + (size_t)2 * a.K);
  // no word of an earlier solve has a number this one waits for
  cudaError_t e = cudaMemsetAsync(exchange, 0, resident_exchange_bytes(a.K), s);
  if (e != cudaSuccess) return e;
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(resident_kernel(method), dim3(p.ctas), dim3(RS_THREADS), args, p.smem, s);
}

}  // namespace pdds
